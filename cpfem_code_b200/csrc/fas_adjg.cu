// fas_adjg.cu -- instantiations of the replay by groups of lanes
// (fas_replay_group.cuh).
#include "fas_replay_group.cuh"
#include "fas_launch.h"

namespace fasdev {

ReplayStepFn replay_step_kernel() { return k_replay_step; }
ReplaySeedFn replay_seed_kernel() { return k_replay_seed; }
ReplayRevFn replay_rev_kernel(int ns) { return ns == 12 ? k_replay_rev<12> : k_replay_rev<32>; }

}  // namespace fasdev
