// fas_adj.cu -- instantiations of the replay kernels (fas_adjoint.cuh).
#include "fas_adjoint.cuh"
#include "fas_launch.h"

namespace fasdev {

ReplayFwdFn replay_fwd_kernel(int ns) { return ns == 12 ? k_replay_fwd<12> : k_replay_fwd<32>; }
ReplayAdjFn replay_adj_kernel(int ns) { return ns == 12 ? k_replay_adj<12> : k_replay_adj<32>; }

}  // namespace fasdev
