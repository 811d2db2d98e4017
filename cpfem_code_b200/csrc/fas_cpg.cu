// fas_cpg.cu -- instantiations of the group pass (fas_cp_group.cuh).
#include "fas_cp_group.cuh"
#include "fas_launch.h"

namespace fasdev {

CpFn cp_kernel(int ns) { return ns == 12 ? k_cp<12> : ns == 32 ? k_cp<32> : k_cp<60>; }
int cp_lanes(int ns) { return ns == 12 ? GpShape<12>::L : ns == 32 ? GpShape<32>::L : GpShape<60>::L; }
CpTangentFn cp_tangent_kernel() { return k_cp_tangent; }
PrepPointsFn prep_points_kernel() { return k_prep_points; }
Prep8Fn prep8_kernel() { return k_prep8; }
PrepqFn prepq_kernel(int nn) { return nn == 20 ? k_prepq<20, 8> : nn == 10 ? k_prepq<10, 4> : k_prepq<15, 6>; }

}  // namespace fasdev
