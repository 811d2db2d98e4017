// fas_cp.cu -- instantiations of the constitutive kernels (fas_cp.cuh).
#include "fas_cp.cuh"
#include "fas_launch.h"

namespace fasdev {

ElemFn elem_kernel(int ns) { return ns == 12 ? k_elem<12> : ns == 32 ? k_elem<32> : k_elem<60>; }
ElemWcFn elem_wc_kernel(int ns) { return ns == 12 ? k_elem_wc<12> : k_elem_wc<32>; }
PointsFn points_kernel(int ns) { return ns == 12 ? k_points<12> : ns == 32 ? k_points<32> : k_points<60>; }
PointsWcFn points_wc_kernel(int ns) { return ns == 12 ? k_points_wc<12> : k_points_wc<32>; }

}  // namespace fasdev
