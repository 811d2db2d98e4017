// fas_cpq.cu -- instantiations of the constitutive kernels of the quadratic
// elements (fas_cp.cuh).
#include "fas_cp.cuh"
#include "fas_launch.h"

namespace fasdev {

template <int NS> static ElemqFn pick(int nn)
{
    return nn == 20 ? k_elemq<NS, 20, 8> : nn == 10 ? k_elemq<NS, 10, 4> : k_elemq<NS, 15, 6>;
}
ElemqFn elemq_kernel(int ns, int nn) { return ns == 12 ? pick<12>(nn) : ns == 32 ? pick<32>(nn) : pick<60>(nn); }

}  // namespace fasdev
