// fas_launch.h -- kernels that live in their own translation units (they take
// minutes to compile): host code takes their launch handles from here.
#pragma once

#include "fas_adjoint_types.cuh"
#include "fas_cp_types.h"
#include "fas_device.cuh"
#include "fas_layout.cuh"

namespace fasdev {

using ElemFn = void (*)(MeshDev, DevMat, DevCtrl, DevGp, const double *, const double *, double *, double, int, int,
                        unsigned long long *, const int *, int *);
using ElemqFn = void (*)(MeshDev, DevMat, DevCtrl, DevGp, const double *, double, const double *, const double *,
                         double *, double, int, int, unsigned long long *, const int *, int *);
using ElemWcFn = void (*)(MeshDev, DevMat, DevCtrl, DevGp, const double *, const double *, double *, double, int, int,
                          unsigned long long *);
using PointsFn = void (*)(DevMat, DevCtrl, DevGp, const int *, double *, double, int, int, unsigned long long *,
                          const int *, int *);
using PointsWcFn = void (*)(DevMat, DevCtrl, DevGp, const int *, double *, double, int, int, unsigned long long *);
using CpFn = void (*)(DevMat, DevCtrl, DevGp, CpWork, int, double, int, int, unsigned long long *);
using CpTangentFn = void (*)(DevGp, CpWork, int);
using PrepPointsFn = void (*)(DevMat, DevGp, CpWork);
using Prep8Fn = void (*)(MeshDev, DevMat, DevCtrl, DevGp, CpWork, const double *, const double *, unsigned long long *);
using PrepqFn = void (*)(MeshDev, DevMat, DevCtrl, DevGp, CpWork, const double *, double, const double *, const double *,
                         unsigned long long *);
using ReplayFwdFn = void (*)(DevMat, DevCtrl, DevGp, const int *, const double *, ReplayDev, double *, double *, int,
                             double *, double *, unsigned long long *);
using ReplayAdjFn = void (*)(DevMat, DevCtrl, DevGp, const int *, ReplayDev, const double *, double *, int, double *,
                             double *, double *, double *, unsigned long long *);

using ReplayStepFn = void (*)(DevMat, DevGp, CpWork, ReplayDev, ReplayRows, int, bool, bool, unsigned long long *);
using ReplaySeedFn = void (*)(DevMat, DevGp, const int *, ReplayDev, double *, double *, double *, double *, double *);
using ReplayRevFn = void (*)(DevMat, DevGp, const int *, ReplayDev, const double *, int, int, int, int, double *, double *,
                             double *, unsigned long long *);

// ns: the compile-time bound on slip systems (12, 32 or 60; 12 or 32 for
// the warp and replay kernels); nn: nodes of a quadratic element (10, 15, 20)
ElemFn elem_kernel(int ns);
ElemqFn elemq_kernel(int ns, int nn);
ElemWcFn elem_wc_kernel(int ns);
PointsFn points_kernel(int ns);
PointsWcFn points_wc_kernel(int ns);
CpFn cp_kernel(int ns);      // the group pass (CTAs of CP_THREADS), ns as above
int cp_lanes(int ns);        // its lanes per Gauss point
CpTangentFn cp_tangent_kernel();
PrepPointsFn prep_points_kernel();
Prep8Fn prep8_kernel();
PrepqFn prepq_kernel(int nn);
ReplayFwdFn replay_fwd_kernel(int ns);
ReplayAdjFn replay_adj_kernel(int ns);
ReplayStepFn replay_step_kernel();
ReplaySeedFn replay_seed_kernel();
ReplayRevFn replay_rev_kernel(int ns);

}  // namespace fasdev
