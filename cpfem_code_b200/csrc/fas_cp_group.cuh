// fas_cp_group.cuh -- the constitutive pass (DSTRSS + CPSTRS) with a group of
// lanes per Gauss point, for materials whose latent hardening is one number.
//
// What bounded the pass.  With one thread per Gauss point the scratch of
// CPSTRS (slip tensors, the active set's matrices) lies in local memory behind
// run-time indices: a point's chain of dependent loads took 1.7 ms however few
// points there were, and 2^20 points 28 ms (0.6 TFLOP/s of FP64).  Here
//   * L lanes serve a point, lane l the slip systems l, l + L, ...: 3 or 4 per
//     lane, with compile-time indices instead of scratch behind run-time ones.  At
//     the 128 registers that four CTAs an SM leave, 1.3 KB (12 systems) to 1.7 KB
//     (32) a thread are still spilled, most of it around the 6 x 6 matrix;
//   * smatrx(i, j) = q for i /= j and its diagonal d_i >= q make the two
//     matrices of the local problem diagonal plus rank one, and the elimination
//     without pivoting of FACTOR and SOLVER (src/fasolt/crys-cons.f90:244-309)
//     becomes the Sherman-Morrison formula (Ann. Math. Statist. 21 (1950)
//     124-127): sums over the systems instead of n^3 / 3 dependent steps.  With
//     rate exponents above zero and hardening coefficients not below, every
//     diagonal term is positive and the formula's denominator at least one;
//   * the logarithm of |gamma| / dt is carried along: it starts as SPOWER's
//     argument and grows by the Newton step, so an inner iteration takes one
//     logarithm and one exponential per system instead of two of each;
//   * three kernels: what a point does once (kinematics, compliance, rotated
//     stress, the elastic branch) runs with a thread per point before the
//     iterations, the inverse of the tangent after them.  In one kernel the
//     unrolled code did not fit the instruction caches: fetching it took 11.6 of
//     18 cycles per instruction, and 2^20 points 15 ms.
// Every lane of a group holds the point's 6-vectors and does the 6 x 6 algebra;
// sums over systems are butterflies inside the group.  The groups of a warp run
// in lockstep, an outer iteration of each at a time.
//
// Constitutive pass before and after: 4,096 FCC points 1.75 and 0.20 ms,
// 100,003 HCP points 5.8 and 3.1 ms, 2^20 FCC points 28.2 and 12.4 ms, a 64^3
// mesh 11 and 2.7 ms.  The iterations are bound by their dependent chains of
// sums, logarithms and divisions (0.3 instructions a cycle and scheduler at 15
// warps an SM), and by fetching their code.  Against the same update in more
// digits the error of the stress and slips fell from 5e-13 to 4e-14: fewer roundings
// than elimination; that of the hardening increments is PLASTC's (below).
//
// The iterations, their stopping tests and error codes are CPSTRS's; sums run
// in another order and the matrices are solved by the formula, so results equal
// the general path's to rounding (fas_device.cuh: dstrss).
#pragma once

#include "fas_cp_math.cuh"

namespace fasdev {

// ------------------------------------------------------------ before the iterations
// What a point does once, by one thread: compliance and rotated stress; the
// elastic branch of DSTRSS (Sig_eps.f90:137-145) completely; a point that takes
// CPSTRS goes to the list of its slip-system class.
__device__ __forceinline__ void cp_prep(const DevMat &M, const DevGp &G, const CpWork &W, int item, int g, const double de[6],
                                        const double r[3])
{
    const int ng = G.ngps;
    const int iel = W.gp_iel[g], mc = (iel < 0 ? -iel : iel) - 1, ns = M.ns[mc];
    double st[6], t[6], s[6], a[3][3], aug[3], S[21];
#pragma unroll
    for (int k = 0; k < 6; ++k) st[k] = G.st[k * ng + g];
    ctmatrx(G.sv[g] + G.dsv[g], G.sv[ng + g] + G.dsv[ng + g], G.sv[2 * ng + g] + G.dsv[2 * ng + g], a, aug);
    elastc_upper(M.e + 9 * mc, a, S);
    tens_rot(r, st, t);
#pragma unroll
    for (int k = 0; k < 6; ++k) s[k] = t[k] + G.ds[k * ng + g];
    const double einit = fj2vom(false, de);
    if (iel > 0 && fj2vom(true, s) > 0.0 && einit > 0.0) {
        cp_enlist(W, ng, item, g, ns, S, t, s, a, 6.0 * einit);
        return;
    }
    double A[36], inv[21], tn[6];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j < 6; ++j) A[6 * i + j] = S[i <= j ? utri(i, j) : utri(j, i)];
    lu6(A);
    lu6_inverse(A, inv);
    G.erepmd[g] = 0.0;
    G.cp_iters[g] = 0;
    G.ops[g] = fas_ops_elastic();
    G.dep[g] = 0.0;
    double *R = W.rec ? W.rec + (size_t)item * W.reclen + W.off_s : nullptr;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        double acc = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) acc = acc + inv[i <= c ? utri(i, c) : utri(c, i)] * de[c];
        tn[i] = acc;
        G.ds[i * ng + g] = acc - st[i];
        if (R) R[i] = acc;
    }
    if (R) {
#pragma unroll
        for (int k = 0; k < 21; ++k) R[8 + k] = inv[k];
    } else {
#pragma unroll
        for (int j = 0; j < 6; ++j)
#pragma unroll
            for (int i = 0; i < 6; ++i) W.chi[(size_t)(i + 6 * j) * ng + g] = inv[i <= j ? utri(i, j) : utri(j, i)];
    }
}

__global__ void __launch_bounds__(128) k_prep_points(DevMat M, DevGp G, CpWork W)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int ng = G.ngps;
    if (g >= ng) return;
    double de[6], r[3];
#pragma unroll
    for (int k = 0; k < 6; ++k) de[k] = G.de[k * ng + g];
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = G.dr[k * ng + g];
    cp_prep(M, G, W, g, g, de, r);
}

// The kinematics of ELVALS (src/fasolt/Elvals.f90:31-120) for 8-node bricks,
// one thread per element: SHAPE_12, the weight and DSTRNS into the element's
// record and G.de, G.dr, then cp_prep.  An element that fails (905, 906, 920)
// goes to no list.
__global__ void __launch_bounds__(128) k_prep8(MeshDev Mh, DevMat M, DevCtrl C, DevGp G, CpWork W,
                                               const double *__restrict__ x, const double *__restrict__ dx,
                                               unsigned long long *errkey)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= Mh.nlmnt || Mh.lt[e] < 9) return;   // tie element: no Gauss point
    using Lr = RecLayout<8>;
    const int ne = Mh.nlmnt;
    const int g = Mh.gpe[e], ng = G.ngps;
    double del[6], r[3];
    {
        double xl[8][3], dxl[8][3], sfd[8][3], defl;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int n = Mh.ln[a * ne + e];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                xl[a][c] = x[3 * n + c];
                dxl[a][c] = dx[3 * n + c];
            }
        }
        const double w = shape12(xl, sfd);
        const int rc = w < 1.e-7 ? 920 : dstrns(sfd, dxl, C.smalr, C.smale, del, r, defl);
        if (rc) {
            atomicMin(errkey, ((unsigned long long)e << 16) | (unsigned long long)rc);
            return;
        }
        double *R = W.rec + (size_t)e * Lr::LEN;
        R[Lr::W] = w;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) R[3 * a + c] = sfd[a][c];
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) G.de[k * ng + g] = del[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) G.dr[k * ng + g] = r[k];
    cp_prep(M, G, W, e, g, del, r);
}

// The same for the quadratic elements, one thread per (element, Gauss point)
// (SHAPE_21, SHAPE_22, SHAPE_23; dnt and wfac as in k_elemq).
template <int NN, int NPG>
__global__ void __launch_bounds__(128) k_prepq(MeshDev Mh, DevMat M, DevCtrl C, DevGp G, CpWork W,
                                               const double *__restrict__ dnt, double wfac,
                                               const double *__restrict__ x, const double *__restrict__ dx,
                                               unsigned long long *errkey)
{
    using Lr = RecLayout<NN>;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= NPG * Mh.nlmnt) return;
    const int e = t / NPG, gq = t - e * NPG;
    if (Mh.lt[e] < 9) return;   // tie element: no Gauss point
    const int ne = Mh.nlmnt;
    const double *dn = dnt + gq * 3 * NN;
    double jac[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int i = 0; i < NN; ++i) {
        const int n = Mh.ln[i * ne + e];
        const double d0 = __ldg(dn + i), d1 = __ldg(dn + NN + i), d2 = __ldg(dn + 2 * NN + i);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double xk = x[3 * n + k];
            jac[0][k] = jac[0][k] + d0 * xk;
            jac[1][k] = jac[1][k] + d1 * xk;
            jac[2][k] = jac[2][k] + d2 * xk;
        }
    }
    double inv[3][3], gr[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    const double w = wfac * invert3(jac, inv);
    double *R = W.rec + (size_t)t * Lr::LEN;
    int rc = w < 1.e-7 ? 920 : 0;
    double del[6], r[3], defl;
    if (!rc) {
        for (int i = 0; i < NN; ++i) {
            const int n = Mh.ln[i * ne + e];
            const double d0 = __ldg(dn + i), d1 = __ldg(dn + NN + i), d2 = __ldg(dn + 2 * NN + i);
            double sf[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                sf[k] = inv[k][0] * d0 + inv[k][1] * d1 + inv[k][2] * d2;
                R[3 * i + k] = sf[k];
            }
#pragma unroll
            for (int bq = 0; bq < 3; ++bq) {
                const double uu = dx[3 * n + bq];
#pragma unroll
                for (int aq = 0; aq < 3; ++aq) gr[aq][bq] = gr[aq][bq] + sf[aq] * uu;
            }
        }
        rc = dstrns_grad(gr, C.smalr, C.smale, del, r, defl);
    }
    if (rc) {
        atomicMin(errkey, ((unsigned long long)t << 16) | (unsigned long long)rc);
        return;
    }
    R[Lr::W] = w;
    const int g = Mh.gpe[gq * ne + e], ng = G.ngps;
#pragma unroll
    for (int k = 0; k < 6; ++k) G.de[k * ng + g] = del[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) G.dr[k * ng + g] = r[k];
    cp_prep(M, G, W, t, g, del, r);
}

// ------------------------------------------------------------ the iterations
// SCALE_IT's factors (Cpstrs.f90:187-230): scale, smult and log(scale).  Out of
// line: rarely needed, and its code would stand in the loop twice.
__device__ __noinline__ double3 scale_factors(double top, double gamcap, double afactor, double amax)
{
    const double scale = gamcap / top;
    double smult = spower(0.9 * scale, afactor * amax);
    if (smult == 0.0) smult = 0.004 / amax;
    return make_double3(scale, smult, log(scale));
}

// CPSTRS of the points in list `cls`.  The outer iterations of a point vary
// from one to nine or more, so a group that is done takes the next entry of the
// list while the others of its warp go on.  What an outer iteration reads once
// (compliance, rotated stress, slip tensors, strain increment) lies in shared
// memory, which leaves room for four warps per scheduler.
template <int NS>
__global__ void __launch_bounds__(CP_THREADS, 4) k_cp(DevMat M, DevCtrl C, DevGp G, CpWork W, int cls, double dt, int inc,
                                                      int nit, unsigned long long *errkey)
{
    constexpr int L = GpShape<NS>::L, P = GpShape<NS>::P, NG = CP_THREADS / L;
    __shared__ double sS[21][NG], sT[6][NG], sE[6][NG], sB[6 * P][CP_THREADS];
    const int n = W.count[cls];
    const int tid = threadIdx.x, lane = tid % L, gi = tid / L, wl = tid & 31;
    const int ng = G.ngps;
    const int nit_ = C.nit_dev ? *C.nit_dev + 1 : nit;
    const double tiny = 1.e-35 * dt;
    bool run = false, more = true;
    int at = 0, item = 0, g = 0, mc = 0, ns = 0, iter = 0, twinsys = 0, timestwinned = 0;
    double s[6] = {0, 0, 0, 0, 0, 0}, s0[P], gh[P], ops = 0.0, gamcap = 0.0, q = 0.0;
    bool on[P], rate = false;
    const double *amp = M.ampar, *sm = M.sm;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        s0[j] = 1.0;
        gh[j] = 0.0;
        on[j] = false;
    }
    // PLASTC's gradh (ela-plas.f90:127-160): constant unless the saturation
    // stress depends on the slip rate (A6)
    auto harden_rate = [&](double sumss) {
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const double *p = amp + 6 * (on[j] ? lane + L * j : 0);
            const double sst = __ldg(p + 4) * pow_exact01(sumss / dt, __ldg(p + 5));
            double arg = sst != 0.0 ? 1.0 - s0[j] / sst : 0.0;
            if (arg < 0.0) arg = 0.0;
            gh[j] = __ldg(p + 2) + __ldg(p + 1) * pow_exact01(arg, __ldg(p + 3));
        }
    };
    bool fresh = false;          // gh of a new point is still to be formed
    while (true) {
        // ---- the groups that are done take the next points
        const bool need = !run && more;
        const unsigned want = __ballot_sync(ALL, need && lane == 0);
        if (want) {
            int base = 0;
            if (wl == 0) base = atomicAdd(W.head + cls, __popc(want));
            base = __shfl_sync(ALL, base, 0);
            const int k0 = base + __popc(want & ((1u << (wl & ~(L - 1))) - 1u));
            if (need && k0 >= n) more = false;
            if (need && more) {
                at = k0;
                item = W.list[cls][at];
                g = W.gp_of ? W.gp_of[item] : item;
                const int iel = W.gp_iel[g];
                mc = (iel < 0 ? -iel : iel) - 1;
                ns = M.ns[mc];
                amp = M.ampar + (size_t)mc * M.tld * 6;
                sm = M.sm + (size_t)mc * M.sld;
                q = M.hq[mc];
                run = fresh = true;
                iter = 0;
                gamcap = W.w[(size_t)CPW_CAP * ng + g];
                twinsys = G.twinsys[g];
                timestwinned = G.timestwinned[g];
                ops = fas_ops_cp_fixed(ns);
#pragma unroll
                for (int k = lane; k < 21; k += L) sS[k][gi] = W.w[(size_t)k * ng + g];
#pragma unroll
                for (int k = lane; k < 6; k += L) {
                    sT[k][gi] = W.w[(size_t)(CPW_T + k) * ng + g];
                    sE[k][gi] = G.de[k * ng + g];
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) s[k] = W.w[(size_t)(CPW_S + k) * ng + g];
                double a[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) a[k] = W.w[(size_t)(CPW_A + k) * ng + g];
                // the lane's systems: BTMATRX (crys_math.f90:75-115)
                rate = false;
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    on[j] = lane + L * j < ns;
                    const int ii = on[j] ? lane + L * j : 0;
                    const double *ab = M.ab + ((size_t)mc * M.tld + ii) * 3, *an = M.an + ((size_t)mc * M.tld + ii) * 3;
                    const double d0 = __ldg(ab), d1 = __ldg(ab + 1), d2 = __ldg(ab + 2);
                    const double n0 = __ldg(an), n1 = __ldg(an + 1), n2 = __ldg(an + 2);
                    double sdr[3], spn[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        sdr[k] = a[k] * d0 + a[3 + k] * d1 + a[6 + k] * d2;
                        spn[k] = a[k] * n0 + a[3 + k] * n1 + a[6 + k] * n2;
                    }
                    sB[6 * j + 0][tid] = sdr[0] * spn[0];
                    sB[6 * j + 1][tid] = sdr[1] * spn[1];
                    sB[6 * j + 2][tid] = sdr[2] * spn[2];
                    sB[6 * j + 3][tid] = sdr[1] * spn[2] + sdr[2] * spn[1];
                    sB[6 * j + 4][tid] = sdr[2] * spn[0] + sdr[0] * spn[2];
                    sB[6 * j + 5][tid] = sdr[0] * spn[1] + sdr[1] * spn[0];
                    s0[j] = G.sv[(3 + ii) * ng + g];
                    rate = rate || (on[j] && __ldg(amp + 6 * ii + 5) != 0.0);
                }
            }
            __syncwarp();
        }
        if (!__any_sync(ALL, run)) {
            if (__any_sync(ALL, more)) continue;
            return;
        }
        // ---- one outer iteration (CPSTRS) of every group that holds a point
        const bool rated = __any_sync(ALL, run && rate);
        ++iter;
        double tau[P], gam[P], lg[P], s1[P];
        bool act[P];
        // resolved shears, SLPINI (crys-cons.f90:143-197)
        double gammax = 0.0;
        int cand = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            tau[j] = sB[6 * j][tid] * s[0] + sB[6 * j + 1][tid] * s[1] + sB[6 * j + 2][tid] * s[2] +
                     sB[6 * j + 3][tid] * s[3] + sB[6 * j + 4][tid] * s[4] + sB[6 * j + 5][tid] * s[5];
            const int i = lane + L * j;
            const double sa = __ldg(M.ssang + (size_t)mc * M.tld + (on[j] ? i : 0));
            const double x = tau[j] / s0[j];
            gam[j] = 0.0;
            lg[j] = 0.0;
            if (on[j] && fabs(sa) > 1.5) {
                if (tau[j] > s0[j] && timestwinned != M.twinlim &&
                    fas_twin_u01(C.seed, g, inc, nit_, iter, i) < M.twinprob)
                    cand = min(cand, i);
            } else if (on[j] && !(sa * x < 0.0) && !(fabs(x) < 1.e-35)) {
                const double p = log(fabs(x)) / __ldg(amp + 6 * i);
                lg[j] = p < -80.0 ? -80.0 : (p > 80.0 ? 80.0 : p);
                gam[j] = dt * copysign(exp(lg[j]), x);
            }
            gammax = fmax(gammax, fabs(gam[j]));
        }
        cand = gmin<L>(cand);
        if (run && twinsys == 0 && cand != 0x7fffffff) {
            twinsys = cand + 1;
            if (lane == 0) *G.tflag = 1;
        }
        gammax = gmax<L>(gammax);
        const double cutoff = 1.e-6 * gammax;
        int nsa = 0;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            act[j] = on[j] && !(fabs(gam[j]) < cutoff);
            if (!act[j]) gam[j] = 0.0;
            nsa += act[j];
        }
        nsa = gisum<L>(nsa);
        // SCALE_IT (amax starts from the first system's am)
        auto scale_it = [&](double top, bool doit) {
            const bool over = doit && top > gamcap;
            if (!__any_sync(ALL, over)) return false;
            int first = 0x7fffffff, big = 0x7fffffff;
#pragma unroll
            for (int j = 0; j < P; ++j)
                if (act[j]) {
                    first = min(first, lane + L * j);
                    if (fabs(gam[j]) == top) big = min(big, lane + L * j);
                }
            first = gmin<L>(first);
            big = gmin<L>(big);
            if (!over) return false;
            const double3 f = scale_factors(top, gamcap, C.afactor, __ldg(amp + 6 * (big == first || big >= ns ? 0 : big)));
#pragma unroll
            for (int k = 0; k < 6; ++k) s[k] = f.y * s[k];
#pragma unroll
            for (int j = 0; j < P; ++j) {
                gam[j] = f.x * gam[j];
                lg[j] += f.z;
                tau[j] = f.y * tau[j];
            }
            return true;
        };
        scale_it(gammax, run);
        // SLPFTA (crys-cons.f90:24-128): Newton on the logarithms of the active
        // slips.  Its matrix is diag(am + dq |g| gradh / s1) + q u v^T with
        // u = 1 / s1, v = gradh |g|.  A last turn after the tests only forms
        // PLASTC's s1 of the final slips.
        const double conv = C.toler * M.amax[mc];
        int inner = 0;
        double tauerr = 0.0;
        bool turn = run;
        while (true) {
            const bool go = __any_sync(ALL, turn);
            if (rated || __any_sync(ALL, fresh)) {
                double ss = 0.0;
#pragma unroll
                for (int j = 0; j < P; ++j) ss += fabs(gam[j]);
                harden_rate(gsum<L>(ss));
                fresh = false;
            }
            double hsum = 0.0;
#pragma unroll
            for (int j = 0; j < P; ++j) hsum += gh[j] * fabs(gam[j]);
            hsum = gsum<L>(hsum);
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const int ii = on[j] ? lane + L * j : 0;
                s1[j] = s0[j] + q * hsum + (__ldg(sm + ii * ns + ii) - q) * (gh[j] * fabs(gam[j]));
            }
            if (!go) break;
            double rr[P], iD[P], u[P], e2 = 0.0, w = 0.0, vr = 0.0;
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const int ii = on[j] ? lane + L * j : 0;
                const double am = __ldg(amp + 6 * ii), dq = __ldg(sm + ii * ns + ii) - q;
                u[j] = 1.0 / s1[j];
                const double ag = fabs(gam[j]), v = ag > 1.e-14 ? gh[j] * ag : 0.0;
                iD[j] = 1.0 / (am + dq * v * u[j]);
                double p = am * lg[j];
                p = p < -80.0 ? -80.0 : (p > 80.0 ? 80.0 : p);
                const bool ok = act[j] && tau[j] * gam[j] > 0.0 && !(ag < tiny);
                rr[j] = ok ? log(fabs(tau[j]) * u[j]) - p : 0.0;
                e2 += rr[j] * rr[j];
                if (act[j]) {
                    vr += v * iD[j] * rr[j];
                    w += v * iD[j] * u[j];
                }
            }
            e2 = gsum<L>(e2);
            vr = gsum<L>(vr);
            w = gsum<L>(w);
            const double te = sqrt(e2), f = q * vr / (1.0 + q * w);
            double top = 0.0;
#pragma unroll
            for (int j = 0; j < P; ++j) {
                rr[j] = act[j] ? (rr[j] - f * u[j]) * iD[j] : 0.0;
                top = fmax(top, fabs(rr[j]));
            }
            top = gmax<L>(top);
            const double scale = top > 5.0 ? 5.0 / top : 1.0;
            if (turn) {
                ++inner;
                tauerr = te;
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const double x = scale * rr[j];
                    if (act[j]) gam[j] = gam[j] * exp(x);
                    lg[j] += x;
                }
                turn = inner < C.maxit && tauerr > conv;
            }
        }
        ops += inner * fas_ops_inner(ns, nsa) + fas_ops_outer(ns, nsa);
        int rc = run && tauerr > 0.5 ? 987 : 0;
        // X = diag(am tau / g + dq tau sgn(g) gradh / s1) + q u v^T with
        // u = tau / s1, v = sgn(g) gradh; as in the reference before SCALE_IT
        double iX[P], u[P], v[P], w = 0.0, top = 0.0;
        bool zero = false;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int ii = on[j] ? lane + L * j : 0;
            const double am = __ldg(amp + 6 * ii), dq = __ldg(sm + ii * ns + ii) - q;
            const double ag = fabs(gam[j]);
            v[j] = ag > 1.e-14 ? copysign(gh[j], gam[j]) : 0.0;
            u[j] = tau[j] / s1[j];
            const double X = (ag > 1.e-12 ? am * tau[j] / gam[j] : am / 1.e-12) + dq * (u[j] * v[j]);
            zero = zero || (act[j] && X == 0.0);
            iX[j] = act[j] ? 1.0 / X : 0.0;
            w += v[j] * iX[j] * u[j];
            if (act[j]) top = fmax(top, ag);
        }
        w = gsum<L>(w);
        if (gisum<L>(zero ? 1 : 0) != 0 && run && !rc) rc = 910;
        const bool scaled = scale_it(gmax<L>(top), run && !rc);
        // plastic strain, djac = b X^-1 b^T + S and the strain error
        double deff, em, A[36];
        bool fin;
        {
            double err[6], pu[6], pv[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                double x = 0.0, y = 0.0, z = 0.0;
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const double bk = sB[6 * j + k][tid];
                    x += bk * gam[j];
                    y += bk * (iX[j] * u[j]);
                    z += bk * (iX[j] * v[j]);
                }
                err[k] = gsum<L>(x);
                pu[k] = gsum<L>(y);
                pv[k] = gsum<L>(z);
            }
            deff = fj2vom(false, err);
            const double f = q / (1.0 + q * w);
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int k = i; k < 6; ++k) {
                    double x = 0.0;
#pragma unroll
                    for (int j = 0; j < P; ++j) x += sB[6 * j + i][tid] * (iX[j] * sB[6 * j + k][tid]);
                    x = gsum<L>(x) + sS[utri(i, k)][gi];
                    A[6 * i + k] = x - f * (pu[i] * pv[k]);
                    if (k > i) A[6 * k + i] = x - f * (pu[k] * pv[i]);
                }
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                double acc = 0.0;
#pragma unroll
                for (int c = 0; c < 6; ++c) acc = acc + sS[k <= c ? utri(k, c) : utri(c, k)][gi] * (s[c] - sT[c][gi]);
                err[k] = sE[k][gi] - err[k] - acc;
            }
            // the tangent's matrix, taken by k_cp_tangent once the point is done
            const double size = fj2vom(true, s);
            const int bad = lu6(A);
            if (bad && run && !rc) rc = 910;
            lu6_solve<0>(A, err);
            em = fj2vom(true, err) / size;
            const double scale = 1.0 / (1.0 + C.alpha * em);
#pragma unroll
            for (int k = 0; k < 6; ++k) s[k] = s[k] + scale * err[k];
            fin = run && (rc != 0 || !(iter < C.maxit && em > C.toler));
            if (fin && !rc && !W.stress) {
#pragma unroll
                for (int k = 0; k < 36; ++k)
                    if (k % L == lane) W.w[(size_t)k * ng + g] = A[k];
            }
        }
        if (!__any_sync(ALL, fin)) continue;
        // ECHROT (crys_math.f90:137-167); the skew part of a slip system in the
        // crystal frame: (a^T d) x (a^T n) = a^T (d x n)
        double rtn[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int ii = on[j] ? lane + L * j : 0;
            const double *ab = M.ab + ((size_t)mc * M.tld + ii) * 3, *an = M.an + ((size_t)mc * M.tld + ii) * 3;
            const double d0 = __ldg(ab), d1 = __ldg(ab + 1), d2 = __ldg(ab + 2);
            const double n0 = __ldg(an), n1 = __ldg(an + 1), n2 = __ldg(an + 2);
            rtn[0] += (d1 * n2 - d2 * n1) / 2.0 * gam[j];
            rtn[1] += (d2 * n0 - d0 * n2) / 2.0 * gam[j];
            rtn[2] += (d0 * n1 - d1 * n0) / 2.0 * gam[j];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) rtn[k] = gsum<L>(rtn[k]);
        // The hardening increments s1 - s0 that are kept: where the slips are small
        // they are a few thousand roundings of s0, and the order of the sum shows in
        // their seventh to ninth digit.  So s1 is added up once more in PLASTC's order
        // (ela-plas.f90:110-201), system by system onto s0.  SCALE_IT in a point's
        // last iteration, which changes the slips after PLASTC, leaves it as it is.
        {
            double sq[P], hd[P];
#pragma unroll
            for (int k = 0; k < P; ++k) {
                sq[k] = s0[k];
                const int ii = on[k] ? lane + L * k : 0;
                hd[k] = __ldg(sm + ii * ns + ii) * gh[k];
            }
#pragma unroll
            for (int k = 0; k < P; ++k) {
                const double hq = on[k] ? q * gh[k] : 0.0, ag = fabs(gam[k]);
#pragma unroll
                for (int l = 0; l < L; ++l) {
                    const double h = __shfl_sync(ALL, hq, l, L), a = __shfl_sync(ALL, ag, l, L);
#pragma unroll
                    for (int m = 0; m < P; ++m) sq[m] = fma(m == k && l == lane ? hd[m] : h, a, sq[m]);
                }
            }
#pragma unroll
            for (int k = 0; k < P; ++k)
                if (!scaled) s1[k] = sq[k];
        }
        if (fin) {
            if (lane == 0) {
                G.cp_iters[g] = rc && W.stress ? -1 : iter;
                G.ops[g] = ops;
                G.twinsys[g] = twinsys;
                G.erepmd[g] = rc ? 0.0 : em;
            }
            if (rc) {
                if (lane == 0) {
                    atomicMin(errkey, ((unsigned long long)item << 16) | (unsigned long long)rc);
                    W.list[cls][at] = -1;
                }
            } else {
                double *R = W.rec ? W.rec + (size_t)item * W.reclen + W.off_s : nullptr;
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    if (k % L == lane) {
                        if (W.stress) W.stress[(size_t)k * ng + g] = s[k];
                        else G.ds[k * ng + g] = s[k] - G.st[k * ng + g];
                        if (R) R[k] = s[k];
                    }
#pragma unroll
                for (int j = 0; j < P; ++j)
                    if (on[j]) {
                        G.srate[(lane + L * j) * ng + g] = fabs(gam[j] / dt);
                        G.dsv[(3 + lane + L * j) * ng + g] = s1[j] - s0[j];
                    }
                if (lane == 0) {
                    G.dep[g] = deff;
                    // the slips' spin, for k_cp_tangent (which knows the Euler angles)
#pragma unroll
                    for (int k = 0; k < 3; ++k) W.w[(size_t)(CPW_SPIN + k) * ng + g] = rtn[k];
                }
            }
            run = false;
        }
    }
}

// ------------------------------------------------------------ after the iterations
// The symmetrised tangent from the factors of djac, and ECHROT's increments of
// the Euler angles (crys_math.f90:137-167), one thread per point of list `cls`.
__global__ void __launch_bounds__(128) k_cp_tangent(DevGp G, CpWork W, int cls)
{
    const int k0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (k0 >= W.count[cls]) return;
    const int item = W.list[cls][k0];
    if (item < 0) return;
    const int g = W.gp_of ? W.gp_of[item] : item, ng = G.ngps;
    {
        double a[3][3], aug[3], dph[3], sk[3], r[3];
        ctmatrx(G.sv[g] + G.dsv[g], G.sv[ng + g] + G.dsv[ng + g], G.sv[2 * ng + g] + G.dsv[2 * ng + g], a, aug);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            sk[k] = W.w[(size_t)(CPW_SPIN + k) * ng + g];
            r[k] = G.dr[k * ng + g];
        }
        echrot(a, aug, sk, r, dph);
#pragma unroll
        for (int k = 0; k < 3; ++k) G.dsv[k * ng + g] = dph[k];
    }
    double A[36], inv[21];
#pragma unroll
    for (int k = 0; k < 36; ++k) A[k] = W.w[(size_t)k * ng + g];
    lu6_inverse(A, inv);
    if (W.rec) {
        double *R = W.rec + (size_t)item * W.reclen + W.off_s + 8;
#pragma unroll
        for (int k = 0; k < 21; ++k) R[k] = inv[k];
    } else {
#pragma unroll
        for (int j = 0; j < 6; ++j)
#pragma unroll
            for (int i = 0; i < 6; ++i) W.chi[(size_t)(i + 6 * j) * ng + g] = inv[i <= j ? utri(i, j) : utri(j, i)];
    }
}

}  // namespace fasdev
