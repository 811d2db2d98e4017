// fas_cp.cuh -- the constitutive kernels: the element passes (kinematics and
// DSTRSS for every Gauss point of a mesh) and the pass over independent
// points, one thread or (opt-in) one warp per Gauss point.
#pragma once

#include "fas_device.cuh"
#include "fas_device_warp.cuh"
#include "fas_layout.cuh"

namespace fasdev {

// The items of a constitutive pass, entry t of the launch order (`order`,
// or the natural order when it is null).  With a device queue (`queue`
// non-null, a persistent grid) every warp takes the next 32 entries until
// the order is exhausted, so the work-sorted order is served heaviest first
// and no CTA slot idles behind one slow warp; otherwise thread t takes
// entry t.
template <typename F>
__device__ __forceinline__ void for_each_item(int n, const int *__restrict__ order, int *queue, F &&f)
{
    if (queue) {
        const int lane = threadIdx.x & 31;
        for (;;) {
            int base = 0;
            if (lane == 0) base = atomicAdd(queue, 32);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= n) return;
            const int t = base + lane;
            if (t < n) f(order ? order[t] : t);
        }
    }
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) f(order ? order[t] : t);
}

// ---------------------------------------------------------------- element pass
// ELVALS per element (src/fasolt/Elvals.f90:31-126): gather, SHAPE_12,
// DSTRNS, DSTRSS, store the GP increments and the element record.
template <int NS>
__global__ void __launch_bounds__(128) k_elem(MeshDev Mh, DevMat M, DevCtrl C, DevGp G,
                                              const double *__restrict__ x,
                                              const double *__restrict__ dx, double *rec,
                                              double dt, int inc, int nit,
                                              unsigned long long *errkey, const int *__restrict__ order,
                                              int *queue)
{
#if FAS_SMEM_TABLES
    extern __shared__ double s_tables[];
    if (M.stage_t > 0) M = stage_tables(M, s_tables);
#endif
    for_each_item(Mh.nlmnt, order, queue, [&](int e) {
        if (Mh.lt[e] < 9) return;   // tie element: no Gauss point
        const int ne = Mh.nlmnt;
        double xl[8][3], dxl[8][3];
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int n = Mh.ln[a * ne + e];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                xl[a][c] = x[3 * n + c];
                dxl[a][c] = dx[3 * n + c];
            }
        }
        double sfd[8][3];
        const double w = shape12(xl, sfd);
        if (w < 1.e-7) {
            atomicMin(errkey, ((unsigned long long)e << 16) | 920ull);
            return;
        }
        double del[6], r[3], defl;
        int rc = dstrns(sfd, dxl, C.smalr, C.smale, del, r, defl);
        if (rc) {
            atomicMin(errkey, ((unsigned long long)e << 16) | (unsigned long long)rc);
            return;
        }
        const int g = Mh.gpe[e];
        const int ng = G.ngps;
        double st[6], ds[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            st[k] = G.st[k * ng + g];
            ds[k] = G.ds[k * ng + g];
        }
        GpOut o;
        rc = dstrss<NS>(M, C, G, g, Mh.le[e], del, r, st, ds, dt, inc, C.nit_dev ? *C.nit_dev + 1 : nit, o);
        if (rc) {
            atomicMin(errkey, ((unsigned long long)e << 16) | (unsigned long long)rc);
            return;
        }
        G.dep[g] = o.deff;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            G.de[k * ng + g] = del[k];
            G.ds[k * ng + g] = ds[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) G.dr[k * ng + g] = r[k];
        double *R = rec + (size_t)e * REC;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) R[3 * a + c] = sfd[a][c];
#pragma unroll
        for (int k = 0; k < 6; ++k) R[REC_S + k] = o.t[k];
        R[REC_W] = w;
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int j = i; j < 6; ++j) R[REC_D + utri(i, j)] = o.chi[i][j];
    });
}

// ELVALS per Gauss point of the quadratic elements (src/fasolt/Elvals.f90:
// 82-126): 10-node tetrahedra with SHAPE_21 (NN 10, NPG 4,
// src/fasolt/Shapef.f90:104-189), 20-node bricks with SHAPE_22 (20, 8,
// :210-342) and 15-node wedges with SHAPE_23 (15, 6, :360-485); one thread
// per (element, GP).  dnt[(g*3 + j)*NN + i] = dndn(j+1, i+1, g+1) is the
// element type's tabulated local-derivative table and wfac its GP weight
// factor (-0.0416667, 1, 0.16666667).  The element's nodes are streamed
// twice -- the Jacobian, then sfd (written straight to the GP record) and
// the displacement gradient -- so no node array is held in registers.
// Errors are keyed by (element, GP) so the first one in the reference's
// loop order wins.
template <int NS, int NN, int NPG>
__global__ void __launch_bounds__(128) k_elemq(MeshDev Mh, DevMat M, DevCtrl C, DevGp G,
                                               const double *__restrict__ dnt, double wfac,
                                               const double *__restrict__ x,
                                               const double *__restrict__ dx, double *rec,
                                               double dt, int inc, int nit,
                                               unsigned long long *errkey, const int *__restrict__ order,
                                               int *queue)
{
#if FAS_SMEM_TABLES
    extern __shared__ double s_tables[];
    if (M.stage_t > 0) M = stage_tables(M, s_tables);
#endif
    using L = RecLayout<NN>;
    for_each_item(NPG * Mh.nlmnt, order, queue, [&](int t) {   // item e*NPG + gq
        const int e = t / NPG, gq = t - e * NPG;
        if (Mh.lt[e] < 9) return;   // tie element: no Gauss point
        const int ne = Mh.nlmnt;
        const unsigned long long key = (unsigned long long)t << 16;
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
        double inv[3][3];
        const double w = wfac * invert3(jac, inv);
        if (w < 1.e-7) {
            atomicMin(errkey, key | 920ull);
            return;
        }
        double *R = rec + (size_t)t * L::LEN;
        double gr[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
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
            for (int b = 0; b < 3; ++b) {
                const double u = dx[3 * n + b];
#pragma unroll
                for (int a = 0; a < 3; ++a) gr[a][b] = gr[a][b] + sf[a] * u;
            }
        }
        double del[6], r[3], defl;
        int rc = dstrns_grad(gr, C.smalr, C.smale, del, r, defl);
        if (rc) {
            atomicMin(errkey, key | (unsigned long long)rc);
            return;
        }
        const int g = Mh.gpe[gq * ne + e];
        const int ng = G.ngps;
        double st[6], ds[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            st[k] = G.st[k * ng + g];
            ds[k] = G.ds[k * ng + g];
        }
        GpOut o;
        rc = dstrss<NS>(M, C, G, g, Mh.le[e], del, r, st, ds, dt, inc, C.nit_dev ? *C.nit_dev + 1 : nit, o);
        if (rc) {
            atomicMin(errkey, key | (unsigned long long)rc);
            return;
        }
        G.dep[g] = o.deff;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            G.de[k * ng + g] = del[k];
            G.ds[k * ng + g] = ds[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) G.dr[k * ng + g] = r[k];
#pragma unroll
        for (int k = 0; k < 6; ++k) R[L::S + k] = o.t[k];
        R[L::W] = w;
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int j = i; j < 6; ++j) R[L::D + utri(i, j)] = o.chi[i][j];
    });
}

// Constitutive update of independent points (no mesh): DSTRSS with the
// stored de / dr; the full tangent goes to chi[36][ngps] (column-major 6x6).
template <int NS>
__global__ void __launch_bounds__(128) k_points(DevMat M, DevCtrl C, DevGp G, const int *gp_iel,
                                                double *chi, double dt, int inc, int nit,
                                                unsigned long long *errkey, const int *__restrict__ order,
                                                int *queue)
{
#if FAS_SMEM_TABLES
    extern __shared__ double s_tables[];
    if (M.stage_t > 0) M = stage_tables(M, s_tables);
#endif
    for_each_item(G.ngps, order, queue, [&](int g) {
        const int ng = G.ngps;
        double de[6], r[3], st[6], ds[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            de[k] = G.de[k * ng + g];
            st[k] = G.st[k * ng + g];
            ds[k] = G.ds[k * ng + g];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = G.dr[k * ng + g];
        GpOut o;
        const int rc = dstrss<NS>(M, C, G, g, gp_iel[g], de, r, st, ds, dt, inc, nit, o);
        if (rc) {
            atomicMin(errkey, ((unsigned long long)g << 16) | (unsigned long long)rc);
            return;
        }
        G.dep[g] = o.deff;
#pragma unroll
        for (int k = 0; k < 6; ++k) G.ds[k * ng + g] = ds[k];
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int j = 0; j < 6; ++j) chi[(i + 6 * j) * (size_t)ng + g] = o.chi[i][j];
    });
}

// ---------------------------------------------------------------- warp-cooperative pass
// ELVALS per element with one warp per element: every lane forms the
// element kinematics (identical values), the warp runs dstrss_wc with lane i
// owning slip system i, and the lanes share out the stores.
template <int NA>
__global__ void __launch_bounds__(128) k_elem_wc(MeshDev Mh, DevMat M, DevCtrl C, DevGp G,
                                                 const double *__restrict__ x,
                                                 const double *__restrict__ dx, double *rec,
                                                 double dt, int inc, int nit,
                                                 unsigned long long *errkey)
{
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (e >= Mh.nlmnt) return;           // whole warps only
    if (Mh.lt[e] < 9) return;            // tie element: no Gauss point
    const int ne = Mh.nlmnt;
    double del[6], r[3], defl;
    double *R = rec + (size_t)e * REC;
    {
        double xl[8][3], dxl[8][3];
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int n = Mh.ln[a * ne + e];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                xl[a][c] = x[3 * n + c];
                dxl[a][c] = dx[3 * n + c];
            }
        }
        double sfd[8][3];
        const double w = shape12(xl, sfd);
        if (w < 1.e-7) {
            if (lane == 0) atomicMin(errkey, ((unsigned long long)e << 16) | 920ull);
            return;
        }
        const int rc = dstrns(sfd, dxl, C.smalr, C.smale, del, r, defl);
        if (rc) {
            if (lane == 0) atomicMin(errkey, ((unsigned long long)e << 16) | (unsigned long long)rc);
            return;
        }
        // record: lanes 0-23 shape derivatives, lane 30 the weight
        double v = 0.0;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (lane == 3 * a + c) v = sfd[a][c];
        if (lane == REC_W) v = w;
        if (lane < 24 || lane == REC_W) R[lane] = v;
    }
    const int g = Mh.gpe[e];
    const int ng = G.ngps;
    double st[6], ds[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        st[k] = G.st[k * ng + g];
        ds[k] = G.ds[k * ng + g];
    }
    wc::GpOutW o;
    const int rc = wc::dstrss_wc<NA>(M, C, G, g, Mh.le[e], del, r, st, ds, dt, inc,
                                     C.nit_dev ? *C.nit_dev + 1 : nit, o);
    if (rc) {
        if (lane == 0) atomicMin(errkey, ((unsigned long long)e << 16) | (unsigned long long)rc);
        return;
    }
    if (lane == 0) G.dep[g] = o.deff;
    if (lane < 6) {
        double dk = 0.0, sk = 0.0, tk = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (k == lane) {
                dk = del[k];
                sk = ds[k];
                tk = o.t[k];
            }
        G.de[lane * ng + g] = dk;
        G.ds[lane * ng + g] = sk;
        R[REC_S + lane] = tk;
        // tangent upper triangle, row `lane`
#pragma unroll
        for (int j = 0; j < 6; ++j)
            if (j >= lane) R[REC_D + utri(lane, j)] = o.chirow[j];
    }
    if (lane < 3) {
        double rk = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (k == lane) rk = r[k];
        G.dr[lane * ng + g] = rk;
    }
}

// Independent points with one warp per point (the micro-benchmark path).
template <int NA>
__global__ void __launch_bounds__(128) k_points_wc(DevMat M, DevCtrl C, DevGp G, const int *gp_iel,
                                                   double *chi, double dt, int inc, int nit,
                                                   unsigned long long *errkey)
{
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (g >= G.ngps) return;
    const int ng = G.ngps;
    double de[6], r[3], st[6], ds[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        de[k] = G.de[k * ng + g];
        st[k] = G.st[k * ng + g];
        ds[k] = G.ds[k * ng + g];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = G.dr[k * ng + g];
    wc::GpOutW o;
    const int rc = wc::dstrss_wc<NA>(M, C, G, g, gp_iel[g], de, r, st, ds, dt, inc, nit, o);
    if (rc) {
        if (lane == 0) atomicMin(errkey, ((unsigned long long)g << 16) | (unsigned long long)rc);
        return;
    }
    if (lane == 0) G.dep[g] = o.deff;
    if (lane < 6) {
        double sk = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (k == lane) sk = ds[k];
        G.ds[lane * ng + g] = sk;
    }
    if (lane < 6) {   // row `lane` of the tangent, column-major 6x6 per point
#pragma unroll
        for (int j = 0; j < 6; ++j) chi[(size_t)(lane + 6 * j) * ng + g] = o.chirow[j];
    }
}

}  // namespace fasdev
