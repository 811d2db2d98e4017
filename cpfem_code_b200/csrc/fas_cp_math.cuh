// fas_cp_math.cuh -- what the group pass (fas_cp_group.cuh) and the replay by
// groups (fas_replay_group.cuh) share: lanes per point, sums over a group,
// ELASTC, 6 x 6 elimination, ECHROT.
#pragma once

#include <type_traits>

#include "fas_device.cuh"
#include "fas_cp_types.h"
#include "fas_layout.cuh"

namespace fasdev {

template <int NS> struct GpShape {
    static constexpr int L = NS <= 12 ? 4 : NS <= 32 ? 8 : 16;   // lanes per point
    static constexpr int P = (NS + L - 1) / L;                   // systems per lane
};

constexpr unsigned ALL = 0xffffffffu;

template <int L> __device__ __forceinline__ double gsum(double v)
{
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(ALL, v, o);
    return v;
}
template <int L> __device__ __forceinline__ double gmax(double v)
{
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v = fmax(v, __shfl_xor_sync(ALL, v, o));
    return v;
}
template <int L> __device__ __forceinline__ int gmin(int v)
{
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v = min(v, __shfl_xor_sync(ALL, v, o));
    return v;
}
template <int L> __device__ __forceinline__ int gisum(int v)
{
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(ALL, v, o);
    return v;
}

// ELASTC (src/fasolt/ela-plas.f90:12-86) from CTMATRX's a, upper triangle
// S[utri(I, J)]; the products of two direction cosines are formed once.
__device__ __forceinline__ void elastc_upper(const double *e, const double a0[3][3], double S[21])
{
    const int pi[6] = {0, 1, 2, 1, 2, 0}, pj[6] = {0, 1, 2, 2, 0, 1};
    double ev[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) ev[k] = __ldg(e + k);
    double d[6][3], x[6][6];   // a_ip a_jp, and a_ip a_jq for the pairs (p, q) = 12, 21, 20, 02, 01, 10
#pragma unroll
    for (int I = 0; I < 6; ++I) {
        const int i = pi[I], j = pj[I];
#pragma unroll
        for (int p = 0; p < 3; ++p) d[I][p] = a0[p][i] * a0[p][j];
        x[I][0] = a0[1][i] * a0[2][j];
        x[I][1] = a0[2][i] * a0[1][j];
        x[I][2] = a0[2][i] * a0[0][j];
        x[I][3] = a0[0][i] * a0[2][j];
        x[I][4] = a0[0][i] * a0[1][j];
        x[I][5] = a0[1][i] * a0[0][j];
    }
#pragma unroll
    for (int I = 0; I < 6; ++I)
#pragma unroll
        for (int J = I; J < 6; ++J) {
            double v = d[I][0] * d[J][0] * ev[0] + d[I][1] * d[J][1] * ev[1] + d[I][2] * d[J][2] * ev[2];
            v += (d[I][1] * d[J][2] + d[I][2] * d[J][1]) * ev[3] + (d[I][2] * d[J][0] + d[I][0] * d[J][2]) * ev[4] +
                 (d[I][0] * d[J][1] + d[I][1] * d[J][0]) * ev[5];
            v += 0.5 * ((x[I][0] * x[J][0] + x[I][1] * x[J][1]) * ev[6] + (x[I][2] * x[J][2] + x[I][3] * x[J][3]) * ev[7] +
                        (x[I][4] * x[J][4] + x[I][5] * x[J][5]) * ev[8]);
            S[utri(I, J)] = I < 3 ? v : 2.0 * v;
        }
}

// 6 x 6 elimination without pivoting (FACTOR), unrolled, with the reciprocal
// pivots kept in place of the pivots; 1 for a zero pivot.
__device__ __forceinline__ int lu6(double A[36])
{
    int bad = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        if (A[7 * k] == 0.0) bad = 1;
        A[7 * k] = 1.0 / A[7 * k];
#pragma unroll
        for (int i = k + 1; i < 6; ++i) {
            const double l = A[6 * i + k] * A[7 * k];
            A[6 * i + k] = l;
#pragma unroll
            for (int j = k + 1; j < 6; ++j) A[6 * i + j] -= l * A[6 * k + j];
        }
    }
    return bad;
}
// Solution of A x = y; `first` is the index of y's first nonzero entry.
template <int FIRST> __device__ __forceinline__ void lu6_solve(const double A[36], double x[6])
{
#pragma unroll
    for (int i = FIRST + 1; i < 6; ++i)
#pragma unroll
        for (int j = FIRST; j < i; ++j) x[i] -= A[6 * i + j] * x[j];
#pragma unroll
    for (int i = 5; i >= 0; --i) {
#pragma unroll
        for (int j = i + 1; j < 6; ++j) x[i] -= A[6 * i + j] * x[j];
        x[i] *= A[7 * i];
    }
}
// The symmetrised inverse (A^-1 + A^-T) / 2, upper triangle.
__device__ __forceinline__ void lu6_inverse(const double A[36], double inv[21])
{
#pragma unroll
    for (int k = 0; k < 21; ++k) inv[k] = 0.0;
    auto column = [&](auto first) {
        constexpr int c = decltype(first)::value;
        double x[6] = {0, 0, 0, 0, 0, 0};
        x[c] = 1.0;
        lu6_solve<c>(A, x);
#pragma unroll
        for (int i = 0; i < 6; ++i) inv[i < c ? utri(i, c) : utri(c, i)] += i == c ? x[i] : 0.5 * x[i];
    };
    column(std::integral_constant<int, 0>{});
    column(std::integral_constant<int, 1>{});
    column(std::integral_constant<int, 2>{});
    column(std::integral_constant<int, 3>{});
    column(std::integral_constant<int, 4>{});
    column(std::integral_constant<int, 5>{});
}

// A point that takes CPSTRS: what its iterations start from, and its place in
// the list of its slip-system class (one atomic per class and warp).
__device__ __forceinline__ void cp_enlist(const CpWork &W, int ng, int item, int g, int ns, const double S[21], const double t[6],
                                          const double s[6], const double a[3][3], double gamcap)
{
#pragma unroll
    for (int k = 0; k < 21; ++k) W.w[(size_t)k * ng + g] = S[k];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        W.w[(size_t)(CPW_T + k) * ng + g] = t[k];
        W.w[(size_t)(CPW_S + k) * ng + g] = s[k];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) W.w[(size_t)(CPW_A + k) * ng + g] = a[k / 3][k % 3];
    W.w[(size_t)CPW_CAP * ng + g] = gamcap;
    const int c = ns <= 12 ? 0 : ns <= 32 ? 1 : 2;
    const unsigned peers = __match_any_sync(__activemask(), c);
    const int me = threadIdx.x & 31, lead = __ffs(peers) - 1;
    int base = 0;
    if (me == lead) base = atomicAdd(W.count + c, __popc(peers));
    base = __shfl_sync(peers, base, lead);
    W.list[c][base + __popc(peers & ((1u << me) - 1u))] = item;
}

// ECHROT (crys_math.f90:137-167): the increments of the Euler angles from the
// slips' spin in the crystal frame and the total spin; a (a^T skew - r) =
// skew - a r.
__device__ __forceinline__ void echrot(const double a[3][3], const double aug[3], const double skew[3], const double r[3],
                                       double dph[3])
{
    double rx[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) rx[k] = skew[k] - (a[k][0] * r[0] + a[k][1] * r[1] + a[k][2] * r[2]);
    const double rz = a[0][2] * skew[0] + a[1][2] * skew[1] + a[2][2] * skew[2] - r[2];
    dph[0] = fabs(aug[2]) < 1.e-5 ? rz : (aug[0] * rx[0] + aug[1] * rx[1]) / aug[2];
    dph[1] = aug[1] * rx[0] - aug[0] * rx[1];
    dph[2] = rx[2] - dph[0] * a[2][2];
}

}  // namespace fasdev
