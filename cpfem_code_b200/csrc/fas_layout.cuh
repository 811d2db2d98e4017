// fas_layout.cuh -- device layouts shared by the kernels: Gauss-point
// records, mesh tables and the block rows of the stiffness matrix.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fasdev {

// Gauss-point record of an NN-node element: sfd (3 NN), stress (6),
// weight, pad, tangent upper triangle (21), pad.
template <int NN> struct RecLayout {
    static constexpr int S = 3 * NN, W = 3 * NN + 6, D = 3 * NN + 8, LEN = 3 * NN + 32;
};
constexpr int REC = RecLayout<8>::LEN;   // 56 doubles per 8-node element record
constexpr int REC_S = RecLayout<8>::S, REC_W = RecLayout<8>::W, REC_D = RecLayout<8>::D;
constexpr int SLOTS = 27;        // node blocks per row of an 8-node brick mesh
constexpr int SLOTS20 = 81;      // node blocks per row of a 20-node brick mesh
constexpr int MAXADJ = 64;       // elements per node the tables allow (bytes of a local-index word)

// block matrix addressing: a row of S slots holds 9 S values padded to a
// multiple of 4 (so FP64 and FP32 rows are both 16-byte multiples, as bulk
// copies need) and S column ids plus the slot count padded to a multiple of 4
__host__ __device__ constexpr int brow_of(int S) { return (S * 9 + 3) / 4 * 4; }
__host__ __device__ constexpr int crow_of(int S) { return (S + 1 + 3) / 4 * 4; }
constexpr int BROW = brow_of(SLOTS);   // 244
constexpr int CROW = crow_of(SLOTS);   // 28
static_assert(BROW == 244 && CROW == 28, "8-node row layout");

// upper-triangle index of chi(i,j), i <= j (0-based)
__host__ __device__ __forceinline__ int utri(int i, int j) { return i * 6 - (i * (i - 1)) / 2 + (j - i); }

struct MeshDev {
    int nlmnt, nnod;
    int nn, npg;         // nodes and Gauss points per element (8, 1 or 20, 8)
    const int *ln;       // [nn][nlmnt] 0-based node ids
    const int *gpe;      // [npg][nlmnt] 0-based GPs of the element
    const int *le;       // [nlmnt]
    const int *lt;       // [nlmnt] element type: the family's (12 or 22), or 1-6 for a tie
    const int *ib;       // [nnod]
    const int *ne_elem;  // [maxadj][nnod] adjacent elements, ascending
    const int *ne_loc;   // [maxadj][nnod] local index of the node in it
    const int *ne_cnt;   // [nnod]
};

struct BlockDev {
    int R;               // rows (= nnod)
    int slots, brow, crow;   // slots per row and the row lengths (brow_of, crow_of)
    const int *perm;     // row -> node
    const int *nslot;    // [R]
    const int *bcol;     // [R][crow] column node of each slot; [slots] = nslot
    const unsigned long long *bloc;   // [R][crow][nbw] byte k: local index of the column node
                                      // in the k-th adjacent element of the row node (0xFF: absent)
    int nbw;             // words of bloc per slot: ceil(elements per node / 8)
    double *blk;         // [R][brow]: value (r, c) of slot s at (r*3+c)*slots + s
    float *blk32;        // FP32 copy of blk (tuned mode), or null
    __host__ __device__ size_t si(int p, int s) const { return (size_t)p * crow + s; }
    __host__ __device__ size_t bi(int p, int s, int q) const { return (size_t)p * brow + (size_t)q * slots + s; }
};

}  // namespace fasdev
