// fas_sor_flow.cuh -- FACSLS (src/fasolt/Stif_sol.f90:161-215) as one
// persistent kernel per solve: multicolour point SOR over spatial tiles, one
// tile and one CTA per SM, with every dependence carried by the data.
//
// What bounds a solve, and what follows for the design.  A sweep reads the
// whole matrix once and has one dependent phase per colour.  With one launch
// per colour, a phase costs about 3 us of launch boundary whatever its size,
// and each phase refills its copy pipeline from empty: 25 us per sweep on a
// 16^3 cube that holds 10 MB, 126 us at 64^3 where the copy engine alone
// needs 72 us.  Here
//   * the block rows of a tile stream through one ring of bulk copies that
//     never stops at a phase: the matrix is constant during a solve, so the
//     producer runs ahead into the next colour and the next sweep, and as
//     many rows as fit stay in shared memory for the whole solve;
//   * the tile's solution values and those of its neighbours' nodes (the
//     halo) live in shared memory, so the gathers of a row take no trip to
//     L2 (27 gathered nodes of 24 bytes cost as many L2 sectors as the row);
//   * a value that another tile needs is published as a 16-byte {value,
//     sweep} pair, one single-copy-atomic access each way: the reader polls
//     the value itself, with no flag, fence or barrier between tiles (880
//     cycles from one SM's store to another SM's register, about a third of
//     a kernel boundary).
//
// Meshes of a few MB run as one thread-block cluster of 16 tiles (CL): a value
// goes from the registers of the row's lanes into the shared memory of each tile
// that reads it (st.async), and the barrier of its colour there counts the
// bytes, so nothing is polled.  The smallest run as one tile.
//
// Order.  Rows of a tile are ordered by colour, those that other tiles need
// first.  In phase c the consumer warps update the tile's rows of colour c
// while the halo warps fetch the neighbours' nodes of colour c; one CTA
// barrier ends the phase.  A row of colour c therefore sees this sweep's
// value of every neighbour of lower colour and the last sweep's of the
// others: the operands of the global colour order, so the iterates equal
// one-launch-per-colour SOR.  A published value is overwritten in place:
// the owner updates node n in sweep s + 1 only after it has fetched the
// values of all of n's neighbours that were computed from n's value of
// sweep s, so every reader has taken it (the pattern is symmetric).  The same
// holds for a value stored into another tile's shared memory, and for its
// colour's barrier: the bytes of sweep s + 1 start to come only after every
// warp of that tile has passed the phase of sweep s.
//
// Stopping test.  Each tile publishes its share of |x_s - x_(s-1)|^2 and
// |x_s|^2 the same way; the control warp of every tile sums all shares in
// tile order, so all tiles reach the same verdict.  Sweep s starts once the
// verdict of sweep s - 2 is known, which costs no wait in practice; when
// sweep j has converged every tile has finished sweep j + 1, and the values
// that sweep j + 1 replaced (`old`) are the iterate of sweep j.
//
// Measured (first FACSLS, us per sweep, one launch per colour against this
// kernel): 8-node cubes 3^3 - / 6.3 (one tile), 8^3 27 / 9.0 (cluster; 11.3 as one
// tile per SM), 12^3 - / 11.2 (11.8), 16^3 25 / 11.8, 32^3 38 / 16.5, 64^3 122 / 83.9 (580
// MB of records: 6.9 TB/s of the 7.4 TB/s that a bare ring of copies reaches);
// FP32 rows 64^3 96.6 / 61.8; 20-node bricks 4^3 - / 21.5 (27.9), 10^3 60 / 28.5, 21 x
// 17 x 23 82 / 43.1, 32^3 205 / 136.  A phase of one tile per SM takes 1.4 us on a
// small mesh: 0.3 us from the barrier to the published values, 0.9 us until the
// neighbours hold them; of a cluster 1.1 us, of one tile 0.8 us, most of it the
// dependent FP64 chain from the late columns to the point update.  Of the 64^3
// phase's 10 us the copies take 9.4.
//
// Every wait is bounded (FLOW_POLLS).  A wait that gives up raises ctl->fault; a CTA
// leaves only at a barrier where all its warps agree, after its own copies
// have landed.
#pragma once

#include "fas_kernels.cuh"

namespace fasdev {

constexpr int FLOW_SYNC = 32 * 14;       // threads of the phase barrier: consumer and halo warps (FlowRow)
constexpr int FLOW_THREADS = FLOW_SYNC + 64;          // + control warp + producer warp: 4 warps and 128
                                                      // registers per thread on each scheduler
constexpr int FLOW_MAXCOL = 64;
constexpr int FLOW_MAXSLOT = 64;         // chunk slots in shared memory
constexpr int FLOW_SMEM = 223 * 1024;    // dynamic part (about 3 KB is static, of 227 KB)
constexpr int FLOW_RING_BYTES = 112 * 1024;   // copies in flight that cover HBM's latency at full rate
// The cluster form: at most 16 tiles, one cluster.  Its control block lies at
// the start of every CTA's dynamic shared memory, at the same offsets: one
// barrier per colour for the halo's bytes, one per slot of the shares, and the
// shares of four sweeps.
constexpr int FLOW_CLUSTER = 16;
constexpr int FLOW_CL_PBAR = FLOW_MAXCOL * 8, FLOW_CL_PART = FLOW_CL_PBAR + 32,
              FLOW_CL_BYTES = (FLOW_CL_PART + 4 * FLOW_CLUSTER * 16 + 127) & ~127;

// Row format of S slots in value type T.  LPR lanes serve a row, lane q the
// positions q, q + LPR, ...
//
// FP64: a row's columns are its early ones (the row's own node first) from
// position 0 up and its late ones, those of the colour before the row's, from
// position S - 1 down, at most LATE of them: the lane's last two positions.
// FP32: positions are the assembled rows' slots, on the lanes of the colour
// kernels, so that the products are summed in their order: FP32 sums in
// another order are as good, but not the same, and differ by 1e-7 in what
// the refinement leaves.  At least 4 and 8 lanes: take() reads a lane's index
// words of a row held in registers 8 at most, and a row has 16 a lane at most.
//
// 27-slot rows store values by position with a fixed pitch, whose distance
// in banks keeps the rows that a warp reads at once off each other's banks;
// 81-slot rows are packed to their own slot count, early then late (a
// mid-edge node has 51 blocks, a corner node 81).  Each lane's tile-local
// column indices are MW words of 16 bits; lane HQ's word past the positions
// is the header, early count | late count << 7 | published << 15, and for
// 81-slot rows the next lane's the row's place in its chunk in 16-byte units.
template <typename T, int S> struct FlowRow {
    static constexpr bool F32 = sizeof(T) == 4;
    static constexpr int LPR32 = tma_lpr<S, float>(), LEAST32 = S == SLOTS ? 4 : 8;
    static constexpr int LPR = F32 ? (LPR32 > LEAST32 ? LPR32 : LEAST32) : S == SLOTS ? 8 : 16;
    static constexpr int SPL = (S + LPR - 1) / LPR;
    static constexpr int JL = F32 ? SPL : SPL - 2;       // first position round that may hold late columns
    static constexpr int LATE = F32 ? 0 : S - JL * LPR;
    // blocks in registers from take() to finish(): the late columns' in FP64,
    // all of a 27-slot row's in FP32; an FP32 81-slot row is read in finish()
    static constexpr bool AHEAD = !F32 || S == SLOTS;
    static constexpr int KEEP = F32 ? (AHEAD ? SPL : 1) : 2;
    static constexpr int MW = SPL + 1 <= 5 ? 4 : SPL <= 8 ? 8 : 16;
    static constexpr int MB = LPR * MW * 2;              // bytes of a row's index words
    static constexpr int HQ = S - (SPL - 1) * LPR;       // lane and word of the header: position S
    static constexpr int RPW = 32 / LPR;                 // rows per warp
    // consumer and halo warps of the fourteen.  A tile polls some tens to hundreds
    // of pairs a phase, three per FP64 node and one per FP32 node, a pair per thread
    // and L2 round trip; more halo warps take more of them in one round trip (us per
    // sweep with 2 / 3 / 4 halo warps: 16^3 13.1 / 12.9 / 12.7, 32^3 18.8 / 17.3 /
    // 16.8, 64^3 84.3 / 85.1 / 84.1, 20-node 10^3 30.2 / 28.6 / 28.5, 21 x 17 x 23
    // 46.3 / 43.8 / 42.6, 32^3 144 / 141 / 136; FP32 64^3 61.8 / 61.7 / 62.7).
    static constexpr int HW = F32 ? 2 : 4;
    static constexpr int CW = FLOW_SYNC / 32 - HW;
    static constexpr int CH = (S == SLOTS ? 8 : 4) * (F32 ? 2 : 1);   // rows per chunk: about 17 or 25 KB
    static constexpr int EW = F32 ? 10 : 6;              // doubles: rhs 3, 1/diagonal 3 (, base 3, pad)
    static constexpr int EB = EW * 8;
    static constexpr int PITCH = S == SLOTS ? (F32 ? 244 : 248) : brow_of(S);   // values of a row (81 slots: at most)
    static constexpr int VB = PITCH * (int)sizeof(T);
    // a chunk's record in memory and its slot in shared memory: the rows'
    // index words, their extras, their values; one bulk copy (three copies a
    // chunk held the producer thread to 349 ns per chunk whatever its size)
    static constexpr int HB = CH * (MB + EB);
    static constexpr int SLOT = HB + CH * VB;
    // Chunk slots that a tile's solution values must leave, or the colour kernels
    // serve the mesh: the copies in flight no longer cover HBM's latency below (us
    // per sweep of the colour kernels against this one with so many slots; 8-node
    // cubes 80^3 233 / 208 (5), 82^3 242 / 262 (4), 86^3 282 / 411 (3); 20-node 44^3
    // 457 / 416 (4), 46^3 525 / 605 (3); FP32 78^3 158 / 146 (4), 80^3 162 / 200 (3),
    // 20-node 42^3 314 / 302 (4), 44^3 328 / 387 (3)).
    static constexpr int LEAST = !F32 && S == SLOTS ? 5 : 4;
    static_assert(VB % 16 == 0 && MB % 16 == 0 && EB % 16 == 0, "bulk copies move 16-byte multiples");
    static_assert(HQ < LPR && (S == SLOTS || HQ + 1 < LPR) && SPL <= MW && LATE < 64, "header words");
    static_assert(!AHEAD || MW <= 8, "take() reads 8 words at most");
    // where a column of position p is stored, for a row of ne early and nl late columns (-1: none)
    __host__ __device__ static constexpr int stored(int p, int ne, int nl)
    {
        return p < ne ? p : S - 1 - p < nl ? (S == SLOTS ? p : ne + (S - 1 - p)) : -1;
    }
};

template <typename T> struct FlowArgs {
    const unsigned char *rec;    // the chunks' records, tile by tile
    const unsigned *voff;        // [R + 1] first value of a row in 16-byte units (81-slot rows)
    const int *trow, *cptr;      // [ntiles + 1] first row and first chunk of a tile
    const int *seg, *hseg;       // [ntiles][ncol + 1] first own row / halo entry of a colour, tile-local
    const int *hptr, *hrow;      // halo entries of a tile: the row (tile order) that holds the node
    const int *node;             // [R]
    ulonglong2 *gx;              // published values: FP64 [R][3] {value, sweep}, FP32 [R] {x, y, z, sweep}
    ulonglong2 *part;            // [4][ntiles][2] {share, sweep}
    const uint16_t *pptr;        // cluster form: [R + ntiles] a row's first destination, tile-local, and each tile's end
    const unsigned *pdst;        // tile << 16 | index of the node's values there
    const int *pfirst;           // [ntiles + 1] first destination of a tile
    double *old;                 // [R][3] the value that the last update replaced
    double *sol;                 // result, node order
    SorCtl *ctl;
    int ntiles, ncol, maxsw;
    int early;                   // 1: groups may be taken before a phase's late columns have come
    double tolerl;
};

__device__ __forceinline__ void st_pair(ulonglong2 *p, unsigned long long a, unsigned long long b)
{
    asm volatile("{ .reg .b128 v; mov.b128 v, {%1, %2}; st.relaxed.gpu.global.b128 [%0], v; }" ::"l"(p), "l"(a), "l"(b)
                 : "memory");
}
__device__ __forceinline__ void st_pair_if(bool on, ulonglong2 *p, unsigned long long a, unsigned long long b)
{
    asm volatile(
        "{ .reg .b128 v; .reg .pred q; setp.ne.s32 q, %3, 0; mov.b128 v, {%1, %2}; @q st.relaxed.gpu.global.b128 [%0], v; }" ::"l"(p),
        "l"(a), "l"(b), "r"((int)on)
        : "memory");
}
__device__ __forceinline__ ulonglong2 ld_pair(const ulonglong2 *p)
{
    ulonglong2 r;
    asm volatile("{ .reg .b128 v; ld.relaxed.gpu.global.b128 v, [%2]; mov.b128 {%0, %1}, v; }"
                 : "=l"(r.x), "=l"(r.y)
                 : "l"(p)
                 : "memory");
    return r;
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// the phase barrier (consumer and halo warps): the OR of every thread's flag
__device__ __forceinline__ bool flow_bar_or(bool flag)
{
    int r;
    __syncwarp();
    asm volatile("{ .reg .pred p, q; setp.ne.s32 p, %1, 0; barrier.cta.red.or.pred q, 1, %2, p; selp.s32 %0, 1, 0, q; }"
                 : "=r"(r)
                 : "r"((int)flag), "n"(FLOW_SYNC)
                 : "memory");
    return r != 0;
}
__device__ __forceinline__ void mbar_arrive_n(uint64_t *bar, unsigned n)
{
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}

// Bound of the looks of one wait: seconds for a poll of another tile (an L2 round
// trip and a sleep each), 0.1 s for a look at shared memory with a 20 ns sleep,
// some tens of ms for one without, which waits for the CTA's own producer only;
// a sweep takes 6 us to 0.2 ms.  None of them spans the time that another kernel
// holds an SM: the CTAs of a cooperative launch, or of a cluster, start together
// (a block of another stream that sat on one SM for 0.5, 6 and 15 s delayed the
// whole solve by as much and changed no result).
constexpr int FLOW_POLLS = 1 << 21;

// Polls `p` until its tag is `tag`; false after the bound or once another
// CTA has raised the fault.
template <int N> __device__ __forceinline__ bool flow_poll(const ulonglong2 *p, unsigned long long tag, int shift,
                                                           const SorCtl *ctl, ulonglong2 (&v)[N])
{
    for (int it = 0; it < FLOW_POLLS; ++it) {
        bool ok = true;
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = ld_pair(p + k);
#pragma unroll
        for (int k = 0; k < N; ++k) ok &= (v[k].y >> shift) == tag;
        if (ok) return true;
        if (it > 8) __nanosleep(it > 64 ? 200 : 40);
        if ((it & 255) == 255 && ((volatile const SorCtl *)ctl)->fault) return false;
    }
    return false;
}

// Cluster form: a value into another CTA's shared memory, counted in bytes by a
// barrier there.
__device__ __forceinline__ unsigned cl_addr(unsigned addr, unsigned rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_push(unsigned addr, double v, unsigned bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cl_push(unsigned addr, float v, unsigned bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cl_push2(unsigned addr, double a, double b, unsigned bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(bar)
                 : "memory");
}
// every thread of every CTA of the cluster
__device__ __forceinline__ void cl_sync()
{
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// Waits for a phase of a barrier that other CTAs complete: at most two seconds,
// and not once another CTA has raised the fault.
__device__ __forceinline__ bool cl_wait(uint64_t *bar, unsigned parity, const SorCtl *ctl)
{
    unsigned long long t0 = 0;
    for (int it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63) == 63) {
            unsigned long long now;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            if (now - t0 > 2000000000ull || ((volatile const SorCtl *)ctl)->fault) return false;
        }
    }
}

template <typename T, int S, bool CL = false>
__global__ void __launch_bounds__(FLOW_THREADS, 1) k_sor_flow(const FlowArgs<T> A)
{
    using L = FlowRow<T, S>;
    constexpr bool F32 = L::F32;
    constexpr int LPR = L::LPR, SPL = L::SPL, CW = L::CW, HW = L::HW;
    using XT = std::conditional_t<F32, float, double>;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ __align__(8) uint64_t s_full[FLOW_MAXSLOT], s_empty[FLOW_MAXSLOT];
    constexpr int NRED = CW * 3;   // shares of a sweep in one CTA
    __shared__ double s_red[2][2][NRED];
    __shared__ int s_seg[FLOW_MAXCOL + 1], s_hseg[FLOW_MAXCOL + 1];
    __shared__ volatile int s_cnt, s_verdict, s_conv, s_quit, s_bad, s_go, s_issued;
    __shared__ int s_base;
    const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ncol = A.ncol, row0 = A.trow[t], n = A.trow[t + 1] - row0;
    const int h0 = A.hptr[t], nh = A.hptr[t + 1] - h0;
    const int nch = (n + L::CH - 1) / L::CH;
    // shared memory: (control block,) own values, halo values, halo rows or
    // destinations, chunk offsets, slots
    size_t o = CL ? FLOW_CL_BYTES : 0;
    uint64_t *s_hal = reinterpret_cast<uint64_t *>(dyn), *s_pbar = reinterpret_cast<uint64_t *>(dyn + FLOW_CL_PBAR);
    double2 *s_part = reinterpret_cast<double2 *>(dyn + FLOW_CL_PART);
    double *xd = reinterpret_cast<double *>(dyn + o);        // FP64: own + halo; FP32: own only
    o += (size_t)(F32 ? n : n + nh) * 24;
    XT *xs = F32 ? reinterpret_cast<XT *>(dyn + o) : reinterpret_cast<XT *>(xd);
    if (F32) o += (size_t)(n + nh) * 12;
    int *s_hrow = reinterpret_cast<int *>(dyn + o);
    const int d0 = CL ? A.pfirst[t] : 0, nd = CL ? A.pfirst[t + 1] - d0 : 0;
    unsigned *s_pdst = reinterpret_cast<unsigned *>(dyn + o);
    if (CL) o += (size_t)nd * 4;
    else o += (size_t)nh * 4;
    unsigned *s_coff = reinterpret_cast<unsigned *>(dyn + o);
    if (S != SLOTS) o += (size_t)(nch + 1) * 4;
    uint16_t *s_pptr = reinterpret_cast<uint16_t *>(dyn + o);
    if (CL) o += (size_t)(n + 1) * 2;
    o = (o + 127) & ~(size_t)127;
    unsigned char *slots = dyn + o;
    const int nslots = min(FLOW_MAXSLOT, (int)((FLOW_SMEM - o) / L::SLOT));
    // the whole tile stays when it fits; otherwise the first chunks stay and
    // the others share a ring, which takes every slot once the tile is so
    // large that keeping a few chunks would save little
    const int nring = nch <= nslots ? 0 : nch > 4 * nslots ? nslots : min(nslots, (FLOW_RING_BYTES + L::SLOT - 1) / L::SLOT);
    const int nres = nring ? nslots - nring : nch;
    const int nstr = nch - nres;

    if (tid == 0) {
        s_cnt = s_verdict = s_conv = s_quit = s_bad = s_go = s_issued = 0;
        const volatile SorCtl *c = A.ctl;
        s_base = c->conv || c->fault ? -1 : c->sweeps;
        for (int k = 0; k < nres + nring; ++k) {
            mbar_init(&s_full[k], 1);
            mbar_init(&s_empty[k], L::CH);
        }
        mbar_fence_init();
    }
    for (int i = tid; i < (F32 ? n : n + nh) * 3; i += FLOW_THREADS) xd[i] = 0.0;
    if (F32)
        for (int i = tid; i < (n + nh) * 3; i += FLOW_THREADS) xs[i] = (XT)0;
    if constexpr (CL) {
        // where the destinations lie in their CTA's shared memory, above its number
        for (int i = tid; i < nd; i += FLOW_THREADS) {
            const unsigned w = A.pdst[d0 + i], rk = w >> 16;
            const unsigned own = F32 ? 24u * (unsigned)(A.trow[rk + 1] - A.trow[rk]) : 0u;
            s_pdst[i] = rk << 20 | (FLOW_CL_BYTES + own + 3u * sizeof(XT) * (w & 0xffffu));
        }
        for (int i = tid; i <= n; i += FLOW_THREADS) s_pptr[i] = A.pptr[row0 + t + i];
    } else {
        for (int i = tid; i < nh; i += FLOW_THREADS) s_hrow[i] = A.hrow[h0 + i];
    }
    for (int i = tid; i <= ncol; i += FLOW_THREADS) {
        s_seg[i] = A.seg[t * (ncol + 1) + i];
        s_hseg[i] = A.hseg[t * (ncol + 1) + i];
    }
    if (S != SLOTS)
        for (int i = tid; i <= nch; i += FLOW_THREADS) s_coff[i] = A.voff[row0 + min(n, i * L::CH)];
    __syncthreads();
    if (s_base < 0) return;      // converged before (a later FP32 cycle), or a wait gave up
    if constexpr (CL) {
        if (tid < ncol) {
            mbar_init(&s_hal[tid], 1);
            mbar_fence_init();
            if (s_hseg[tid + 1] > s_hseg[tid])
                mbar_expect_tx(&s_hal[tid], (unsigned)(s_hseg[tid + 1] - s_hseg[tid]) * 3u * sizeof(XT));
        } else if (tid >= FLOW_MAXCOL && tid < FLOW_MAXCOL + 4) {
            mbar_init(&s_pbar[tid - FLOW_MAXCOL], 1);
            mbar_fence_init();
            mbar_expect_tx(&s_pbar[tid - FLOW_MAXCOL], 16u * A.ntiles);
        }
        __syncthreads();
        cl_sync();               // every CTA's barriers and zeros stand
    }
    const unsigned dyn0 = smem_u32(dyn);
    const unsigned long long base = (unsigned)s_base;

    if (warp < CW) {
        // ------------------------------------------------------ consumers
        const int row = lane / LPR, q = lane % LPR, lead = lane - q;
        // position / nring by its reciprocal: exact below 2^26 positions
        const unsigned rcp = nring ? (unsigned)((0x100000000ull + nring - 1) / nring) : 0u;
        double v0 = 0.0, v1 = 0.0;
        bool bad = false, use_old = false;
        // The group of rows in hand.  take() multiplies the early columns and
        // reads the blocks of the late ones, whose values the halo warps may
        // still be fetching, into registers; finish() adds the late ones and
        // updates the rows.  So a warp takes its first group of a phase before
        // the barrier that ends the phase before, and only the late columns, the
        // join of the lanes and the point update remain between one tile's
        // published value and the next's.
        T b[L::KEEP][9];
        int mi[L::KEEP];
        bool late[L::KEEP];
        XT f0 = 0, f1 = 0, f2 = 0;
        double oq = 0.0, bq = 0.0;
        int i = 0, issued = 0, st = S;
        bool live = false, pub = false;
        const T *row_vals = nullptr;             // FP32 81-slot rows: the row in its slot
        const uint16_t *row_words = nullptr;
        int row_n = 0, hold_n = 1;
        uint64_t *hold = nullptr;
        // The point update x += 1.2 (t - x) of the three DOFs in turn, as
        // corrections d = 1.2 / D times the DOF's residual, with the residual's
        // share of the old values taken out before the row's sum a is known:
        // d0 = g0 (h0 - a0), d1 = g1 (h1 - a1 - k10 d0),
        // d2 = g2 (h2 - a2 - k20 d0 - k21 d1): seven dependent operations after
        // the sum where the quotients in turn take 24, and the rounding of g
        // scales a correction only (FP32 holds the right-hand side, the
        // reciprocals and the old values in their place).
        double hh0 = 0.0, hh1 = 0.0, hh2 = 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0, k10 = 0.0, k20 = 0.0, k21 = 0.0;
        auto take = [&](int g, int c1, int sw, bool block) -> bool {
            i = g + row;
            live = i < c1;
            const unsigned ii = live ? i : g;
            const int k = (int)(ii / L::CH), ri = (int)(ii % L::CH);
            int slot = k;
            bool ready = true;
            if (k >= nres || sw == 1) {
                unsigned par = 0;
                if (k >= nres) {
                    const int p = (sw - 1) * nstr + k - nres, w = (int)__umulhi((unsigned)p, rcp);
                    slot = nres + (p - w * nring);
                    par = (unsigned)w & 1u;
                    // the parity tells only the slot's current round from the one
                    // before: the copy must have been issued, i.e. the slot's last
                    // round read, before the wait means this round
                    if (issued <= p) {
                        issued = s_issued;
                        for (int it = 0; block && it < FLOW_POLLS && issued <= p; ++it) issued = s_issued;
                        __threadfence_block();
                    }
                    ready = issued > p;
                }
                if (ready) ready = block ? mbar_wait_bounded(&s_full[slot], par) : mbar_test(&s_full[slot], par);
            }
            if (!__all_sync(0xffffffffu, ready)) return false;
            const unsigned char *ch = slots + (size_t)slot * L::SLOT;
            const uint16_t *meta = reinterpret_cast<const uint16_t *>(ch + ri * L::MB);
            const int head = meta[L::HQ * L::MW + SPL - 1];
            unsigned wd[L::MW];
            if constexpr (L::MW == 4) {
                const uint2 w = reinterpret_cast<const uint2 *>(meta)[q];
                wd[0] = w.x & 0xffffu, wd[1] = w.x >> 16, wd[2] = w.y & 0xffffu, wd[3] = w.y >> 16;
            } else {
                const uint4 w = reinterpret_cast<const uint4 *>(meta + q * L::MW)[0];
                wd[0] = w.x & 0xffffu, wd[1] = w.x >> 16, wd[2] = w.y & 0xffffu, wd[3] = w.y >> 16;
                wd[4] = w.z & 0xffffu, wd[5] = w.z >> 16, wd[6] = w.w & 0xffffu, wd[7] = w.w >> 16;
            }
            const int ne = head & 0x7f, nl = (head >> 7) & 0x3f;
            pub = (head & 0x8000) != 0;
            st = S == SLOTS ? S : ne + nl;
            const T *vals = reinterpret_cast<const T *>(
                ch + L::HB + (S == SLOTS ? ri * L::VB : 16 * (int)meta[(L::HQ + 1) * L::MW + SPL - 1]));
            const double *e = reinterpret_cast<const double *>(ch + L::CH * L::MB + ri * L::EB);
            const double2 e01 = reinterpret_cast<const double2 *>(e)[0], e23 = reinterpret_cast<const double2 *>(e)[1],
                          e45 = reinterpret_cast<const double2 *>(e)[2];
            const double *own = xd + 3 * ii;
            const double o0 = own[0], o1 = own[1], o2 = own[2];
            oq = q == 0 ? o0 : q == 1 ? o1 : o2;
            // every load is issued whatever the position (an absent column reads the
            // diagonal and counts with a zero), so that none waits for a branch
            if constexpr (F32) {
                bq = e[6 + (q < 3 ? q : 0)];
                hh0 = e01.x, hh1 = e01.y, hh2 = e23.x, g0 = e23.y, g1 = e45.x, g2 = e45.y;
                k10 = o0, k20 = o1, k21 = o2;
                if constexpr (L::AHEAD) {
#pragma unroll
                    for (int j = 0; j < SPL; ++j) {
                        const int p = q + LPR * j;
                        late[j] = p >= 1 && p < ne;
                        mi[j] = late[j] ? (int)wd[j] : 0;
#pragma unroll
                        for (int z = 0; z < 9; ++z) b[j][z] = vals[(late[j] ? p : 0) + z * S];
                    }
                } else {
                    row_vals = vals;
                    row_words = meta + q * L::MW;
                    row_n = ne;
                    hold = k >= nres ? &s_empty[slot] : nullptr;
                    hold_n = i == n - 1 ? L::CH - ri : 1;
                }
            } else {
                f0 = f1 = f2 = 0;
#pragma unroll
                for (int j = 0; j < SPL; ++j) {
                    const int p = q + LPR * j;
                    const bool early = p >= 1 && p < ne;
                    const bool lt = j >= L::JL && S - 1 - p >= 0 && S - 1 - p < nl;
                    const int at = early ? p : lt ? (S == SLOTS ? p : ne + S - 1 - p) : 0;
                    const T *v = vals + at;
                    T w[9];
#pragma unroll
                    for (int z = 0; z < 9; ++z) w[z] = v[z * st];
                    const XT *y = xs + 3 * (early ? (int)wd[j] : 0);
                    XT y0 = y[0], y1 = y[1], y2 = y[2];
                    y0 = early ? y0 : (XT)0, y1 = early ? y1 : (XT)0, y2 = early ? y2 : (XT)0;
                    f0 += w[0] * y0 + w[1] * y1 + w[2] * y2;
                    f1 += w[3] * y0 + w[4] * y1 + w[5] * y2;
                    f2 += w[6] * y0 + w[7] * y1 + w[8] * y2;
                    if (j == 0) {   // lane 0's first position is the row's own block
                        g0 = 1.2 * e23.y, g1 = 1.2 * e45.x, g2 = 1.2 * e45.y;
                        hh0 = e01.x - (w[0] * o0 + w[1] * o1 + w[2] * o2);
                        hh1 = e01.y - (w[3] * o0 + w[4] * o1 + w[5] * o2);
                        hh2 = e23.x - (w[6] * o0 + w[7] * o1 + w[8] * o2);
                        k10 = w[3], k20 = w[6], k21 = w[7];
                    }
                    if (j >= L::JL) {
                        constexpr int J0 = L::JL;
                        late[(j - J0) & 1] = lt;
                        mi[(j - J0) & 1] = lt ? (int)wd[j] : 0;
#pragma unroll
                        for (int z = 0; z < 9; ++z) b[(j - J0) & 1][z] = w[z];
                    }
                }
            }
            // the row is read: its share of the slot (the tile's last row also gives
            // the places that a short last chunk leaves empty), so that the ring
            // goes on while the group waits for its late columns
            if constexpr (L::AHEAD) {
                __syncwarp();
                if (q == 0 && live && k >= nres) mbar_arrive_n(&s_empty[slot], i == n - 1 ? L::CH - ri : 1);
            }
            return true;
        };
        auto finish = [&](int sw, int c) {
            double a0, a1, a2, x0, x1, x2;
            if constexpr (F32) {
                // FP32 products and lane sums in slot order, joined in FP64, and the
                // quotients in turn, from the correctly rounded reciprocals with an exact
                // remainder (Markstein, IBM J. Res. Dev. 34 (1990) 111-119): the same
                // rounding as the colour kernels throughout
                f0 = f1 = f2 = 0;
                T D[9];
#pragma unroll
                for (int j = 0; j < SPL; ++j) {
                    bool on;
                    int m;
                    T w[9];
                    if constexpr (L::AHEAD) {
                        on = late[j];
                        m = mi[j];
#pragma unroll
                        for (int z = 0; z < 9; ++z) w[z] = b[j][z];
                    } else {
                        const int p = q + LPR * j;
                        on = p >= 1 && p < row_n;
                        m = on ? row_words[j] : 0;
#pragma unroll
                        for (int z = 0; z < 9; ++z) w[z] = row_vals[(on ? p : 0) + z * st];
                    }
                    const XT *y = xs + 3 * m;
                    XT y0 = y[0], y1 = y[1], y2 = y[2];
                    y0 = on ? y0 : (XT)0, y1 = on ? y1 : (XT)0, y2 = on ? y2 : (XT)0;
                    f0 += w[0] * y0 + w[1] * y1 + w[2] * y2;
                    f1 += w[3] * y0 + w[4] * y1 + w[5] * y2;
                    f2 += w[6] * y0 + w[7] * y1 + w[8] * y2;
                    if (j == 0)
#pragma unroll
                        for (int z = 0; z < 9; ++z) D[z] = w[z];
                }
                if constexpr (!L::AHEAD) {
                    __syncwarp();
                    if (q == 0 && live && hold) mbar_arrive_n(hold, hold_n);
                }
                a0 = f0, a1 = f1, a2 = f2;
#pragma unroll
                for (int u = 1; u < LPR; u <<= 1) {
                    a0 += __shfl_xor_sync(0xffffffffu, a0, u);
                    a1 += __shfl_xor_sync(0xffffffffu, a1, u);
                    a2 += __shfl_xor_sync(0xffffffffu, a2, u);
                }
                x0 = k10, x1 = k20, x2 = k21;
                double nm = hh0 - (a0 + (double)D[1] * x1 + (double)D[2] * x2);
                double q0 = nm * g0;
                double tt = fma(fma(-q0, (double)D[0], nm), g0, q0);
                x0 = x0 + 1.2 * (tt - x0);
                nm = hh1 - (a1 + (double)D[3] * x0 + (double)D[5] * x2);
                q0 = nm * g1;
                tt = fma(fma(-q0, (double)D[4], nm), g1, q0);
                x1 = x1 + 1.2 * (tt - x1);
                nm = hh2 - (a2 + (double)D[6] * x0 + (double)D[7] * x1);
                q0 = nm * g2;
                tt = fma(fma(-q0, (double)D[8], nm), g2, q0);
                x2 = x2 + 1.2 * (tt - x2);
            } else {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (!__any_sync(0xffffffffu, late[j])) continue;
                    const XT *y = xs + 3 * mi[j];
                    XT y0 = y[0], y1 = y[1], y2 = y[2];
                    y0 = late[j] ? y0 : (XT)0, y1 = late[j] ? y1 : (XT)0, y2 = late[j] ? y2 : (XT)0;
                    f0 += b[j][0] * y0 + b[j][1] * y1 + b[j][2] * y2;
                    f1 += b[j][3] * y0 + b[j][4] * y1 + b[j][5] * y2;
                    f2 += b[j][6] * y0 + b[j][7] * y1 + b[j][8] * y2;
                }
                a0 = f0, a1 = f1, a2 = f2;
#pragma unroll
                for (int u = 1; u < LPR; u <<= 1) {
                    a0 += __shfl_xor_sync(0xffffffffu, a0, u);
                    a1 += __shfl_xor_sync(0xffffffffu, a1, u);
                    a2 += __shfl_xor_sync(0xffffffffu, a2, u);
                }
                x0 = g0 * (hh0 - a0);
                x1 = g1 * ((hh1 - a1) - k10 * x0);
                x2 = g2 * (((hh2 - a2) - k20 * x0) - k21 * x1);
            }
            // lane q < 3 publishes and stores component q
            const double t0 = __shfl_sync(0xffffffffu, x0, lead), t1 = __shfl_sync(0xffffffffu, x1, lead),
                         t2 = __shfl_sync(0xffffffffu, x2, lead);
            const double tq = q == 0 ? t0 : q == 1 ? t1 : t2;
            const double xq = F32 ? tq : oq + tq, dq = F32 ? tq - oq : tq;
            const bool mine = live && q < 3;
            const size_t r = (size_t)row0 + i;
            if constexpr (CL) {
                if (pub && mine) {
                    const int k1 = s_pptr[i + 1];
                    for (int k = s_pptr[i]; k < k1; ++k) {
                        const unsigned w = s_pdst[k], rk = w >> 20;
                        cl_push(cl_addr(dyn0 + (w & 0xfffffu) + (unsigned)sizeof(XT) * q, rk), (XT)xq, cl_addr(dyn0 + 8u * c, rk));
                    }
                }
            } else if constexpr (F32)
                st_pair_if(pub && mine && q == 0, A.gx + r,
                           (unsigned long long)__float_as_uint((float)x0) |
                               ((unsigned long long)__float_as_uint((float)x1) << 32),
                           (unsigned long long)__float_as_uint((float)x2) | ((base + (unsigned)sw) << 32));
            else
                st_pair_if(pub && mine, A.gx + 3 * r + q, __double_as_longlong(xq), base + (unsigned)sw);
            if (mine) {
                xd[3 * i + q] = xq;
                if constexpr (F32) xs[3 * i + q] = (float)xq;
                A.old[3 * r + q] = oq;
                v0 += dq * dq;
                const double xb = F32 ? xq + bq : xq;
                v1 += xb * xb;
            }
        };
        bool taken = false;
        // A phase's groups begin at the warp after the last one of the phase
        // before, so that the warps of a phase of few rows have taken their rows
        // while others finished the phase before (us per sweep with every phase
        // beginning at warp 0: clusters 8^3 11.0, 20-node 4^3 27.9 against 9.0, 21.5; 32^3
        // 17.0 against 16.5).  Not in tiles that stream all their rows, whose phases
        // have several groups a warp: 21 x 17 x 23 20-node bricks 43.1 against 45.7.
        const bool rotate = CL || nring < nslots;
        int w0 = 0, g = s_seg[0] + warp * L::RPW, c1 = s_seg[1];
        for (int s = 1; s <= A.maxsw; ++s) {
            for (int c = 0; c < ncol; ++c) {
                for (; g < c1; g += CW * L::RPW) {
                    if (!taken && !take(g, c1, s, true)) {
                        bad = true;
                        break;
                    }
                    taken = false;
                    finish(s, c);
                }
                const bool last = c + 1 == ncol;
                if (last) {
                    // the sweep's shares; sweep s + 1 may start once the verdict of
                    // sweep s - 1 is known
#pragma unroll
                    for (int u = LPR; u < 32; u <<= 1) {
                        v0 += __shfl_xor_sync(0xffffffffu, v0, u);
                        v1 += __shfl_xor_sync(0xffffffffu, v1, u);
                    }
                    if (lane < 3) {
                        s_red[s & 1][0][3 * warp + lane] = v0;
                        s_red[s & 1][1][3 * warp + lane] = v1;
                    }
                    v0 = v1 = 0.0;
                    if (tid == 0 && s > 1) {
                        for (int it = 0; s_verdict < s - 1 && !s_bad && it < FLOW_POLLS; ++it) __nanosleep(20);
                        s_go = (s_bad || s_verdict < s - 1) ? 2 : (s_conv != 0 && s_conv <= s - 1 ? 1 : 0);
                    }
                }
                const int cn = last ? 0 : c + 1, sn = last ? s + 1 : s;
                if (rotate) w0 = (w0 + (c1 - s_seg[c] + L::RPW - 1) / L::RPW) % CW;
                g = s_seg[cn] + (warp - w0 + (warp < w0 ? CW : 0)) * L::RPW;
                c1 = s_seg[cn + 1];
                if (L::AHEAD && A.early && !bad && g < c1 && sn <= A.maxsw) {
                    __syncwarp();
                    taken = take(g, c1, sn, false);
                }
                bad = flow_bar_or(bad);
                if (bad) break;
            }
            if (bad) break;
            if (tid == 0) s_cnt = s;
            const int go = s_go;
            bad = go == 2;
            use_old = go == 1;
            if (go) break;
        }
        if (bad) {
            if (tid == 0) atomicExch(&A.ctl->fault, 1);
        } else {
            for (int i = tid; i < n; i += 32 * CW) {
                const int nd = A.node[row0 + i];
#pragma unroll
                for (int z = 0; z < 3; ++z)
                    A.sol[3 * (size_t)nd + z] = use_old ? __ldcg(A.old + 3 * (size_t)(row0 + i) + z) : xd[3 * (size_t)i + z];
            }
        }
        if (tid == 0) s_quit = 1;
    } else if (warp < CW + HW) {
        // ------------------------------------------------------ halo
        const int hl = tid - 32 * CW;
        for (int s = 1; s <= A.maxsw; ++s) {
            const unsigned long long tag = base + (unsigned)s;
            bool bad = false;
            for (int c = 0; c < ncol; ++c) {
                if constexpr (CL) {
                    const int nc = s_hseg[c + 1] - s_hseg[c];
                    if (nc > 0) {
                        bad = !cl_wait(&s_hal[c], (unsigned)(s - 1) & 1u, A.ctl);
                        // no value of the next sweep's colour c completes its phase before
                        // this: the barrier's one arrival is still to come
                        if (hl == 0 && !bad) mbar_expect_tx(&s_hal[c], (unsigned)nc * 3u * sizeof(XT));
                    }
                    bad = flow_bar_or(bad);
                    if (bad) break;
                    continue;
                }
                // one pair per thread: neighbouring pairs share their L2 requests
                constexpr int W = F32 ? 1 : 3;
                for (int b = W * s_hseg[c] + hl; b < W * s_hseg[c + 1] && !bad; b += 32 * HW) {
                    const int hb = b / W, z = b - hb * W;
                    XT *y = xs + 3 * (size_t)(n + hb);
                    ulonglong2 v[1];
                    bad = !flow_poll<1>(A.gx + W * (size_t)s_hrow[hb] + z, tag, F32 ? 32 : 0, A.ctl, v);
                    if constexpr (F32) {
                        y[0] = __uint_as_float((unsigned)v[0].x);
                        y[1] = __uint_as_float((unsigned)(v[0].x >> 32));
                        y[2] = __uint_as_float((unsigned)v[0].y);
                    } else {
                        y[z] = __longlong_as_double(v[0].x);
                    }
                }
                bad = flow_bar_or(bad);
                if (bad) break;
            }
            if (bad || s_go) break;
        }
    } else if (warp == CW + HW) {
        // ------------------------------------------------------ control
        for (int s = 1; s <= A.maxsw; ++s) {
            int it = 0;
            while (s_cnt < s && !s_quit && ++it < FLOW_POLLS) __nanosleep(20);
            if (!__all_sync(0xffffffffu, s_cnt >= s)) {
                if (lane == 0) s_bad = 1;
                break;
            }
            __threadfence_block();
            double a = 0.0, b = 0.0;
            for (int w = lane; w < NRED; w += 32) {
                a += s_red[s & 1][0][w];
                b += s_red[s & 1][1][w];
            }
#pragma unroll
            for (int u = 16; u > 0; u >>= 1) {
                a += __shfl_xor_sync(0xffffffffu, a, u);
                b += __shfl_xor_sync(0xffffffffu, b, u);
            }
            bool ok = true;
            if constexpr (CL) {
                const int sl = s & 3;
                if (lane < A.ntiles)
                    cl_push2(cl_addr(dyn0 + FLOW_CL_PART + 16u * (unsigned)(sl * FLOW_CLUSTER + t), lane), a, b,
                             cl_addr(dyn0 + FLOW_CL_PBAR + 8u * sl, lane));
                // the k-th use of slot sl, k = (s - 1) / 4 from sweep 1 on
                ok = cl_wait(&s_pbar[sl], (unsigned)((s - 1) >> 2) & 1u, A.ctl);
                const double2 v = lane < A.ntiles ? s_part[sl * FLOW_CLUSTER + lane] : make_double2(0.0, 0.0);
                a = v.x, b = v.y;
                __syncwarp();
                if (lane == 0 && ok) mbar_expect_tx(&s_pbar[sl], 16u * A.ntiles);
            } else {
                ulonglong2 *ps = A.part + (size_t)(s & 3) * A.ntiles * 2;
                const unsigned long long tag = base + (unsigned)s;
                if (lane == 0) {
                    st_pair(ps + 2 * t, __double_as_longlong(a), tag);
                    st_pair(ps + 2 * t + 1, __double_as_longlong(b), tag);
                }
                a = b = 0.0;
                for (int j = lane; j < A.ntiles && ok; j += 32) {
                    ulonglong2 v[2];
                    ok = flow_poll<2>(ps + 2 * j, tag, 0, A.ctl, v);
                    a += __longlong_as_double(v[0].x);
                    b += __longlong_as_double(v[1].x);
                }
            }
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) s_bad = 1;
                break;
            }
#pragma unroll
            for (int u = 16; u > 0; u >>= 1) {
                a += __shfl_xor_sync(0xffffffffu, a, u);
                b += __shfl_xor_sync(0xffffffffu, b, u);
            }
            const double err = a / b;
            const bool conv = err < A.tolerl;
            if (lane == 0) {
                if (t == 0 && (conv || s == A.maxsw)) {
                    A.ctl->err = err;
                    A.ctl->sweeps = (int)base + s;
                    A.ctl->conv = conv ? 1 : 0;
                }
                if (conv) s_conv = s;
                __threadfence_block();
                s_verdict = s;
            }
            if (conv) break;
        }
    } else if (lane == 0) {
        // ------------------------------------------------------ producer
        const uint64_t pol = l2_evict_first();
        const int c0 = A.cptr[t];
        auto issue = [&](int k, int slot) {
            const unsigned bytes = S == SLOTS ? L::SLOT : L::HB + 16u * (s_coff[k + 1] - s_coff[k]);
            const size_t at = S == SLOTS ? (size_t)(c0 + k) * L::SLOT : (size_t)(c0 + k) * L::HB + (size_t)s_coff[k] * 16;
            mbar_expect_tx(&s_full[slot], bytes);
            bulk_g2s(slots + (size_t)slot * L::SLOT, A.rec + at, bytes, &s_full[slot], pol);
        };
        for (int k = 0; k < nres; ++k) issue(k, k);
        int issued = 0, rs = 0;
        unsigned par = 1;        // the first round finds every slot empty
        bool go = nring > 0;
        for (int s = 1; s <= A.maxsw && go; ++s)
            for (int k = nres; k < nch && go; ++k) {
                if (issued >= nring) {
                    bool free = false;
                    for (int it = 0; it < FLOW_POLLS && !free && !s_quit; ++it) free = mbar_try_wait(&s_empty[nres + rs], par);
                    if (!free) {
                        go = false;
                        break;
                    }
                }
                issue(k, nres + rs);
                __threadfence_block();
                s_issued = ++issued;
                if (++rs == nring) {
                    rs = 0;
                    par ^= 1u;
                }
            }
        // no copy may be in flight when the CTA's shared memory is released
        for (int k = 0; k < nres; ++k) mbar_wait_bounded(&s_full[k], 0u);
        for (int j = max(0, issued - nring); j < issued; ++j)
            mbar_wait_bounded(&s_full[nres + j % nring], (unsigned)((j / nring) & 1));
    }
    if constexpr (CL) {
        // No CTA leaves while another may still write to it.  A solve that ends
        // has waited for every value sent to it; one that gave up leaves some in
        // flight, so its CTAs wait a millisecond, where a value takes less than
        // a microsecond.
        cl_sync();
        if (((volatile const SorCtl *)A.ctl)->fault)
            for (int k = 0; k < 1000; ++k) __nanosleep(1000);
    }
}

// Place of row r of the tile with rows [r0, ...) and chunks from c0 on: its
// chunk's record and its row in the chunk.
template <typename T, int S>
__device__ __forceinline__ unsigned char *flow_record(unsigned char *rec, int r, int r0, int c0, const unsigned *voff, int &ri)
{
    using L = FlowRow<T, S>;
    const int k = (r - r0) / L::CH;
    ri = (r - r0) % L::CH;
    return rec + (S == SLOTS ? (size_t)(c0 + k) * L::SLOT : (size_t)(c0 + k) * L::HB + (size_t)voff[r0 + k * L::CH] * 16);
}

// The assembled rows in tile order and format, with the right-hand side and
// the correctly rounded reciprocals of the diagonal in the row's extras (the
// FP32 solve's first residual is the right-hand side and its base zero);
// one warp per row.
template <typename T, int S>
__global__ void __launch_bounds__(256) k_flow_pack(BlockDev B, const int *__restrict__ src, const unsigned *__restrict__ voff,
                                                   const int *__restrict__ tile_of_row, const int *__restrict__ trow,
                                                   const int *__restrict__ cptr, const unsigned char *__restrict__ from,
                                                   const double *__restrict__ rhs, unsigned char *__restrict__ rec)
{
    using L = FlowRow<T, S>;
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < B.R; r += gridDim.x * wpb) {
        const int p = src[r], t = tile_of_row[r], r0 = trow[t];
        int ri;
        unsigned char *ch = flow_record<T, S>(rec, r, r0, cptr[t], voff, ri);
        const double *b = B.blk + (size_t)p * brow_of(S);
        const unsigned char *f = from + (size_t)r * S;
        if (S == SLOTS) {
            T *d = reinterpret_cast<T *>(ch + L::HB + ri * L::VB);
            const int o = lane >= S ? 0xFF : !L::F32 ? f[lane] : lane < B.nslot[p] ? lane : 0xFF;
#pragma unroll
            for (int z = 0; z < 9; ++z)
                if (lane < S) d[z * S + lane] = o < S ? (T)b[z * S + o] : (T)0;
        } else {
            const int ns = B.nslot[p];
            T *d = reinterpret_cast<T *>(ch + L::HB + (size_t)(voff[r] - voff[r - ri]) * 16);
            for (int sl = lane; sl < ns; sl += 32) {
                const int o = L::F32 ? sl : f[sl];
#pragma unroll
                for (int z = 0; z < 9; ++z) d[z * ns + sl] = (T)b[z * S + o];
            }
        }
        if (lane < L::EW) {
            double *e = reinterpret_cast<double *>(ch + L::CH * L::MB + ri * L::EB);
            const int nd = B.perm[p];
            e[lane] = lane < 3 ? rhs[3 * nd + lane] : lane < 6 ? 1.0 / (double)(T)b[4 * (lane - 3) * S] : 0.0;
        }
    }
}

// Index words of every row (FlowRow) from the tile-local columns lcol[R][S]
// in storage order and the rows' headers; eoff[node] (when set) receives the
// place of the node's extras in the records, in doubles.
template <typename T, int S>
__global__ void k_flow_meta(int R, const uint16_t *__restrict__ lcol, const uint16_t *__restrict__ head,
                            const unsigned char *__restrict__ from, const unsigned *__restrict__ voff,
                            const int *__restrict__ tile_of_row, const int *__restrict__ trow,
                            const int *__restrict__ cptr, const int *__restrict__ node,
                            unsigned char *__restrict__ rec, unsigned *__restrict__ eoff)
{
    using L = FlowRow<T, S>;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int r = (int)(tid / L::LPR), q = (int)(tid % L::LPR);
    if (r >= R) return;
    const int t = tile_of_row[r];
    int ri;
    unsigned char *ch = flow_record<T, S>(rec, r, trow[t], cptr[t], voff, ri);
    const int ne = head[r] & 0x7f, nl = (head[r] >> 7) & 0x3f;
    uint16_t *m = reinterpret_cast<uint16_t *>(ch + ri * L::MB) + q * L::MW;
    for (int j = 0; j < L::MW; ++j) {
        const int p = q + L::LPR * j;
        int at = j < L::SPL && p < S ? L::stored(p, L::F32 ? ne + nl : ne, L::F32 ? 0 : nl) : -1;
        if (L::F32 && at >= 0)      // FP32 rows keep the slots' order
            for (int k = 0; k < S; ++k)
                if (from[(size_t)r * S + k] == p) at = k;
        m[j] = at >= 0 ? lcol[(size_t)r * S + at] : 0;
    }
    if (q == L::HQ) m[L::SPL - 1] = (uint16_t)(L::F32 ? (ne + nl) | (head[r] & 0x8000) : head[r]);
    if (S != SLOTS && q == L::HQ + 1) m[L::SPL - 1] = (uint16_t)(voff[r] - voff[r - ri]);
    if (eoff && q == 0) eoff[node[r]] = (unsigned)((ch + L::CH * L::MB + ri * L::EB - rec) / 8);
}

}  // namespace fasdev
