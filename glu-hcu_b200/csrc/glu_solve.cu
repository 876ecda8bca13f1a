// Triangular solves with the factors, on the device.
//
// The reference solves on the CPU in FP32 (Symbolic_Matrix::solve,
// src/symbolic.cc:200-251): permute/scale b, unit-L column sweep (:226-229),
// U column sweep with the diagonal divide (:232-239), permute/scale back.
// Here the same sweeps run on the GPU:
//
//  * sparse columns (in front of the dense trailing block) are processed level
//    by level, with level sets of each sweep's own dependency graph computed
//    once per pattern (the L and U sweeps by supernodes, glu_solve_snode.cu,
//    unless those are off): a level with many items, chunks of a column's or
//    row's entries, gets its own launch (a warp per item); a run of thin levels
//    executes inside one thread-block cluster that steps from level to level
//    with hardware cluster barriers.  All four sweeps scatter (x_i -= L(i,j)
//    x_j with atomics; the transposed ones along the rows);
//  * the dense trailing block is solved by row blocks of 64: a block adds the
//    contribution of every finished earlier block (one 64 x 64 tile each, in
//    registers) and then multiplies by the inverse of its diagonal tile; blocks
//    are claimed in order through a ticket and wait (bounded) for the entries
//    they read;
//  * the coupling between the two (U entries of tail columns in sparse rows)
//    is one parallel scatter over the tail columns.
#include <cooperative_groups.h>

#include <algorithm>

#include "glu_common.cuh"
#include "glu_kernels.h"
#include "glu_tri.cuh"

namespace cg = cooperative_groups;

namespace glu {


// ------------------------------------------------------------ sparse sweeps --
// Every sweep is in scatter form: once x_j is final, the entries of its
//   SWEEP_L : CSC column j below the diagonal   (x_j = y_j)
//   SWEEP_U : CSC column j above the diagonal   (x_j = y_j / U(j,j))
//   SWEEP_UT: CSR row j right of the diagonal    (x_j = y_j / U(j,j))
//   SWEEP_LT: CSR row j left of the diagonal     (x_j = y_j)
// are subtracted: y_target -= entry * x_j.  A long column or row is split into
// items of kSweepChunk entries that run in parallel; every item of j reads
// the same y_j (nothing writes y_j while its level runs) and the dividing
// sweeps store the finished x_j to xo (item 0 of j).
//
// What bounds them is the chain of dependent loads of a level (item, entry,
// CSC position, value, then y_j) and the updates' way through L2, so all but
// y_j is read ahead: by a level's launch before it waits for the previous
// one, in the cluster kernel while the level before runs (its items' records
// one level earlier still).  n = 100,000 transposed: 5.5 -> 3.7 us per level
// launch, the runs of thin levels 30 -> 23 us, the three solves
// and refinements of an adjoint 822 -> 590 us.
struct SweepItem {
    uint2 at;       // j, first entry
    uint32_t info;  // entries | kSweepFirst; ~0u: none
};
template <int kMode>
struct SweepEntries {
    static constexpr int kK = kSweepChunk / 32;
    uint32_t j, count, tgt[kK];
    float v[kK], d;
    bool first;

    __device__ __forceinline__ void load(const DevPattern &P, const float *__restrict__ val, const SweepItem &I,
                                         uint32_t lane) {
        constexpr bool kDiv = (kMode == SWEEP_U || kMode == SWEEP_UT);
        constexpr bool kRow = (kMode == SWEEP_UT || kMode == SWEEP_LT);
        j = I.at.x;
        count = I.info & (kSweepFirst - 1u);
        first = (I.info & kSweepFirst) != 0;
        d = kDiv ? __ldg(val + __ldg(P.diag + j)) : 1.0f;
        uint32_t pos[kK];
#pragma unroll
        for (int k = 0; k < kK; ++k) {
            const uint32_t e = I.at.y + lane + 32 * k;
            if (lane + 32 * k < count) {
                tgt[k] = __ldg((kRow ? P.cidx : P.ridx) + e);
                pos[k] = kRow ? __ldg(P.cpos + e) : e;
            }
        }
#pragma unroll
        for (int k = 0; k < kK; ++k)
            if (lane + 32 * k < count) v[k] = __ldg(val + pos[k]);
    }
    __device__ __forceinline__ void apply(float *y, float *xo, uint32_t nrhs, uint32_t n, uint32_t lane) const {
        constexpr bool kDiv = (kMode == SWEEP_U || kMode == SWEEP_UT);
        for (uint32_t r = 0; r < nrhs; ++r) {
            float *yr = y + size_t(r) * n;
            float xj = __ldcg(yr + j);
            if (kDiv) {
                xj = xj / d;
                if (first && lane == 0) xo[size_t(r) * n + j] = xj;
            }
            if (xj == 0.0f) continue;
#pragma unroll
            for (int k = 0; k < kK; ++k)
                if (lane + 32 * k < count) atomicAdd(yr + tgt[k], -__fmul_rn(v[k], xj));
        }
    }
};
__device__ __forceinline__ SweepItem sweep_item(const uint2 *__restrict__ items, const uint16_t *__restrict__ info,
                                                uint32_t i, uint32_t end) {
    if (i >= end) return SweepItem{make_uint2(0u, 0u), ~0u};
    return SweepItem{__ldg(items + i), __ldg(info + i)};
}

// One level, own launch: warps over its items [i0, i1).
template <int kMode>
__global__ void __launch_bounds__(256) k_sweep_level(DevPattern P, const float *__restrict__ val, float *y, float *xo,
                                                     uint32_t nrhs, const uint2 *__restrict__ items,
                                                     const uint16_t *__restrict__ info, uint32_t i0, uint32_t i1,
                                                     uint64_t vstride, uint64_t ystride) {
    pdl_release();
    val += blockIdx.z * vstride;  // value set blockIdx.z, its right-hand sides
    y += blockIdx.z * ystride;
    xo += blockIdx.z * ystride;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nw = gridDim.x * (blockDim.x >> 5);
    uint32_t i = i0 + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    SweepEntries<kMode> E;
    if (i < i1) E.load(P, val, sweep_item(items, info, i, i1), lane);
    pdl_wait();  // the previous level's y
    while (i < i1) {
        E.apply(y, xo, nrhs, P.n, lane);
        i += nw;
        if (i < i1) E.load(P, val, sweep_item(items, info, i, i1), lane);
    }
}

// A run of thin levels [l0, l1) inside one cluster; cluster barrier between
// levels; values of y written by other blocks are read through L2.
template <int kMode>
__global__ void __launch_bounds__(kSolveChainThreads) k_sweep_chain(DevPattern P, const float *__restrict__ val,
                                                                    float *y, float *xo, uint32_t nrhs,
                                                                    const uint2 *__restrict__ items,
                                                                    const uint16_t *__restrict__ info,
                                                                    const uint32_t *__restrict__ level_off,
                                                                    uint32_t l0, uint32_t l1, uint64_t vstride,
                                                                    uint64_t ystride) {
    pdl_release();
    val += blockIdx.z * vstride;  // value set blockIdx.z, its right-hand sides
    y += blockIdx.z * ystride;
    xo += blockIdx.z * ystride;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t nblk = cluster.num_blocks();
    const uint32_t rank = cluster.block_rank();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t wpb = blockDim.x >> 5;
    const uint32_t w0 = rank * wpb + (threadIdx.x >> 5), nw = nblk * wpb;
    // this level's items [o0, o1), the next level's [o1, o2): this warp's first
    // ones' entries (E, F), and the record of its first one after those
    uint32_t o0 = __ldg(level_off + l0), o1 = __ldg(level_off + l0 + 1);
    uint32_t o2 = l0 + 1 < l1 ? __ldg(level_off + l0 + 2) : o1;
    SweepEntries<kMode> E, F;
    {
        const SweepItem I = sweep_item(items, info, o0 + w0, o1);
        if (I.info != ~0u) E.load(P, val, I, lane);
    }
    SweepItem I = sweep_item(items, info, o1 + w0, o2);
    pdl_wait();  // y
    for (uint32_t l = l0; l < l1; ++l) {
        const uint32_t o3 = l + 2 < l1 ? __ldg(level_off + l + 3) : o2;
        if (I.info != ~0u) F.load(P, val, I, lane);
        I = sweep_item(items, info, o2 + w0, o3);
        if (o0 + w0 < o1) E.apply(y, xo, nrhs, P.n, lane);
        for (uint32_t i = o0 + w0 + nw; i < o1; i += nw) {
            E.load(P, val, sweep_item(items, info, i, o1), lane);
            E.apply(y, xo, nrhs, P.n, lane);
        }
        cluster.sync();
        E = F;
        o0 = o1, o1 = o2, o2 = o3;
    }
}

// Coupling of the dense tail with the sparse unknowns, tail columns / rows j
// (x_j final): y_i -= U(i,j) x_j for the U entries of tail column j in rows i <
// t (kRow = false, before the sparse U sweep), or y_c -= L(j,c) x_j for the L
// entries of tail row j in columns c < t (kRow = true, before the sparse L^T
// sweep).  A warp takes the entries [64 blockIdx.x, 64 blockIdx.x + 64) of
// kCoupleCols neighbouring columns.
// What bounds it is the updates in L2, many on the same unknowns: neighbouring
// tail columns mostly hold the same rows at the same places, so a lane sums up
// their products as long as the row stays the same and issues one update.  The
// entries are read while the dense sweep before still runs (a chained launch).
// After its sweep: order 3,968 66 -> 55 us, order 1,100 20 -> 8 us (a warp per
// column and an update per entry); order 9,216, 12 value sets of four
// right-hand sides 1,141 -> 640 us.
constexpr int kCoupleCols = 8;
constexpr int kCoupleEach = 2;  // entries of a column per lane
constexpr uint32_t kCoupleRhs = 4;
template <bool kRow>
__global__ void __launch_bounds__(256) k_tail_coupling(DevPattern P, uint32_t t, uint32_t m,
                                                       const uint32_t *__restrict__ tail_start,
                                                       const float *__restrict__ val, float *y, uint32_t nrhs,
                                                       uint64_t vstride, uint64_t ystride) {
    pdl_release();
    // value set and kCoupleRhs right-hand sides of it
    const uint32_t shares = (nrhs + kCoupleRhs - 1) / kCoupleRhs, z = blockIdx.z / shares;
    const uint32_t v0 = (blockIdx.z - z * shares) * kCoupleRhs, v1 = min(v0 + kCoupleRhs, nrhs);
    val += z * vstride;
    y += z * ystride;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t j0 = (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kCoupleCols;
    const uint32_t n = P.n, off = blockIdx.x * (32 * kCoupleEach);
    // lane g: column j0 + g, its entries from `off` on
    const bool own = lane < uint32_t(kCoupleCols) && j0 + lane < m;
    uint32_t b = 0, e = 0;
    if (own) {
        b = __ldg((kRow ? P.rptr : P.cptr) + t + j0 + lane) + off;
        e = __ldg(tail_start + j0 + lane);
    }
    const bool any = __any_sync(0xffffffffu, b < e);
    uint32_t tgt[kCoupleCols][kCoupleEach];
    float v[kCoupleCols][kCoupleEach];
    if (any) {
        uint32_t pos[kCoupleCols][kCoupleEach];
#pragma unroll
        for (int g = 0; g < kCoupleCols; ++g) {
            const uint32_t bg = __shfl_sync(0xffffffffu, b, g), eg = __shfl_sync(0xffffffffu, e, g);
#pragma unroll
            for (int u = 0; u < kCoupleEach; ++u) {
                const uint32_t p = bg + 32 * u + lane;
                tgt[g][u] = p < eg ? __ldg((kRow ? P.cidx : P.ridx) + p) : 0xffffffffu;
                pos[g][u] = p < eg ? (kRow ? __ldg(P.cpos + p) : p) : 0u;
            }
        }
#pragma unroll
        for (int g = 0; g < kCoupleCols; ++g)
#pragma unroll
            for (int u = 0; u < kCoupleEach; ++u) v[g][u] = tgt[g][u] != 0xffffffffu ? __ldg(val + pos[g][u]) : 0.0f;
    }
    pdl_wait();  // the tail's unknowns
    if (!any) return;
    float xs[kCoupleRhs];
#pragma unroll
    for (int q = 0; q < int(kCoupleRhs); ++q)
        xs[q] = (own && v0 + q < v1) ? __ldcg(y + size_t(v0 + q) * n + t + j0 + lane) : 0.0f;
#pragma unroll
    for (int q = 0; q < int(kCoupleRhs); ++q) {
        if (v0 + q >= v1) break;
        float *yr = y + size_t(v0 + q) * n;
        const float x = xs[q];
        float sum[kCoupleEach];
        uint32_t row[kCoupleEach];
#pragma unroll
        for (int u = 0; u < kCoupleEach; ++u) sum[u] = 0.0f, row[u] = 0xffffffffu;
#pragma unroll
        for (int g = 0; g < kCoupleCols; ++g) {
            const float xj = __shfl_sync(0xffffffffu, x, g);
            if (xj == 0.0f) continue;
#pragma unroll
            for (int u = 0; u < kCoupleEach; ++u) {
                if (tgt[g][u] == 0xffffffffu) continue;
                if (tgt[g][u] != row[u]) {
                    if (row[u] != 0xffffffffu) atomicAdd(yr + row[u], -sum[u]);
                    sum[u] = 0.0f;
                    row[u] = tgt[g][u];
                }
                sum[u] = fmaf(v[g][u], xj, sum[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kCoupleEach; ++u)
            if (row[u] != 0xffffffffu) atomicAdd(yr + row[u], -sum[u]);
    }
}

// y[j] = xo[j] for the sparse unknowns j < t (after a dividing sweep).
__global__ void k_copy_sparse(const float *__restrict__ xo, float *y, uint32_t t, uint32_t n) {
    const size_t off = size_t(blockIdx.y) * n;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < t; j += gridDim.x * blockDim.x) y[off + j] = xo[off + j];
}

template <int kMode>
static cudaError_t run_sweep(const DevPattern &P, const SolvePlanDev &S, const float *val, float *y, float *xo,
                             uint32_t nrhs, const SolveBatch &B, cudaStream_t st) {
    const SweepPlan &sw = S.sweep[kMode];
    const uint64_t ystride = uint64_t(nrhs) * P.n;
    // blocks per value set of a wide level: a warp per item, at most about
    // eight blocks per SM in all
    const uint32_t most = std::max<uint32_t>(1u, (148u * 8u + B.count - 1) / B.count);
    for (uint32_t i = 0; i < sw.nsteps; ++i) {
        const SweepStep &s = sw.steps[i];
        if (s.kind == 0) {
            const cudaError_t e = launch_chained(k_sweep_level<kMode>, dim3(std::min(most, (s.i1 - s.i0 + 7) / 8), 1, B.count),
                                                 dim3(256), 0, st, P, val, y, xo, nrhs, sw.items, sw.info, s.i0, s.i1,
                                                 B.vstride, ystride);
            if (e != cudaSuccess) return e;
        } else {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(S.cluster, 1, B.count);
            cfg.blockDim = dim3(kSolveChainThreads, 1, 1);
            cfg.stream = st;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = S.cluster;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 2;
            cudaError_t e = cudaLaunchKernelEx(&cfg, k_sweep_chain<kMode>, P, val, y, xo, nrhs, sw.items, sw.info,
                                               sw.level_off, s.l0, s.l1, B.vstride, ystride);
            if (e != cudaSuccess) return e;
        }
    }
    if ((kMode == SWEEP_U || kMode == SWEEP_UT) && S.t > 0) {
        uint32_t bx = (S.t + 255) / 256;
        if (bx > 1024) bx = 1024;
        k_copy_sparse<<<dim3(bx, nrhs * B.count, 1), 256, 0, st>>>(xo, y, S.t, P.n);
    }
    return cudaGetLastError();
}

// --------------------------------------------------------- dense tail sweeps --
// Solve T x = r on the dense block (entries [t, t + m) of the vectors), where
//   kMode 0: T = L   (unit lower,      T(i,c) = val[doff[c] + i])
//   kMode 1: T = U   (upper,           T(i,c) = val[doff[c] + i])
//   kMode 2: T = U^T (lower,           T(i,c) = val[doff[i] + c])
//   kMode 3: T = L^T (unit upper,      T(i,c) = val[doff[i] + c])
// A block of threads owns 64 rows of up to R right-hand sides of one value
// set; these items are claimed in solve order (ascending for lower, descending
// for upper) through a ticket, interleaved over the value sets and the groups
// of right-hand sides, so every chain advances at once and an item waits only
// on items of smaller tickets, which are running or done.
//
// What bounds it: the chain of m / 64 blocks, each of which needs the one
// before.  Hence
//  * a solved entry is its own flag: the output starts as kUnsolved (a NaN
//    pattern no solution holds) and a reader polls the value it needs, which
//    saves the fence, the flag and the second trip to L2 on every link;
//  * a warp polls, stages and multiplies its own columns: no barrier of the
//    block while the finished blocks' tiles stream by (the next tile and its x
//    are in flight meanwhile);
//  * the diagonal block's solve is a product with its inverse (dinv, computed
//    once per factorization by k_dense_diag_inv), a parallel mat-vec instead
//    of 64 dependent steps; two block barriers per link remain.  It stands
//    column-major, so a warp's load of it is one line (row-major its 32 lines
//    per load took as long as a link).
// Measured (B200): a link takes 0.82 us at order 1,920 with one right-hand side
// (24.7 us a sweep; 26.5 us with row-major inverses, 87 us with a flag per block
// and three barriers per tile), and 32 right-hand sides take 36 us (8.5 ms as
// groups of four one after another inside the block); transposed, order 3,776,
// 54 us (193 us).  Blocks of 128 rows take 22, 34 and 39 us, but their inverses
// cost 10 us more per factorization than these, which a step pays every time.
// The forward sweep reads y and writes xo, the backward sweep reads xo and
// writes y: the forward one leaves kUnsolved in the rows of y it has read, and
// the transform in front of the solve leaves it in xo (SolveInit).
constexpr int kRB = 64;
constexpr int kRHSChunk = 4;

__device__ __forceinline__ float ld_poll(const float *p) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool unsolved(float v) { return __float_as_uint(v) == kUnsolved; }
__device__ __forceinline__ void publish(float *p, float v) {
    // (arithmetic gives the canonical NaN, never this pattern; an input may)
    if (unsolved(v)) v = __uint_as_float(0x7FFFFFFFu);
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// Polls the warp's N values per lane (v[k] at at(k); entries that are not
// needed hold 0) until all are solved; bounded, a wait that sees another's
// timeout gives up early.  Only the block whose turn is next polls without a
// pause: the others' polls go to the same L2 slice as its own (transposed,
// order 3,776: 54 us, 59 without the pause).
template <int N, class At>
__device__ __forceinline__ void wait_solved(float (&v)[N], At &&at, bool next, uint32_t *status, uint32_t limit) {
    for (uint32_t spins = 0;; ++spins) {
        bool open = false;
#pragma unroll
        for (int k = 0; k < N; ++k) open |= unsolved(v[k]);
        if (!__any_sync(0xffffffffu, open)) return;
        if (spins >= limit) {
            if ((threadIdx.x & 31) == 0) atomicOr(status, DEV_TIMEOUT);
            return;
        }
        if (!next) __nanosleep(60);
        if ((spins & 1023u) == 1023u && (ld_acquire_gpu(status) & DEV_TIMEOUT)) return;
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (unsolved(v[k])) v[k] = ld_poll(at(k));
    }
}

// Inverses of the 64 x 64 diagonal blocks of the dense tail: blockIdx.y = 0
// the unit lower L_bb, 1 the upper U_bb; dinv[z][b][which] column-major (rows
// past the tail's end are the identity).  blockIdx.z selects the value set.
__global__ void __launch_bounds__(256) k_dense_diag_inv(const float *__restrict__ val, uint64_t dstride,
                                                         const uint32_t *__restrict__ doff, uint32_t m,
                                                         float *__restrict__ dinv) {
    __shared__ TriInverse T;
    const uint32_t b = blockIdx.x, which = blockIdx.y;
    const uint32_t nb = (m + kRB - 1) / kRB;
    val += blockIdx.z * dstride;
    const uint32_t rb0 = b * kRB, rows = min(uint32_t(kRB), m - rb0);
    tri_invert(T, which, rows, dinv + ((size_t(blockIdx.z) * nb + b) * 2 + which) * kRB * kRB,
               [&](uint32_t i, uint32_t c) { return val[doff[rb0 + c] + rb0 + i]; });
}

// One item: its value set, first right-hand side and block (in solve order).
struct TrsvItem {
    uint32_t z, v0, tk;
};
__device__ __forceinline__ TrsvItem trsv_item(uint32_t tg, uint32_t count, uint32_t chunks, uint32_t R) {
    const uint32_t per = count * chunks, rem = tg % per;
    return TrsvItem{rem / chunks, (rem % chunks) * R, tg / per};
}

// T = L (kMode 0) or U (kMode 1): T(i, c) down the columns.  Warp w: rows
// 32 (w & 1) + lane, columns 16 (w >> 1) .. + 15 of every tile, in registers;
// the 16 x R values of x go through a stretch of shared memory of the warp's
// own, read back as broadcasts.
template <int kMode, int R>
__global__ void __launch_bounds__(256, R == 1 ? 4 : 3)
    k_dense_trsv(const float *__restrict__ val, const uint32_t *__restrict__ doff, uint32_t t, uint32_t m, float *rin,
                 float *out, uint32_t n, uint32_t nrhs, uint32_t chunks, uint32_t count, uint32_t *ticket,
                 uint32_t *status, uint32_t spin_limit, uint32_t ticket_base, uint64_t dstride, uint64_t ystride,
                 const float *__restrict__ dinv) {
    constexpr bool kLower = kMode == 0;
    constexpr int kW = 16;               // columns per warp and tile
    constexpr int kX = R == 1 ? 1 : R / 2;  // x values a lane polls: kW * R of them on 32 lanes
    __shared__ __align__(16) float xs[8][2][kW * R];
    __shared__ float part[2][4][kRB][R];
    __shared__ uint32_t s_item;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nb = (m + kRB - 1) / kRB;
    pdl_release();  // the coupling after an upper sweep reads its entries meanwhile
    if (tid == 0) s_item = atomicAdd(ticket, 1u) + ticket_base;
    __syncthreads();
    if (s_item >= nb * count * chunks) return;
    const TrsvItem it = trsv_item(s_item, count, chunks, R);
    const uint32_t tk = it.tk, nr = min(uint32_t(R), nrhs - it.v0);
    val += it.z * dstride;
    rin += it.z * ystride + size_t(it.v0) * n + t;
    out += it.z * ystride + size_t(it.v0) * n + t;
    const uint32_t b = kLower ? tk : nb - 1 - tk;
    const uint32_t rb0 = b * kRB, rows = min(uint32_t(kRB), m - rb0);
    const uint32_t row = tid & (kRB - 1), q = tid / kRB, col0 = q * kW;
    const float *inv = dinv + ((size_t(it.z) * nb + b) * 2 + kMode) * kRB * kRB + col0 * kRB + row;
    // lane's x values: column lane % 16, right-hand sides lane / 16 + 2 k
    const uint32_t xc = lane & 15, xr = lane >> 4;
    const bool rowok = row < rows;
    auto load_tile = [&](uint32_t s, float (&tv)[kW]) {
        const uint32_t cb = (kLower ? s : nb - 1 - s) * kRB + col0;
        const uint32_t off = cb + xc < m ? __ldg(doff + cb + xc) : 0u;
#pragma unroll
        for (int k = 0; k < kW; ++k) {
            const uint32_t o = __shfl_sync(0xffffffffu, off, k);
            tv[k] = (rowok && cb + k < m) ? __ldg(val + o + rb0 + row) : 0.0f;
        }
    };
    auto x_at = [&](uint32_t s, int k) -> const float * {
        const uint32_t c = (kLower ? s : nb - 1 - s) * kRB + col0 + xc;
        return out + size_t(R == 1 ? 0u : xr + 2 * k) * n + c;
    };
    auto load_x = [&](uint32_t s, float (&v)[kX]) {
        const uint32_t c = (kLower ? s : nb - 1 - s) * kRB + col0 + xc;
#pragma unroll
        for (int k = 0; k < kX; ++k) v[k] = (c < m && (R == 1 ? 0u : xr + 2 * k) < nr) ? ld_poll(x_at(s, k)) : 0.0f;
    };
    auto stage = [&](float *dst, const float (&v)[kX]) {
#pragma unroll
        for (int k = 0; k < kX; ++k)
            if (R > 1 || xr == 0) dst[xc * R + (R == 1 ? 0u : xr + 2 * k)] = v[k];
        __syncwarp();
    };
    auto multiply = [&](float (&acc)[R], const float (&tv)[kW], const float *src) {
        const float4 *s4 = reinterpret_cast<const float4 *>(src);
        if (R == 1) {
#pragma unroll
            for (int k = 0; k < kW; k += 4) {
                const float4 v = s4[k / 4];
                acc[0] = fmaf(tv[k], v.x, acc[0]);
                acc[0] = fmaf(tv[k + 1], v.y, acc[0]);
                acc[0] = fmaf(tv[k + 2], v.z, acc[0]);
                acc[0] = fmaf(tv[k + 3], v.w, acc[0]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < kW; ++k)
#pragma unroll
                for (int r = 0; r < R; r += 4) {
                    const float4 v = s4[(k * R + r) / 4];
                    acc[r % R] = fmaf(tv[k], v.x, acc[r % R]);
                    acc[(r + 1) % R] = fmaf(tv[k], v.y, acc[(r + 1) % R]);
                    acc[(r + 2) % R] = fmaf(tv[k], v.z, acc[(r + 2) % R]);
                    acc[(r + 3) % R] = fmaf(tv[k], v.w, acc[(r + 3) % R]);
                }
        }
    };
    // the right-hand sides of the columns this warp takes in the diagonal product
    float rv[kX];
#pragma unroll
    for (int k = 0; k < kX; ++k) {
        const uint32_t r = R == 1 ? 0u : xr + 2 * k;
        rv[k] = (col0 + xc < rows && r < nr) ? __ldcg(rin + size_t(r) * n + rb0 + col0 + xc) : 0.0f;
    }
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0f;
    float tv[kW], xv[kX];
    if (tk > 0) {
        load_tile(0, tv);
        load_x(0, xv);
    } else {
#pragma unroll
        for (int k = 0; k < kW; ++k) tv[k] = __ldg(inv + k * kRB);
    }
    for (uint32_t s = 0; s < tk; ++s) {
        float tn[kW], xn[kX];
        if (s + 1 < tk) {  // the next tile and a first look at its x, else the diagonal's inverse
            load_tile(s + 1, tn);
            load_x(s + 1, xn);
        } else {
#pragma unroll
            for (int k = 0; k < kW; ++k) tn[k] = __ldg(inv + k * kRB);
#pragma unroll
            for (int k = 0; k < kX; ++k) xn[k] = 0.0f;
        }
        wait_solved(xv, [&](int k) { return x_at(s, k); }, s + 1 == tk, status, spin_limit);
        float *buf = xs[warp][s & 1];
        stage(buf, xv);
        multiply(acc, tv, buf);
#pragma unroll
        for (int k = 0; k < kW; ++k) tv[k] = tn[k];
#pragma unroll
        for (int k = 0; k < kX; ++k) xv[k] = xn[k];
    }
    // r = b - (contributions) for the block's rows, then x = T_bb^-1 r
#pragma unroll
    for (int r = 0; r < R; ++r) part[0][q][row][r] = acc[r];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kX; ++k) {
        const uint32_t c = col0 + xc, r = R == 1 ? 0u : xr + 2 * k;
        xv[k] = rv[k] - ((part[0][0][c][r] + part[0][1][c][r]) + (part[0][2][c][r] + part[0][3][c][r]));
    }
    float *buf = xs[warp][tk & 1];
    stage(buf, xv);
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0f;
    multiply(acc, tv, buf);
#pragma unroll
    for (int r = 0; r < R; ++r) part[1][q][row][r] = acc[r];
    __syncthreads();
    for (uint32_t e = tid; e < uint32_t(kRB * R); e += 256) {
        const uint32_t i = e % kRB, r = e / kRB;
        if (i < rows && r < nr) {
            publish(out + size_t(r) * n + rb0 + i,
                    (part[1][0][i][r] + part[1][1][i][r]) + (part[1][2][i][r] + part[1][3][i][r]));
            if (kLower) rin[size_t(r) * n + rb0 + i] = __uint_as_float(kUnsolved);  // read by all warps: output of the backward sweep
        }
    }
}

// Sums of N values per lane over the warp: lane L returns with the sum of
// value L % N (N = 8 or 32, the sums repeat every N lanes).  Each halving
// step keeps one half of the values and adds the partner's.
template <int N>
__device__ __forceinline__ float warp_transpose_sum(float (&v)[N], uint32_t lane) {
#pragma unroll
    for (int h = N / 2; h > 0; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float keep = up ? v[k + h] : v[k], give = up ? v[k] : v[k + h];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, give, h);
        }
    }
    float s = v[0];
#pragma unroll
    for (int h = N; h < 32; h <<= 1) s += __shfl_xor_sync(0xffffffffu, s, h);
    return s;
}

// T = U^T (kMode 2) or L^T (kMode 3): T(i, c) along c.  Warp w: rows 8 w ..
// 8 w + 7, lane: columns lane and lane + 32 of every tile; a lane polls the x
// of its own two columns and the row sums are reduced once, after the last
// tile.
template <int kMode, int R>
__global__ void __launch_bounds__(256, R == 1 ? 3 : 2)
    k_dense_trsv_trans(const float *__restrict__ val, const uint32_t *__restrict__ doff, uint32_t t, uint32_t m,
                       float *rin, float *out, uint32_t n, uint32_t nrhs, uint32_t chunks, uint32_t count,
                       uint32_t *ticket, uint32_t *status, uint32_t spin_limit, uint32_t ticket_base,
                       uint64_t dstride, uint64_t ystride, const float *__restrict__ dinv) {
    constexpr bool kLower = kMode == 2;
    constexpr int kRows = 8;
    constexpr int kWhich = kMode == 3 ? 0 : 1;  // inverse of L or of U
    __shared__ float rs[kRB][R];
    __shared__ uint32_t s_item;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nb = (m + kRB - 1) / kRB;
    pdl_release();  // the coupling after an upper sweep reads its entries meanwhile
    if (tid == 0) s_item = atomicAdd(ticket, 1u) + ticket_base;
    __syncthreads();
    if (s_item >= nb * count * chunks) return;
    const TrsvItem it = trsv_item(s_item, count, chunks, R);
    const uint32_t tk = it.tk, nr = min(uint32_t(R), nrhs - it.v0);
    val += it.z * dstride;
    rin += it.z * ystride + size_t(it.v0) * n + t;
    out += it.z * ystride + size_t(it.v0) * n + t;
    const uint32_t b = kLower ? tk : nb - 1 - tk;
    const uint32_t rb0 = b * kRB, rows = min(uint32_t(kRB), m - rb0);
    const uint32_t i0 = warp * kRows;
    const float *inv = dinv + ((size_t(it.z) * nb + b) * 2 + kWhich) * kRB * kRB;
    uint32_t base[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) base[i] = i0 + i < rows ? __ldg(doff + rb0 + i0 + i) : 0u;
    auto load_tile = [&](uint32_t s, float (&tv)[2 * kRows]) {
        const uint32_t c = (kLower ? s : nb - 1 - s) * kRB + lane;
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            tv[2 * i] = (i0 + i < rows && c < m) ? __ldg(val + base[i] + c) : 0.0f;
            tv[2 * i + 1] = (i0 + i < rows && c + 32 < m) ? __ldg(val + base[i] + c + 32) : 0.0f;
        }
    };
    // row i of T_bb^-1 is column i of the stored inverse
    auto load_inv = [&](float (&tv)[2 * kRows]) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < kRows; ++i) tv[2 * i + h] = __ldg(inv + (i0 + i) * kRB + lane + 32 * h);
    };
    auto x_at = [&](uint32_t s, int k) -> const float * {
        return out + size_t(k >> 1) * n + (kLower ? s : nb - 1 - s) * kRB + lane + 32 * (k & 1);
    };
    auto load_x = [&](uint32_t s, float (&v)[2 * R]) {
        const uint32_t c = (kLower ? s : nb - 1 - s) * kRB + lane;
#pragma unroll
        for (int k = 0; k < 2 * R; ++k)
            v[k] = (c + 32 * (k & 1) < m && uint32_t(k >> 1) < nr) ? ld_poll(x_at(s, k)) : 0.0f;
    };
    float acc[kRows * R];
    auto multiply = [&](const float (&tv)[2 * kRows], const float (&xv)[2 * R]) {
#pragma unroll
        for (int i = 0; i < kRows; ++i)
#pragma unroll
            for (int r = 0; r < R; ++r)
                acc[i * R + r] = fmaf(tv[2 * i + 1], xv[2 * r + 1], fmaf(tv[2 * i], xv[2 * r], acc[i * R + r]));
    };
    // after the reduction lane L holds row i0 + (L % (8 R)) / R, right-hand side L % R
    const uint32_t li = (lane % (kRows * R)) / R, lr = lane % R;
    const bool mine = lane < uint32_t(kRows * R) && i0 + li < rows && lr < nr;
    const float rv = mine ? __ldcg(rin + size_t(lr) * n + rb0 + i0 + li) : 0.0f;
#pragma unroll
    for (int e = 0; e < kRows * R; ++e) acc[e] = 0.0f;
    float tv[2 * kRows], xv[2 * R];
    if (tk > 0) {
        load_tile(0, tv);
        load_x(0, xv);
    } else {
        load_inv(tv);
    }
    for (uint32_t s = 0; s < tk; ++s) {
        float tn[2 * kRows], xn[2 * R];
        if (s + 1 < tk) {
            load_tile(s + 1, tn);
            load_x(s + 1, xn);
        } else {
            load_inv(tn);
#pragma unroll
            for (int k = 0; k < 2 * R; ++k) xn[k] = 0.0f;
        }
        wait_solved(xv, [&](int k) { return x_at(s, k); }, s + 1 == tk, status, spin_limit);
        multiply(tv, xv);
#pragma unroll
        for (int k = 0; k < 2 * kRows; ++k) tv[k] = tn[k];
#pragma unroll
        for (int k = 0; k < 2 * R; ++k) xv[k] = xn[k];
    }
    const float r0 = rv - warp_transpose_sum(acc, lane);
    if (lane < uint32_t(kRows * R)) rs[i0 + li][lr] = r0;  // zero for rows and right-hand sides that are not there
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        xv[2 * r] = rs[lane][r];
        xv[2 * r + 1] = rs[lane + 32][r];
    }
#pragma unroll
    for (int e = 0; e < kRows * R; ++e) acc[e] = 0.0f;
    multiply(tv, xv);
    const float x = warp_transpose_sum(acc, lane);
    if (mine) {
        publish(out + size_t(lr) * n + rb0 + i0 + li, x);
        if (kLower) rin[size_t(lr) * n + rb0 + i0 + li] = __uint_as_float(kUnsolved);
    }
}

cudaError_t launch_dense_diag_inv(const float *dval, uint64_t dstride, uint32_t count, const uint32_t *doff,
                                  uint32_t m, float *dinv, cudaStream_t st) {
    if (m == 0) return cudaSuccess;
    k_dense_diag_inv<<<dim3((m + kRB - 1) / kRB, 2, count), 256, 0, st>>>(dval, dstride, doff, m, dinv);
    return cudaGetLastError();
}

// The forward sweeps (modes 0, 2) read y and write xo with ticket 0, the
// backward ones (1, 3) read xo and write y with ticket 1.  Right-hand sides in
// groups of one, or of kRHSChunk when there are several.
template <int kMode>
static cudaError_t dense_sweep(const SolvePlanDev &S, const float *dval, float *y, float *xo, uint32_t n,
                               uint32_t nrhs, uint32_t *tickets, uint32_t *status, const SolveBatch &B,
                               cudaStream_t st) {
    if (S.m == 0) return cudaSuccess;
    constexpr bool kForward = kMode == 0 || kMode == 2;
    const uint32_t nb = (S.m + kRB - 1) / kRB;
    const uint32_t chunks = nrhs == 1 ? 1u : (nrhs + kRHSChunk - 1) / kRHSChunk;
    const uint64_t items = uint64_t(nb) * chunks * B.count;
    if (items > 0x7FFFFFFFu) return cudaErrorInvalidValue;
    auto go = [&](auto kern) {
        kern<<<uint32_t(items), 256, 0, st>>>(dval, S.doff, S.t, S.m, kForward ? y : xo, kForward ? xo : y, n, nrhs,
                                              chunks, B.count, tickets + (kForward ? 0 : 1), status, S.spin_limit,
                                              S.ticket_base, B.dstride, uint64_t(nrhs) * n, B.dinv);
    };
    if constexpr (kMode >= 2) {
        if (nrhs == 1)
            go(k_dense_trsv_trans<kMode, 1>);
        else
            go(k_dense_trsv_trans<kMode, kRHSChunk>);
    } else {
        if (nrhs == 1)
            go(k_dense_trsv<kMode, 1>);
        else
            go(k_dense_trsv<kMode, kRHSChunk>);
    }
    return cudaGetLastError();
}

static cudaError_t tail_coupling(const DevPattern &P, const SolvePlanDev &S, const float *val, float *y,
                                 uint32_t nrhs, bool rows, const SolveBatch &B, cudaStream_t st) {
    if (S.m == 0 || S.t == 0) return cudaSuccess;
    const uint32_t longest = std::max<uint32_t>(1u, rows ? S.tail_row_longest : S.tail_longest), each = 32 * kCoupleEach;
    const dim3 grid((longest + each - 1) / each, (S.m + 8 * kCoupleCols - 1) / (8 * kCoupleCols),
                    B.count * ((nrhs + kCoupleRhs - 1) / kCoupleRhs));
    const uint64_t ystride = uint64_t(nrhs) * P.n;
    return rows ? launch_chained(k_tail_coupling<true>, grid, dim3(256), 0, st, P, S.t, S.m, S.tail_row_start, val, y,
                                 nrhs, B.vstride, ystride)
                : launch_chained(k_tail_coupling<false>, grid, dim3(256), 0, st, P, S.t, S.m, S.tail_start, val, y, nrhs,
                                 B.vstride, ystride);
}

cudaError_t solve_lower_unit(const DevPattern &P, const SolvePlanDev &S, const float *val,
                             const float *dval, float *y, float *xo, uint32_t nrhs, uint32_t *tickets,
                             uint32_t *ticket, uint32_t *status, const SolveBatch &B, cudaStream_t st) {
    cudaError_t e = S.sn[0].nlev ? run_sn_sweep(P, S.sn[0], false, S.t, val, y, xo, nrhs, B, B.sweep_done, ticket,
                                                status, S.spin_limit, st)
                                 : run_sweep<SWEEP_L>(P, S, val, y, xo, nrhs, B, st);
    if (e != cudaSuccess) return e;
    return dense_sweep<0>(S, dval, y, xo, P.n, nrhs, tickets, status, B, st);
}

cudaError_t solve_upper(const DevPattern &P, const SolvePlanDev &S, const float *val,
                        const float *dval, float *y, float *xo, uint32_t nrhs, uint32_t *tickets,
                        uint32_t *ticket, uint32_t *status, const SolveBatch &B, cudaStream_t st) {
    cudaError_t e = dense_sweep<1>(S, dval, y, xo, P.n, nrhs, tickets, status, B, st);
    if (e == cudaSuccess) e = tail_coupling(P, S, val, y, nrhs, false, B, st);
    if (e == cudaSuccess)
        e = S.sn[1].nlev ? run_sn_sweep(P, S.sn[1], true, S.t, val, y, xo, nrhs, B, B.sweep_done, ticket, status,
                                        S.spin_limit, st)
                         : run_sweep<SWEEP_U>(P, S, val, y, xo, nrhs, B, st);
    return e;
}

cudaError_t solve_upper_trans(const DevPattern &P, const SolvePlanDev &S, const float *val,
                              const float *dval, float *y, float *xo, uint32_t nrhs, uint32_t *tickets,
                              uint32_t *ticket, uint32_t *status, const SolveBatch &B, cudaStream_t st) {
    cudaError_t e = run_sweep<SWEEP_UT>(P, S, val, y, xo, nrhs, B, st);
    if (e == cudaSuccess) e = dense_sweep<2>(S, dval, y, xo, P.n, nrhs, tickets, status, B, st);
    return e;
}

cudaError_t solve_lower_unit_trans(const DevPattern &P, const SolvePlanDev &S, const float *val,
                                   const float *dval, float *y, float *xo, uint32_t nrhs, uint32_t *tickets,
                                   uint32_t *ticket, uint32_t *status, const SolveBatch &B, cudaStream_t st) {
    cudaError_t e = dense_sweep<3>(S, dval, y, xo, P.n, nrhs, tickets, status, B, st);
    if (e == cudaSuccess) e = tail_coupling(P, S, val, y, nrhs, true, B, st);
    if (e == cudaSuccess) e = run_sweep<SWEEP_LT>(P, S, val, y, xo, nrhs, B, st);
    return e;
}

// --------------------------------------------------------------- transforms --
// What the dense tail sweeps find at their start (SolveInit), written along
// with entry j of vector blockIdx.y of a solve's input transform.
__device__ __forceinline__ void solve_init(const SolveInit &I, size_t off, uint32_t j) {
    if (I.xo && j >= I.t) I.xo[off + j] = __uint_as_float(kUnsolved);
    if (I.tickets && j == 0 && blockIdx.y == 0) I.tickets[0] = I.tickets[1] = 0u;
}

__global__ void k_transform_f32(const uint32_t *__restrict__ idx, const double *__restrict__ scale,
                                const float *__restrict__ in, float *__restrict__ out, uint32_t n, SolveInit I) {
    const size_t off = size_t(blockIdx.y) * n;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        solve_init(I, off, j);
        float v = in[off + idx[j]];
        // float * double evaluated in double, stored as float (symbolic.cc:219,244)
        out[off + j] = scale ? static_cast<float>(static_cast<double>(v) * scale[j]) : v;
    }
}

__global__ void k_transform_f64_to_f32(const uint32_t *__restrict__ idx, const double *__restrict__ scale,
                                       const double *__restrict__ in, float *__restrict__ out, uint32_t n,
                                       SolveInit I) {
    const size_t off = size_t(blockIdx.y) * n;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        solve_init(I, off, j);
        double v = in[off + idx[j]];
        out[off + j] = static_cast<float>(scale ? v * scale[j] : v);
    }
}

__global__ void k_transform_f32_to_f64(const uint32_t *__restrict__ idx, const double *__restrict__ scale,
                                       const float *__restrict__ in, double *__restrict__ x, uint32_t n,
                                       int accumulate) {
    const size_t off = size_t(blockIdx.y) * n;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        double v = static_cast<double>(in[off + idx[j]]);
        if (scale) v *= scale[j];
        x[off + j] = accumulate ? x[off + j] + v : v;
    }
}

static inline dim3 tgrid(uint32_t n, uint32_t nrhs) {
    uint32_t bx = (n + 255) / 256;
    if (bx > 1024) bx = 1024;
    return dim3(bx, nrhs, 1);
}

cudaError_t launch_transform_f32(const uint32_t *idx, const double *scale, const float *in,
                                 float *out, uint32_t n, uint32_t nrhs, const SolveInit &init, cudaStream_t st) {
    k_transform_f32<<<tgrid(n, nrhs), 256, 0, st>>>(idx, scale, in, out, n, init);
    return cudaGetLastError();
}
cudaError_t launch_transform_f64_to_f32(const uint32_t *idx, const double *scale, const double *in,
                                        float *out, uint32_t n, uint32_t nrhs, const SolveInit &init,
                                        cudaStream_t st) {
    k_transform_f64_to_f32<<<tgrid(n, nrhs), 256, 0, st>>>(idx, scale, in, out, n, init);
    return cudaGetLastError();
}
cudaError_t launch_transform_f32_to_f64_add(const uint32_t *idx, const double *scale,
                                            const float *in, double *x, uint32_t n, uint32_t nrhs,
                                            int accumulate, cudaStream_t st) {
    k_transform_f32_to_f64<<<tgrid(n, nrhs), 256, 0, st>>>(idx, scale, in, x, n, accumulate);
    return cudaGetLastError();
}

// ---------------------------------------------------------- FP64 residuals --
// r = b - A0 x with A0 in CSR form (a_rptr/a_cidx; a_vmap gives the CSC
// position of each CSR entry in ax0), kLanes lanes per row (circuit and grid
// rows hold five to ten entries: with a warp per row most lanes had none and
// the rows' loads waited for each other), deterministic order within a row.
// norms[2v] += sum r^2, norms[2v+1] = max |r| for right-hand side v, one
// atomic each per block (one per warp of a large launch queued at the one
// address).  Measured, n = 490,000: 120 us with a warp per row and an atomic per
// warp, 20 us now.
constexpr int kResidualThreads = 256;
template <int kLanes>
__global__ void __launch_bounds__(kResidualThreads) k_residual(const uint32_t *__restrict__ rptr,
                                                               const uint32_t *__restrict__ cidx,
                                                               const uint32_t *__restrict__ vmap,
                                                               const double *__restrict__ ax0, uint32_t n,
                                                               const double *__restrict__ b,
                                                               const double *__restrict__ x, double *__restrict__ r,
                                                               double *norms, uint32_t nrhs_per_set,
                                                               uint64_t ax0_stride) {
    __shared__ double s_ss[kResidualThreads / 32], s_mx[kResidualThreads / 32];
    const uint32_t sub = threadIdx.x % kLanes;
    const uint32_t v = blockIdx.y;
    const size_t off = size_t(v) * n;
    ax0 += (v / nrhs_per_set) * ax0_stride;  // the value set of vector v
    double ss = 0.0, mx = 0.0;
    const uint32_t step = gridDim.x * (kResidualThreads / kLanes);
    // (every lane of a warp makes the same number of rounds, for the shuffles)
    for (uint32_t row0 = blockIdx.x * (kResidualThreads / kLanes) + (threadIdx.x & ~31u) / kLanes; row0 < n; row0 += step) {
        const uint32_t row = row0 + (threadIdx.x & 31) / kLanes;
        const bool in = row < n;
        double acc = 0.0;
        if (in)
            for (uint32_t e = rptr[row] + sub; e < rptr[row + 1]; e += kLanes)
                acc = fma(ax0[vmap[e]], x[off + cidx[e]], acc);
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (in && sub == 0) {
            const double rv = b[off + row] - acc;
            r[off + row] = rv;
            ss += rv * rv;
            mx = fmax(mx, fabs(rv));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s_ss[threadIdx.x / 32] = ss;
        s_mx[threadIdx.x / 32] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kResidualThreads / 32; ++w) {
            ss += s_ss[w];
            mx = fmax(mx, s_mx[w]);
        }
        atomicAdd(norms + 2 * v, ss);
        // non-negative doubles order like their bit patterns
        atomicMax(reinterpret_cast<unsigned long long *>(norms + 2 * v + 1),
                  static_cast<unsigned long long>(__double_as_longlong(mx)));
    }
}

cudaError_t launch_residual(const uint32_t *a_rptr, const uint32_t *a_cidx, const uint32_t *a_vmap,
                            const double *ax0, uint32_t n, const double *b, const double *x,
                            double *r, uint32_t nvec, uint32_t nrhs_per_set, uint64_t ax0_stride,
                            double *norms, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(norms, 0, sizeof(double) * 2 * nvec, st);
    if (e != cudaSuccess) return e;
    // lanes per row by the mean row length (ax0_stride entries in n rows)
    const double mean = double(ax0_stride) / std::max<uint32_t>(n, 1);
    const uint32_t lanes = mean <= 6 ? 4 : mean <= 14 ? 8 : 32;
    const uint32_t rows = kResidualThreads / lanes;
    uint32_t blocks = (n + rows - 1) / rows;
    // about eight blocks per SM in all
    const uint32_t cap = std::max<uint32_t>(1u, (148u * 8u + nvec - 1) / nvec);
    if (blocks > cap) blocks = cap;
    auto go = [&](auto kern) {
        kern<<<dim3(blocks, nvec, 1), kResidualThreads, 0, st>>>(a_rptr, a_cidx, a_vmap, ax0, n, b, x, r, norms,
                                                                 std::max<uint32_t>(nrhs_per_set, 1u), ax0_stride);
    };
    if (lanes == 4)
        go(k_residual<4>);
    else if (lanes == 8)
        go(k_residual<8>);
    else
        go(k_residual<32>);
    return cudaGetLastError();
}

__global__ void k_norms(const double *__restrict__ v, uint32_t n, double *norms) {
    const size_t off = size_t(blockIdx.y) * n;
    double ss = 0.0, mx = 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double a = v[off + i];
        ss += a * a;
        mx = fmax(mx, fabs(a));
    }
    for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(norms + 2 * blockIdx.y, ss);
        atomicMax(reinterpret_cast<unsigned long long *>(norms + 2 * blockIdx.y + 1),
                  static_cast<unsigned long long>(__double_as_longlong(mx)));
    }
}

cudaError_t launch_norms(const double *v, uint32_t n, uint32_t nvec, double *norms,
                         cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(norms, 0, sizeof(double) * 2 * nvec, st);
    if (e != cudaSuccess) return e;
    uint32_t blocks = (n + 255) / 256;
    if (blocks > 256) blocks = 256;
    k_norms<<<dim3(blocks, nvec, 1), 256, 0, st>>>(v, n, norms);
    return cudaGetLastError();
}

}  // namespace glu
