// The whole dense trailing block factored by one launch: a dataflow of 64 x 64
// tiles.
//
// The blocked algorithm of glu_factor_dense.cu takes a panel kernel, an
// operand pack and an update kernel (three with look-ahead) per 64 columns.
// On trailing blocks of a few thousand columns those are bound by their own
// latency, not by their work: the panel's serial 64-pivot LU repeated in every
// block, C read and written once per panel, a launch and a drain each.  Here a
// block of threads owns one tile (i, j) for good:
//   for s < min(i, j): C -= L(i, s) U(s, j), as the two tiles become ready
//   i == j: C = L11 U11;  i > j: L = C U11^-1;  i < j: U = L11^-1 C
// (left-looking per tile), so C is read and written once, tiles of later
// columns are updated while the diagonal chain advances, and a column step
// costs the chain diagonal LU -> one triangular solve -> one tile product
// instead of three kernels.
//
// Tiles are claimed in the order of min(i, j), the diagonal tile first,
// interleaved over the value sets (a ticket); a tile needs only tiles claimed
// before it, so every wait is for a running or finished block.  Besides its
// place in the factor a finished tile is written to a workspace, K-major and
// contiguous (16 KB; the diagonal tile as both operand layouts of the solves).
// What is on the chain is handed on in quarters: 16 columns of the diagonal
// tile's LU while the next 16 are factored (by warps that have no columns
// left), 16 columns of a solved tile while it solves the next; the solve and
// the last product in front of a diagonal tile start on them.  A publisher warp
// releases the pieces (their count is the tile's flag), so no computing warp
// waits for its stores; a producer warp waits for the flags and brings the
// operands in by bulk copies, two stages ahead of the products.  The
// workspace is the block's size again; the rule that chooses this kernel is
// in glu_engine.cpp (dense_flow).
//
// The waits for the flags are the only ones on another block.  They are bounded
// (the handle's wait limit, at least kFlowPolls polls); one that runs out sets
// DEV_TIMEOUT, and from then on its block's stages pass through without a
// copy: every barrier of the block still gets the arrivals that it expects, the
// computing warps run to their end with whatever the stages hold, the block's
// pieces are released, and so the launch drains.
//
// A column step of the chain takes 13 us (order 1,920, one block per SM), 7 of
// them the LU; 16.5 us with whole tiles handed on (LU 7.0, publishing it 1.5,
// flag and copy 1.1, triangular solve 2.6, publishing 0.8, flag and copy 1.2,
// product 1.9), 50 us in panel, pack and update kernels.  The whole block: 0.40
// ms, 0.49 ms and 1.51 ms.
//
// FP32 fused multiply-add throughout; the 64 products of a step are summed by
// themselves and subtracted from the entry once (relative error against 64 bits of random
// filled blocks, order 1,920: 1.8e-7; one at a time 7.9e-7, panels and updates
// 4.5e-7).
//
// The reference's counterpart is the per-column work of RL_onecol_factorizeCurrentCol
// and RL_onecol_updateSubmat (src/numeric.cu:205-319).
#include <algorithm>

#include "glu_common.cuh"
#include "glu_kernels.h"
#include "glu_tri.cuh"

namespace glu {
namespace {

constexpr int kT = kFlowTile;                        // 64
constexpr int kStages = 2;
constexpr uint32_t kTileBytes = kT * kT * 4;         // 16 KB
constexpr uint32_t kDiagBytes = kT * kTriML * 4;     // 17 KB: rows of 64 and the pivot's reciprocal, padded
constexpr uint32_t kStageBytes = 2 * kTileBytes;
constexpr int kLdW = kT + 1;                         // solve tile, [k][vector]
constexpr size_t kWorkBytes = sizeof(float) * kT * kLuLD;  // LU tile, or solve tile
constexpr size_t kSmem = kStages * kStageBytes + kWorkBytes;
constexpr size_t kSmemAlone = 120 * 1024;  // keeps a second block off the SM
constexpr int kThreads = kTriThreads + 64;           // eight computing warps, the producer and the publisher
constexpr int kPieces = 4;                           // of a tile: 16 of its 64 k each, ready one after another
constexpr uint32_t kPieceBytes = kTileBytes / kPieces, kDiagPieceBytes = kDiagBytes / kPieces;
static_assert(kFlowTile == kTriMax && kFlowDiagFloats == kT * kTriML, "layouts");
static_assert(kDiagBytes <= kStageBytes && kLdW <= kLuLD, "the diagonal tile fits a stage");

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void bar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// For another warp of the block or a copy of the block's own: both end by
// themselves, so the bound is a fixed one that a sound block never meets.
__device__ __forceinline__ void bar_wait(uint64_t *bar, uint32_t parity, uint32_t *status) {
#pragma unroll 1
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return;
    }
    atomicOr(status, DEV_TIMEOUT);
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// Between the acquire of a tile's flag and its bulk copy: the tile was written
// by ordinary stores, the copy reads through the asynchronous proxy.
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }

// A tile waits here while blocks in front of it still factor: about a step of
// the chain (12.5 us), a few milliseconds in the largest blocks.  A wait limit
// that suits the solves' waits (a link of theirs takes a microsecond) must not
// end that, so the limit counts from this many polls (about 0.1 s) on.
constexpr uint32_t kFlowPolls = 1u << 17;

// Bounded wait until `pieces` pieces of a tile are ready (one thread); false if
// it ran out, or another wait did.
__device__ __forceinline__ bool wait_tile(const uint32_t *flag, uint32_t pieces, uint32_t *status, uint32_t limit) {
#pragma unroll 1
    for (uint32_t spins = 0; ld_acquire_gpu(flag) < pieces; ++spins) {
        if (spins >= limit) {
            atomicOr(status, DEV_TIMEOUT);
            return false;
        }
        if ((spins & 255u) == 255u && (ld_acquire_gpu(status) & DEV_TIMEOUT)) return false;
    }
    return true;
}

// x M = a for the 64 vectors of W ([k][vector], leading dimension kLdW) by 256
// threads: chunks of 16, each solved a vector per thread (64 threads), then
// applied to the columns behind it by all.  M row-major, leading dimension
// kTriML (kDiv: with the pivots' reciprocals in the padding).  before(cb) waits
// for rows 16 cb .. + 15 of M; after(cb) is called by all threads once chunk cb
// of the result stands in W.
template <bool kDiv, class Before, class After>
__device__ __forceinline__ void solve_tile(float *W, const float *M, uint32_t tid, Before &&before, After &&after) {
    const uint32_t v = tid & 63, q = tid >> 6;
#pragma unroll 1
    for (uint32_t cb = 0; cb < 4; ++cb) {
        before(cb);
        if (tid < 64) {
            float x[kTriChunk];
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) x[k] = W[(cb * kTriChunk + k) * kLdW + v];
            tri_chunk_solve<kDiv>(x, M, cb, kT);
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) W[(cb * kTriChunk + k) * kLdW + v] = x[k];
        }
        tri_sync();
        after(cb);
        // columns 16 (cb + 1) .. 63: four groups of 4 (3 - cb)
        for (uint32_t g = 0; g < 3 - cb; ++g) {
            const uint32_t j0 = (cb + 1) * kTriChunk + q * 4 * (3 - cb) + 4 * g;
            float y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = W[(j0 + e) * kLdW + v];
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) {
                const float x = W[(cb * kTriChunk + k) * kLdW + v];
                const float4 t = *reinterpret_cast<const float4 *>(M + (cb * kTriChunk + k) * kTriML + j0);
                y[0] = fmaf(-x, t.x, y[0]);
                y[1] = fmaf(-x, t.y, y[1]);
                y[2] = fmaf(-x, t.z, y[2]);
                y[3] = fmaf(-x, t.w, y[3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) W[(j0 + e) * kLdW + v] = y[e];
        }
        tri_sync();
    }
}

struct FlowTile {
    uint32_t i, j, k;  // tile row and column, k = min
};
// Tile number idx of nt x nt in the order of the tickets.
__device__ __forceinline__ FlowTile flow_tile(uint32_t idx, uint32_t nt) {
    const uint32_t left = nt * nt - idx;  // tiles from here on: (nt - k)^2 at the start of step k
    uint32_t s = uint32_t(sqrtf(float(left)));
    while (s * s < left) ++s;
    while (s > 1 && (s - 1) * (s - 1) >= left) --s;
    const uint32_t k = nt - s, o = s * s - left;  // o-th tile of step k
    FlowTile t{k, k, k};
    if (o & 1)
        t.i = k + (o + 1) / 2;
    else
        t.j = k + o / 2;
    return t;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 2)
    k_dense_flow(float *val_base, uint64_t stride, const uint32_t *__restrict__ doff, uint32_t m, uint32_t nt,
                 uint32_t count, const float *pert_z, float *work, uint64_t work_stride, uint32_t *ctl,
                 uint32_t *status, uint32_t spin_limit, uint32_t ticket_base) {
    extern __shared__ __align__(128) unsigned char flow_smem[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], last_full[kPieces], diag_full[kPieces];
    __shared__ __align__(8) uint64_t written[kPieces];  // one phase each: a piece may be written before the last is released
    __shared__ uint32_t s_item;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        s_item = atomicAdd(ctl, 1u) + ticket_base;
        const uint32_t item = s_item;
        const FlowTile t0 = item < nt * nt * count ? flow_tile(item / count, nt) : FlowTile{0, 0, 0};
        for (int s = 0; s < kStages; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], kTriThreads / 32);
        }
        for (int p = 0; p < kPieces; ++p) {
            bar_init(&last_full[p], 1);
            bar_init(&diag_full[p], 1);
            bar_init(&written[p], t0.i == t0.j ? 3 : kTriThreads / 32);  // the warps that write a piece
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= nt * nt * count) return;
    const uint32_t z = item % count;
    const FlowTile t = flow_tile(item / count, nt);
    uint32_t *ready = ctl + 4 + size_t(z) * nt * nt;             // pieces of each tile that are ready
    float *tiles = work + z * work_stride;                       // [i][j][k][v]
    float *diags = tiles + size_t(nt) * nt * kT * kT;            // [k][0: U rows, 1: L columns]
    if (warp == kTriThreads / 32) {  // producer: operands as they become ready
        if (lane == 0) {
            bool ok = true;  // until a wait for a tile gives up: then arrivals without copies
            for (uint32_t s = 0; s < t.k; ++s) {
                const uint32_t st = s % kStages;
                unsigned char *dst = flow_smem + st * kStageBytes;
                const float *srcL = tiles + (size_t(t.i) * nt + s) * kT * kT, *srcU = tiles + (size_t(s) * nt + t.j) * kT * kT;
                const uint32_t *fL = ready + size_t(t.i) * nt + s, *fU = ready + size_t(s) * nt + t.j;
                if (s >= uint32_t(kStages)) bar_wait(&empty[st], (s / kStages - 1) & 1, status);
                if (s + 1 < t.k) {
                    ok = ok && wait_tile(fL, kPieces, status, spin_limit) && wait_tile(fU, kPieces, status, spin_limit);
                    if (ok) {
                        proxy_fence();
                        bar_expect(&full[st], 2 * kTileBytes);
                        bulk_load(dst, srcL, kTileBytes, &full[st]);
                        bulk_load(dst + kTileBytes, srcU, kTileBytes, &full[st]);
                    } else {
                        bar_arrive(&full[st]);
                    }
                } else {  // the last step's operands may be in the making: piece by piece
                    for (uint32_t p = 0; p < uint32_t(kPieces); ++p) {
                        ok = ok && wait_tile(fL, p + 1, status, spin_limit) && wait_tile(fU, p + 1, status, spin_limit);
                        if (ok) {
                            proxy_fence();
                            bar_expect(&last_full[p], 2 * kPieceBytes);
                            bulk_load(dst + p * kPieceBytes, srcL + p * (kPieceBytes / 4), kPieceBytes, &last_full[p]);
                            bulk_load(dst + kTileBytes + p * kPieceBytes, srcU + p * (kPieceBytes / 4), kPieceBytes,
                                      &last_full[p]);
                        } else {
                            bar_arrive(&last_full[p]);
                        }
                    }
                }
            }
            if (t.i != t.j) {
                const uint32_t st = t.k % kStages;
                if (t.k >= uint32_t(kStages)) bar_wait(&empty[st], (t.k / kStages - 1) & 1, status);
                const float *src = diags + (size_t(t.k) * 2 + (t.i > t.j ? 0 : 1)) * kFlowDiagFloats;
                for (uint32_t p = 0; p < uint32_t(kPieces); ++p) {
                    ok = ok && wait_tile(ready + size_t(t.k) * nt + t.k, p + 1, status, spin_limit);
                    if (ok) {
                        proxy_fence();
                        bar_expect(&diag_full[p], kDiagPieceBytes);
                        bulk_load(flow_smem + st * kStageBytes + p * kDiagPieceBytes, src + p * (kDiagPieceBytes / 4),
                                  kDiagPieceBytes, &diag_full[p]);
                    } else {
                        bar_arrive(&diag_full[p]);
                    }
                }
            }
            // the block must not end with copies in flight
            for (uint32_t s = t.k > uint32_t(kStages) + 1 ? t.k - 1 - kStages : 0; s + 1 < t.k; ++s)
                bar_wait(&full[s % kStages], (s / kStages) & 1, status);
            for (int p = 0; p < kPieces; ++p) {
                if (t.k) bar_wait(&last_full[p], 0, status);
                if (t.i != t.j) bar_wait(&diag_full[p], 0, status);
            }
        }
        return;
    }
    if (warp == kTriThreads / 32 + 1) {  // publisher: releases each piece once it is written
        if (lane == 0 && (t.i != t.j || t.k + 1 < nt))
            for (uint32_t p = 0; p < uint32_t(kPieces); ++p) {
                bar_wait(&written[p], 0, status);
                st_release_gpu(ready + size_t(t.i) * nt + t.j, p + 1);
            }
        return;
    }
    float *val = val_base + z * stride;
    const uint32_t tr = tid & 15, tc = tid >> 4;
    const uint32_t r0 = t.i * kT, c0 = t.j * kT;
    const uint32_t rows = min(uint32_t(kT), m - r0), cols = min(uint32_t(kT), m - c0);
    // C: rows 4 tr .. + 3, columns 4 tc .. + 3 (the identity past the block's end)
    float acc[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const uint32_t c = tc * 4 + b;
        const float *src = c < cols ? val + doff[c0 + c] + r0 + tr * 4 : nullptr;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const uint32_t r = tr * 4 + a;
            acc[a][b] = (src && r < rows) ? ld_cg(src + a) : (t.i == t.j && r == c ? 1.0f : 0.0f);
        }
    }
    for (uint32_t s = 0; s < t.k; ++s) {
        const uint32_t st = s % kStages;
        const bool last = s + 1 == t.k;
        if (!last) bar_wait(&full[st], (s / kStages) & 1, status);
        const float *sL = reinterpret_cast<const float *>(flow_smem + st * kStageBytes) + tr * 4;
        const float *sU = reinterpret_cast<const float *>(flow_smem + st * kStageBytes + kTileBytes) + tc * 4;
        // the 64 products in a sum of their own, subtracted once: its roundings
        // are relative to the sum, not to C
        float sum[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) sum[a][b] = 0.0f;
#pragma unroll 1
        for (int p = 0; p < kPieces; ++p) {
            if (last) bar_wait(&last_full[p], 0, status);
#pragma unroll
            for (int kk = 0; kk < kT / kPieces; ++kk) {
                const int k = p * (kT / kPieces) + kk;
                const float4 av = *reinterpret_cast<const float4 *>(sL + k * kT);
                const float4 bv = *reinterpret_cast<const float4 *>(sU + k * kT);
                const float ar[4] = {av.x, av.y, av.z, av.w}, br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b) sum[a][b] = fmaf(ar[a], br[b], sum[a][b]);
            }
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&empty[st]);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] -= sum[a][b];
    }
    float *W = reinterpret_cast<float *>(flow_smem + kStages * kStageBytes);
    if (t.i == t.j) {
#pragma unroll
        for (int b = 0; b < 4; ++b)
            *reinterpret_cast<float4 *>(W + (tc * 4 + b) * kLuLD + tr * 4) =
                make_float4(acc[0][b], acc[1][b], acc[2][b], acc[3][b]);
        tri_sync();
        // piece p by warps 5 .. 7: rows 16 p .. + 15 of U with the pivots'
        // reciprocals, columns 16 p .. + 15 of L
        float *du = diags + size_t(t.k) * 2 * kFlowDiagFloats, *dl = du + kFlowDiagFloats;
        auto publish = [&](uint32_t p) {
            if (t.k + 1 == nt) return;
            for (uint32_t e = tid - 5 * 32; e < 256u; e += 96) {
                const uint32_t a = 16 * p + (e & 15), b = (e >> 4) * 4;  // row a of U, columns b .. b + 3
                *reinterpret_cast<float4 *>(du + a * kTriML + b) =
                    make_float4(W[b * kLuLD + a], W[(b + 1) * kLuLD + a], W[(b + 2) * kLuLD + a], W[(b + 3) * kLuLD + a]);
                const uint32_t c = 16 * p + (e >> 4), r = (e & 15) * 4;  // column c of L, rows r .. r + 3
                *reinterpret_cast<float4 *>(dl + c * kTriML + r) = *reinterpret_cast<const float4 *>(W + c * kLuLD + r);
                if (e < 16u) du[a * kTriML + kT] = 1.0f / W[a * kLuLD + a];
            }
            __syncwarp();
            if (lane == 0) bar_arrive(&written[p]);
        };
        tri_lu_smem(W, rows, t.k + 1 < nt, pert_z ? pert_z[z] : 0.0f, publish);
#pragma unroll 4
        for (uint32_t e = tid; e < uint32_t(kT * kT); e += kTriThreads) {
            const uint32_t c = e >> 6, r = e & 63;
            if (c < cols && r < rows) st_cg(val + doff[c0 + c] + r0 + r, W[c * kLuLD + r]);
        }
        return;
    }
    // solve: [k][vector]; L: k = column, vector = row; U: k = row, vector = column
    const bool lower = t.i > t.j;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint32_t k = (lower ? tc * 4 + b : tr * 4 + a), v = (lower ? tr * 4 + a : tc * 4 + b);
            W[k * kLdW + v] = acc[a][b];
        }
    tri_sync();
    const float *M = reinterpret_cast<const float *>(flow_smem + (t.k % kStages) * kStageBytes);
    float *out = tiles + (size_t(t.i) * nt + t.j) * kT * kT;
    auto before = [&](uint32_t p) { bar_wait(&diag_full[p], 0, status); };
    auto after = [&](uint32_t p) {  // piece p of the tile
        const uint32_t k = 16 * p + (tid >> 4), v = (tid & 15) * 4;
        const float *w = W + k * kLdW + v;
        *reinterpret_cast<float4 *>(out + k * kT + v) = make_float4(w[0], w[1], w[2], w[3]);
        __syncwarp();
        if (lane == 0) bar_arrive(&written[p]);
    };
    if (lower)
        solve_tile<true>(W, M, tid, before, after);
    else
        solve_tile<false>(W, M, tid, before, after);
#pragma unroll 4
    for (uint32_t e = tid; e < uint32_t(kT * kT); e += kTriThreads) {
        const uint32_t c = e >> 6, r = e & 63;  // down the columns
        if (c < cols && r < rows)
            st_cg(val + doff[c0 + c] + r0 + r, lower ? W[c * kLdW + r] : W[r * kLdW + c]);
    }
}

size_t dense_flow_floats(uint32_t m) {
    const size_t nt = (m + kT - 1) / kT;
    return nt * nt * kT * kT + nt * 2 * kFlowDiagFloats;
}
size_t dense_flow_ctl_words(uint32_t m, uint32_t count) {
    const size_t nt = (m + kT - 1) / kT;
    return 4 + nt * nt * count;
}

cudaError_t launch_dense_flow(float *val, uint64_t stride, uint32_t count, const uint32_t *doff, uint32_t m,
                              const float *pert_z, float *work, uint32_t *ctl, uint32_t *status, uint32_t spin_limit,
                              uint32_t ticket_base, cudaStream_t st) {
    static PerDeviceOnce attr;
    cudaError_t e = attr.run([] {
        return cudaFuncSetAttribute(k_dense_flow, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemAlone));
    });
    if (e != cudaSuccess) return e;
    const uint32_t nt = (m + kT - 1) / kT;
    e = cudaMemsetAsync(ctl, 0, sizeof(uint32_t) * dense_flow_ctl_words(m, count), st);
    if (e != cudaSuccess) return e;
    // One block per SM while the diagonal chain is what takes the time (a
    // second block's products slow its LU down), two when the tiles' products
    // do.  Measured with whole tiles handed on, one against two: order 1,920 0.49
    // / 0.57 ms, order 3,000 0.90 / 1.02, four of order 1,920 0.81 / 0.75, 96 of
    // order 576 0.73 / 0.59; equal at order 3,968 and sixteen of 641.
    const size_t smem = uint64_t(nt) * nt * count <= 3000 ? kSmemAlone : kSmem;
    k_dense_flow<<<nt * nt * count, kThreads, smem, st>>>(val, stride, doff, m, nt, count, pert_z, work,
                                                           dense_flow_floats(m), ctl, status,
                                                           std::max(spin_limit, kFlowPolls), ticket_base);
    return cudaGetLastError();
}

}  // namespace glu
