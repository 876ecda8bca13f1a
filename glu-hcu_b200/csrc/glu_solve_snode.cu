// Supernodal form of the sparse L and U sweeps of the triangular solves.
//
// The reference sweeps column by column (Symbolic_Matrix::solve,
// src/symbolic.cc:226-239).  With the factor's supernodes (runs of columns
// [s, s+w) with a dense diagonal block and a common lower pattern) a sweep
// step is a whole supernode: its w unknowns are solved against the dense
// diagonal block (wide ones: a product with the block's inverse, computed once
// per factorization by k_sn_diag_inv; else, or where that product is not finite,
// a chain over the columns by one warp) and their off-diagonal entries are then scattered into the unknowns
// they feed:
//   L (forward, unit):  x_S = L11^-1 y_S;  y_r -= L21(r,:) x_S for the m rows
//                       below the block (one thread per row, dot over w);
//   U (backward):       x_S = U11^-1 y_S;  y_i -= U(i,c) x_c for the entries
//                       of the supernode's columns above the block.
// Supernodes are leveled by the sweep's dependencies: L — a supernode waits
// for the supernodes whose L21 rows fall in it; U — for the supernodes that
// hold its update targets.  Finished unknowns go to xo (another block of the
// same supernode may still read y_S) and are copied back after the sweep.
// Every block finds its supernode and part through a precomputed map; small
// supernodes (width <= kSnSmallWidth with at most 32 off-diagonal rows or
// entries) go eight to a block, one warp each.
//
// What bounds the sweeps is the chain of levels, each a launch chained to the
// one before, so the time from a level's last scatter to the next one's counts:
// a block reads everything that does not depend on the unknowns (plan,
// pattern, factors, inverse) before it waits for the previous level, and
// between that wait and its own scatter there is one read of y, the solve
// against the diagonal block and the products.  Several right-hand sides are
// spread over the grid's second dimension.  (FP32 solve of a 251 x 251 grid, 70
// levels: 656 -> 399 us against waiting first and solving the block by a chain
// with divisions; 32 right-hand sides at n = 4,960: 576 -> 286 us.)
#include <algorithm>

#include "glu_common.cuh"
#include "glu_kernels.h"
#include "glu_tri.cuh"

namespace glu {

namespace {
constexpr int kLD = kSnMaxWidth + 1;
constexpr uint32_t kFull = 0xffffffffu;

// Right-hand sides [q0, q1) of a block: blockIdx.y's share of nrhs.
struct Rhs {
    uint32_t q0, q1;
};
__device__ __forceinline__ Rhs rhs_share(uint32_t nrhs) {
    const uint32_t per = (nrhs + gridDim.y - 1) / gridDim.y, q0 = blockIdx.y * per;
    return Rhs{q0, min(q0 + per, nrhs)};
}

// L sweep of one small supernode (w <= kSnSmallWidth, m <= 32) by one warp:
// lane k holds unknown s+k and L21 row k; the entries it needs are loaded
// before the dependency chain starts.
__device__ __forceinline__ void sn_sweep_l_small(const DevPattern &P, const SnSweepPlan &W,
                                                 const float *__restrict__ val, float *y, float *xo, Rhs Q,
                                                 uint32_t i, uint32_t lane) {
    constexpr int SW = int(kSnSmallWidth);
    const uint4 md = W.meta[i];
    const uint32_t s = md.x, w = md.y, lbase = md.z, m = md.w, l = s + w - 1, n = P.n;
    if (w == 1) {
        const bool in = lane < m;
        const float lv = in ? __ldg(val + lbase + lane) : 0.0f;
        const uint32_t target = in ? __ldg(P.ridx + lbase + lane) : 0u;
        pdl_wait();  // the previous level's x
        for (uint32_t q = Q.q0; q < Q.q1; ++q) {
            float *yq = y + size_t(q) * n;
            const float x = __ldcg(yq + s);
            if (lane == 0) xo[size_t(q) * n + s] = x;
            const float u = __fmul_rn(lv, x);
            if (in && u != 0.0f) atomicAdd(yq + target, -u);
        }
        return;
    }
    const uint32_t dl = lane < w ? P.diag[s + lane] : 0u;
    float lrow[SW], l21[SW];
#pragma unroll
    for (int c = 0; c < SW; ++c) {
        const uint32_t dc = __shfl_sync(kFull, dl, c);
        lrow[c] = (uint32_t(c) < lane && lane < w) ? __ldg(val + dc + (lane - c)) : 0.0f;
        if (m) l21[c] = (lane < m && uint32_t(c) < w) ? __ldg(val + dc + (l + 1 - (s + c)) + lane) : 0.0f;
    }
    const uint32_t target = lane < m ? __ldg(P.ridx + lbase + lane) : 0u;
    pdl_wait();  // the previous level's x
    for (uint32_t q = Q.q0; q < Q.q1; ++q) {
        float *yq = y + size_t(q) * n;
        float v = lane < w ? __ldcg(yq + s + lane) : 0.0f;
#pragma unroll
        for (int c = 0; c + 1 < SW; ++c) {
            if (uint32_t(c) + 1 >= w) break;
            const float xc = __shfl_sync(kFull, v, c);
            if (lane > uint32_t(c) && lane < w) v = __fsub_rn(v, __fmul_rn(lrow[c], xc));
        }
        if (lane < w) xo[size_t(q) * n + s + lane] = v;
        if (m == 0) continue;
        float acc = 0.0f;
#pragma unroll
        for (int c = 0; c < SW; ++c) {
            if (uint32_t(c) >= w) break;
            acc = fmaf(l21[c], __shfl_sync(kFull, v, c), acc);
        }
        if (lane < m && acc != 0.0f) atomicAdd(yq + target, -acc);
    }
}

// Groups of tiny supernodes (one column, at most eight off-diagonal entries):
// eight lanes each, 32 to a block.  They are most of a grid's leaves, and a
// warp each left most lanes without an entry.
__device__ __forceinline__ void sn_sweep_l_tiny(const DevPattern &P, const SnSweepPlan &W,
                                                const float *__restrict__ val, float *y, float *xo, Rhs Q, uint2 bi) {
    const uint32_t g = threadIdx.x >> 3, sub = threadIdx.x & 7;
    if (g >= (bi.y & kSnGroupCount)) return;
    const uint4 md = W.meta[W.small[bi.x + g]];
    const uint32_t s = md.x, lbase = md.z, m = md.w;
    const bool in = sub < m;
    const float l21 = in ? __ldg(val + lbase + sub) : 0.0f;
    const uint32_t target = in ? __ldg(P.ridx + lbase + sub) : 0u;
    pdl_wait();  // the previous level's x
    for (uint32_t q = Q.q0; q < Q.q1; ++q) {
        float *yq = y + size_t(q) * P.n;
        const float x = __ldcg(yq + s);
        if (sub == 0) xo[size_t(q) * P.n + s] = x;
        const float u = __fmul_rn(l21, x);
        if (in && u != 0.0f) atomicAdd(yq + target, -u);
    }
}
__device__ __forceinline__ void sn_sweep_u_tiny(const DevPattern &P, const SnSweepPlan &W,
                                                const float *__restrict__ val, float *y, float *xo, Rhs Q, uint2 bi) {
    const uint32_t g = threadIdx.x >> 3, sub = threadIdx.x & 7;
    if (g >= (bi.y & kSnGroupCount)) return;
    const uint4 md = W.meta[W.small[bi.x + g]];
    const uint32_t s = md.x, cp = md.z, dk = md.w;
    const bool in = cp + sub < dk;
    const float u = in ? __ldg(val + cp + sub) : 0.0f;
    const uint32_t target = in ? __ldg(P.ridx + cp + sub) : 0u;
    const float piv = __ldg(val + dk);
    pdl_wait();  // the previous level's x
    for (uint32_t q = Q.q0; q < Q.q1; ++q) {
        float *yq = y + size_t(q) * P.n;
        const float x = __ldcg(yq + s) / piv;
        if (sub == 0) xo[size_t(q) * P.n + s] = x;
        if (in && x != 0.0f) atomicAdd(yq + target, -__fmul_rn(u, x));
    }
}

// U sweep of one small supernode (w <= kSnSmallWidth, at most 32 entries above
// the block) by one warp: lane k holds unknown s+k and above-block entry k.
__device__ __forceinline__ void sn_sweep_u_small(const DevPattern &P, const SnSweepPlan &W,
                                                 const float *__restrict__ val, float *y, float *xo, Rhs Q,
                                                 uint32_t i, uint32_t lane) {
    constexpr int SW = int(kSnSmallWidth);
    const uint4 md = W.meta[i];
    const uint32_t s = md.x, w = md.y, n = P.n;
    if (w == 1) {
        const bool in = md.z + lane < md.w;
        const float uv = in ? __ldg(val + md.z + lane) : 0.0f;
        const uint32_t target = in ? __ldg(P.ridx + md.z + lane) : 0u;
        const float piv = __ldg(val + md.w);
        pdl_wait();  // the previous level's x
        for (uint32_t q = Q.q0; q < Q.q1; ++q) {
            float *yq = y + size_t(q) * n;
            const float x = __ldcg(yq + s) / piv;
            if (lane == 0) xo[size_t(q) * n + s] = x;
            if (in && x != 0.0f) atomicAdd(yq + target, -__fmul_rn(uv, x));
        }
        return;
    }
    const uint32_t dl = lane < w ? P.diag[s + lane] : 0u;
    const uint32_t cp = lane < w ? P.cptr[s + lane] : 0u;
    const uint32_t cnt = lane < w ? (dl - lane) - cp : 0u;  // entries of column s+lane above the block
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= uint32_t(o)) incl += v;
    }
    const uint32_t pre = incl - cnt, total = __shfl_sync(kFull, incl, 31);
    uint32_t col = 0;  // column of entry `lane`: the last c < w with pre_c <= lane
#pragma unroll
    for (int c = 1; c < SW; ++c) {
        const uint32_t pc = __shfl_sync(kFull, pre, c);
        if (uint32_t(c) < w && pc <= lane) col = c;
    }
    const uint32_t pcol = __shfl_sync(kFull, cp, col) + (lane - __shfl_sync(kFull, pre, col));
    const bool ev = lane < total;
    const uint32_t tg = ev ? __ldg(P.ridx + pcol) : 0u;
    const float ue = ev ? __ldg(val + pcol) : 0.0f;
    float urow[SW];  // U(s+lane, s+cc) for cc > lane, at diag[s+cc] - (cc - lane)
#pragma unroll
    for (int cc = 0; cc < SW; ++cc) {
        const uint32_t dcc = __shfl_sync(kFull, dl, cc);
        urow[cc] = (lane < uint32_t(cc) && uint32_t(cc) < w) ? __ldg(val + dcc - (cc - lane)) : 0.0f;
    }
    const float piv = lane < w ? __ldg(val + dl) : 1.0f;
    // reciprocals before the chain, unless a pivot is too large or too small
    // (or, below, an unknown turns out not to be finite)
    const float mag = fabsf(piv), rec = lu_reciprocal(piv);
    const bool quick = __all_sync(kFull, mag > 1e-30f && mag < 1e30f);
    pdl_wait();  // the previous level's x
    for (uint32_t q = Q.q0; q < Q.q1; ++q) {
        float *yq = y + size_t(q) * n;
        const float v0 = lane < w ? __ldcg(yq + s + lane) : 0.0f;
        float v = v0;
        bool solved = false;
        if (quick) {
#pragma unroll
            for (int cc = SW - 1; cc >= 0; --cc) {
                if (uint32_t(cc) >= w) continue;
                // every lane divides its own value, so that the step is one shuffle long
                const float xc = __shfl_sync(kFull, lu_quotient(v, piv, rec), cc);
                if (lane == uint32_t(cc)) v = xc;
                if (lane < uint32_t(cc)) v = __fsub_rn(v, __fmul_rn(urow[cc], xc));
            }
            solved = __all_sync(kFull, isfinite(v));
        }
        if (!solved) {
            v = v0;
#pragma unroll
            for (int cc = SW - 1; cc >= 0; --cc) {
                if (uint32_t(cc) >= w) continue;
                const float xc = __shfl_sync(kFull, v / piv, cc);
                if (lane == uint32_t(cc)) v = xc;
                if (lane < uint32_t(cc)) v = __fsub_rn(v, __fmul_rn(urow[cc], xc));
            }
        }
        if (lane < w) xo[size_t(q) * n + s + lane] = v;
        const float xe = __shfl_sync(kFull, v, col);
        if (ev && xe != 0.0f) atomicAdd(yq + tg, -__fmul_rn(ue, xe));
    }
}
// A group of small supernodes: tiny ones, or one per warp.
__device__ __forceinline__ void sn_sweep_l_group(const DevPattern &P, const SnSweepPlan &W,
                                                 const float *__restrict__ val, float *y, float *xo, Rhs Q, uint2 bi) {
    const uint32_t wi = threadIdx.x >> 5;
    if (bi.y & kSnTinyFlag)
        sn_sweep_l_tiny(P, W, val, y, xo, Q, bi);
    else if (wi < (bi.y & kSnGroupCount))
        sn_sweep_l_small(P, W, val, y, xo, Q, W.small[bi.x + wi], threadIdx.x & 31);
}
__device__ __forceinline__ void sn_sweep_u_group(const DevPattern &P, const SnSweepPlan &W,
                                                 const float *__restrict__ val, float *y, float *xo, Rhs Q, uint2 bi) {
    const uint32_t wi = threadIdx.x >> 5;
    if (bi.y & kSnTinyFlag)
        sn_sweep_u_tiny(P, W, val, y, xo, Q, bi);
    else if (wi < (bi.y & kSnGroupCount))
        sn_sweep_u_small(P, W, val, y, xo, Q, W.small[bi.x + wi], threadIdx.x & 31);
}

// Fused sweeps: the block's item and value set from one ticket counter of the
// launch, handed out item-major over the value sets (ticket = item * count +
// set, so every set's sweep advances at once), and a wait (thread 0, bounded)
// until every supernode it solves has received all its releases; a block
// waits only on items of smaller tickets.  Returns {map index, value set},
// the index UINT32_MAX when the ticket is past the end.  Per-level launches
// use {b0 + blockIdx.x, blockIdx.z} instead.
__device__ __forceinline__ uint2 sweep_block(const SnSweepPlan &W, uint32_t b0, const uint32_t *done,
                                             uint32_t *ticket, uint32_t *status, uint32_t spin_limit) {
    if (!done) return make_uint2(b0 + blockIdx.x, blockIdx.z);
    __shared__ uint32_t s_blk, s_z;
    if (threadIdx.x == 0) {
        const uint32_t k = atomicAdd(ticket, 1u);
        const uint32_t blk = k / gridDim.z, z = k % gridDim.z;
        if (blk < W.nblocks) {
            const uint32_t *dz = done + size_t(z) * W.ns;
            for (uint32_t e = W.wait_off[blk]; e < W.wait_off[blk + 1]; ++e) {
                const uint32_t q = W.wait_idx[e];
                wait_count(dz + q, W.indeg[q], status, spin_limit);
            }
        }
        s_blk = blk;
        s_z = z;
    }
    __syncthreads();
    return make_uint2(s_blk < W.nblocks ? s_blk : UINT32_MAX, s_z);
}

// After the block's scatter: one release for every supernode it updated (its
// atomics are made visible first: barrier, then a device-scope fence).
__device__ __forceinline__ void sweep_release(const SnSweepPlan &W, uint32_t blk, uint32_t *done) {
    if (!done) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        for (uint32_t e = W.rel_off[blk]; e < W.rel_off[blk + 1]; ++e) atomicAdd(done + W.rel_idx[e], 1u);
    }
}
}  // namespace

// x = T^-1 v of a wide supernode by all 256 threads: thread (row, quarter) holds
// the inverse's 16 entries iv of its row and quarter; v (w values, zero beyond)
// in shared memory before the call, x in xs after it (two barriers inside).
__device__ __forceinline__ void wide_solve(const float (&iv)[16], const float *vs, float (*part)[kSnMaxWidth], float *xs,
                                           uint32_t tid) {
    const uint32_t row = tid & 63, q = tid >> 6;
    const float4 *v4 = reinterpret_cast<const float4 *>(vs + q * 16);
    float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
        const float4 v = v4[k / 4];
        a0 = fmaf(iv[k], v.x, a0);
        a1 = fmaf(iv[k + 1], v.y, a1);
        a0 = fmaf(iv[k + 2], v.z, a0);
        a1 = fmaf(iv[k + 3], v.w, a1);
    }
    part[q][row] = a0 + a1;
    __syncthreads();
    if (tid < kSnMaxWidth) xs[tid] = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
    __syncthreads();
}
// Whether that x is finite, the same to all warps; else it is solved for by
// substitution: an inverse can overflow where that does not (a block graded by
// its rows' and columns' scales), and an infinite v makes every unknown NaN.
// (Asked beside the products with x, not in front of them: a vote in the barrier
// took a solve of a 251 x 251 grid from 291 to 297 us.)
__device__ __forceinline__ bool wide_finite(const float *xs, uint32_t tid) {
    return __all_sync(kFull, isfinite(xs[tid & 31]) && isfinite(xs[(tid & 31) + 32]));
}
__device__ __forceinline__ void load_inverse(float (&iv)[16], const float *__restrict__ inv, uint32_t tid) {
    inv += (tid >> 6) * 16 * kSnMaxWidth + (tid & 63);
#pragma unroll
    for (int k = 0; k < 16; ++k) iv[k] = __ldg(inv + k * kSnMaxWidth);
}

// kInv: the wide supernodes' inverses are there (invs).  Without them the kernels need
// fewer registers, and more blocks fit on an SM, which is what bounds the sweeps
// of many value sets (64 of a hundred filled 40 x 40 blocks, where the inverses are
// over their budget: L 150 -> 87 us, U 93 -> 77 us a launch with kernels of
// their own and the rows of L21 behind a branch).
// kBlocks of them per SM: three (85 registers, a few spilled) once there are
// kManyBlocks of the launch, for which the rate counts; with fewer the time of one does (64 x 64
// blocks, per launch: 63 of them 7.3 us at three and 5.9 at two, 1,008 20.5 and 19.5,
// 4,032 70 and 83).
constexpr uint64_t kManyBlocks = 12 * 148;
template <bool kInv, int kBlocks>
__global__ void __launch_bounds__(256, kBlocks) k_sn_sweep_l(DevPattern P, SnSweepPlan W, const float *__restrict__ val,
                                                    float *y, float *xo, uint32_t nrhs, uint32_t b0,
                                                    uint64_t vstride, uint64_t ystride,
                                                    const float *__restrict__ invs, uint64_t inv_stride, uint32_t *done,
                                                    uint32_t *ticket, uint32_t *status, uint32_t spin_limit) {
    pdl_release();
    const uint2 bz = sweep_block(W, b0, done, ticket, status, spin_limit);
    const uint32_t blk = bz.x;
    val += bz.y * vstride;  // value set bz.y, its right-hand sides
    y += bz.y * ystride;
    xo += bz.y * ystride;
    if (done) done += size_t(bz.y) * W.ns;
    if (blk == UINT32_MAX) return;
    const Rhs Q = rhs_share(nrhs);
    __shared__ float sT[kSnMaxWidth * kLD];
    __shared__ __align__(16) float xs[kSnMaxWidth], vs[kSnMaxWidth];
    float(*part)[kSnMaxWidth] = reinterpret_cast<float(*)[kSnMaxWidth]>(sT);
    const uint2 bi = W.map[blk];
    if (bi.y & kSnSmallFlag) {  // a group of small supernodes, one per warp
        sn_sweep_l_group(P, W, val, y, xo, Q, bi);
        sweep_release(W, blk, done);
        return;
    }
    const uint4 md = W.meta[bi.x];
    const uint32_t s = md.x, w = md.y, lbase = md.z, m = md.w, t = bi.y;
    const uint32_t l = s + w - 1;
    const uint32_t tid = threadIdx.x, n = P.n;
    const uint32_t wide = (kInv && w > kSnSmallWidth) ? __ldg(W.wide + bi.x) : UINT32_MAX;
    __shared__ uint32_t sB[kSnMaxWidth];
    if (tid < w) sB[tid] = P.diag[s + tid];
    __syncthreads();
    // This thread's L21 row and its target: they do not depend on x, so they
    // are loaded before the dependency chain (and serve every right-hand side).
    // (Behind a branch: warps without rows, all of a block diagonal matrix, skip it and the products.)
    const uint32_t r = t * blockDim.x + tid;  // L21 row of this thread
    float lr[kSnMaxWidth];
    uint32_t target = 0;
    if (r < m) {
        target = __ldg(P.ridx + lbase + r);
#pragma unroll
        for (int c = 0; c < int(kSnMaxWidth); ++c)
            lr[c] = uint32_t(c) < w ? __ldg(val + sB[c] + (l + 1 - (s + c)) + r) : 0.0f;
    }
    float iv[16];
    if (kInv && wide != UINT32_MAX) {
        load_inverse(iv, invs + bz.y * inv_stride + (size_t(wide) * 2) * kSnMaxWidth * kSnMaxWidth, tid);
    } else {
        // L11, strictly lower: L(s+k, s+c) at diag[s+c] + (k - c); eight loads in flight per thread
        for (uint32_t e0 = 0; e0 < w * kSnMaxWidth; e0 += 8 * 256) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t e = e0 + u * 256 + tid, c = e >> 6, k = e & 63;
                v[u] = (c < w && k < w && k > c) ? __ldg(val + sB[c] + (k - c)) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t e = e0 + u * 256 + tid, c = e >> 6, k = e & 63;
                if (c < w && k < w && k > c) sT[c * kLD + k] = v[u];
            }
        }
        if (tid < kSnMaxWidth) xs[tid] = 0.0f;
        __syncthreads();
    }
    pdl_wait();  // the previous level's x
    for (uint32_t q = Q.q0; q < Q.q1; ++q) {
        float *yq = y + size_t(q) * n;
        // the chain over the columns, by one warp, from the block in sT
        auto substitute = [&] {
            if (tid < 32) {
                const uint32_t k0 = tid, k1 = tid + 32;
                float v0 = k0 < w ? __ldcg(yq + s + k0) : 0.0f;
                float v1 = k1 < w ? __ldcg(yq + s + k1) : 0.0f;
                for (uint32_t c = 0; c + 1 < w; ++c) {
                    const float xc = __shfl_sync(0xffffffffu, c < 32 ? v0 : v1, c & 31);
                    if (k0 > c && k0 < w) v0 = __fsub_rn(v0, __fmul_rn(sT[c * kLD + k0], xc));
                    if (k1 > c && k1 < w) v1 = __fsub_rn(v1, __fmul_rn(sT[c * kLD + k1], xc));
                }
                if (k0 < w) xs[k0] = v0;
                if (k1 < w) xs[k1] = v1;
                if (t == 0) {
                    if (k0 < w) xo[size_t(q) * n + s + k0] = v0;
                    if (k1 < w) xo[size_t(q) * n + s + k1] = v1;
                }
            }
            __syncthreads();
        };
        if (kInv && wide != UINT32_MAX) {
            if (tid < kSnMaxWidth) vs[tid] = tid < w ? __ldcg(yq + s + tid) : 0.0f;
            __syncthreads();
            wide_solve(iv, vs, part, xs, tid);
        } else {
            substitute();
        }
        // four sums: one chain of 64 multiply-adds would take as long as the solve
        auto product = [&] {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            const float4 *x4 = reinterpret_cast<const float4 *>(xs);
#pragma unroll
            for (int c = 0; c < int(kSnMaxWidth); c += 4) {
                if (uint32_t(c) >= w) break;
                const float4 x = x4[c / 4];
                acc[0] = fmaf(lr[c], x.x, acc[0]);
                acc[1] = fmaf(lr[c + 1], x.y, acc[1]);
                acc[2] = fmaf(lr[c + 2], x.z, acc[2]);
                acc[3] = fmaf(lr[c + 3], x.w, acc[3]);
            }
            return (acc[0] + acc[1]) + (acc[2] + acc[3]);
        };
        float sum = 0.0f;
        if (r < m) sum = product();
        if (kInv && wide != UINT32_MAX && !wide_finite(xs, tid)) {
            __syncthreads();  // all warps have read xs
#pragma unroll 1
            for (uint32_t e = tid; e < w * kSnMaxWidth; e += 256) {
                const uint32_t c = e >> 6, k = e & 63;
                if (k < w && k > c) sT[c * kLD + k] = __ldg(val + sB[c] + (k - c));
            }
            if (tid < kSnMaxWidth) xs[tid] = 0.0f;
            __syncthreads();
            substitute();
            if (r < m) sum = product();
        }
        if (kInv && wide != UINT32_MAX && t == 0 && tid < w) xo[size_t(q) * n + s + tid] = xs[tid];
        if (sum != 0.0f) atomicAdd(yq + target, -sum);
        if (q + 1 < Q.q1) __syncthreads();
    }
    sweep_release(W, blk, done);
}

// The L sweep's parts of narrow supernodes (w <= kSnSmallWidth, 256 rows of L21
// each, a row per thread in 16 registers) and groups of small ones.
__global__ void __launch_bounds__(256, 4) k_sn_sweep_l_narrow(DevPattern P, SnSweepPlan W, const float *__restrict__ val,
                                                           float *y, float *xo, uint32_t nrhs, uint32_t b0,
                                                           uint64_t vstride, uint64_t ystride) {
    constexpr int SW = int(kSnSmallWidth);
    __shared__ uint32_t sB[SW];
    __shared__ __align__(16) float sT[SW * (SW + 1)], xs[SW];
    pdl_release();
    val += blockIdx.z * vstride;
    y += blockIdx.z * ystride;
    xo += blockIdx.z * ystride;
    const Rhs Q = rhs_share(nrhs);
    const uint2 bi = W.map[b0 + blockIdx.x];
    if (bi.y & kSnSmallFlag) {
        sn_sweep_l_group(P, W, val, y, xo, Q, bi);
        return;
    }
    const uint4 md = W.meta[bi.x];
    const uint32_t s = md.x, w = md.y, lbase = md.z, m = md.w, t = bi.y;
    const uint32_t l = s + w - 1;
    const uint32_t tid = threadIdx.x, n = P.n;
    if (tid < w) sB[tid] = P.diag[s + tid];
    __syncthreads();
    const uint32_t r = t * blockDim.x + tid;  // L21 row of this thread
    float lr[SW];
#pragma unroll
    for (int c = 0; c < SW; ++c)
        lr[c] = (r < m && uint32_t(c) < w) ? __ldg(val + sB[c] + (l + 1 - (s + c)) + r) : 0.0f;
    const uint32_t target = r < m ? __ldg(P.ridx + lbase + r) : 0u;
    {   // L11, strictly lower: L(s+k, s+c) at diag[s+c] + (k - c)
        const uint32_t c = tid / SW, k = tid % SW;
        sT[c * (SW + 1) + k] = (c < w && k < w && k > c) ? __ldg(val + sB[c] + (k - c)) : 0.0f;
    }
    if (tid < SW) xs[tid] = 0.0f;
    __syncthreads();
    pdl_wait();  // the previous level's x
    for (uint32_t q = Q.q0; q < Q.q1; ++q) {
        float *yq = y + size_t(q) * n;
        if (tid < 32) {
            float v = tid < w ? __ldcg(yq + s + tid) : 0.0f;
            for (uint32_t c = 0; c + 1 < w; ++c) {
                const float xc = __shfl_sync(kFull, v, c);
                if (tid > c && tid < w) v = __fsub_rn(v, __fmul_rn(sT[c * (SW + 1) + tid], xc));
            }
            if (tid < w) xs[tid] = v;
            if (t == 0 && tid < w) xo[size_t(q) * n + s + tid] = v;
        }
        __syncthreads();
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const float4 *x4 = reinterpret_cast<const float4 *>(xs);
#pragma unroll
        for (int c = 0; c < SW; c += 4) {
            const float4 x = x4[c / 4];
            acc[0] = fmaf(lr[c], x.x, acc[0]);
            acc[1] = fmaf(lr[c + 1], x.y, acc[1]);
            acc[2] = fmaf(lr[c + 2], x.z, acc[2]);
            acc[3] = fmaf(lr[c + 3], x.w, acc[3]);
        }
        const float sum = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        if (r < m && sum != 0.0f) atomicAdd(yq + target, -sum);
        if (q + 1 < Q.q1) __syncthreads();
    }
}

template <bool kInv>
__global__ void __launch_bounds__(256, kInv ? 3 : 4) k_sn_sweep_u(DevPattern P, SnSweepPlan W, const float *__restrict__ val,
                                                    float *y, float *xo, uint32_t nrhs, uint32_t b0,
                                                    uint64_t vstride, uint64_t ystride,
                                                    const float *__restrict__ invs, uint64_t inv_stride, uint32_t *done,
                                                    uint32_t *ticket, uint32_t *status, uint32_t spin_limit) {
    pdl_release();
    const uint2 bz = sweep_block(W, b0, done, ticket, status, spin_limit);
    const uint32_t blk = bz.x;
    val += bz.y * vstride;  // value set bz.y, its right-hand sides
    y += bz.y * ystride;
    xo += bz.y * ystride;
    if (done) done += size_t(bz.y) * W.ns;
    if (blk == UINT32_MAX) return;
    const Rhs Q = rhs_share(nrhs);
    __shared__ float sT[kSnMaxWidth * kLD];
    __shared__ __align__(16) float xs[kSnMaxWidth], vs[kSnMaxWidth];
    __shared__ uint32_t pre[kSnMaxWidth + 1];
    float(*part)[kSnMaxWidth] = reinterpret_cast<float(*)[kSnMaxWidth]>(sT);
    const uint2 bi = W.map[blk];
    if (bi.y & kSnSmallFlag) {  // a group of small supernodes, one per warp
        sn_sweep_u_group(P, W, val, y, xo, Q, bi);
        sweep_release(W, blk, done);
        return;
    }
    const uint32_t s = W.meta[bi.x].x, w = W.meta[bi.x].y, t = bi.y;
    const uint32_t tid = threadIdx.x, n = P.n;
    const uint32_t wide = (kInv && w > kSnSmallWidth) ? __ldg(W.wide + bi.x) : UINT32_MAX;
    __shared__ uint32_t sB[kSnMaxWidth], sC[kSnMaxWidth];
    if (tid < 32) {
        // entries of column s+c above the block: positions cptr[s+c] .. diag[s+c]-c-1
        const uint32_t c0 = tid, c1 = tid + 32;
        const uint32_t d0 = c0 < w ? P.diag[s + c0] : 0u, d1 = c1 < w ? P.diag[s + c1] : 0u;
        const uint32_t p0 = c0 < w ? P.cptr[s + c0] : 0u, p1 = c1 < w ? P.cptr[s + c1] : 0u;
        if (c0 < w) {
            sB[c0] = d0;
            sC[c0] = p0;
        }
        if (c1 < w) {
            sB[c1] = d1;
            sC[c1] = p1;
        }
        const uint32_t n0 = c0 < w ? (d0 - c0) - p0 : 0u, n1 = c1 < w ? (d1 - c1) - p1 : 0u;
        uint32_t a0 = n0, a1 = n1;  // inclusive warp scans
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y0 = __shfl_up_sync(0xffffffffu, a0, o), y1 = __shfl_up_sync(0xffffffffu, a1, o);
            if (tid >= uint32_t(o)) {
                a0 += y0;
                a1 += y1;
            }
        }
        const uint32_t tot0 = __shfl_sync(0xffffffffu, a0, 31);
        if (c0 < w) pre[c0] = a0 - n0;
        if (c1 < w) pre[c1] = tot0 + a1 - n1;
        if (c0 == w - 1) pre[w] = a0;
        if (c1 == w - 1) pre[w] = tot0 + a1;
    }
    __syncthreads();
    float iv[16];
    if (kInv && wide != UINT32_MAX) {
        load_inverse(iv, invs + bz.y * inv_stride + (size_t(wide) * 2 + 1) * kSnMaxWidth * kSnMaxWidth, tid);
    } else {
        // U11 with its diagonal: U(s+k, s+c), k <= c, at diag[s+c] - (c - k); eight loads in flight
        for (uint32_t e0 = 0; e0 < w * kSnMaxWidth; e0 += 8 * 256) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t e = e0 + u * 256 + tid, c = e >> 6, k = e & 63;
                v[u] = (c < w && k <= c) ? __ldg(val + sB[c] - (c - k)) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t e = e0 + u * 256 + tid, c = e >> 6, k = e & 63;
                if (c < w && k <= c) sT[c * kLD + k] = v[u];
            }
        }
        __syncthreads();
    }
    const uint32_t e0 = t * kSnSweepAbove, e1 = min(e0 + kSnSweepAbove, pre[w]);
    // kSnSweepAbove / 256 entries above the block per thread: column, target
    // and value do not depend on x, so they are loaded before the chain
    constexpr int kPer = int(kSnSweepAbove / 256);
    uint32_t ecol[kPer], etg[kPer];
    float eval[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const uint32_t e = e0 + tid + u * 256;
        ecol[u] = kSnMaxWidth;  // none
        etg[u] = 0u;
        eval[u] = 0.0f;
        if (e < e1) {
            uint32_t lo = 0, hi = w;  // last c with pre[c] <= e
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (pre[mid] <= e)
                    lo = mid;
                else
                    hi = mid;
            }
            const uint32_t p = sC[lo] + (e - pre[lo]);
            ecol[u] = lo;
            etg[u] = __ldg(P.ridx + p);
            eval[u] = __ldg(val + p);
        }
    }
    // the chain's lanes: pivots and reciprocals of columns tid and tid + 32
    float pv0 = 1.0f, pv1 = 1.0f;
    if (wide == UINT32_MAX && tid < 32) {
        if (tid < w) pv0 = sT[tid * kLD + tid];
        if (tid + 32 < w) pv1 = sT[(tid + 32) * kLD + tid + 32];
    }
    const float rc0 = lu_reciprocal(pv0), rc1 = lu_reciprocal(pv1);
    const float g0 = fabsf(pv0), g1 = fabsf(pv1);
    const bool quick =
        __all_sync(kFull, wide == UINT32_MAX && g0 > 1e-30f && g0 < 1e30f && g1 > 1e-30f && g1 < 1e30f);
    pdl_wait();  // the previous level's x
    for (uint32_t q = Q.q0; q < Q.q1; ++q) {
        float *yq = y + size_t(q) * n;
        // the chain over the columns, by one warp, from the block in sT
        auto substitute = [&] {
            if (tid < 32) {
                const uint32_t k0 = tid, k1 = tid + 32;
                const float b0 = k0 < w ? __ldcg(yq + s + k0) : 0.0f, b1 = k1 < w ? __ldcg(yq + s + k1) : 0.0f;
                float v0 = b0, v1 = b1;
                auto step = [&](uint32_t cc, float quotient) {
                    const float xc = __shfl_sync(kFull, quotient, cc & 31);
                    if (k0 == cc) v0 = xc;
                    if (k1 == cc) v1 = xc;
                    if (k0 < cc) v0 = __fsub_rn(v0, __fmul_rn(sT[cc * kLD + k0], xc));
                    if (k1 < cc) v1 = __fsub_rn(v1, __fmul_rn(sT[cc * kLD + k1], xc));
                };
                bool solved = false;
                if (quick) {
                    // every lane divides its own value, so that the step is one shuffle long
                    for (uint32_t cc = w; cc-- > 0;)
                        step(cc, cc < 32 ? lu_quotient(v0, pv0, rc0) : lu_quotient(v1, pv1, rc1));
                    solved = __all_sync(kFull, isfinite(v0) && isfinite(v1));
                }
                if (!solved) {
                    v0 = b0, v1 = b1;
                    for (uint32_t cc = w; cc-- > 0;) step(cc, (cc < 32 ? v0 : v1) / sT[cc * kLD + cc]);
                }
                if (k0 < w) xs[k0] = v0;
                if (k1 < w) xs[k1] = v1;
            }
            __syncthreads();
        };
        if (kInv && wide != UINT32_MAX) {
            if (tid < kSnMaxWidth) vs[tid] = tid < w ? __ldcg(yq + s + tid) : 0.0f;
            __syncthreads();
            wide_solve(iv, vs, part, xs, tid);
            if (!wide_finite(xs, tid)) {
                __syncthreads();  // all warps have read xs
#pragma unroll 1
                for (uint32_t e = tid; e < w * kSnMaxWidth; e += 256) {
                    const uint32_t c = e >> 6, k = e & 63;
                    if (k <= c) sT[c * kLD + k] = __ldg(val + sB[c] - (c - k));
                }
                __syncthreads();
                substitute();
            }
        } else {
            substitute();
        }
        if (t == 0 && tid < w) xo[size_t(q) * n + s + tid] = xs[tid];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            if (ecol[u] >= kSnMaxWidth) continue;
            const float xc = xs[ecol[u]];
            if (xc != 0.0f) atomicAdd(yq + etg[u], -__fmul_rn(eval[u], xc));
        }
        if (q + 1 < Q.q1) __syncthreads();
    }
    sweep_release(W, blk, done);
}

// Per-level launches of the small-supernode groups alone: blocks
// [b0, b0 + gridDim.x) of the map are all groups, one small supernode per
// warp.  Without the full kernels' 64-wide register rows and shared tiles
// four (L: 64 registers) or five (U: 48) blocks stay resident per SM instead of
// two or four, so the wide first levels of the L sweep (a quarter of a million
// leaf supernodes on the 700 x 700 mesh) take half the waves.  Each warp's
// chain is latency-bound (plan, pattern and factor loads, then w dependent
// steps), so resident warps set the rate.
__global__ void __launch_bounds__(256, 4) k_sn_sweep_l_small(DevPattern P, SnSweepPlan W, const float *__restrict__ val,
                                                          float *y, float *xo, uint32_t nrhs, uint32_t b0,
                                                          uint64_t vstride, uint64_t ystride) {
    pdl_release();
    sn_sweep_l_group(P, W, val + blockIdx.z * vstride, y + blockIdx.z * ystride, xo + blockIdx.z * ystride,
                     rhs_share(nrhs), W.map[b0 + blockIdx.x]);
}

__global__ void __launch_bounds__(256, 5) k_sn_sweep_u_small(DevPattern P, SnSweepPlan W, const float *__restrict__ val,
                                                          float *y, float *xo, uint32_t nrhs, uint32_t b0,
                                                          uint64_t vstride, uint64_t ystride) {
    pdl_release();
    sn_sweep_u_group(P, W, val + blockIdx.z * vstride, y + blockIdx.z * ystride, xo + blockIdx.z * ystride,
                     rhs_share(nrhs), W.map[b0 + blockIdx.x]);
}

// Inverses of the diagonal blocks of the wide supernodes (blockIdx.x; first
// column and width): blockIdx.y = 0 L, 1 U, blockIdx.z the value set.
__global__ void __launch_bounds__(256) k_sn_diag_inv(DevPattern P, const uint2 *__restrict__ wide,
                                                      const float *__restrict__ val, uint64_t vstride,
                                                      float *__restrict__ invs, uint64_t inv_stride) {
    __shared__ TriInverse T;
    __shared__ uint32_t sB[kSnMaxWidth];
    const uint2 d = wide[blockIdx.x];
    val += blockIdx.z * vstride;
    if (threadIdx.x < d.y) sB[threadIdx.x] = P.diag[d.x + threadIdx.x];
    __syncthreads();
    tri_invert(T, blockIdx.y, d.y,
               invs + blockIdx.z * inv_stride + (size_t(blockIdx.x) * 2 + blockIdx.y) * kSnMaxWidth * kSnMaxWidth,
               [&](uint32_t i, uint32_t c) { return val[sB[c] + i - c]; });
}

cudaError_t launch_sn_diag_inv(const DevPattern &P, const uint2 *wide, uint32_t nwide, const float *val,
                               uint64_t vstride, uint32_t count, float *invs, uint64_t inv_stride, cudaStream_t st) {
    k_sn_diag_inv<<<dim3(nwide, 2, count), 256, 0, st>>>(P, wide, val, vstride, invs, inv_stride);
    return cudaGetLastError();
}

__global__ void k_sn_copy(const float *__restrict__ xo, float *y, uint32_t t, uint32_t n) {
    const size_t off = size_t(blockIdx.y) * n;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < t; j += gridDim.x * blockDim.x) y[off + j] = xo[off + j];
}

cudaError_t run_sn_sweep(const DevPattern &P, const SnSweepPlan &W, bool upper, uint32_t t, const float *val,
                         float *y, float *xo, uint32_t nrhs, const SolveBatch &B, uint32_t *done, uint32_t *ticket,
                         uint32_t *status, uint32_t spin_limit, cudaStream_t st) {
    const uint64_t ystride = uint64_t(nrhs) * P.n;
    // blocks per level and value set over which the right-hand sides are
    // spread: as many as leave about four blocks per SM in all
    auto shares = [&](uint32_t blocks) {
        const uint64_t have = std::max<uint64_t>(uint64_t(blocks) * B.count, 1);
        return uint32_t(std::min<uint64_t>(nrhs, std::max<uint64_t>(1, 4 * 148 / have)));
    };
    auto full = [&](uint32_t blocks) {
        if (upper) return B.sn_inv ? k_sn_sweep_u<true> : k_sn_sweep_u<false>;
        if (B.sn_inv) return k_sn_sweep_l<true, 2>;
        return uint64_t(blocks) * B.count > kManyBlocks ? k_sn_sweep_l<false, 3> : k_sn_sweep_l<false, 2>;
    };
    if (W.fused && done && W.nblocks) {
        // one launch: blocks in map order by ticket, supernodes wait for their releases
        cudaError_t e = cudaMemsetAsync(done, 0, sizeof(uint32_t) * size_t(W.ns) * B.count, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(ticket, 0, sizeof(uint32_t) * B.count, st);
        if (e != cudaSuccess) return e;
        const dim3 grid(W.nblocks, 1, B.count);
        full(W.nblocks)<<<grid, 256, 0, st>>>(P, W, val, y, xo, nrhs, 0, B.vstride, ystride, B.sn_inv, B.sn_inv_stride, done,
                                   ticket, status, spin_limit);
    } else {
        // one launch per level (up to three where its narrow parts or its
        // small-supernode groups get their own), each chained to the one
        // before (its blocks start while the previous launch drains, and wait
        // for its x); the supernodes of one level do not feed each other, so
        // its launches may run in any order
        for (uint32_t l = 0; l < W.nlev; ++l) {
            const SnSweepLevel &lv = W.levels[l];
            const uint3 k3 = sn_sweep_level_launches(lv, upper);
            cudaError_t e = cudaSuccess;
            const uint32_t rest = k3.z ? lv.big : lv.blocks;  // blocks not in the small-group launch
            if (k3.x) {  // the full kernel: every block that no other launch takes
                const uint32_t nblk = k3.y ? lv.wide : rest;
                const dim3 grid(nblk, shares(nblk), B.count);
                e = launch_chained(full(nblk), grid, dim3(256), 0, st, P, W, val, y, xo, nrhs, lv.b0, B.vstride, ystride,
                                   B.sn_inv, B.sn_inv_stride, (uint32_t *)nullptr, (uint32_t *)nullptr, status,
                                   spin_limit);
                if (e != cudaSuccess) return e;
            }
            if (k3.y) {  // L: the narrow parts (and the groups, unless they launch apart)
                const uint32_t nblk = rest - lv.wide;
                const dim3 grid(nblk, shares(nblk), B.count);
                e = launch_chained(k_sn_sweep_l_narrow, grid, dim3(256), 0, st, P, W, val, y, xo, nrhs, lv.b0 + lv.wide,
                                   B.vstride, ystride);
                if (e != cudaSuccess) return e;
            }
            if (k3.z) {  // the small-supernode groups
                const dim3 grid(lv.blocks - lv.big, shares(lv.blocks - lv.big), B.count);
                if (upper)
                    e = launch_chained(k_sn_sweep_u_small, grid, dim3(256), 0, st, P, W, val, y, xo, nrhs,
                                       lv.b0 + lv.big, B.vstride, ystride);
                else
                    e = launch_chained(k_sn_sweep_l_small, grid, dim3(256), 0, st, P, W, val, y, xo, nrhs,
                                       lv.b0 + lv.big, B.vstride, ystride);
                if (e != cudaSuccess) return e;
            }
        }
    }
    if (t > 0) {  // the vectors of all value sets are contiguous: nrhs * count of them
        uint32_t bx = (t + 255) / 256;
        if (bx > 1024) bx = 1024;
        k_sn_copy<<<dim3(bx, nrhs * B.count, 1), 256, 0, st>>>(xo, y, t, P.n);
    }
    return cudaGetLastError();
}

}  // namespace glu
