// Small dense triangular kernels shared by the supernodal and the dense
// trailing-block factorization: the LU of a w x w diagonal block (w <= 64)
// and the triangular solves of the rows of L21 and the columns of U12 against
// it.  Both follow the right-looking column algorithm of the reference
// (src/numeric.cu:10-345): every entry receives its updates in increasing
// column order, then (L entries) its division by the pivot; products are
// fused multiply-adds.
//
// The code is written as short loops over 16-column chunks whose bodies are
// unrolled (register arrays need static indices): a fully unrolled 64-step
// form is tens of kilobytes of straight-line code that every block fetches
// once, and stalls on instruction fetch.
#pragma once

#include "glu_common.cuh"

namespace glu {

constexpr int kTriMax = 64;        // largest block width
constexpr int kTriChunk = 16;      // columns per unrolled chunk
constexpr int kTriThreads = 256;   // threads of the diagonal-block LU
constexpr int kTriML = kTriMax + 4;  // leading dimension of the operand matrix (16-byte rows)

#ifdef __CUDACC__

// Barrier of the first 256 threads of a block (a block may hold further warps
// with other work).
__device__ __forceinline__ void tri_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// Leading dimension of the block in shared memory: 16-byte columns, two
// neighbours' float4 at four rows apart on different banks.
constexpr int kLuLD = kTriMax + 16;

constexpr int kLuChunk = 8;         // columns per step of the block LU

// a / p from r, p's reciprocal to about one unit in the last place: the
// quotient's estimate corrected by its remainder (Markstein, IBM J. Res. Dev.
// 34, 1990).  For finite quotients: an infinite one, which the division gives
// as such, comes out as NaN here (its remainder is infinite too), so whoever
// uses it looks for values that are not finite and divides instead, or takes
// lu_quotient_wide, which is infinite where the estimate is.
__device__ __forceinline__ float lu_quotient(float a, float p, float r) {
    const float q = a * r;
    return fmaf(fmaf(-q, p, a), r, q);
}
__device__ __forceinline__ float lu_quotient_wide(float a, float p, float r) {
    const float q = a * r;
    return isfinite(q) ? fmaf(fmaf(-q, p, a), r, q) : q;
}
__device__ __forceinline__ float lu_reciprocal(float p) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(p));
    return r;
}

// Columns [base, base + 8) of the 64 x 64 block S (column-major, leading
// dimension kLuLD) factored by one warp.  Every lane keeps the 8 x 8 diagonal
// block in registers and factors it for itself, so the chain of pivots holds
// no shuffle and no trip through shared memory, only reciprocal, quotient and
// multiply-add; each lane carries two of the rows below along.
// kDivide: quotients by division; otherwise by lu_quotient, and nothing is
// stored and false returned when a pivot is too large or too small for it.
// (Entries of the diagonal block that are not finite make a pivot of it so; the
// rows below have none and take lu_quotient_wide, off the chain of pivots. A
// vote on them in front of the stores took a level of the grids 0.7 us longer.)
template <bool kDivide>
__device__ __forceinline__ bool lu_panel_try(float *S, uint32_t base, uint32_t w, bool last_l, float pert,
                                             uint32_t lane) {
    constexpr int N = kLuChunk;
    float d[N][N], a0[N], a1[N];  // d[row][column]
    const uint32_t r0 = base + N + lane, r1 = r0 + 32;
    // (rows past the block: the last row once more, not stored)
    float *p0 = S + base * kLuLD + min(r0, uint32_t(kTriMax) - 1), *p1 = S + base * kLuLD + min(r1, uint32_t(kTriMax) - 1);
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const float4 *s4 = reinterpret_cast<const float4 *>(S + (base + c) * kLuLD + base);
#pragma unroll
        for (int v = 0; v < N / 4; ++v) {
            const float4 t = s4[v];
            d[4 * v][c] = t.x, d[4 * v + 1][c] = t.y, d[4 * v + 2][c] = t.z, d[4 * v + 3][c] = t.w;
        }
        a0[c] = p0[c * kLuLD];
        a1[c] = p1[c * kLuLD];
    }
    bool ok = true;  // the same in all lanes, as the diagonal block is
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const uint32_t next = base + c + 1;
        if (pert > 0.0f && (next < w || (next == w && last_l)) && fabsf(d[c][c]) < pert) d[c][c] = pert;
        const float p = d[c][c], mag = fabsf(p);
        ok = ok && mag > 1e-30f && mag < 1e30f;
        const float r = kDivide ? 0.0f : lu_reciprocal(p);
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i > c) d[i][c] = kDivide ? d[i][c] / p : lu_quotient(d[i][c], p, r);
        a0[c] = kDivide ? a0[c] / p : lu_quotient_wide(a0[c], p, r);
        a1[c] = kDivide ? a1[c] / p : lu_quotient_wide(a1[c], p, r);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (j <= c) continue;
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i > c) d[i][j] = fmaf(-d[i][c], d[c][j], d[i][j]);
            a0[j] = fmaf(-a0[c], d[c][j], a0[j]);
            a1[j] = fmaf(-a1[c], d[c][j], a1[j]);
        }
    }
    if (!kDivide && !ok) return false;
    __syncwarp();  // every lane has read the panel
    if (r0 < uint32_t(kTriMax)) {
#pragma unroll
        for (int c = 0; c < N; ++c) p0[c * kLuLD] = a0[c];
    }
    if (r1 < uint32_t(kTriMax)) {
#pragma unroll
        for (int c = 0; c < N; ++c) p1[c * kLuLD] = a1[c];
    }
    // lane 2 c + v stores rows 4 v .. 4 v + 3 of column c, chosen by selects (a
    // branch per value, or one lane storing all of them, takes longer)
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float t[N];
#pragma unroll
        for (int c = 0; c < N; ++c) t[c] = (lane & 1) ? d[4 + e][c] : d[e][c];
#pragma unroll
        for (int c = 0; c < N / 2; ++c) t[c] = (lane & 2) ? t[2 * c + 1] : t[2 * c];
#pragma unroll
        for (int c = 0; c < N / 4; ++c) t[c] = (lane & 4) ? t[2 * c + 1] : t[2 * c];
        o[e] = (lane & 8) ? t[1] : t[0];
    }
    if (lane < 2 * N)
        *reinterpret_cast<float4 *>(S + (base + (lane >> 1)) * kLuLD + base + 4 * (lane & 1)) =
            make_float4(o[0], o[1], o[2], o[3]);
    return true;
}
// (out of line: its divisions would take the common path's registers)
static __device__ __noinline__ void lu_panel_divide(float *S, uint32_t base, uint32_t w, bool last_l, float pert,
                                                    uint32_t lane) {
    lu_panel_try<true>(S, base, w, last_l, pert, lane);
}
__device__ __forceinline__ void lu_panel(float *S, uint32_t base, uint32_t w, bool last_l, float pert, uint32_t lane) {
    if (!lu_panel_try<false>(S, base, w, last_l, pert, lane)) lu_panel_divide(S, base, w, last_l, pert, lane);
}

// Columns j and j + 1 of the block behind columns [base, base + 8), by eight
// threads: each solves the columns' 8 entries of U (L11 x = a, the same values
// in all eight) and updates the rows base + 8 + 4 q + 32 g .. + 3 with them.
// (Shared-memory loads bound it: an entry of L serves two columns.)
__device__ __forceinline__ void lu_columns(float *S, uint32_t base, uint32_t j, uint32_t q) {
    constexpr int N = kLuChunk;
    float *col[2] = {S + j * kLuLD + base, S + (j + 1) * kLuLD + base};
    // rows of this thread, relative to base (past the block: the last four, not stored)
    const uint32_t last = uint32_t(kTriMax) - 4 - base, r0 = N + 4 * q, r1 = r0 + 32;
    const uint32_t o0 = min(r0, last), o1 = min(r1, last);
    float x[2][N];
    float4 c[2][2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        const float4 u = *reinterpret_cast<const float4 *>(col[b]), v = *reinterpret_cast<const float4 *>(col[b] + 4);
        x[b][0] = u.x, x[b][1] = u.y, x[b][2] = u.z, x[b][3] = u.w;
        x[b][4] = v.x, x[b][5] = v.y, x[b][6] = v.z, x[b][7] = v.w;
        c[b][0] = *reinterpret_cast<const float4 *>(col[b] + o0);
        c[b][1] = *reinterpret_cast<const float4 *>(col[b] + o1);
    }
    const float *lp = S + base * kLuLD + base;
#pragma unroll
    for (int k = 0; k + 1 < N; ++k) {
        const float4 u = *reinterpret_cast<const float4 *>(lp + k * kLuLD);
        const float4 v = *reinterpret_cast<const float4 *>(lp + k * kLuLD + 4);
        const float l[N] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
        for (int r = 0; r < N; ++r)
            if (r > k) {
                x[0][r] = fmaf(-l[r], x[0][k], x[0][r]);
                x[1][r] = fmaf(-l[r], x[1][k], x[1][r]);
            }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const float4 l0 = *reinterpret_cast<const float4 *>(lp + k * kLuLD + o0);
        const float4 l1 = *reinterpret_cast<const float4 *>(lp + k * kLuLD + o1);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            c[b][0].x = fmaf(-l0.x, x[b][k], c[b][0].x);
            c[b][0].y = fmaf(-l0.y, x[b][k], c[b][0].y);
            c[b][0].z = fmaf(-l0.z, x[b][k], c[b][0].z);
            c[b][0].w = fmaf(-l0.w, x[b][k], c[b][0].w);
            c[b][1].x = fmaf(-l1.x, x[b][k], c[b][1].x);
            c[b][1].y = fmaf(-l1.y, x[b][k], c[b][1].y);
            c[b][1].z = fmaf(-l1.z, x[b][k], c[b][1].z);
            c[b][1].w = fmaf(-l1.w, x[b][k], c[b][1].w);
        }
    }
    __syncwarp();  // the eight threads of the columns have read them
    if (r0 <= last) {
#pragma unroll
        for (int b = 0; b < 2; ++b) *reinterpret_cast<float4 *>(col[b] + r0) = c[b][0];
    }
    if (r1 <= last) {
#pragma unroll
        for (int b = 0; b < 2; ++b) *reinterpret_cast<float4 *>(col[b] + r1) = c[b][1];
    }
    if (q == 0) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            *reinterpret_cast<float4 *>(col[b]) = make_float4(x[b][0], x[b][1], x[b][2], x[b][3]);
            *reinterpret_cast<float4 *>(col[b] + 4) = make_float4(x[b][4], x[b][5], x[b][6], x[b][7]);
        }
    }
}

// Column j of the block behind columns [base, base + 8), by one warp: every lane
// solves the column's 8 entries of U and updates rows base + 8 + lane and
// base + 40 + lane with them.
__device__ __forceinline__ void lu_one_column(float *S, uint32_t base, uint32_t j, uint32_t lane) {
    constexpr int N = kLuChunk;
    float *col = S + j * kLuLD + base;
    const float *lp = S + base * kLuLD + base;
    // (rows past the block: the last one once more, not stored)
    const uint32_t last = uint32_t(kTriMax) - 1 - base, r0 = N + lane, r1 = r0 + 32;
    const uint32_t o0 = min(r0, last), o1 = min(r1, last);
    const float4 u = *reinterpret_cast<const float4 *>(col), v = *reinterpret_cast<const float4 *>(col + 4);
    float x[N] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    float c0 = col[o0], c1 = col[o1], l0[N], l1[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        l0[k] = lp[k * kLuLD + o0];
        l1[k] = lp[k * kLuLD + o1];
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const float4 lu = *reinterpret_cast<const float4 *>(lp + k * kLuLD);
        const float4 lv = *reinterpret_cast<const float4 *>(lp + k * kLuLD + 4);
        const float l[N] = {lu.x, lu.y, lu.z, lu.w, lv.x, lv.y, lv.z, lv.w};
#pragma unroll
        for (int r = 0; r < N; ++r)
            if (r > k) x[r] = fmaf(-l[r], x[k], x[r]);
        c0 = fmaf(-l0[k], x[k], c0);
        c1 = fmaf(-l1[k], x[k], c1);
    }
    __syncwarp();  // every lane has read the column
    if (r0 <= last) col[r0] = c0;
    if (r1 <= last) col[r1] = c1;
    if (lane == 0) {
        *reinterpret_cast<float4 *>(col) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4 *>(col + 4) = make_float4(x[4], x[5], x[6], x[7]);
    }
}

// LU of the w x w block (w <= 64) in shared memory, S column-major with leading
// dimension kLuLD, 256 threads; rows and columns >= w must hold the identity.
// Right-looking by chunks of 8 columns.  Behind a chunk, each warp first takes
// one column of the next chunk (lu_one_column); then warp 0 factors that chunk
// (lu_panel) while the others update the columns further right (lu_columns).
// Every entry receives its updates in increasing column order, then (L
// entries) its division by the pivot, GESP as numeric.cu:139-140 (a pivot
// whose column has an L part: c < w - 1, or c = w - 1 and last_l).
// A 64-wide block takes 12,100 cycles on its own; 30,700 with a row per four
// threads, a barrier and a division per pivot (the division's slow path is
// taken for every zero of a sparse or padded row).
// The caller has a barrier between its writes of S and the call; on return the
// block is complete for all 256 threads.  done(p) is called by warps 5, 6 and 7,
// which have no columns left by then, as soon as columns 16 p .. 16 p + 15 of L
// and rows 16 p .. 16 p + 15 of U are final (p = 0 .. 3, for w = 64 only).
struct TriNothing {
    __device__ __forceinline__ void operator()(uint32_t) const {}
};
template <class Done = TriNothing>
__device__ __forceinline__ void tri_lu_smem(float *S, uint32_t w, bool last_l, float pert, Done &&done = Done()) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t end = (w + kLuChunk - 1) / kLuChunk * kLuChunk;  // columns to factor
    if (warp == 0) lu_panel(S, 0, w, last_l, pert, lane);
    tri_sync();
#pragma unroll 1
    for (uint32_t base = 0; base + kLuChunk < end; base += kLuChunk) {
        lu_one_column(S, base, base + kLuChunk + warp, lane);
        tri_sync();
        if (warp == 0)
            lu_panel(S, base + kLuChunk, w, last_l, pert, lane);
        else if (base + kLuChunk * (warp + 1) < end)
            lu_columns(S, base, base + kLuChunk * (warp + 1) + 2 * (lane >> 3), lane & 7);
        else if (warp >= 5 && w == uint32_t(kTriMax) && base >= 16 && (base & 15) == 0)
            done(base / 16 - 1);
        tri_sync();
    }
    if (warp >= 5 && w == uint32_t(kTriMax)) done(3);
}

// Solve within chunk cb of one row: x = the chunk's N <= 16 entries after the
// updates of the earlier chunks; for c = 16 cb + k < w in increasing order,
// x[k] *= 1 / M(c, c) (kDiv) and x[p] -= x[k] M(c, 16 cb + p) for p > k.
// M row-major in shared memory with leading dimension kTriML; with kDiv the
// row's padding holds the pivot's reciprocal, M[c * kTriML + kTriMax] = 1 /
// M(c, c) (correctly rounded), so that the solve's dependency chain is a
// multiply and a fused multiply-add per column instead of a division (one
// extra rounding of each L entry).  The row's entries before `first` are
// structural zeros: they are not multiplied, as M may not be finite there.
template <bool kDiv, int N>
__device__ __forceinline__ void tri_chunk_solve(float (&x)[N], const float *sM, uint32_t cb, uint32_t w,
                                                uint32_t first = 0) {
    static_assert(N <= kTriChunk, "one chunk");
    constexpr int NV = (N + 3) / 4;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const uint32_t c = cb * kTriChunk + k;
        if (c >= w) break;
        const float4 *m4 = reinterpret_cast<const float4 *>(sM + c * kTriML + cb * kTriChunk);
        float mr[4 * NV];
#pragma unroll
        for (int v = k / 4; v < NV; ++v) {
            const float4 t = m4[v];
            mr[4 * v] = t.x; mr[4 * v + 1] = t.y; mr[4 * v + 2] = t.z; mr[4 * v + 3] = t.w;
        }
        if (kDiv) x[k] = x[k] * sM[c * kTriML + kTriMax];
#pragma unroll
        for (int p = k + 1; p < N; ++p)
            if (c >= first) x[p] = fmaf(-x[k], mr[p], x[p]);
    }
}

// y (chunk cj) -= x (solved chunk cb) times M(chunk cb rows, chunk cj columns),
// rows of M in increasing order, from `first` on.
__device__ __forceinline__ void tri_chunk_update(float (&y)[kTriChunk], const float (&x)[kTriChunk], const float *sM,
                                                 uint32_t cb, uint32_t cj, uint32_t w, uint32_t first = 0) {
#pragma unroll
    for (int k = 0; k < kTriChunk; ++k) {
        const uint32_t c = cb * kTriChunk + k;
        if (c >= w) break;
        const float4 *m4 = reinterpret_cast<const float4 *>(sM + c * kTriML + cj * kTriChunk);
#pragma unroll
        for (int v = 0; v < kTriChunk / 4; ++v) {
            const float4 t = m4[v];
            if (c < first) continue;
            y[4 * v] = fmaf(-x[k], t.x, y[4 * v]);
            y[4 * v + 1] = fmaf(-x[k], t.y, y[4 * v + 1]);
            y[4 * v + 2] = fmaf(-x[k], t.z, y[4 * v + 2]);
            y[4 * v + 3] = fmaf(-x[k], t.w, y[4 * v + 3]);
        }
    }
}

// Solve x M = a for one row per thread (kDiv: M upper triangular; else
// unit upper triangular, which with M = L^T is the column solve L x = a),
// w <= 64.  The row lives in shared memory, entry c at sW[c * ldw + t];
// entries >= w are never stored back and never used as multipliers.
template <bool kDiv>
__device__ __forceinline__ void tri_rows_solve(float *sW, uint32_t ldw, uint32_t t, const float *sM, uint32_t w) {
    const uint32_t nch = (w + kTriChunk - 1) / kTriChunk;
    for (uint32_t cb = 0; cb < nch; ++cb) {
        float x[kTriChunk];
#pragma unroll
        for (int k = 0; k < kTriChunk; ++k) x[k] = sW[(cb * kTriChunk + k) * ldw + t];
        tri_chunk_solve<kDiv>(x, sM, cb, w);
#pragma unroll
        for (int k = 0; k < kTriChunk; ++k) sW[(cb * kTriChunk + k) * ldw + t] = x[k];
        for (uint32_t cj = cb + 1; cj < nch; ++cj) {
            float y[kTriChunk];
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) y[k] = sW[(cj * kTriChunk + k) * ldw + t];
            tri_chunk_update(y, x, sM, cb, cj, w);
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) sW[(cj * kTriChunk + k) * ldw + t] = y[k];
        }
    }
}

// Two rows t0, t1 of one thread, w = 64: an entry of M read from shared memory
// (four bytes to every lane, which is what bounds the solves of many rows)
// serves both.
template <bool kDiv>
__device__ __forceinline__ void tri_two_rows_solve(float *sW, uint32_t ldw, uint32_t t0, uint32_t t1, const float *sM) {
    constexpr uint32_t kCh = kTriMax / kTriChunk;
#pragma unroll 1
    for (uint32_t cb = 0; cb < kCh; ++cb) {
        float x[2][kTriChunk];
        const float *m = sM + cb * kTriChunk * kTriML;  // the chunk's rows of M
        float *w = sW + cb * kTriChunk * ldw;
#pragma unroll
        for (int k = 0; k < kTriChunk; ++k) x[0][k] = w[k * ldw + t0], x[1][k] = w[k * ldw + t1];
#pragma unroll
        for (int k = 0; k < kTriChunk; ++k) {
            const float4 *m4 = reinterpret_cast<const float4 *>(m + k * kTriML + cb * kTriChunk);
            float mr[kTriChunk];
#pragma unroll
            for (int v = k / 4; v < kTriChunk / 4; ++v) {
                const float4 t = m4[v];
                mr[4 * v] = t.x, mr[4 * v + 1] = t.y, mr[4 * v + 2] = t.z, mr[4 * v + 3] = t.w;
            }
            if (kDiv) {
                const float d = m[k * kTriML + kTriMax];
                x[0][k] *= d, x[1][k] *= d;
            }
#pragma unroll
            for (int p = k + 1; p < kTriChunk; ++p) {
                x[0][p] = fmaf(-x[0][k], mr[p], x[0][p]);
                x[1][p] = fmaf(-x[1][k], mr[p], x[1][p]);
            }
        }
#pragma unroll
        for (int k = 0; k < kTriChunk; ++k) w[k * ldw + t0] = x[0][k], w[k * ldw + t1] = x[1][k];
#pragma unroll 1
        for (uint32_t cj = cb + 1; cj < kCh; ++cj) {
            float y[2][kTriChunk];
            float *wj = sW + cj * kTriChunk * ldw;
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) y[0][k] = wj[k * ldw + t0], y[1][k] = wj[k * ldw + t1];
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) {
                const float4 *m4 = reinterpret_cast<const float4 *>(m + k * kTriML + cj * kTriChunk);
#pragma unroll
                for (int v = 0; v < kTriChunk / 4; ++v) {
                    const float4 t = m4[v];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        y[r][4 * v] = fmaf(-x[r][k], t.x, y[r][4 * v]);
                        y[r][4 * v + 1] = fmaf(-x[r][k], t.y, y[r][4 * v + 1]);
                        y[r][4 * v + 2] = fmaf(-x[r][k], t.z, y[r][4 * v + 2]);
                        y[r][4 * v + 3] = fmaf(-x[r][k], t.w, y[r][4 * v + 3]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) wj[k * ldw + t0] = y[0][k], wj[k * ldw + t1] = y[1][k];
        }
    }
}

// The same as tri_rows_solve with two threads per row (half 0 or 1; all 2 x rows threads of the
// block take part): chunk cj belongs to half cj % 2, which applies the earlier
// chunks to it and solves it, so the two halves share the updates and only a
// solved chunk is waited for (a block barrier each).  The caller has a barrier
// between its writes and the call and before it reads the result.
template <bool kDiv>
__device__ __forceinline__ void tri_rows_solve_halves(float *sW, uint32_t ldw, uint32_t t, uint32_t half, const float *sM,
                                                      uint32_t w, uint32_t first = 0) {
    const uint32_t nch = (w + kTriChunk - 1) / kTriChunk;
    for (uint32_t cb = 0; cb < nch; ++cb) {
        if (half == (cb & 1)) {
            float x[kTriChunk];
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) x[k] = sW[(cb * kTriChunk + k) * ldw + t];
            tri_chunk_solve<kDiv>(x, sM, cb, w, first);
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) sW[(cb * kTriChunk + k) * ldw + t] = x[k];
        }
        if (cb + 1 == nch) break;
        __syncthreads();
        float x[kTriChunk];
#pragma unroll
        for (int k = 0; k < kTriChunk; ++k) x[k] = sW[(cb * kTriChunk + k) * ldw + t];
        for (uint32_t cj = cb + 1 + ((cb + 1 + half) & 1); cj < nch; cj += 2) {
            float y[kTriChunk];
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) y[k] = sW[(cj * kTriChunk + k) * ldw + t];
            tri_chunk_update(y, x, sM, cb, cj, w, first);
#pragma unroll
            for (int k = 0; k < kTriChunk; ++k) sW[(cj * kTriChunk + k) * ldw + t] = y[k];
        }
    }
}

// Working arrays of tri_invert.
struct TriInverse {
    float M[kTriMax][kTriMax + 1], X[kTriMax][kTriMax + 1], W[kTriMax / 2][kTriMax / 2 + 1];
};

// The inverse of a factored diagonal block of w <= 64 columns by 256 threads,
// column-major 64 x 64 at out (the identity past w): which = 0 the unit lower L,
// 1 the upper U; at(i, c) reads the block's entry.  U is taken as its
// transpose, so both are the inverse of a lower triangular M: the four 16 x 16
// diagonal blocks by substitution (a column per thread, in registers), then
// twice the off-diagonal block of a pair, X21 = -X22 M21 X11, as products over
// all threads -- 16 dependent steps instead of 64 (a launch at order 128: 8.3
// us, 28 us with 64 threads of serial substitution).
template <class At>
__device__ __forceinline__ void tri_invert(TriInverse &T, uint32_t which, uint32_t w, float *__restrict__ out, At &&at) {
    auto &M = T.M;
    auto &X = T.X;
    auto &W = T.W;
    const uint32_t tid = threadIdx.x;
#pragma unroll 4
    for (uint32_t e = tid; e < uint32_t(kTriMax * kTriMax); e += 256) {
        const uint32_t c = e / kTriMax, i = e % kTriMax;
        float v = i == c ? 1.0f : 0.0f;
        if (i < w && c < w && (which == 0 ? i > c : i <= c)) v = at(i, c);
        if (which == 0)
            M[i][c] = v;
        else
            M[c][i] = v;
        X[i][c] = 0.0f;
    }
    __syncthreads();
    if (tid < uint32_t(kTriMax)) {  // column j of the 16 x 16 block at g
        const uint32_t g = tid & ~15u, j = tid & 15u;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k < i; ++k) acc = fmaf(M[g + i][g + k], x[k], acc);
            // zero above the diagonal: x[k] = 0 for k < j
            x[i] = (uint32_t(i) == j ? 1.0f : uint32_t(i) > j ? -acc : 0.0f) / M[g + i][g + i];
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) X[g + i][g + j] = x[i];
    }
    __syncthreads();
    // pairs of 16-blocks: 2 x 256 outputs; W = M21 X11, X21 = -X22 W
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const uint32_t g = u * 32, i = tid / 16, j = tid % 16;
        float acc = 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) acc = fmaf(M[g + 16 + i][g + k], X[g + k][g + j], acc);
        W[u * 16 + i][j] = acc;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const uint32_t g = u * 32, i = tid / 16, j = tid % 16;
        float acc = 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) acc = fmaf(X[g + 16 + i][g + 16 + k], W[u * 16 + k][j], acc);
        X[g + 16 + i][g + j] = -acc;
    }
    __syncthreads();
    // the pair of 32-blocks
    const uint32_t j = tid % 32, i0 = tid / 32;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
        const float xv = X[k][j];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = fmaf(M[32 + i0 + 8 * u][k], xv, acc[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        W[i0 + 8 * u][j] = acc[u];
        acc[u] = 0.0f;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
        const float wv = W[k][j];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = fmaf(X[32 + i0 + 8 * u][32 + k], wv, acc[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) X[32 + i0 + 8 * u][j] = -acc[u];
    __syncthreads();
#pragma unroll 4
    for (uint32_t e = tid; e < uint32_t(kTriMax * kTriMax); e += 256)
        out[e] = which == 0 ? X[e % kTriMax][e / kTriMax] : X[e / kTriMax][e % kTriMax];
}

// Four-byte asynchronous copy global -> shared (completes at tri_async_wait).
__device__ __forceinline__ void tri_async_copy(float *dst, const float *src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void tri_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tri_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

#endif  // __CUDACC__

}  // namespace glu
