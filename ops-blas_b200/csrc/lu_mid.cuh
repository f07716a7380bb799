// Blocked LU of one matrix of order 33..128 held in shared memory, in blocks of 16 columns whose
// rows are spread over the lanes of one warp (row lane + 32 t, t < R = ceil(n / 32)). Shared by the
// batched kernel (getrf_mid.cu) and the grouped persistent kernel (grouped.cu).
//
// Left-looking over the blocks: a block is loaded into registers once, takes every earlier panel's
// update, is factored by its warp alone and goes back to shared memory, so a column needs no
// barrier of more than a warp. Rows never move: S holds every value at its physical row, `pos` is a
// row's index in the reference's in-place matrix (sgetrf_batched_kernel.cpp:106-150) and rowof the
// inverse. Every element receives one fmaf per step in increasing step order and multipliers are the
// correctly rounded quotients, so the factors are the reference order's bits.
//
// A row that has become a pivot is poisoned with NaN in the registers of the blocks still to be
// factored (its true values are in S or in the panel's row buffer by then): it never wins the pivot
// search and needs no masks in the updates.
#pragma once

#include <cuda_runtime.h>

#include "f32x2.cuh"
#include "quotient.cuh"
#include "small_common.cuh"

namespace opsblas {

constexpr int kMidNB = 16;    // columns of a block
constexpr int kMidULd = 20;   // row stride of the update's U rows (16-byte rows, conflict-free by eights)
constexpr int kMidMaxN = 128;

__host__ __device__ constexpr int mid_blocks(int n) { return (n + kMidNB - 1) / kMidNB; }

// Shared memory of one matrix of NBLK blocks factored by W warps. Constant strides: every address in
// the unrolled code is a register plus an immediate.
//   S: 16 NBLK columns of LD floats (LD is odd in units of 4: accesses along a row spread over
//      eight banks); columns beyond n hold anything, no other column ever depends on them
//   u: per warp, 16 rows of the block being worked on
//   rowof: physical row of every position; ipiv: pivot positions; posn: per panel, the position of
//   every row after it; stop: columns eliminated (n, or the column of an exactly-zero pivot)
template <int NBLK, int W>
struct MidSmem {
    static constexpr int R = (NBLK + 1) / 2;  // rows per lane
    static constexpr int LD = kMidNB * NBLK + 4;
    static constexpr int NP = kMidNB * NBLK;
    float S[NP * LD];
    float u[W][kMidNB * kMidULd];
    int rowof[NP], ipiv[NP];
    unsigned char posn[NBLK][32 * R];
    int stop, pad[3];
};

// max over the warp of |v|; NaN lanes are ignored unless all are NaN
__device__ __forceinline__ float warp_absmax(float v)
{
    float r;
    asm volatile("redux.sync.max.abs.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// A block in registers: p[t][h] = columns 2h, 2h + 1 of row lane + 32 t, packed for the f32x2 unit
// (kept packed everywhere: moving pairs in and out of scalars cost two moves per packed fma).
template <int R>
using MidBlock = f32x2[R][kMidNB / 2];

// The block of columns k0... Rows beyond n are NaN (dead).
template <int NBLK, int W>
__device__ __forceinline__ void mid_load(MidBlock<MidSmem<NBLK, W>::R>& p, const MidSmem<NBLK, W>& M, int n, int k0,
                                         int lane)
{
    constexpr int R = MidSmem<NBLK, W>::R, LD = MidSmem<NBLK, W>::LD;
    const float* s = M.S + lane + k0 * LD;
#pragma unroll
    for (int h = 0; h < kMidNB / 2; h++)
#pragma unroll
        for (int t = 0; t < R; t++) p[t][h] = f2_pack(s[32 * t + 2 * h * LD], s[32 * t + (2 * h + 1) * LD]);
    if (lane + 32 * (R - 1) >= n) {  // n > 32 (R - 1): only the last tile has such rows
#pragma unroll
        for (int h = 0; h < kMidNB / 2; h++) p[R - 1][h] = f2_dup(__int_as_float(0x7fffffff));
    }
}

// Row t of the block to 16 consecutive floats.
template <int R>
__device__ __forceinline__ void mid_put_row(const MidBlock<R>& p, int t, float* dst)
{
    ulonglong2* w = reinterpret_cast<ulonglong2*>(dst);
#pragma unroll
    for (int q = 0; q < kMidNB / 4; q++) w[q] = make_ulonglong2(p[t][2 * q], p[t][2 * q + 1]);
}

// Row t of the block to its 16 columns of S.
template <int R, int LD>
__device__ __forceinline__ void mid_put_columns(const MidBlock<R>& p, int t, float* s)
{
#pragma unroll
    for (int h = 0; h < kMidNB / 2; h++) {
        float x, y;
        f2_unpack(p[t][h], x, y);
        s[2 * h * LD] = x;
        s[(2 * h + 1) * LD] = y;
    }
}

// p[t][*] += u[*] * l[t], u 16 floats of shared memory
template <int R>
__device__ __forceinline__ void mid_rank1(MidBlock<R>& p, const float* uk, const f32x2 (&l)[R])
{
    const ulonglong2* w = reinterpret_cast<const ulonglong2*>(uk);
#pragma unroll
    for (int q = 0; q < kMidNB / 4; q++) {
        const ulonglong2 v = w[q];
#pragma unroll
        for (int t = 0; t < R; t++) {
            p[t][2 * q] = f2_fma(v.x, l[t], p[t][2 * q]);
            p[t][2 * q + 1] = f2_fma(v.y, l[t], p[t][2 * q + 1]);
        }
    }
}

// Applies the first K columns of panel b to the block at column k0: its U rows (solved with a lane
// per column, both halves of the warp alike) go to S, the rows below take the rank-K update, and the
// panel's pivot rows die. u: this warp's buffer (the U rows, negated).
template <int NBLK, int W>
__device__ __forceinline__ void mid_apply(MidBlock<MidSmem<NBLK, W>::R>& p, MidSmem<NBLK, W>& M, float* u, int b,
                                          int K, int k0, int lane)
{
    constexpr int R = MidSmem<NBLK, W>::R, LD = MidSmem<NBLK, W>::LD;
    const int q0 = b * kMidNB;
    bool dies[R];
#pragma unroll
    for (int t = 0; t < R; t++) {
        const int d = (int)M.posn[b][lane + 32 * t] - q0;
        dies[t] = (unsigned)d < (unsigned)K;
        if (dies[t]) mid_put_row<R>(p, t, u + d * kMidULd);
    }
    __syncwarp();
    {
        const int col = lane & (kMidNB - 1);
        int r[kMidNB];
#pragma unroll
        for (int q = 0; q < kMidNB / 4; q++) {
            const int4 v = reinterpret_cast<const int4*>(M.rowof + q0)[q];
            r[4 * q] = v.x;
            r[4 * q + 1] = v.y;
            r[4 * q + 2] = v.z;
            r[4 * q + 3] = v.w;
        }
        float x[kMidNB];
#pragma unroll
        for (int i = 0; i < kMidNB; i++) x[i] = u[i * kMidULd + col];
        const float* l11 = M.S + q0 * LD;
#pragma unroll
        for (int i = 1; i < kMidNB; i++) {
#pragma unroll
            for (int c = 0; c < kMidNB; c++)
                if (c < i) x[i] = fmaf(-l11[r[i] + c * LD], x[c], x[i]);  // rows from K on are not used
        }
        __syncwarp();
        if (lane < kMidNB) {
            float* s = M.S + (k0 + col) * LD;
#pragma unroll
            for (int i = 0; i < kMidNB; i++) {
                u[i * kMidULd + col] = -x[i];
                if (i < K) s[r[i]] = x[i];
            }
        }
        __syncwarp();
    }
    const float* l = M.S + lane + q0 * LD;
    f32x2 ll[R];
#pragma unroll 3
    for (int k = 0; k + 1 < K; k++) {
#pragma unroll
        for (int t = 0; t < R; t++) ll[t] = f2_dup(l[32 * t]);
        mid_rank1<R>(p, u, ll);
        l += LD;
        u += kMidULd;
    }
#pragma unroll
    for (int t = 0; t < R; t++) ll[t] = f2_dup(dies[t] ? __int_as_float(0x7fffffff) : l[32 * t]);
    mid_rank1<R>(p, u, ll);
    __syncwarp();  // u is read before the next panel's rows overwrite it
}

// Factors block jb's cw columns and publishes it: values to S, posn, rowof, ipiv. Returns the number
// of columns eliminated (cw, or the column of the block at which the pivot is exactly zero).
// Multipliers are quotients by one reciprocal (quotient.cuh).
template <int NBLK, bool PIVOT, int W>
__device__ __forceinline__ int mid_factor(MidBlock<MidSmem<NBLK, W>::R>& p, MidSmem<NBLK, W>& M, float* u, int n,
                                          int jb, int cw, int lane)
{
    constexpr int R = MidSmem<NBLK, W>::R, LD = MidSmem<NBLK, W>::LD;
    const int k0 = jb * kMidNB;
    int pos[R];    // the rows' positions (255: no row)
    bool live[R];  // rows of the panel: alive before it
#pragma unroll
    for (int t = 0; t < R; t++) {
        const int r = lane + 32 * t;
        pos[t] = r >= n ? 255 : (jb == 0 ? r : (int)M.posn[jb - 1][r]);
        live[t] = r < n && pos[t] >= k0;
    }
    int done = cw;
#pragma unroll
    for (int c = 0; c < kMidNB; c++) {
        if (c >= cw) break;
        const int k = k0 + c;
        float a[R];
#pragma unroll
        for (int t = 0; t < R; t++) a[t] = f2_get(p[t][c / 2], c & 1);
        // first maximum of |a| over the live rows (dead ones are NaN): magnitude, then the lowest
        // position; nothing above zero (zeros, NaN): the row at position k
        int ppos = k;
        bool usual = false;  // the quotients' range, warp-uniform
        float y = 0.0f;
        if (PIVOT) {
            float best = fabsf(a[0]);
#pragma unroll
            for (int t = 1; t < R; t++) best = fmaxf(best, fabsf(a[t]));
            const float mx = warp_absmax(best);
            y = qt_reciprocal(mx);
            usual = qt_usual(mx);
            unsigned cand = 0xffffffffu;
#pragma unroll
            for (int t = 0; t < R; t++)
                if (fabsf(a[t]) == mx) cand = min(cand, (unsigned)pos[t]);
            const unsigned first = __reduce_min_sync(0xffffffffu, cand);
            ppos = mx > 0.0f ? (int)first : k;
            if (lane == 0) M.ipiv[k] = ppos;
        }
        bool hit[R];
#pragma unroll
        for (int t = 0; t < R; t++) {
            hit[t] = pos[t] == ppos;
            if (hit[t]) mid_put_row<R>(p, t, u + c * kMidULd);
        }
        __syncwarp();
        f32x2 uu[kMidNB / 2];
#pragma unroll
        for (int q = c / 4; q < kMidNB / 4; q++) {
            const ulonglong2 v = reinterpret_cast<const ulonglong2*>(u + c * kMidULd)[q];
            uu[2 * q] = v.x;
            uu[2 * q + 1] = v.y;
        }
        const float pv = f2_get(uu[c / 2], c & 1);
        if (!usual && pv == 0.0f) {  // warp-uniform: stop before the interchange
            done = c;
            break;
        }
        float l[R];
        if (!PIVOT) {
            usual = qt_usual(pv);
            y = qt_reciprocal(pv);
        }
        qt_quotients<PIVOT, R>(a, pv, copysignf(y, pv), usual, l);
#pragma unroll
        for (int t = 0; t < R; t++) {
            if (pos[t] == k) pos[t] = ppos;
            if (hit[t]) pos[t] = k;
            const float v = hit[t] ? __int_as_float(0x7fffffff) : -l[t];
            float x, z;
            f2_unpack(p[t][c / 2], x, z);
            if (c & 1)
                p[t][c / 2] = f2_pack(x, l[t]);
            else
                p[t][c / 2] = f2_pack(l[t], fmaf(f2_get(uu[c / 2], 1), v, z));
            const f32x2 nl = f2_dup(v);
#pragma unroll
            for (int h = c / 2 + 1; h < kMidNB / 2; h++) p[t][h] = f2_fma(uu[h], nl, p[t][h]);
        }
    }
    // the block back to S: live rows from the registers, the panel's pivot rows from their buffer;
    // after a stop the rows that are left keep the positions they have
    const int known = done < cw ? n : k0 + done;
#pragma unroll
    for (int t = 0; t < R; t++) {
        if (live[t] && pos[t] >= k0 + done) mid_put_columns<R, LD>(p, t, M.S + lane + 32 * t + k0 * LD);
        M.posn[jb][lane + 32 * t] = (unsigned char)pos[t];
        if (live[t] && pos[t] < known) M.rowof[pos[t]] = lane + 32 * t;
    }
    __syncwarp();
    if (lane < kMidNB) {
        float* s = M.S + (k0 + lane) * LD;
#pragma unroll
        for (int i = 0; i < kMidNB; i++)
            if (i < done) s[M.rowof[k0 + i]] = u[i * kMidULd + lane];
    }
    return done;
}

// The hand-over barrier of panel b among the W warps of a team. W ids serve all panels: panel b + W
// cannot be published before the warps of panels b + 1 .. b + W - 1, all of b's waiters, have passed
// b's. BASE > 0: ids BASE .. BASE + W - 1 as constants (a barrier named by a register claims all
// sixteen of the CTA, which limits the CTAs of an SM); BASE 0: from the register `base`, for the
// kernel that has one CTA an SM. The arriving side goes on at once.
template <int W, int BASE, bool WAIT>
__device__ __forceinline__ void mid_barrier(int base, int b, int threads)
{
#define OPSBLAS_MID_BAR(OPERAND, VALUE)                                                                             \
    if (WAIT)                                                                                                       \
        asm volatile("bar.sync %0, %1;" ::OPERAND(VALUE), "r"(threads) : "memory");                                 \
    else                                                                                                            \
        asm volatile("bar.arrive %0, %1;" ::OPERAND(VALUE), "r"(threads) : "memory");
    const int i = b & (W - 1);
    if (BASE == 0) {
        OPSBLAS_MID_BAR("r", base + i)
    } else if (i == 0) {
        OPSBLAS_MID_BAR("n", BASE)
    } else if (i == 1) {
        OPSBLAS_MID_BAR("n", BASE + 1)
    } else if (i == 2) {
        OPSBLAS_MID_BAR("n", BASE + 2)
    } else {
        OPSBLAS_MID_BAR("n", BASE + 3)
    }
#undef OPSBLAS_MID_BAR
}

// Factors the matrix in M.S with W warps (1, 2 or 4), block jb by warp jb % W. A panel's warp arrives at
// its barrier, the others with a block after it wait there the first time they need the panel. S and
// M.stop = n must be visible to the team before the call; the caller synchronises it after.
template <int NBLK, bool PIVOT, int W, int BASE>
__device__ __forceinline__ void mid_getrf(MidSmem<NBLK, W>& M, int n, int warp, int lane, int base)
{
    constexpr int R = MidSmem<NBLK, W>::R;
    float* u = M.u[W == 1 ? 0 : warp];
    MidBlock<R> p;
    int seen = 0;  // panels below this one are known to this warp
    for (int jb = W == 1 ? 0 : warp; jb < NBLK; jb += W) {
        const int k0 = jb * kMidNB;
        mid_load<NBLK, W>(p, M, n, k0, lane);
        int stop = n;
        for (int b = 0; b < jb; b++) {
            if (W > 1 && b >= seen) {
                // the warps with a block after b: W, or as many as blocks are left
                if (b % W != warp) mid_barrier<W, BASE, true>(base, b, 32 * (min(W - 1, NBLK - 1 - b) + 1));
                seen = b + 1;
            }
            if (stop < n) continue;
            stop = *reinterpret_cast<volatile int*>(&M.stop);
            const int K = min(kMidNB, stop - b * kMidNB);
            if (K > 0) mid_apply<NBLK, W>(p, M, u, b, K, k0, lane);
            if (stop >= (b + 1) * kMidNB) stop = n;  // a later panel's stop is not this panel's matter
        }
        if (stop == n) {
            const int cw = min(kMidNB, n - k0);
            const int done = mid_factor<NBLK, PIVOT, W>(p, M, u, n, jb, cw, lane);
            if (done < cw && lane == 0) *reinterpret_cast<volatile int*>(&M.stop) = k0 + done;
        } else {  // a block after a stop: rows that are still alive back to S
#pragma unroll
            for (int t = 0; t < R; t++) {
                const int r = lane + 32 * t;
                if (r < n && (int)M.posn[stop / kMidNB][r] >= stop)
                    mid_put_columns<R, MidSmem<NBLK, W>::LD>(p, t, M.S + r + k0 * MidSmem<NBLK, W>::LD);
            }
        }
        __syncwarp();
        if (W > 1 && jb + 1 < NBLK) {
            __threadfence_block();
            mid_barrier<W, BASE, false>(base, jb, 32 * (min(W - 1, NBLK - 1 - jb) + 1));
        }
    }
}

// A (n x n, leading dimension lda) into S by cp.async, W warps, and valid entries in rowof; the caller
// waits (cp_async_wait_all) and synchronises.
template <int NBLK, int W>
__device__ __forceinline__ void mid_stage(MidSmem<NBLK, W>& M, const float* A, int lda, int n, int warp, int lane)
{
    constexpr int LD = MidSmem<NBLK, W>::LD;
    for (int i = warp * 32 + lane; i < kMidNB * NBLK; i += 32 * W) M.rowof[i] = i;
    if ((lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0) {
        // lanes in groups of G, a group a column at a time, a 16-byte copy a lane
        constexpr int G = NBLK <= 4 ? 16 : 32;
        const int q = lane & (G - 1), rows = n - 4 * q;
        for (int j = warp * (32 / G) + lane / G; j < n; j += W * (32 / G)) {
            const float* a = A + 4 * q + (long long)j * lda;
            float* s = M.S + 4 * q + j * LD;
            if (rows >= 4)
                cp_async16(s, a);
            else
                for (int e = 0; e < rows; e++) cp_async4(s + e, a + e);
        }
    } else {
        for (int j = warp; j < n; j += W)
            for (int i = lane; i < n; i += 32) cp_async4(M.S + i + j * LD, A + i + (long long)j * lda);
    }
}

// The factors to A, pivots to pm (nullptr: none): row i of the result is physical row rowof[i].
template <int NBLK, int W>
__device__ __forceinline__ void mid_store(const MidSmem<NBLK, W>& M, float* A, int lda, int n, int* pm, int warp,
                                          int lane)
{
    constexpr int R = MidSmem<NBLK, W>::R, LD = MidSmem<NBLK, W>::LD;
    int r[R];
#pragma unroll
    for (int t = 0; t < R; t++) r[t] = lane + 32 * t < n ? M.rowof[lane + 32 * t] : 0;
    const float* s = M.S + warp * LD;
    float* a = A + lane + (long long)warp * lda;
    const bool last = lane + 32 * (R - 1) < n;
#pragma unroll 4
    for (int j = warp; j < n; j += W) {
#pragma unroll
        for (int t = 0; t < R; t++)
            if (t + 1 < R || last) a[32 * t] = s[r[t]];
        s += W * LD;
        a += (long long)W * lda;
    }
    if (pm != nullptr) {
        const int stop = M.stop;  // entries past a stop are 0
        for (int i = warp * 32 + lane; i < n; i += 32 * W) pm[i] = i <= stop ? M.ipiv[i] + 1 : 0;
    }
}

// C right-hand sides solved by one warp from the factors in M.S, in the reference getrs's order (trans N):
// y[c][t] enters as b[rowof[lane + 32 t]] and leaves as x[lane + 32 t]. A step is a chain of a broadcast, an
// fma and in the U sweep a division: four columns at a time hide it (us, orders 80, 8 columns, 100 instances
// in one grouped launch: 158 with one at a time, 107).
template <int NBLK, int W, int C>
__device__ __forceinline__ void mid_solve(const MidSmem<NBLK, W>& M, int n, int lane,
                                          float (&y)[C][MidSmem<NBLK, W>::R])
{
    constexpr int R = MidSmem<NBLK, W>::R, LD = MidSmem<NBLK, W>::LD;
    const float* s[R];
#pragma unroll
    for (int t = 0; t < R; t++) s[t] = M.S + (lane + 32 * t < n ? M.rowof[lane + 32 * t] : 0);
#pragma unroll
    for (int q = 0; q < R; q++) {
#pragma unroll 4
        for (int l = 0; l < 32; l++) {
            const int k = 32 * q + l;
            if (k >= n) break;
            float m[R];
#pragma unroll
            for (int t = q; t < R; t++) m[t] = -s[t][k * LD];
#pragma unroll
            for (int c = 0; c < C; c++) {
                const float yk = __shfl_sync(0xffffffffu, y[c][q], l);
                if (lane > l) y[c][q] = fmaf(m[q], yk, y[c][q]);
#pragma unroll
                for (int t = q + 1; t < R; t++) y[c][t] = fmaf(m[t], yk, y[c][t]);
            }
        }
    }
#pragma unroll
    for (int q = R - 1; q >= 0; q--) {
        const int d = min(lane + 32 * q, n - 1);
        const float diag = s[q][d * LD];
#pragma unroll 4
        for (int l = min(31, n - 1 - 32 * q); l >= 0; l--) {
            const int k = 32 * q + l;
            float m[R];
#pragma unroll
            for (int t = 0; t <= q; t++) m[t] = -s[t][k * LD];
#pragma unroll
            for (int c = 0; c < C; c++) {
                const float xk = __shfl_sync(0xffffffffu, y[c][q] / diag, l);
                y[c][q] = lane == l ? xk : (lane < l ? fmaf(m[q], xk, y[c][q]) : y[c][q]);
#pragma unroll
                for (int t = 0; t < q; t++) y[c][t] = fmaf(m[t], xk, y[c][t]);
            }
        }
    }
}

}  // namespace opsblas
