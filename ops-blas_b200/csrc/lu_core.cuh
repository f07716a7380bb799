// LU building blocks shared by the batched kernels (getrf.cu) and the grouped
// persistent kernel (grouped.cu). Each block restates the reference's unblocked right-looking
// LU (sgetrf_batched_kernel.cpp:106-150): first-maximum pivot, whole-row interchange,
// multipliers by true division, one fmaf per update in column order, stop at the first
// exactly-zero pivot. Whatever kernel runs them, the factors are the same bits.
#pragma once

#include <cuda_runtime.h>

#include "small_common.cuh"

namespace opsblas {

// =============================================================================================
// Register LU for n <= 32: one warp segment per matrix (SEG lanes, 32/SEG matrices per warp).
// Lane r of a segment holds row r of its matrix in registers a4 (float4 chunks, zero padded).
// Pivoting is implicit: rows never move between lanes; `pos` is the row index the lane's row
// has in the reference's in-place matrix at the current step. Per column k:
//   1. argmax of |a[k]| over lanes with pos >= k (redux.sync), ties to the lowest pos --
//      the reference's first-maximum rule; zero and NaN are never chosen;
//   2. the pivot lane publishes its row (from column k on) in shared memory; every lane
//      reads it back with broadcast 16-byte loads;
//   3. lanes below the pivot form l = a[k] / pivot and update a[j] -= l * u[j], j > k.
// =============================================================================================
template <int N>
__device__ __forceinline__ float qget(const float4 (&v)[(N + 3) / 4], int j)
{
    return f4get(v[j >> 2], j & 3);
}

template <int N>
__device__ __forceinline__ void qset(float4 (&v)[(N + 3) / 4], int j, float x)
{
    float4& c = v[j >> 2];
    if ((j & 3) == 0) c.x = x;
    else if ((j & 3) == 1) c.y = x;
    else if ((j & 3) == 2) c.z = x;
    else c.w = x;
}

// a[j] -= l * u[j] on the pairs (x, y) / (z, w) of a float4 chunk, one packed fma per pair;
// fma(u, -l, a) == fma(-l, u, a) exactly.
__device__ __forceinline__ void ffma2_lo(float4& a, float ux, float uy, float2 nl)
{
    const float2 r = __ffma2_rn(make_float2(ux, uy), nl, make_float2(a.x, a.y));
    a.x = r.x;
    a.y = r.y;
}

__device__ __forceinline__ void ffma2_hi(float4& a, float uz, float uw, float2 nl)
{
    const float2 r = __ffma2_rn(make_float2(uz, uw), nl, make_float2(a.z, a.w));
    a.z = r.x;
    a.w = r.y;
}

// Factors the segment's matrix held in a4. rowbuf: this warp's 2 x 32 floats of shared memory
// (16-byte aligned). On return: pos = the lane row's final row index, mypiv = 1-based pivot of
// column r (0 when r >= info), inf = info (uniform within the segment).
template <int N, bool PIVOT, int SEG>
__device__ __forceinline__ void small_getrf_core(float4 (&a4)[(N + 3) / 4], int& pos, int& mypiv, int& inf,
                                                 float* rowbuf, int seg, int r, bool mvalid, bool rvalid)
{
    constexpr int NC = (N + 3) / 4;
    constexpr bool UNIFORM = SEG == 32;  // one matrix per warp: segment state is warp-uniform
    pos = r;
    mypiv = 0;
    inf = 0;
#pragma unroll
    for (int k = 0; k < N; k++) {
        float* buf = rowbuf + (k & 1) * 32 + seg * SEG;
        const bool live = UNIFORM ? rvalid : (rvalid && inf == 0);
        const float ak = qget<N>(a4, k);
        int prow = k;
        bool ispiv;
        if (PIVOT) {
            const bool elig = live && pos >= k;
            const float v = fabsf(ak);
            const unsigned key = (elig && v > 0.0f) ? __float_as_uint(v) : 0u;
            prow = (int)seg_argmax<SEG>(key, elig ? (unsigned)pos : 0xffffffffu, seg);
            ispiv = elig && pos == prow;
        } else {
            ispiv = live && pos == k;
        }
        if (ispiv) {
#pragma unroll
            for (int c = k / 4; c < NC; c++) reinterpret_cast<float4*>(buf)[c] = a4[c];
        }
        __syncwarp();
        const float4 ck = reinterpret_cast<const float4*>(buf)[k / 4];
        const float pv = f4get(ck, k % 4);
        if (UNIFORM) {
            if (PIVOT && r == k) mypiv = prow + 1;
            if (pv == 0.0f) {  // warp-uniform: every lane read the same pivot
                inf = k + 1;
                break;
            }
        } else if (mvalid && inf == 0) {
            if (PIVOT && r == k) mypiv = prow + 1;
            if (pv == 0.0f) inf = k + 1;
        }
        if (UNIFORM ? live : (live && inf == 0)) {
            if (ispiv)
                pos = k;
            else if (pos == k)
                pos = prow;
            if (pos > k) {
                // Multiplier by true division, then a[j] -= l * u[j] for j > k, one fma each.
                const float l = ak / pv;
                qset<N>(a4, k, l);
                const float2 nl = make_float2(-l, -l);
#pragma unroll
                for (int c = k / 4; c < NC; c++) {
                    const float4 u = (c == k / 4) ? ck : reinterpret_cast<const float4*>(buf)[c];
                    // columns 4c..4c+3 that lie right of k
                    if (4 * c > k) {
                        ffma2_lo(a4[c], u.x, u.y, nl);
                    } else if (4 * c + 1 > k) {
                        a4[c].y = fmaf(-l, u.y, a4[c].y);
                    }
                    if (4 * c + 2 > k && 4 * c + 2 < N) {
                        ffma2_hi(a4[c], u.z, u.w, nl);
                    } else if (4 * c + 3 > k && 4 * c + 3 < N) {
                        a4[c].w = fmaf(-l, u.w, a4[c].w);
                    }
                }
            }
        }
    }
}

// Solves one right-hand side with the factors left in registers by small_getrf_core, in the
// reference getrs's order (sgetrs_batched_kernel.cpp:83-200, trans N): b permuted by the row
// interchanges, unit-L forward sweep j = 0..n-1, U backward sweep j = n-1..0 with x_j = y_j /
// U(j,j), one fmaf per update. The lane of original row r enters with y = b[r] (b[r] sits at
// position pos after the interchanges) and leaves with y = x[pos]. owner: this segment's SEG
// ints of shared memory, filled here with the lane of each position. All 32 lanes call this.
template <int N, int SEG>
__device__ __forceinline__ float small_solve_core(const float4 (&a4)[(N + 3) / 4], int pos, bool rvalid, int seg,
                                                  int r, int* owner, float y)
{
    if (rvalid) owner[pos] = r;
    __syncwarp();
    const int base = seg * SEG;
#pragma unroll
    for (int k = 0; k < N; k++) {
        const float yk = __shfl_sync(0xffffffffu, y, base + owner[k]);
        if (rvalid && pos > k) y = fmaf(-qget<N>(a4, k), yk, y);
    }
#pragma unroll
    for (int k = N - 1; k >= 0; k--) {
        const float t = (rvalid && pos == k) ? y / qget<N>(a4, k) : 0.0f;
        const float xk = __shfl_sync(0xffffffffu, t, base + owner[k]);
        if (rvalid) {
            if (pos == k)
                y = xk;
            else if (pos < k)
                y = fmaf(-qget<N>(a4, k), xk, y);
        }
    }
    __syncwarp();
    return y;
}

// Barrier over the team: bar < 0 means the team is the whole CTA; a one-warp team needs only
// the warp barrier.
template <int NT>
__device__ __forceinline__ void team_sync(int bar)
{
    if (NT == 32)
        __syncwarp();
    else if (bar < 0)
        __syncthreads();
    else
        asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "n"(NT) : "memory");
}

}  // namespace opsblas
