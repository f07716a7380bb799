// Triangular sweeps with LU factors for a block of right-hand-side columns held by one warp: rows over
// the lanes (row lane + 32 t, t < R = ceil(n / 32)), CW columns of them in registers. The factors
// arrive panel by panel (16 columns) in shared memory and serve every warp of the CTA.
//
// Per panel the 16 rows of the diagonal block go through shared memory to a lane per column, are
// solved there, and the rows that remain take one fmaf per column of the panel: ascending columns in
// the L sweep, descending in the U sweep, each element in the reference's order
// (sgetrs_batched_kernel.cpp:83-200, getri_batched_kernel.cpp:39-308), so the results are its bits.
#pragma once

#include <cuda_runtime.h>

#include "small_common.cuh"

namespace opsblas {

constexpr int kSvNB = 16;  // panel columns

template <int CW>
constexpr int kSvULd = CW + 4;  // row stride of the panel's solved rows

// p[t][*] -= P(row, k) * u[k][*] for the tiles T0 <= t < T1, k ascending over [klo, khi) or descending
template <int R, int CW, int T0, int T1, bool UP>
__device__ __forceinline__ void sv_gemm(float2 (&p)[R][CW / 2], const float* P, int ldp, const float* u, int klo,
                                        int khi, int lane)
{
#pragma unroll 2
    for (int i = klo; i < khi; i++) {
        const int k = UP ? i : khi - 1 - (i - klo);
        float2 nl[R];
#pragma unroll
        for (int t = T0; t < T1; t++) {
            const float v = -P[lane + 32 * t + k * ldp];
            nl[t] = make_float2(v, v);
        }
        const float4* uk = reinterpret_cast<const float4*>(u + k * kSvULd<CW>);
#pragma unroll
        for (int q = 0; q < CW / 4; q++) {
            const float4 v = uk[q];
#pragma unroll
            for (int t = T0; t < T1; t++) {
                p[t][2 * q] = __ffma2_rn(make_float2(v.x, v.y), nl[t], p[t][2 * q]);
                p[t][2 * q + 1] = __ffma2_rn(make_float2(v.z, v.w), nl[t], p[t][2 * q + 1]);
            }
        }
    }
}

template <int R, int CW, int T>
__device__ __forceinline__ void sv_gemm_below(float2 (&p)[R][CW / 2], const float* P, int ldp, const float* u, int t0,
                                              int lane)
{
    if constexpr (T < R) {
        if (t0 == T)
            sv_gemm<R, CW, T, R, true>(p, P, ldp, u, 0, kSvNB, lane);
        else
            sv_gemm_below<R, CW, T + 1>(p, P, ldp, u, t0, lane);
    }
}

template <int R, int CW, int T>
__device__ __forceinline__ void sv_gemm_above(float2 (&p)[R][CW / 2], const float* P, int ldp, const float* u, int t1,
                                              int klo, int khi, int lane)
{
    if constexpr (T > 0) {
        if (t1 == T)
            sv_gemm<R, CW, 0, T, false>(p, P, ldp, u, klo, khi, lane);
        else
            sv_gemm_above<R, CW, T - 1>(p, P, ldp, u, t1, klo, khi, lane);
    }
}

// Rows k0 .. k0 + 15 of the block to u, or back from it.
template <int R, int CW>
__device__ __forceinline__ void sv_rows_out(const float2 (&p)[R][CW / 2], float* u, int k0, int lane)
{
#pragma unroll
    for (int t = 0; t < R; t++) {
        const int i = lane + 32 * t - k0;
        if ((unsigned)i < 16u) {
            float4* w = reinterpret_cast<float4*>(u + i * kSvULd<CW>);
#pragma unroll
            for (int q = 0; q < CW / 4; q++)
                w[q] = make_float4(p[t][2 * q].x, p[t][2 * q].y, p[t][2 * q + 1].x, p[t][2 * q + 1].y);
        }
    }
    __syncwarp();
}

template <int R, int CW>
__device__ __forceinline__ void sv_rows_in(float2 (&p)[R][CW / 2], const float* u, int k0, int lane)
{
#pragma unroll
    for (int t = 0; t < R; t++) {
        const int i = lane + 32 * t - k0;
        if ((unsigned)i < 16u) {
            const float4* w = reinterpret_cast<const float4*>(u + i * kSvULd<CW>);
#pragma unroll
            for (int q = 0; q < CW / 4; q++) {
                const float4 v = w[q];
                p[t][2 * q] = make_float2(v.x, v.y);
                p[t][2 * q + 1] = make_float2(v.z, v.w);
            }
        }
    }
    __syncwarp();
}

// One panel of the unit-L sweep: P holds columns k0.. (row i at P[i + c * ldp], rows from k0 on).
template <int R, int CW>
__device__ __forceinline__ void sv_forward(float2 (&p)[R][CW / 2], const float* P, int ldp, float* u, int k0, int n,
                                           int lane)
{
    sv_rows_out<R, CW>(p, u, k0, lane);
    const int kw = min(kSvNB, n - k0);
    if (lane < CW) {
        float x[kSvNB];
#pragma unroll
        for (int i = 0; i < kSvNB; i++) x[i] = u[i * kSvULd<CW> + lane];
#pragma unroll
        for (int c = 0; c + 1 < kSvNB; c++) {
            if (c + 1 >= kw) break;
            const float4* l = reinterpret_cast<const float4*>(P + k0 + c * ldp);
#pragma unroll
            for (int q = (c + 1) / 4; q < kSvNB / 4; q++) {
                const float4 v = l[q];
                const float lv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (4 * q + e > c) x[4 * q + e] = fmaf(-lv[e], x[c], x[4 * q + e]);
            }
        }
#pragma unroll
        for (int i = 0; i < kSvNB; i++) u[i * kSvULd<CW> + lane] = x[i];
    }
    __syncwarp();
    if (kw == kSvNB) {  // rows below: the panel's own tile only when rows of it are below
        sv_gemm_below<R, CW, 0>(p, P, ldp, u, (k0 + kSvNB) >> 5, lane);
        __syncwarp();
    }
    sv_rows_in<R, CW>(p, u, k0, lane);  // also over what the update did to the panel's own rows
}

// One panel of the U sweep over its columns above `stop` (-1: all of them), descending.
template <int R, int CW>
__device__ __forceinline__ void sv_backward(float2 (&p)[R][CW / 2], const float* P, int ldp, float* u, int k0, int n,
                                            int stop, int lane)
{
    sv_rows_out<R, CW>(p, u, k0, lane);
    const int kw = min(kSvNB, n - k0), klo = max(0, stop + 1 - k0);
    if (lane < CW) {
        float x[kSvNB];
#pragma unroll
        for (int i = 0; i < kSvNB; i++) x[i] = u[i * kSvULd<CW> + lane];
#pragma unroll
        for (int j = kSvNB - 1; j >= 0; j--) {
            if (j >= kw || j < klo) continue;
            const float4* c = reinterpret_cast<const float4*>(P + k0 + j * ldp);
            const float4 d = c[j / 4];
            x[j] = x[j] / f4get(d, j % 4);
#pragma unroll
            for (int q = 0; q <= j / 4; q++) {
                const float4 v = q == j / 4 ? d : c[q];
                const float uv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (4 * q + e < j) x[4 * q + e] = fmaf(-uv[e], x[j], x[4 * q + e]);
            }
        }
#pragma unroll
        for (int i = 0; i < kSvNB; i++) u[i * kSvULd<CW> + lane] = x[i];
    }
    __syncwarp();
    sv_gemm_above<R, CW, R>(p, P, ldp, u, (k0 + 31) >> 5, klo, kw, lane);
    __syncwarp();
    sv_rows_in<R, CW>(p, u, k0, lane);
}

// Rows [r0, r1) of columns k0 .. k0 + 15 (those inside the matrix) into P by cp.async, one commit group.
__device__ __forceinline__ void sv_stage(float* P, int ldp, const float* A, int lda, int n, int k0, int r0, int r1,
                                         bool vec, int tid, int threads)
{
    const int kw = min(kSvNB, n - k0);
    // sixteen threads a column: r0 is a multiple of 16, so 16-byte copies start aligned
    for (int c = tid >> 4; c < kw; c += threads >> 4) {
        const float* a = A + (long long)(k0 + c) * lda;
        float* s = P + c * ldp;
        int i = r0 + (tid & 15) * 4;
        if (vec) {
            for (; i + 3 < r1; i += 64) cp_async16(s + i, a + i);
            for (; i < r1; i++) cp_async4(s + i, a + i);
        } else {
            for (; i < r1; i += 64)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (i + e < r1) cp_async4(s + i + e, a + i + e);
        }
    }
    cp_async_commit();
}

}  // namespace opsblas
