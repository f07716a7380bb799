// A column of M rows in one lane's registers as packed row pairs (2h, 2h + 1), for the QR kernels whose
// lanes own columns. Sums run in row order with every product rounded before it is added; products and
// updates take two rows an instruction.
#pragma once

#include <cuda_runtime.h>

#include "f32x2.cuh"

namespace opsblas {

template <int M>
using QrCol = f32x2[(M + 1) / 2];

// s + sum over rows r >= R0 of v_r x_r, in row order
template <int M, int R0>
__device__ __forceinline__ float qc_dot(float s, const QrCol<M>& v, const QrCol<M>& x)
{
    if (R0 < M && (R0 & 1)) s = __fadd_rn(s, __fmul_rn(f2_get(v[R0 / 2], 1), f2_get(x[R0 / 2], 1)));
#pragma unroll
    for (int h = (R0 + 1) / 2; 2 * h + 1 < M; h++) {
        float a, b;
        f2_unpack(f2_mul(v[h], x[h]), a, b);
        s = __fadd_rn(__fadd_rn(s, a), b);
    }
    if ((M & 1) && M - 1 >= R0) s = __fadd_rn(s, __fmul_rn(f2_get(v[M / 2], 0), f2_get(x[M / 2], 0)));
    return s;
}

// x_r -= c v_r for rows r >= R0, product and difference each rounded. The difference is an fma by -1 (exact, so
// one rounding), which leaves no sum of a product to be joined: the ptxas of CUDA 12.9 makes one fma of a
// packed product and the packed sum that it feeds, in spite of their .rn. Packed pairs of both against
// differences one by one: 24 x 17 x 30000 109 us, 119.
template <int M, int R0>
__device__ __forceinline__ void qc_axmy(QrCol<M>& x, const QrCol<M>& v, float c)
{
    if (R0 < M && (R0 & 1)) {
        float a, b;
        f2_unpack(x[R0 / 2], a, b);
        x[R0 / 2] = f2_pack(a, __fsub_rn(b, __fmul_rn(c, f2_get(v[R0 / 2], 1))));
    }
    const f32x2 cc = f2_dup(c), minus = f2_dup(-1.0f);
#pragma unroll
    for (int h = (R0 + 1) / 2; 2 * h < M; h++) x[h] = f2_fma(f2_mul(cc, v[h]), minus, x[h]);
}

template <int M>
__device__ __forceinline__ float qc_get(const QrCol<M>& x, int r)
{
    return f2_get(x[r / 2], r & 1);
}

template <int M>
__device__ __forceinline__ void qc_set(QrCol<M>& x, int r, float f)
{
    float a, b;
    f2_unpack(x[r / 2], a, b);
    x[r / 2] = (r & 1) ? f2_pack(a, f) : f2_pack(f, b);
}

// Rows from R0's 16-byte chunk on to / from a 16-byte aligned buffer indexed by row (a multiple of 4
// rows long); on reading, rows below R0 of that chunk come along.
template <int M, int R0>
__device__ __forceinline__ void qc_put(float* buf, const QrCol<M>& x)
{
#pragma unroll
    for (int c = R0 / 4; c < (M + 3) / 4; c++)
        reinterpret_cast<ulonglong2*>(buf)[c] =
            make_ulonglong2(x[2 * c], 2 * c + 1 < (M + 1) / 2 ? x[2 * c + 1 < (M + 1) / 2 ? 2 * c + 1 : 0] : 0ull);
}

template <int M, int R0>
__device__ __forceinline__ void qc_take(QrCol<M>& x, const float* buf)
{
#pragma unroll
    for (int c = R0 / 4; c < (M + 3) / 4; c++) {
        const ulonglong2 f = reinterpret_cast<const ulonglong2*>(buf)[c];
        x[2 * c] = f.x;
        if (2 * c + 1 < (M + 1) / 2) x[2 * c + 1 < (M + 1) / 2 ? 2 * c + 1 : 0] = f.y;
    }
}

// M consecutive floats of global memory; vec: 16-byte aligned. A lane reads its own column, so every
// instruction touches 32 lines: four rows at a time instead of one is a quarter of the L1 time.
template <int M>
__device__ __forceinline__ void qc_load(QrCol<M>& x, const float* p, bool vec)
{
    constexpr int F = M / 4;  // whole chunks
    if (vec) {
#pragma unroll
        for (int c = 0; c < F; c++) {
            const ulonglong2 f = reinterpret_cast<const ulonglong2*>(p)[c];
            x[2 * c] = f.x;
            x[2 * c + 1] = f.y;
        }
    } else {
#pragma unroll
        for (int h = 0; h < 2 * F; h++) x[h] = f2_pack(p[2 * h], p[2 * h + 1]);
    }
#pragma unroll
    for (int h = 2 * F; h < (M + 1) / 2; h++) x[h] = f2_pack(p[2 * h], 2 * h + 1 < M ? p[2 * h + 1] : 0.0f);
}

template <int M>
__device__ __forceinline__ void qc_store(const QrCol<M>& x, float* p, bool vec)
{
    constexpr int F = M / 4;
    if (vec) {
#pragma unroll
        for (int c = 0; c < F; c++) reinterpret_cast<ulonglong2*>(p)[c] = make_ulonglong2(x[2 * c], x[2 * c + 1]);
    }
#pragma unroll
    for (int r = 0; r < M; r++)
        if (r >= 4 * F || !vec) p[r] = qc_get<M>(x, r);
}

}  // namespace opsblas
