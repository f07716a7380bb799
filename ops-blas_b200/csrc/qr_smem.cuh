// Householder reflectors of one matrix held row by row in shared memory, columns over the lanes of the
// CTA's warps (column c at lane c % 32 of its 64-column warp, two a lane). Shared by geqrf and gels for
// shapes beyond their register kernels. Every sum runs down one column in row order with each product
// rounded before it is added, as the register kernels and the oracle have it; a column's sum of squares
// for the next reflector is formed while the column is updated.
#pragma once

#include <cuda_runtime.h>

#include "small_common.cuh"

namespace opsblas {

constexpr int kQsMaxCols = 256;  // four warps
constexpr int kQsMaxBytes = 200 * 1024;

__host__ __device__ inline int qs_ld(int cols) { return cols | 1; }  // odd: a column's rows hit every bank
__host__ __device__ inline int qs_warps(int cols) { return (cols + 63) / 64; }
__host__ __device__ inline size_t qs_bytes(int m, int cols)
{
    return ((size_t)m * qs_ld(cols) + ((m + 7) & ~7) + 8) * 4;
}
inline bool qs_supported(int m, int cols) { return cols <= kQsMaxCols && qs_bytes(m, cols) <= kQsMaxBytes; }

struct QsSmem {
    float* a;  // a[r * ld + c]
    float* v;  // the reflector's rows (16-byte aligned, index r)
    float* s;  // sum of squares below the diagonal of the next column; spare
    int ld;
    __device__ __forceinline__ QsSmem(float* base, int m, int cols)
    {
        v = base;
        s = v + ((m + 7) & ~7);
        a = s + 8;
        ld = qs_ld(cols);
    }
};

__device__ __forceinline__ void qs_sync(int warps)
{
    if (warps == 1)
        __syncwarp();
    else
        __syncthreads();
}

// f(r, c) for every element of m rows and n columns, column after column over the CTA's threads, so that a
// warp is full on any number of rows and a thread's elements do not wait for each other (a warp a column,
// each load waiting for its store, left few columns on their way and few lanes at work: us, geqrf
// 33 x 33 x 148 64 -> 45, 64 x 48 x 4096 377 -> 297, 1 x 64 x 148 23 -> 6).
template <class F>
__device__ __forceinline__ void qs_columns(int m, int n, int threads, int tid, F f)
{
    const int dr = threads % m, dc = threads / m;
    int r = tid % m, c = tid / m;
#pragma unroll 4
    for (int e = tid; e < m * n; e += threads) {
        f(r, c);
        r += dr;
        c += dc;
        if (r >= m) {
            r -= m;
            c++;
        }
    }
}

// Applies the reflector (v rows i+1 .., t) to this lane's columns c0 and c0 + 32 (those in (i, cols)) and
// returns their sums of squares below row i + 1. GELS: w = v . a + a(i), a(i) -= t w, a += (-t w) v;
// else: dot = a(i) + v . a, coef = t dot, a -= coef v, a(i) -= coef.
template <bool GELS>
__device__ __forceinline__ void qs_apply(const QsSmem& M, int m, int i, int cols, int c0, float t, float (&ss)[2])
{
    const int ld = M.ld;
    const bool on[2] = {c0 > i && c0 < cols, c0 + 32 > i && c0 + 32 < cols};
    float* p = M.a + i * ld + c0;
    float head[2], w[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        head[h] = on[h] ? p[32 * h] : 0.0f;
        w[h] = GELS ? 0.0f : head[h];
        ss[h] = 0.0f;
    }
    const float* q = p + ld;
#pragma unroll 8
    for (int r = i + 1; r < m; r++, q += ld) {
        const float vr = M.v[r];
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (on[h]) w[h] = __fadd_rn(w[h], __fmul_rn(vr, q[32 * h]));
    }
    float coef[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (GELS) w[h] = __fadd_rn(w[h], head[h]);
        coef[h] = __fmul_rn(t, w[h]);
        if (on[h]) p[32 * h] = __fsub_rn(head[h], coef[h]);
    }
    float* u = p + ld;
    if (i + 1 < m) {  // row i + 1: the next column's own diagonal, outside its sum
        const float vr = M.v[i + 1];
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (on[h])
                u[32 * h] = GELS ? __fadd_rn(u[32 * h], __fmul_rn(-coef[h], vr)) : __fsub_rn(u[32 * h], __fmul_rn(coef[h], vr));
        u += ld;
    }
#pragma unroll 4
    for (int r = i + 2; r < m; r++, u += ld) {
        const float vr = M.v[r];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (on[h]) {
                const float x = GELS ? __fadd_rn(u[32 * h], __fmul_rn(-coef[h], vr)) : __fsub_rn(u[32 * h], __fmul_rn(coef[h], vr));
                u[32 * h] = x;
                ss[h] = __fadd_rn(ss[h], __fmul_rn(x, x));
            }
        }
    }
}

// The sum of squares of column c below its diagonal, by one thread.
__device__ __forceinline__ float qs_squares(const QsSmem& M, int m, int c)
{
    float ss = 0.0f;
    for (int r = c + 1; r < m; r++) ss = __fadd_rn(ss, __fmul_rn(M.a[r * M.ld + c], M.a[r * M.ld + c]));
    return ss;
}

// Reflectors 0 .. k - 1 over the columns [0, cols). REFLECT(ss, akk, t, head, v): forms a reflector from
// the sum of squares and the diagonal (tau, the new diagonal, and how an element becomes v); returns
// false when it is skipped. TAU(i, t) records tau.
template <bool GELS, class Reflect, class Scale, class Tau>
__device__ __forceinline__ void qs_factor(const QsSmem& M, int m, int k, int cols, int warps, int tid, Reflect reflect,
                                          Scale scale, Tau put_tau)
{
    const int c0 = (tid >> 5) * 64 + (tid & 31), threads = warps * 32;
    if (c0 == 0) M.s[0] = qs_squares(M, m, 0);
    qs_sync(warps);
    for (int i = 0; i < k; i++) {
        // every thread forms the same reflector
        float t, head, sc;
        const float akk = M.a[i * M.ld + i];
        const bool used = reflect(M.s[i & 1], akk, t, head, sc);
        if (tid == 0) put_tau(i, used ? t : 0.0f);
        if (used) {
            for (int r = i + 1 + tid; r < m; r += threads) {
                const float x = scale(M.a[r * M.ld + i], sc);
                M.v[r] = x;
                M.a[r * M.ld + i] = x;
            }
            qs_sync(warps);
            if (tid == 0) M.a[i * M.ld + i] = head;
            float ss[2];
            qs_apply<GELS>(M, m, i, cols, c0, t, ss);
            if (c0 == i + 1) M.s[(i + 1) & 1] = ss[0];
            if (c0 + 32 == i + 1) M.s[(i + 1) & 1] = ss[1];
        } else if (c0 == i + 1 || c0 + 32 == i + 1) {
            M.s[(i + 1) & 1] = i + 1 < k ? qs_squares(M, m, i + 1) : 0.0f;
        }
        qs_sync(warps);
    }
}

}  // namespace opsblas
