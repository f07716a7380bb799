// aclblasSgetrsBatched for 32 < n <= 128, all transpositions: LU staged whole in shared memory, one thread
// per right-hand side (sgetrs_batched_kernel.cpp:83-388 runs a thread per right-hand side too).
//
// A CTA holds as many matrices as give a warp 32 right-hand sides, or as fit a third of an SM's shared
// memory; LU crosses HBM once, in 16-byte asynchronous copies. Lane = right-hand side in each of the
// CTA's four warps; x stays in shared memory (stride odd in 16-byte units: conflict-free) and the warps
// share out its blocks of eight rows: a solved block's columns update the blocks that remain (L and
// U^T ascending, U descending). The L^T sweep chains every element to the next in the reference's order
// and is one thread's. With one or two right-hand sides of trans N a warp takes one, rows over lanes.
// Bound by latency at the 12 matrices (n = 64) to 3 (n = 128) that an SM's shared memory holds. B200,
// CUDA events, us, before (a thread per right-hand side reading LU through L1, or a CTA of 256 threads
// for one matrix) -> now: N, n = 64, 8 columns x 65536: 1670 -> 905; n = 100, 1 x 4096: 365 -> 127;
// n = 128, 16 x 4096: 1610 -> 422, 100 x 600: 498 -> 365; T, n = 64, 8 x 65536: 1551 -> 1200; n = 100,
// 1 x 4096: 847 -> 309.
// Every element takes one fmaf per term in the reference's order and is divided as there, so the
// results are its bits. Rows and columns past n are zero: -0 * 0 added to a sum leaves it as it is.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "f32x2.cuh"
#include "internal.h"
#include "small_common.cuh"

namespace opsblas {

constexpr int kSgMaxN = 128;
constexpr int kSgThreads = 128;
constexpr int kSgRowsMaxRhs = 2;      // trans N: up to here a warp per right-hand side
constexpr int kSgBudget = 75 * 1024;  // bytes a CTA aims at: three an SM

struct SgShape {
    int n8, region, xs, per, cols;  // rows rounded to 8; floats a matrix; floats an x; matrices and columns a CTA
    size_t smem;
    SgShape(int n, int nrhs, int batch)
    {
        n8 = (n + 7) & ~7;
        region = n8 * n8 + 4;  // odd in 16-byte units: the matrices of a warp are read from different banks
        xs = n8 + 4;
        // equal blocks of at most 32 columns, a CTA each: with 128 in one, x takes as much shared memory as
        // LU and an SM holds one CTA (us, n = 128, 128 columns x 300: N 442 -> 205, T 737 -> 328;
        // n = 33, T, 128 x 1: 70 -> 25)
        const int blocks = (nrhs + 31) / 32;
        cols = (nrhs + blocks - 1) / blocks;
        const int bytes = (region + n8 + cols * xs) * 4;
        per = std::max(1, std::min(32 / cols, kSgBudget / bytes));
        per = std::max(1, std::min(per, batch / (3 * sm_count())));  // a small batch spreads over the SMs first
        smem = (size_t)per * bytes;
    }
};

__device__ __forceinline__ void sg_get8(const float* s, float (&v)[8])
{
    const float4 a = reinterpret_cast<const float4*>(s)[0], b = reinterpret_cast<const float4*>(s)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

__device__ __forceinline__ void sg_put8(float* s, const float (&v)[8])
{
    reinterpret_cast<float4*>(s)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(s)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

__device__ __forceinline__ void sg_load_acc(f32x2 (&acc)[4], const float* x)
{
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(x);
    acc[0] = p[0].x, acc[1] = p[0].y, acc[2] = p[1].x, acc[3] = p[1].y;
}

// x[r0 .. r0 + 7] -= M(r0 .. r0 + 7, k) x[k] for the eight columns from k0, ascending or descending
template <bool UP>
__device__ __forceinline__ void sg_update_n(const float* m, int ld, float* x, int r0, int k0)
{
    f32x2 acc[4];
    sg_load_acc(acc, x + r0);
    float xv[8];
    sg_get8(x + k0, xv);
    const float* c = m + r0 + k0 * ld;
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int k = UP ? e : 7 - e;
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(c + k * ld);
        const ulonglong2 a = p[0], b = p[1];
        const f32x2 nx = f2_dup(-xv[k]);
        acc[0] = f2_fma(a.x, nx, acc[0]);
        acc[1] = f2_fma(a.y, nx, acc[1]);
        acc[2] = f2_fma(b.x, nx, acc[2]);
        acc[3] = f2_fma(b.y, nx, acc[3]);
    }
    ulonglong2* p = reinterpret_cast<ulonglong2*>(x + r0);
    p[0] = make_ulonglong2(acc[0], acc[1]);
    p[1] = make_ulonglong2(acc[2], acc[3]);
}

// x[r0 .. r0 + 7] -= U(j, r0 .. r0 + 7) x[j] for the eight rows j from k0, ascending
__device__ __forceinline__ void sg_update_t(const float* m, int ld, float* x, int r0, int k0)
{
    float v[8], xv[8];
    sg_get8(x + r0, v);
    sg_get8(x + k0, xv);
    const float* c = m + k0 + r0 * ld;
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float4 a = *reinterpret_cast<const float4*>(c + 4 * h + i * ld);
            v[i] = fmaf(-a.x, xv[4 * h], v[i]);
            v[i] = fmaf(-a.y, xv[4 * h + 1], v[i]);
            v[i] = fmaf(-a.z, xv[4 * h + 2], v[i]);
            v[i] = fmaf(-a.w, xv[4 * h + 3], v[i]);
        }
    sg_put8(x + r0, v);
}

// The triangle of the block at r0. LOWER: unit L; UPPER: U; UPPER_T: U^T.
enum class SgTri { LOWER, UPPER, UPPER_T };
template <SgTri T>
__device__ __forceinline__ void sg_triangle(const float* m, int ld, float* x, int r0, int n)
{
    float v[8];
    sg_get8(x + r0, v);
    const float* c = m + r0 + r0 * ld;
    if (T == SgTri::LOWER) {
#pragma unroll
        for (int j = 0; j < 7; j++) {
            float l[8];
            sg_get8(c + j * ld, l);
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (i > j) v[i] = fmaf(-l[i], v[j], v[i]);
        }
    } else if (T == SgTri::UPPER) {
#pragma unroll
        for (int j = 7; j >= 0; j--) {
            float u[8];
            sg_get8(c + j * ld, u);
            if (r0 + j < n) {
                v[j] = v[j] / u[j];
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (i < j) v[i] = fmaf(-u[i], v[j], v[i]);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            float u[8];
            sg_get8(c + i * ld, u);
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (j < i) v[i] = fmaf(-u[j], v[j], v[i]);
            if (r0 + i < n) v[i] = v[i] / u[i];
        }
    }
    if (r0 + 8 > n) {  // 0 * inf or NaN may have come into the rows past n
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (r0 + i >= n) v[i] = 0.0f;
    }
    sg_put8(x + r0, v);
}

// One sweep by the CTA's warps: blocks of eight rows dealt out over them (block b: warp b % 4), a
// barrier a block. The block after the current one is brought up to date and solved first, by its
// warp, before that warp's other blocks. work: this thread has a right-hand side.
template <SgTri T>
__device__ __forceinline__ void sg_sweep(const float* m, int ld, float* x, int n, int warp, bool work)
{
    constexpr int WARPS = kSgThreads / 32;
    constexpr bool UP = T != SgTri::UPPER;
    const int nb = ld >> 3;
    auto row = [&](int b) { return UP ? 8 * b : 8 * (nb - 1 - b); };  // step b's block
    if (warp == 0 && work) sg_triangle<T>(m, ld, x, row(0), n);
    __syncthreads();
    for (int b = 0; b + 1 < nb; b++) {
        if (work) {
            int j = b + 1 + ((warp - (b + 1)) & (WARPS - 1));  // this warp's first block after b
            for (; j < nb; j += WARPS) {
                if (T == SgTri::UPPER_T)
                    sg_update_t(m, ld, x, row(j), row(b));
                else
                    sg_update_n<UP>(m, ld, x, row(j), row(b));
                if (j == b + 1) sg_triangle<T>(m, ld, x, row(j), n);
            }
        }
        __syncthreads();
    }
}

// L^T by one thread: x_j -= sum_{i > j} L(i,j) x_i with i ascending from j + 1, each sum a chain that
// starts from the element solved just before.
__device__ __forceinline__ void sg_lower_t(const float* m, int ld, float* x, int n)
{
    for (int r0 = ld - 4; r0 >= 0; r0 -= 4) {
        const float4 x4 = *reinterpret_cast<const float4*>(x + r0);
        float v[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
        for (int j = 3; j >= 0; j--) {
            const float* col = m + (r0 + j) * ld;
            const float4 l4 = *reinterpret_cast<const float4*>(col + r0);
            const float l[4] = {l4.x, l4.y, l4.z, l4.w};
            float s = v[j];
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (i > j) s = fmaf(-l[i], v[i], s);
            const float4* lq = reinterpret_cast<const float4*>(col + r0 + 4);
            const float4* xq = reinterpret_cast<const float4*>(x + r0 + 4);
#pragma unroll 8
            for (int q = (ld - r0) / 4 - 1; q > 0; q--, lq++, xq++) {
                const float4 a = *lq, b = *xq;
                s = fmaf(-a.x, b.x, s);
                s = fmaf(-a.y, b.y, s);
                s = fmaf(-a.z, b.z, s);
                s = fmaf(-a.w, b.w, s);
            }
            v[j] = r0 + j < n ? s : 0.0f;
        }
        *reinterpret_cast<float4*>(x + r0) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// The interchanges k = 0 .. n - 1 (or in reverse) on one vector; pv: 0-based, invalid pivots k itself.
template <bool REVERSE>
__device__ __forceinline__ void sg_interchange(float* x, const int* pv, int n8)
{
    for (int q = 0; q < n8; q += 4) {
        const int k4 = REVERSE ? n8 - 4 - q : q;
        const int4 v = *reinterpret_cast<const int4*>(pv + k4);
        const int p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int u = REVERSE ? 3 - e : e;
            const float a = x[k4 + u], b = x[p[u]];
            x[p[u]] = a;
            x[k4 + u] = b;
        }
    }
}

// One right-hand side solved by a warp, rows over the lanes (few right-hand sides: the chain of a thread
// that has one to itself would be n times as long).
template <int R>
__device__ __forceinline__ void sg_rows_n(const float* m, int ld, float* x, int n, int lane)
{
    float y[R];
#pragma unroll
    for (int t = 0; t < R; t++) y[t] = lane + 32 * t < ld ? x[lane + 32 * t] : 0.0f;
    const float* s = m + lane;
#pragma unroll
    for (int q = 0; q < R; q++) {
        const float* c = s + 32 * q * ld;
        const int steps = min(32, n - 32 * q);
#pragma unroll 8
        for (int l = 0; l < steps; l++, c += ld) {
            const float yk = __shfl_sync(0xffffffffu, y[q], l);
            if (lane > l) y[q] = fmaf(-c[32 * q], yk, y[q]);
#pragma unroll
            for (int t = q + 1; t < R; t++) y[t] = fmaf(-c[32 * t], yk, y[t]);
        }
    }
#pragma unroll
    for (int q = R - 1; q >= 0; q--) {
        const int last = min(31, n - 1 - 32 * q);
        const float diag = m[min(lane + 32 * q, n - 1) * (ld + 1)];
        const float* c = s + (32 * q + last) * ld;
#pragma unroll 8
        for (int l = last; l >= 0; l--, c -= ld) {
            const float xk = __shfl_sync(0xffffffffu, y[q] / diag, l);
            if (lane < l) y[q] = fmaf(-c[32 * q], xk, y[q]);
            if (lane == l) y[q] = xk;
#pragma unroll
            for (int t = 0; t < q; t++) y[t] = fmaf(-c[32 * t], xk, y[t]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < R; t++)
        if (lane + 32 * t < ld) x[lane + 32 * t] = y[t];
}

// MODE 0: trans N, a thread per right-hand side; 1: trans T; 2..4: trans N, a warp per right-hand side
// with MODE rows a lane.
template <int MODE>
__global__ void __launch_bounds__(kSgThreads)
getrs_staged_kernel(const float* const* __restrict__ Aarray, int n, int lda, const int* __restrict__ ipiv,
                    float* const* __restrict__ Barray, int ldb, int nrhs, int batch, int n8, int region, int xs,
                    int per, int cols, int first)
{
    constexpr bool TR = MODE == 1;
    constexpr int WARPS = kSgThreads / 32;
    extern __shared__ __align__(16) float sm[];
    float* xall = sm + per * region;
    int* pv = reinterpret_cast<int*>(xall + per * cols * xs);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long m0 = (long long)blockIdx.x * per;
    const int c0 = first + (int)blockIdx.y * cols, cw = min(cols, nrhs - c0);

    // LU of the CTA's matrices on its way; those without a right-hand side (NULL) are skipped
    bool any = false;
    for (int g = 0; g < per; g++) {
        if (m0 + g >= batch || Barray[m0 + g] == nullptr) continue;
        any = true;
        const float* A = Aarray[m0 + g];
        float* s = sm + g * region;
        if ((lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0) {
            // half a warp a column while that covers it
            const int half = n <= 64 ? 16 : 32, i = 4 * (lane & (half - 1));
            const int step = WARPS * (32 / half);
            int j = warp * (32 / half) + lane / half;
            const float* a = A + i + (long long)j * lda;
            float* d = s + i + j * n8;
            const int rows = n - i;
#pragma unroll 4
            for (; j < n; j += step, a += (long long)step * lda, d += step * n8) {
                if (rows >= 4)
                    cp_async16(d, a);
                else
                    for (int e = 0; e < rows; e++) cp_async4(d + e, a + e);
            }
        } else {
            for (int j = warp; j < n; j += WARPS)
                for (int i = lane; i < n; i += 32) cp_async4(s + i + j * n8, A + i + (long long)j * lda);
        }
        if (n != n8) {
            for (int j = warp; j < n8; j += WARPS)
                if (j >= n)
                    for (int i = lane; i < n8; i += 32) s[i + j * n8] = 0.0f;
                else if (lane < n8 - n)
                    s[n + lane + j * n8] = 0.0f;
        }
    }
    if (!any) return;  // nothing to solve (a refinement's converged matrices), for the whole CTA
    // B behind it; pivots of rows past n and invalid ones swap nothing
    for (int v = warp; v < per * cw; v += WARPS) {
        const int g = v / cw, c = v - g * cw;
        const float* B = m0 + g < batch ? Barray[m0 + g] : nullptr;
        float* x = xall + (g * cols + c) * xs;
        const float* b = B + (long long)(c0 + c) * ldb;
        for (int i = lane; i < n8; i += 32)
            if (B != nullptr && i < n)
                cp_async4(x + i, b + i);
            else
                x[i] = 0.0f;
    }
    for (int e = tid; e < per * n8; e += kSgThreads) {
        const int g = e / n8, k = e - g * n8;
        int q = k;
        if (ipiv != nullptr && k < n && m0 + g < batch) {
            q = ipiv[(m0 + g) * n + k] - 1;
            if ((unsigned)q >= (unsigned)n) q = k;
        }
        pv[e] = q;
    }
    cp_async_wait_all();
    __syncthreads();
    if constexpr (MODE < 2) {
        // lane = right-hand side, in every warp alike
        const int g = lane / cw, c = lane - g * cw;
        const bool work = lane < per * cw && m0 + g < batch && Barray[m0 + g] != nullptr;
        const float* m = sm + (work ? g : 0) * region;
        float* x = xall + (work ? g * cols + c : 0) * xs;
        const int* p = pv + (work ? g : 0) * n8;
        if (TR) {
            sg_sweep<SgTri::UPPER_T>(m, n8, x, n, warp, work);
            if (warp == 0 && work) {
                sg_lower_t(m, n8, x, n);
                sg_interchange<true>(x, p, n8);
            }
        } else {
            if (warp == 0 && work) sg_interchange<false>(x, p, n8);
            sg_sweep<SgTri::LOWER>(m, n8, x, n, warp, work);
            sg_sweep<SgTri::UPPER>(m, n8, x, n, warp, work);
        }
    } else {
        for (int v = warp; v < per * cw; v += WARPS) {
            const int g = v / cw, c = v - g * cw;
            if (m0 + g < batch && Barray[m0 + g] != nullptr) {
                float* x = xall + (g * cols + c) * xs;
                if (lane == 0) sg_interchange<false>(x, pv + g * n8, n8);
                __syncwarp();
                sg_rows_n<MODE>(sm + g * region, n8, x, n, lane);
            }
        }
    }
    __syncthreads();
    for (int v = warp; v < per * cw; v += WARPS) {
        const int g = v / cw, c = v - g * cw;
        float* B = m0 + g < batch ? Barray[m0 + g] : nullptr;
        if (B == nullptr) continue;
        const float* x = xall + (g * cols + c) * xs;
        for (int i = lane; i < n; i += 32) B[i + (long long)(c0 + c) * ldb] = x[i];
    }
}

bool getrs_staged_supported(int n) { return n > 32 && n <= kSgMaxN; }

cudaError_t getrs_staged_launch(cudaStream_t st, bool trans, int n, int nrhs, const float* const* Aarray, int lda,
                                const int* ipiv, float* const* Barray, int ldb, int batch)
{
    const SgShape s(n, nrhs, batch);
    auto kernel = trans ? getrs_staged_kernel<1>
                  : nrhs > kSgRowsMaxRhs ? getrs_staged_kernel<0>
                  : n <= 64 ? getrs_staged_kernel<2>
                  : n <= 96 ? getrs_staged_kernel<3>
                            : getrs_staged_kernel<4>;
    const cudaError_t e = ensure_smem_limit(kernel, 200 * 1024);
    if (e != cudaSuccess) return e;
    // one launch for as many column blocks as a grid's second dimension takes
    for (long long first = 0; first < nrhs; first += (long long)kMaxGridY * s.cols) {
        const long long blocks = std::min<long long>((nrhs - first + s.cols - 1) / s.cols, kMaxGridY);
        const dim3 grid((unsigned)((batch + (long long)s.per - 1) / s.per), (unsigned)blocks);
        kernel<<<grid, kSgThreads, s.smem, st>>>(Aarray, n, lda, ipiv, Barray, ldb, nrhs, batch, s.n8, s.region, s.xs,
                                                 s.per, s.cols, (int)first);
    }
    return cudaGetLastError();
}

}  // namespace opsblas
