// aclblasSgetrsBatched, trans N, 128 < n <= 256: every warp holds CW right-hand sides of one matrix in
// registers, rows over the lanes, and the CTA's warps share the factors' panels of 16 columns, staged two
// deep by cp.async (lu_solve.cuh). B is gathered through the interchanges once and written back once;
// LU crosses HBM once. Bit-identical to the reference's order (sgetrs_batched_kernel.cpp:83-200).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "internal.h"
#include "lu_solve.cuh"
#include "small_common.cuh"

namespace opsblas {

constexpr int kGbMaxWarps = 4;

template <int R, int CW>
__global__ void __launch_bounds__(kGbMaxWarps * 32, CW > 8 ? (R > 6 ? 2 : 3) : 4)
getrs_block_kernel(const float* const* __restrict__ Aarray, int n, int lda, const int* __restrict__ ipiv,
                   float* const* __restrict__ Barray, int ldb, int nrhs, int first)
{
    constexpr int LDP = 32 * R + 4;
    extern __shared__ __align__(16) float sm[];
    float* panel[2] = {sm, sm + kSvNB * LDP};
    const int tid = threadIdx.x, threads = blockDim.x, warp = tid >> 5, lane = tid & 31;
    float* u = sm + 2 * kSvNB * LDP + warp * kSvNB * kSvULd<CW>;
    int* src = reinterpret_cast<int*>(sm + 2 * kSvNB * LDP + (threads >> 5) * kSvNB * kSvULd<CW>);
    int* pv = src + 32 * R;
    const long long m = blockIdx.x;
    float* B = Barray[m];
    if (B == nullptr) return;  // a NULL right-hand side skips the matrix
    const float* A = Aarray[m];
    const bool vec = (reinterpret_cast<uintptr_t>(A) & 15) == 0 && (lda & 3) == 0;
    const int nb = (n + kSvNB - 1) / kSvNB;
    sv_stage(panel[0], LDP, A, lda, n, 0, 0, n, vec, tid, threads);
    for (int i = tid; i < n; i += threads) {
        pv[i] = ipiv ? ipiv[m * n + i] - 1 : i;
        src[i] = i;
    }
    __syncthreads();
    if (tid == 0) {  // src[i]: the row that the interchanges bring to position i (invalid pivots skipped)
#pragma unroll 4
        for (int k = 0; k < n; k++) {
            const int q = pv[k];
            if ((unsigned)q < (unsigned)n) {
                const int a = src[k];
                src[k] = src[q];
                src[q] = a;
            }
        }
    }
    __syncthreads();
    const long long c0l = first + ((long long)blockIdx.y * (threads >> 5) + warp) * CW;
    const bool work = c0l < nrhs;
    const int c0 = work ? (int)c0l : nrhs;  // this warp's right-hand sides
    float2 p[R][CW / 2];
    int row[R];
#pragma unroll
    for (int t = 0; t < R; t++) row[t] = lane + 32 * t < n ? src[lane + 32 * t] : -1;
    // columns past nrhs repeat the last one: zeros would send their lanes, and so the warp, through the
    // division's special case in every row (with that and registers spilled, n = 160, 8 columns x 1500: 301 us, 169)
#pragma unroll
    for (int c = 0; c < CW; c += 2) {
        const float* b0 = B + (long long)min(c0 + c, nrhs - 1) * ldb;
        const float* b1 = B + (long long)min(c0 + c + 1, nrhs - 1) * ldb;
#pragma unroll
        for (int t = 0; t < R; t++)
            p[t][c / 2] = make_float2(row[t] >= 0 ? b0[row[t]] : 0.0f, row[t] >= 0 ? b1[row[t]] : 0.0f);
    }
    int buf = 0;
    for (int b = 0; b < nb; b++, buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();
        if (b + 1 < nb)
            sv_stage(panel[buf ^ 1], LDP, A, lda, n, (b + 1) * kSvNB, (b + 1) * kSvNB, n, vec, tid, threads);
        else
            sv_stage(panel[buf ^ 1], LDP, A, lda, n, b * kSvNB, 0, n, vec, tid, threads);
        if (work) sv_forward<R, CW>(p, panel[buf], LDP, u, b * kSvNB, n, lane);
    }
    for (int b = nb - 1; b >= 0; b--, buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();
        const int k0 = b * kSvNB;
        if (b > 0) sv_stage(panel[buf ^ 1], LDP, A, lda, n, k0 - kSvNB, 0, k0, vec, tid, threads);
        if (work) sv_backward<R, CW>(p, panel[buf], LDP, u, k0, n, -1, lane);
    }
#pragma unroll
    for (int c = 0; c < CW; c++) {
        if (c0 + c < nrhs) {
            float* col = B + (long long)(c0 + c) * ldb;
#pragma unroll
            for (int t = 0; t < R; t++)
                if (lane + 32 * t < n) col[lane + 32 * t] = (c & 1) ? p[t][c / 2].y : p[t][c / 2].x;
        }
    }
}

// A warp per 16 right-hand sides needs enough of them to hide its latency. Up to 16 columns are one pass of
// the CTA of 256 threads for one matrix (getrs_blk.cu), three of which an SM holds: that is faster until a
// second wave of them (us, there and here: n = 160, 8 columns x 300 59, 82, x 500 96, 82; n = 256,
// 16 x 444 121, 133, x 500 190, 135). More columns are passes in turn there: here from two warps an SM on
// (n = 129, 17 x 148 80, 59; n = 256, 40 x 148 207, 145).
bool getrs_block_preferred(int n, int nrhs, int batch)
{
    if (n <= 128 || n > 256) return false;
    return nrhs <= 16 ? batch > 3 * sm_count() : (long long)batch * ((nrhs + 15) / 16) >= 2 * sm_count();
}

template <int R, int CW>
static cudaError_t launch_block(cudaStream_t st, int n, int nrhs, const float* const* Aarray, int lda, const int* ipiv,
                                float* const* Barray, int ldb, int batch)
{
    const int blocks = (int)((nrhs + (long long)CW - 1) / CW);
    const int parts = (blocks + kGbMaxWarps - 1) / kGbMaxWarps, warps = (blocks + parts - 1) / parts;
    const size_t smem = (size_t)(2 * kSvNB * (32 * R + 4) + warps * kSvNB * kSvULd<CW> + 2 * 32 * R) * 4;
    const cudaError_t e = ensure_smem_limit(getrs_block_kernel<R, CW>, 64 * 1024);
    if (e != cudaSuccess) return e;
    // one launch for as many CTAs a matrix as a grid's second dimension takes
    for (int p0 = 0; p0 < parts; p0 += kMaxGridY) {
        const dim3 grid((unsigned)batch, (unsigned)std::min(parts - p0, kMaxGridY));
        getrs_block_kernel<R, CW><<<grid, warps * 32, smem, st>>>(Aarray, n, lda, ipiv, Barray, ldb, nrhs,
                                                                  p0 * warps * CW);
    }
    return cudaGetLastError();
}

template <int R>
static cudaError_t launch_block(cudaStream_t st, int n, int nrhs, const float* const* Aarray, int lda, const int* ipiv,
                                float* const* Barray, int ldb, int batch)
{
    return nrhs <= 4 ? launch_block<R, 4>(st, n, nrhs, Aarray, lda, ipiv, Barray, ldb, batch)
                     : launch_block<R, 16>(st, n, nrhs, Aarray, lda, ipiv, Barray, ldb, batch);
}

cudaError_t getrs_block_launch(cudaStream_t st, int n, int nrhs, const float* const* Aarray, int lda, const int* ipiv,
                               float* const* Barray, int ldb, int batch)
{
    return n <= 192 ? launch_block<6>(st, n, nrhs, Aarray, lda, ipiv, Barray, ldb, batch)
                    : launch_block<8>(st, n, nrhs, Aarray, lda, ipiv, Barray, ldb, batch);
}

}  // namespace opsblas
