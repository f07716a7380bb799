// aclblasSgetrfBatched for 32 < n <= 128: the blocked shared-memory LU of lu_mid.cuh, one matrix a CTA.
//
// Bound by the serial chain of the columns (pivot search, row broadcast, division): a warp issues one
// instruction in about five cycles, and shared memory limits the matrices of an SM (18 at n = 48, 11 at
// 64, 3 at 128). The former kernel kept the matrix in the registers of 2 to 8 warps with a CTA barrier
// a column. B200, CUDA events, us, before -> now: n = 64 x 65536 2460 -> 1620, n = 100 x 4096 1180 -> 452,
// n = 128 x 2048 743 -> 365.
#include <cuda_runtime.h>

#include "internal.h"
#include "lu_mid.cuh"

namespace opsblas {

// CTAs of an SM that the shared memory allows, at most 16 warps: the registers follow from it.
template <int NBLK, int W>
constexpr int kMidPerSm = 232448 / ((int)sizeof(MidSmem<NBLK, W>) + 1024) < 16 / W
                              ? 232448 / ((int)sizeof(MidSmem<NBLK, W>) + 1024)
                              : 16 / W;

template <int NBLK, bool PIVOT, int W>
__global__ void __launch_bounds__(W * 32, (kMidPerSm<NBLK, W>))
getrf_mid_kernel(float* const* __restrict__ Aarray, int n, int lda, int* __restrict__ piv, int* __restrict__ info)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    auto& M = *reinterpret_cast<MidSmem<NBLK, W>*>(dyn);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long m = blockIdx.x;
    float* A = Aarray[m];
    mid_stage<NBLK, W>(M, A, lda, n, warp, lane);
    if (threadIdx.x == 0) M.stop = n;
    cp_async_wait_all();
    __syncthreads();
    mid_getrf<NBLK, PIVOT, W, 1>(M, n, warp, lane, 1);
    __syncthreads();
    mid_store<NBLK, W>(M, A, lda, n, PIVOT ? piv + m * n : nullptr, warp, lane);
    if (threadIdx.x == 0 && info != nullptr) info[m] = M.stop < n ? M.stop + 1 : 0;
}

bool getrf_mid_supported(int n) { return n > 32 && n <= kMidMaxN; }

template <int NBLK, bool PIVOT, int W>
static cudaError_t launch_mid(cudaStream_t st, float* const* Aarray, int n, int lda, int* piv, int* info, int batch)
{
    constexpr int smem = (int)sizeof(MidSmem<NBLK, W>);
    const cudaError_t e = ensure_smem_limit(getrf_mid_kernel<NBLK, PIVOT, W>, smem);
    if (e != cudaSuccess) return e;
    getrf_mid_kernel<NBLK, PIVOT, W><<<(unsigned)batch, W * 32, smem, st>>>(Aarray, n, lda, piv, info);
    return cudaGetLastError();
}

template <int NBLK, int W>
static cudaError_t launch_mid(cudaStream_t st, float* const* Aarray, int n, int lda, int* piv, int* info, int batch)
{
    return piv != nullptr ? launch_mid<NBLK, true, W>(st, Aarray, n, lda, piv, info, batch)
                          : launch_mid<NBLK, false, W>(st, Aarray, n, lda, piv, info, batch);
}

// Warps per matrix: one below 65 rows (eleven matrices an SM already), two up to 112, four above, where
// the shared memory holds three matrices an SM (us for 16384 / 8192 / 4096 / 4096 matrices of n = 64 /
// 96 / 112 / 128 with 1, 2, 4 warps, measured alike: 428, 451, 698 / 858, 680, 740 / 717, 586, 651 /
// 1161, 967, 807).
cudaError_t getrf_mid_launch(cudaStream_t st, float* const* Aarray, int n, int lda, int* piv, int* info, int batch)
{
    switch (mid_blocks(n)) {
        case 3: return launch_mid<3, 1>(st, Aarray, n, lda, piv, info, batch);
        case 4: return launch_mid<4, 1>(st, Aarray, n, lda, piv, info, batch);
        case 5: return launch_mid<5, 2>(st, Aarray, n, lda, piv, info, batch);
        case 6: return launch_mid<6, 2>(st, Aarray, n, lda, piv, info, batch);
        case 7: return launch_mid<7, 2>(st, Aarray, n, lda, piv, info, batch);
        case 8: return launch_mid<8, 4>(st, Aarray, n, lda, piv, info, batch);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace opsblas
