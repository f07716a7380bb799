// aclblasSgeqrfBatched: batched Householder QR, FP32, column-major, LAPACK storage (R in the
// upper triangle, the Householder vectors below the diagonal with an implicit unit head, tau).
//
// Replaces blas/geqrf_batched/arch35/sgeqrf_batched_host.cpp:19-141 (host) and
// sgeqrf_batched_kernel.cpp:44-190 (device) of the reference. Its arithmetic, per column i:
// sigma = sum_{r>i} A(r,i)^2; sigma == 0 gives tau = 0 and no update; otherwise
// alpha = -sign(x1) sqrt(sigma + x1^2), tau = (alpha - x1) / alpha, v = A(i+1:, i) / (x1 - alpha),
// A(i,i) = alpha, and every column c > i gets dot = A(i,c) + v . A(i+1:, c), coef = tau * dot,
// A(i+1:, c) -= coef v, A(i,c) -= coef. The reference sums by thread trees; these kernels sum in
// row order with every product rounded before it is added (no contraction), the order of the
// CPU oracle they match bit for bit. Parity with the reference is its own test rule:
// MIXED_TOLERANCE against LAPACK sgeqrf_.
//   m, n <= 32 : geqrf_col_kernel<M>, one warp per matrix, lane c = column c in registers (every
//                sum local, in row order), the reflector published through shared memory with
//                its divisions one row per lane, the column update in packed f32x2 operations;
//   1 < n <= 256, m > 1 and the matrix in shared memory: geqrf_smem_kernel, a warp per 64 columns;
//   otherwise  : geqrf_generic_kernel, one CTA per matrix in global memory (correctness path):
//                thread 0 forms the reflector, thread t updates columns i+1+t, i+1+t+256, ...
#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

#include "internal.h"
#include "qr_col.cuh"
#include "qr_smem.cuh"
#include "small_common.cuh"

namespace opsblas {

constexpr int kQrWarps = 8;

// Reflector I of the warp's matrix. Lane c holds column c; every sum runs locally in row order, so the
// arithmetic is the row-order restatement's. The reflector's divisions are shared out one row per lane
// through the warp's shared-memory column buffer. Packed pairs and 16-byte column loads: 32 x 32 x 65536
// 971 -> 545 us, 24 x 17 x 32768 174 -> 125 us.
template <int M, int I>
__device__ __forceinline__ void qr_col_step(QrCol<M>& col, float& mytau, float* vb, int lane, int n)
{
    // sigma = sum_{r>I} A(r,I)^2 (every lane forms it for its own column; lane I's is used)
    const float sigma = __shfl_sync(0xffffffffu, qc_dot<M, I + 1>(0.0f, col, col), I);
    const float x1 = __shfl_sync(0xffffffffu, qc_get<M>(col, I), I);
    float t, alpha;
    if (sigma == 0.0f) {
        t = 0.0f;
        alpha = x1;
    } else {
        const float normx = sqrtf(__fadd_rn(sigma, __fmul_rn(x1, x1)));
        alpha = x1 >= 0.0f ? -normx : normx;
        t = __fdiv_rn(__fsub_rn(alpha, x1), alpha);
    }
    if (lane == I) mytau = t;
    if (t == 0.0f) return;  // uniform: A(I,I) stays x1 == alpha, no update
    const float vscale = __fsub_rn(x1, alpha);
    // v_r = A(r,I) / vscale for r > I: lane I publishes its column, lane r divides row r
    if (lane == I) qc_put<M, I + 1>(vb, col);
    __syncwarp();
    if (lane > I && lane < M) vb[lane] = __fdiv_rn(vb[lane], vscale);
    __syncwarp();
    QrCol<M> v;
    qc_take<M, I + 1>(v, vb);
    if (lane == I) {
        const float above = I & 1 ? qc_get<M>(col, I - 1 > 0 ? I - 1 : 0) : 0.0f;  // shares I's pair
#pragma unroll
        for (int h = (I + 2) / 2; h < (M + 1) / 2; h++) col[h] = v[h];
        col[I / 2] = I & 1 ? f2_pack(above, alpha)
                           : f2_pack(alpha, I + 1 < M ? qc_get<M>(v, I + 1 < M ? I + 1 : 0) : 0.0f);
    } else if (lane > I && lane < n) {
        // dot = A(I,c) + sum_{r>I} v_r A(r,c) in row order, then A(r,c) -= coef v_r, A(I,c) -= coef
        const float head = qc_get<M>(col, I);
        const float coef = __fmul_rn(t, qc_dot<M, I + 1>(head, v, col));
        qc_axmy<M, I + 1>(col, v, coef);
        qc_set<M>(col, I, __fsub_rn(head, coef));
    }
    __syncwarp();  // the buffer is read before the next reflector writes it
}

// Reflectors 0 .. min(m, n) - 1, one instantiation per row index.
template <int M, int... I>
__device__ __forceinline__ void qr_col_all(QrCol<M>& col, float& mytau, float* vb, int lane, int n,
                                           std::integer_sequence<int, I...>)
{
    ((I < n ? qr_col_step<M, I>(col, mytau, vb, lane, n) : void()), ...);
}

template <int M>
__global__ void __launch_bounds__(kQrWarps * 32)
geqrf_col_kernel(float* const* __restrict__ Aarray, int n, int lda, float* const* __restrict__ TauArray, int batch)
{
    __shared__ __align__(16) float vbuf[kQrWarps][32];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const long long b = (long long)blockIdx.x * kQrWarps + warp;
    if (b >= batch) return;  // warp-uniform
    float* A = Aarray[b];
    float* tau = TauArray[b];
    const bool cv = lane < n;
    const bool vec = (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    QrCol<M> col;
    float* Ac = A + (long long)lane * lda;
    if (cv) {
        qc_load<M>(col, Ac, vec);
    } else {
#pragma unroll
        for (int h = 0; h < (M + 1) / 2; h++) col[h] = 0ull;
    }
    float mytau = 0.0f;
    qr_col_all<M>(col, mytau, vbuf[warp], lane, n, std::make_integer_sequence<int, M>{});
    if (cv) qc_store<M>(col, Ac, vec);
    if (lane < M && lane < n) tau[lane] = mytau;
}

// Larger shapes that fit shared memory: one matrix a CTA, a warp per 64 columns (qr_smem.cuh). Bound by
// instruction issue and the row-order sums. us, the generic kernel's thread-0 reflector over global memory
// -> this: 64 x 48 x 4096 3542 -> 297, 33 x 33 x 148 55 -> 45, 33 x 33 x 4096 365 -> 103.
__global__ void __launch_bounds__(128)
geqrf_smem_kernel(float* const* __restrict__ Aarray, int m, int n, int lda, float* const* __restrict__ TauArray)
{
    extern __shared__ __align__(16) float dyn[];
    const int tid = threadIdx.x, warps = blockDim.x >> 5;
    const QsSmem M(dyn, m, n);
    float* A = Aarray[blockIdx.x];
    float* tau = TauArray[blockIdx.x];
    qs_columns(m, n, warps * 32, tid, [&](int r, int c) { cp_async4(M.a + r * M.ld + c, A + r + (long long)c * lda); });
    cp_async_wait_all();
    qs_sync(warps);
    qs_factor<false>(
        M, m, m < n ? m : n, n, warps, tid,
        [](float sigma, float x1, float& t, float& alpha, float& sc) {
            if (sigma == 0.0f) return false;
            const float normx = sqrtf(__fadd_rn(sigma, __fmul_rn(x1, x1)));
            alpha = x1 >= 0.0f ? -normx : normx;
            t = __fdiv_rn(__fsub_rn(alpha, x1), alpha);
            sc = __fsub_rn(x1, alpha);
            return t != 0.0f;
        },
        [](float x, float sc) { return __fdiv_rn(x, sc); }, [&](int i, float t) { tau[i] = t; });
    qs_columns(m, n, warps * 32, tid, [&](int r, int c) { A[r + (long long)c * lda] = M.a[r * M.ld + c]; });
}

constexpr int kQrThreads = 256;

__global__ void __launch_bounds__(kQrThreads)
geqrf_generic_kernel(float* const* __restrict__ Aarray, int m, int n, int lda, float* const* __restrict__ TauArray)
{
    __shared__ float s_par[3];  // tau, alpha, x1 - alpha
    float* A = Aarray[blockIdx.x];
    float* tau = TauArray[blockIdx.x];
    const int tid = threadIdx.x;
    const int k = m < n ? m : n;
    for (int i = 0; i < k; i++) {
        float* ci = A + (long long)i * lda;
        if (tid == 0) {
            float sigma = 0.0f;
            for (int r = i + 1; r < m; r++) sigma = __fadd_rn(sigma, __fmul_rn(ci[r], ci[r]));
            const float x1 = ci[i];
            float t, alpha;
            if (sigma == 0.0f) {
                t = 0.0f;
                alpha = x1;
            } else {
                const float normx = sqrtf(__fadd_rn(sigma, __fmul_rn(x1, x1)));
                alpha = x1 >= 0.0f ? -normx : normx;
                t = __fdiv_rn(__fsub_rn(alpha, x1), alpha);
            }
            tau[i] = t;
            s_par[0] = t;
            s_par[1] = alpha;
            s_par[2] = __fsub_rn(x1, alpha);
        }
        __syncthreads();
        const float t = s_par[0], alpha = s_par[1], vscale = s_par[2];
        if (t != 0.0f) {
            for (int r = i + 1 + tid; r < m; r += kQrThreads) ci[r] = __fdiv_rn(ci[r], vscale);
            __syncthreads();
            for (int c = i + 1 + tid; c < n; c += kQrThreads) {
                float* cc = A + (long long)c * lda;
                float dot = cc[i];
                for (int r = i + 1; r < m; r++) dot = __fadd_rn(dot, __fmul_rn(ci[r], cc[r]));
                const float coef = __fmul_rn(t, dot);
                for (int r = i + 1; r < m; r++) cc[r] = __fsub_rn(cc[r], __fmul_rn(coef, ci[r]));
                cc[i] = __fsub_rn(cc[i], coef);
            }
            if (tid == 0) ci[i] = alpha;
        }
        __syncthreads();  // s_par and column i+1 ready for the next step
    }
}

}  // namespace opsblas

using namespace opsblas;

extern "C" aclblasStatus_t aclblasSgeqrfBatched(aclblasHandle_t handle, int m, int n, float* const Aarray[], int lda,
                                                float* const TauArray[], int* info, int batchSize)
{
    static const char* kApi = "aclblasSgeqrfBatched";
    if (handle == nullptr) {
        log_error(kApi, "handle is nullptr");
        return ACLBLAS_STATUS_HANDLE_IS_NULLPTR;
    }
    if (info == nullptr) {
        log_error(kApi, "info must not be nullptr");
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    // ValidateGeqrfBatchedParams (sgeqrf_batched_host.cpp:21-58): LAPACK-style -position in the
    // host info, counting m=1, n=2, Aarray=3, lda=4, TauArray=5, batchSize=6.
    if (m < 0) {
        log_error(kApi, "m must be >= 0, got %d", m);
        *info = ACLBLAS_LAPACK_INFO_ARG_1;
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (n < 0) {
        log_error(kApi, "n must be >= 0, got %d", n);
        *info = ACLBLAS_LAPACK_INFO_ARG_2;
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (lda < max1(m)) {
        log_error(kApi, "lda must be >= max(1, m), got lda=%d, m=%d", lda, m);
        *info = ACLBLAS_LAPACK_INFO_ARG_4;
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (batchSize < 0) {
        log_error(kApi, "batchSize must be >= 0, got %d", batchSize);
        *info = ACLBLAS_LAPACK_INFO_ARG_6;
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (batchSize > 0 && Aarray == nullptr) {
        log_error(kApi, "Aarray must not be nullptr when batchSize > 0");
        *info = ACLBLAS_LAPACK_INFO_ARG_3;
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (batchSize > 0 && m > 0 && n > 0 && TauArray == nullptr) {
        log_error(kApi, "TauArray must not be nullptr when batchSize > 0 and min(m,n) > 0");
        *info = ACLBLAS_LAPACK_INFO_ARG_5;
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (m == 0 || n == 0 || batchSize == 0) {
        *info = ACLBLAS_LAPACK_INFO_OK;
        return ACLBLAS_STATUS_SUCCESS;
    }

    cudaStream_t st = handle->stream;
    if (m <= 32 && n <= 32) {
        const unsigned grid = (unsigned)((batchSize + kQrWarps - 1) / kQrWarps);
        switch (m) {
#define OPSBLAS_GEQRF_CASE(MM)                                                                                      \
    case MM:                                                                                                        \
        geqrf_col_kernel<MM><<<grid, kQrWarps * 32, 0, st>>>(Aarray, n, lda, TauArray, batchSize);                  \
        break;
            OPSBLAS_FOR_N_1_32(OPSBLAS_GEQRF_CASE)
#undef OPSBLAS_GEQRF_CASE
            default:
                break;
        }
    } else if (m > 1 && n > 1 && qs_supported(m, n)) {
        // one reflector is not worth the way through shared memory (us, generic and this: 33 x 1 x 148 6 and 8,
        // 100 x 1 x 8000 31 and 37; 33 x 2 x 8000 47 and 27)
        const cudaError_t e = ensure_smem_limit(geqrf_smem_kernel, kQsMaxBytes);
        if (e != cudaSuccess) return launch_status(kApi, e);
        geqrf_smem_kernel<<<(unsigned)batchSize, qs_warps(n) * 32, qs_bytes(m, n), st>>>(Aarray, m, n, lda, TauArray);
    } else {
        geqrf_generic_kernel<<<(unsigned)batchSize, kQrThreads, 0, st>>>(Aarray, m, n, lda, TauArray);
    }
    const aclblasStatus_t status = launch_status(kApi, cudaGetLastError());
    if (status == ACLBLAS_STATUS_SUCCESS) *info = ACLBLAS_LAPACK_INFO_OK;
    return status;
}
