// Blocked batched LU on the matrix stored by rows, panels of 32 columns, two variants:
//   * plain FP32 getrf for 128 < n <= 1024 (aclblasSgetrfBatched, getrf_rows_launch): the
//     reference's arithmetic -- first-maximum pivot on exact magnitudes, true division, stop at
//     the first exactly-zero pivot -- and a tiled CUDA-core trailing update that applies the
//     rank-1 updates one fmaf at a time in the reference's order: bit-identical to it;
//   * mixed precision for 256 < n <= 1024 (aclblasSgetrfsRefineBatchedEx with
//     ACLBLAS_COMPUTE_32F_FAST_TF32, once the matrix no longer fits one SM's tensor memory:
//     getrf_tmem.cu covers n <= 256; getrf_blocked_tc_launch): the trailing update on the tcgen05
//     tensor cores in split TF32.
// Both work on the matrix stored by rows (T(i, j) at LU[j + i * ldlu]): a row is contiguous, so
// pivot rows, interchanges and the panel's rows are whole cache lines, where by columns every row
// element is a separate sector. The steps below describe the mixed variant. The plain one has the same
// panel, except that a stop keeps the reference's semantics and no TF32 planes are written
// (lu_panel_kernel's EXACT), and runs lu_rows_update_kernel as its update.
//   0. lu_rows_in_kernel: A (by columns) into LU by rows, 32 x 32 tiles through shared memory.
//   Per panel k0 = 0, 32, ...:
//   1. lu_panel_kernel, one CTA per matrix, two panel rows a thread:
//      * factors the panel (rows k0..n-1, columns k0..k0+31) in FP32 in registers, in two halves of
//        16 columns, with implicit pivoting (`pos` tracks the reference's in-place order): the
//        reference's first maximum of the exact magnitudes, correctly rounded multipliers, one CTA
//        barrier per column; 1-based pivots in LAPACK's sequential-swap convention;
//      * writes the factored panel at the final positions and moves the rest of every row whose
//        position changed (at most 64 rows: the whole-row interchanges of the reference,
//        SwapRows, applied once per panel);
//      * L21 (rows below the diagonal block, K-contiguous) and U12 = L11^-1 * (the pivot rows'
//        trailing entries) into scratch as TF32 high and low planes; U12 also into its final rows;
//   2. gemm_tc_lu_update: T22 -= L21 * U12 on the tensor cores (split TF32, three products, FP32
//      accumulation), as the column-major product U12^T * L21^T on the by-rows storage;
//   and lu_rows_out_kernel transposes LU in place back to columns. On an exactly-zero pivot the
//   matrix stops (info = column + 1); its later updates change nothing.
#include <cuda_runtime.h>

#include "f32x2.cuh"
#include "internal.h"
#include "lu_mid.cuh"
#include "quotient.cuh"
#include "small_common.cuh"
#include "tc_common.cuh"

namespace opsblas {

constexpr int kBpW = 32;  // panel width = the update's K

constexpr int kBpH = 16;  // columns factored at a time: half a panel, so that its unrolled code is run twice

template <int NW>
struct __align__(16) BpSmem {
    union {
        float crow[kBpH][NW][kBpH];  // per column and warp: the warp's pivot candidate row
        float l11[kBpW][kBpW];       // after the factorisation: L11 negated
    };
    uint2 slot[2][NW];           // per column parity and warp: its best magnitude (bits) and position
    int win[kBpH];               // the warp whose candidate became column c's pivot row
    float u[kBpH][kBpH + 4];     // the first half's pivot rows, second half
    int mv_src[2 * kBpW];     // rows whose position changed: memory row and destination row
    int mv_dst[2 * kBpW];
    int mv_cnt;
};

// Scratch per matrix (byte offsets): L21 (n - 32 rows x 32, row-major) as its TF32 high plane
// followed by its low plane; U12 (32 x (n - 32), column-major: n - 32 "rows" of 32) the same way.
// A plane is (n - 32) x 32 floats, so each low plane starts n - 32 rows after its high plane.
struct BpScratch {
    long long plane, l21, u12, per_matrix;
    explicit BpScratch(int n)
    {
        plane = (long long)(n - kBpW) * kBpW * 4;
        l21 = 0;
        u12 = (2 * plane + 255) / 256 * 256;
        per_matrix = u12 + (2 * plane + 255) / 256 * 256;
    }
};

// 16-byte cp.async that reads src_bytes (0 or 16) and zero-fills the rest.
__device__ __forceinline__ void cp_async16_zf(uint32_t saddr, const void* gmem, int src_bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(gmem), "r"(src_bytes) : "memory");
}

// hi = x rounded to TF32 (nearest even), lo = (x - hi) rounded to TF32.
__device__ __forceinline__ void tf32_split(float x, float& hi, float& lo)
{
    hi = tf32_rne(x);
    lo = tf32_rne(x - hi);
}

// The transposes move 64 x 64 tiles with 256 threads: each thread has four 16-byte loads (or
// sixteen 4-byte loads when rows are not 16-byte aligned) of a tile in flight, the tile is
// re-read across from shared memory (row stride 65: conflict-free) and written as columns.
constexpr int kTpT = 64;

// tile (r0, c0) of the column-major matrix X (ld) into s[c][r] (r, c < 64, zeros outside n x n)
__device__ __forceinline__ void tp_load(float (*s)[kTpT + 1], const float* X, long long ld, int r0, int c0, int n,
                                        bool vec)
{
    const int tid = threadIdx.x;
    if (vec && r0 + kTpT <= n) {
        constexpr int K = kTpT * kTpT / 4 / 256;
        float4 v[K];  // every load in flight before the first store
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int e = tid + 256 * k, c = e / (kTpT / 4), rq = (e % (kTpT / 4)) * 4;
            v[k] = c0 + c < n ? *reinterpret_cast<const float4*>(X + (r0 + rq) + (long long)(c0 + c) * ld)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int e = tid + 256 * k, c = e / (kTpT / 4), rq = (e % (kTpT / 4)) * 4;
            s[c][rq] = v[k].x;
            s[c][rq + 1] = v[k].y;
            s[c][rq + 2] = v[k].z;
            s[c][rq + 3] = v[k].w;
        }
    } else {
        constexpr int K = kTpT * kTpT / 256;
        float v[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int e = tid + 256 * k, c = e / kTpT, r = e % kTpT;
            v[k] = (r0 + r < n && c0 + c < n) ? X[(r0 + r) + (long long)(c0 + c) * ld] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int e = tid + 256 * k;
            s[e / kTpT][e % kTpT] = v[k];
        }
    }
}

// Y(r0 + r, c0 + c) = s[r][c] (the transpose of the tile s holds), column-major Y (ld)
__device__ __forceinline__ void tp_store(const float (*s)[kTpT + 1], float* Y, long long ld, int r0, int c0, int n,
                                         bool vec)
{
    const int tid = threadIdx.x;
    if (vec && r0 + kTpT <= n) {
#pragma unroll
        for (int k = 0; k < kTpT * kTpT / 4 / 256; k++) {
            const int e = tid + 256 * k, c = e / (kTpT / 4), rq = (e % (kTpT / 4)) * 4;
            if (c0 + c < n)
                *reinterpret_cast<float4*>(Y + (r0 + rq) + (long long)(c0 + c) * ld) =
                    make_float4(s[rq][c], s[rq + 1][c], s[rq + 2][c], s[rq + 3][c]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < kTpT * kTpT / 256; k++) {
            const int e = tid + 256 * k, c = e / kTpT, r = e % kTpT;
            if (r0 + r < n && c0 + c < n) Y[(r0 + r) + (long long)(c0 + c) * ld] = s[r][c];
        }
    }
}

// T(i, j) = A(i, j): A by columns (lda) into LU by rows (ldt), i.e. the storage of T is the
// transpose of A's. One 64 x 64 tile (blockIdx.y) of one matrix (blockIdx.x).
__global__ void __launch_bounds__(256)
lu_rows_in_kernel(const float* const* __restrict__ Aarr, int lda, float* const* __restrict__ Tarr, int ldt, int n)
{
    __shared__ float tile[kTpT][kTpT + 1];
    const int nt = (n + kTpT - 1) / kTpT;
    const int i0 = (int)(blockIdx.y % nt) * kTpT, j0 = (int)(blockIdx.y / nt) * kTpT;
    const float* A = Aarr[blockIdx.x];
    float* T = Tarr[blockIdx.x];
    const bool vec = (reinterpret_cast<uintptr_t>(A) & 15) == 0 && (lda & 3) == 0 &&
                     (reinterpret_cast<uintptr_t>(T) & 15) == 0 && (ldt & 3) == 0;
    tp_load(tile, A, lda, i0, j0, n, vec);  // tile[c][r] = A(i0 + r, j0 + c)
    __syncthreads();
    tp_store(tile, T, ldt, j0, i0, n, vec);  // storage (j0 + r, i0 + c) = tile[r][c] = A(i0 + c, j0 + r)
}

// In-place transpose of the n x n storage matrix S(r, c) = LU[r + c * ld]: the by-rows factors
// become the by-columns LU (and back). One pair of 64 x 64 tiles (I, J), I <= J, per CTA
// (blockIdx.y).
__global__ void __launch_bounds__(256)
lu_rows_out_kernel(float* const* __restrict__ LUarr, int ld, int n)
{
    __shared__ float ta[kTpT][kTpT + 1], tb[kTpT][kTpT + 1];
    const int nt = (n + kTpT - 1) / kTpT;
    int p = (int)blockIdx.y, I = 0;
    while (p >= nt - I) {
        p -= nt - I;
        I++;
    }
    const int J = I + p;
    float* S = LUarr[blockIdx.x];
    const bool vec = (reinterpret_cast<uintptr_t>(S) & 15) == 0 && (ld & 3) == 0;
    const int a0 = I * kTpT, b0 = J * kTpT;
    tp_load(ta, S, ld, a0, b0, n, vec);                 // ta[c][r] = S(a0 + r, b0 + c)
    if (I != J) tp_load(tb, S, ld, b0, a0, n, vec);     // tb[c][r] = S(b0 + r, a0 + c)
    __syncthreads();
    if (I != J) tp_store(tb, S, ld, a0, b0, n, vec);    // S'(a0 + r, b0 + c) = tb[r][c] = S(b0 + c, a0 + r)
    tp_store(ta, S, ld, b0, a0, n, vec);                // S'(b0 + r, a0 + c) = ta[r][c] = S(a0 + c, b0 + r)
}

// Rows moved a round by the panel kernel's interchange step: 64 rows x MVC columns (64 for CTAs of 128 and
// 256 threads, else 32, so that shared memory lets 512 threads of them share an SM).
template <int NT>
struct PanelMv {
    static constexpr int MVC = NT == 128 || NT == 256 ? 64 : 32;  // two buffers of 64 x MVC floats
};

__device__ __forceinline__ void bp_take_row(f32x2 (&p)[kBpH / 2], const float* s)
{
#pragma unroll
    for (int q = 0; q < kBpH / 4; q++) {
        const ulonglong2 v = reinterpret_cast<const ulonglong2*>(s)[q];
        p[2 * q] = v.x;
        p[2 * q + 1] = v.y;
    }
}

// Factors hw columns (k .. of half h) of the panel held in p: one CTA barrier per column. Each warp finds
// its first maximum (two redux), publishes magnitude, position and the row; after the barrier every
// warp takes the best of the warps' (two redux) and reads the pivot row. Returns the columns eliminated.
// Multipliers are correctly rounded quotients by one reciprocal (quotient.cuh), and a row that has become a
// pivot is poisoned with NaN until the half is done (as in lu_mid.cuh: masks cost more than the updates).
template <int NT, int RPT, bool PIVOT>
__device__ __forceinline__ int lu_panel_half(f32x2 (&p)[RPT][kBpH / 2], int (&pos)[RPT], BpSmem<NT / 32>& S, int k,
                                             int hw, int* __restrict__ piv, int tid, int warp, int lane)
{
    constexpr int NW = NT / 32;
    int done = hw;
#pragma unroll
    for (int c = 0; c < kBpH; c++, k++) {
        if (c >= hw) break;
        float a[RPT];
#pragma unroll
        for (int r = 0; r < RPT; r++) a[r] = f2_get(p[r][c / 2], c & 1);
        int ppos = k, bw = 0;
        bool usual = false;
        float y = 0.0f;
        if (PIVOT) {
            float best = fabsf(a[0]);
#pragma unroll
            for (int r = 1; r < RPT; r++) best = fmaxf(best, fabsf(a[r]));
            const float wm = warp_absmax(best);  // (NaN, the dead rows' value, never wins)
            unsigned cand = 0x7fffffffu;
#pragma unroll
            for (int r = 0; r < RPT; r++)
                if (fabsf(a[r]) == wm) cand = min(cand, (unsigned)pos[r]);
            if (!(wm > 0.0f)) {  // nothing above zero: the warp's lowest live position (warp-uniform)
#pragma unroll
                for (int r = 0; r < RPT; r++)
                    if (pos[r] >= k) cand = min(cand, (unsigned)pos[r]);
            }
            const int wp = (int)__reduce_min_sync(0xffffffffu, cand);
            if (lane == 0) S.slot[c & 1][warp] = make_uint2(wm > 0.0f ? __float_as_uint(wm) : 0u, (unsigned)wp);
#pragma unroll
            for (int r = 0; r < RPT; r++)
                if (pos[r] == wp) {
                    ulonglong2* d = reinterpret_cast<ulonglong2*>(S.crow[c][warp]);
#pragma unroll
                    for (int q = 0; q < kBpH / 4; q++) d[q] = make_ulonglong2(p[r][2 * q], p[r][2 * q + 1]);
                }
            __syncthreads();
            const uint2 sl = lane < NW ? S.slot[c & 1][lane] : make_uint2(0u, 0x7fffffffu);
            const unsigned g = __reduce_max_sync(0xffffffffu, sl.x);
            ppos = (int)__reduce_min_sync(0xffffffffu, sl.x == g ? sl.y : 0x7fffffffu);
            bw = __ffs(__ballot_sync(0xffffffffu, sl.y == (unsigned)ppos)) - 1;
            const float mx = __uint_as_float(g);
            y = qt_reciprocal(mx);
            usual = qt_usual(mx);
        } else {  // the row at position k, published by its warp
#pragma unroll
            for (int r = 0; r < RPT; r++)
                if (pos[r] == k) {
                    S.win[c] = warp;
                    ulonglong2* d = reinterpret_cast<ulonglong2*>(S.crow[c][warp]);
#pragma unroll
                    for (int q = 0; q < kBpH / 4; q++) d[q] = make_ulonglong2(p[r][2 * q], p[r][2 * q + 1]);
                }
            __syncthreads();
            bw = S.win[c];
        }
        const float* prow = S.crow[c][bw];
        f32x2 u[kBpH / 2];
#pragma unroll
        for (int q = c / 4; q < kBpH / 4; q++) {
            const ulonglong2 v = reinterpret_cast<const ulonglong2*>(prow)[q];
            u[2 * q] = v.x;
            u[2 * q + 1] = v.y;
        }
        const float pv = f2_get(u[c / 2], c & 1);
        if (tid == 0) {
            if (PIVOT) {
                piv[k] = ppos + 1;
                S.win[c] = bw;
            }
        }
        if (!usual && pv == 0.0f) {  // exactly-zero pivot: stop here, before the interchange (uniform)
            done = c;
            break;
        }
        float l[RPT];
        if (!PIVOT) {
            usual = qt_usual(pv);
            y = qt_reciprocal(pv);
        }
        qt_quotients<PIVOT, RPT>(a, pv, copysignf(y, pv), usual, l);
#pragma unroll
        for (int r = 0; r < RPT; r++) {
            const bool hit = pos[r] == ppos;
            if (pos[r] == k) pos[r] = ppos;
            if (hit) pos[r] = k;
            const float v = hit ? __int_as_float(0x7fffffff) : -l[r];
            float x, z;
            f2_unpack(p[r][c / 2], x, z);
            if (c & 1)
                p[r][c / 2] = f2_pack(x, l[r]);
            else
                p[r][c / 2] = f2_pack(l[r], fmaf(f2_get(u[c / 2], 1), v, z));
            const f32x2 nl = f2_dup(v);
#pragma unroll
            for (int h = c / 2 + 1; h < kBpH / 2; h++) p[r][h] = f2_fma(u[h], nl, p[r][h]);
        }
    }
    // the half's pivot rows, overwritten after they were published
#pragma unroll
    for (int r = 0; r < RPT; r++) {
        const int i = pos[r] - (k - done);
        if (pos[r] >= k - done && pos[r] < k) bp_take_row(p[r], S.crow[i][warp]);
    }
    return done;
}

// One CTA per matrix; thread t holds memory rows k0 + t + r * NT (r < RPT) of the panel. NT x RPT
// covers the panel's rows; 128 registers a thread, so that 512 / NT CTAs share an SM. The panel is
// factored in two halves of 16 columns by the same code (a whole panel's unrolled columns are more code
// than the instruction cache holds: half of the former kernel's time was waiting for instructions).
// The pivot search is the reference's first maximum of the exact magnitudes, the multipliers are
// correctly rounded, every update one fmaf in column order.
// EXACT (the plain FP32 factorisation): after a stop at column kk of the panel only the U rows above kk
// are formed (the trailing update then takes rows from kk on with K = kk - k0); no TF32 planes (the
// update reads L21 and U12 from LU). Otherwise (mixed): TF32 planes, and a stop zeroes the update.
// PIVOT = false: no pivoting (the reference's no-pivot variant). st[m]: the matrix's info code so far
// (0, or the stop column + 1); info, when not nullptr, receives the same.
template <int NT, int RPT, bool EXACT, bool PIVOT>
__global__ void __launch_bounds__(NT, 512 / NT)
lu_panel_kernel(float* const* __restrict__ LUarr, int n, int ldt, int k0, int* __restrict__ piv,
                int* __restrict__ info, int* __restrict__ st, char* __restrict__ scratch, long long l21_off,
                long long u12_off, long long per_matrix)
{
    constexpr int NW = NT / 32;
    __shared__ BpSmem<NW> S;
    constexpr int kMvCols = PanelMv<NT>::MVC;
    __shared__ __align__(16) float mvbuf[2][2 * kBpW * kMvCols];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long m = blockIdx.x;
    float* T = LUarr[m];  // by rows: T(i, j) = T[j + i * ldt]
    int* pm = PIVOT ? piv + m * n : nullptr;
    const int mp = n - k0;                      // panel rows
    const int pw = mp < kBpW ? mp : kBpW;       // panel columns
    const int ntr = n - k0 - kBpW;              // trailing rows and columns
    const long long lo = (long long)(n - kBpW) * kBpW;  // floats from a high plane to its low plane
    float* L21 = EXACT ? nullptr : reinterpret_cast<float*>(scratch + m * per_matrix + l21_off);
    float* U12 = EXACT ? nullptr : reinterpret_cast<float*>(scratch + m * per_matrix + u12_off);
    const int inf0 = st[m];
    // whole rows as float4 when every row start is 16-byte aligned (uniform per matrix)
    const bool vec = (reinterpret_cast<uintptr_t>(T) & 15) == 0 && (ldt & 3) == 0 && pw == kBpW;

    if (tid == 0) S.mv_cnt = 0;
    if (inf0 != 0) {  // stopped at an earlier zero pivot
        if (!EXACT) {  // this step's update must change nothing
            for (int e = tid; e < (ntr > 0 ? ntr : 0) * kBpW; e += NT) {
                L21[e] = 0.0f;
                L21[lo + e] = 0.0f;
                U12[e] = 0.0f;
                U12[lo + e] = 0.0f;
            }
        }
        return;
    }

    // 1. this thread's panel rows (zeros outside the matrix; no position: -1): cur is the half being
    //    factored, oth the other one
    int pos[RPT];
    f32x2 cur[RPT][kBpH / 2], oth[RPT][kBpH / 2];
#pragma unroll
    for (int r = 0; r < RPT; r++) {
        const bool valid = tid + r * NT < mp;
        pos[r] = valid ? k0 + tid + r * NT : -1;
#pragma unroll
        for (int h = 0; h < kBpH / 2; h++) cur[r][h] = oth[r][h] = f2_dup(__int_as_float(0x7fffffff));
        if (valid) {
            const float* row = T + (long long)pos[r] * ldt + k0;
            if (vec) {
#pragma unroll
                for (int q = 0; q < kBpH / 4; q++) {
                    const ulonglong2 v = reinterpret_cast<const ulonglong2*>(row)[q];
                    const ulonglong2 x = reinterpret_cast<const ulonglong2*>(row + kBpH)[q];
                    cur[r][2 * q] = v.x, cur[r][2 * q + 1] = v.y;
                    oth[r][2 * q] = x.x, oth[r][2 * q + 1] = x.y;
                }
            } else {
#pragma unroll
                for (int h = 0; h < kBpH / 2; h++) {
                    const int c = 2 * h, e = kBpH + 2 * h;
                    cur[r][h] = f2_pack(c < pw ? row[c] : 0.0f, c + 1 < pw ? row[c + 1] : 0.0f);
                    oth[r][h] = f2_pack(e < pw ? row[e] : 0.0f, e + 1 < pw ? row[e + 1] : 0.0f);
                }
            }
        }
    }
    __syncthreads();

    // 2. factor, half by half; the second half first takes the first's update
    int done = 0, first = 0;  // first: the columns eliminated in the first half
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        const int hw = max(0, min(kBpH, pw - half * kBpH));
        const int d = lu_panel_half<NT, RPT, PIVOT>(cur, pos, S, k0 + half * kBpH, hw, pm, tid, warp, lane);
        done += d;
        if (half == 1) break;
#pragma unroll
        for (int r = 0; r < RPT; r++)
#pragma unroll
            for (int h = 0; h < kBpH / 2; h++) {
                const f32x2 x = cur[r][h];
                cur[r][h] = oth[r][h];
                oth[r][h] = x;
            }
        // the second half's entries of the first half's pivot rows, solved by a lane per column, then
        // one fmaf per pivot row for the rows below (after a stop: the rows before it only)
        if (pw > kBpH) {
#pragma unroll
            for (int r = 0; r < RPT; r++)
                if (pos[r] >= k0 && pos[r] < k0 + d) {
                    ulonglong2* x = reinterpret_cast<ulonglong2*>(S.u[pos[r] - k0]);
#pragma unroll
                    for (int q = 0; q < kBpH / 4; q++) x[q] = make_ulonglong2(cur[r][2 * q], cur[r][2 * q + 1]);
                }
            __syncthreads();
            if (tid < kBpH) {
                float x[kBpH];
#pragma unroll
                for (int i = 0; i < kBpH; i++) x[i] = i < d ? S.u[i][tid] : 0.0f;
#pragma unroll
                for (int i = 1; i < kBpH; i++) {
                    if (i < d) {
                        const float* l = S.crow[i][S.win[i]];
#pragma unroll
                        for (int c = 0; c < kBpH; c++)
                            if (c < i) x[i] = fmaf(-l[c], x[c], x[i]);
                        S.u[i][tid] = x[i];
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kBpH; i++) {
                if (i < d) {
                    const ulonglong2* ui = reinterpret_cast<const ulonglong2*>(S.u[i]);
                    f32x2 nl[RPT];
#pragma unroll
                    for (int r = 0; r < RPT; r++) nl[r] = f2_dup(-f2_get(oth[r][i / 2], i & 1));
#pragma unroll
                    for (int q = 0; q < kBpH / 4; q++) {
                        const ulonglong2 v = ui[q];
#pragma unroll
                        for (int r = 0; r < RPT; r++) {
                            cur[r][2 * q] = f2_fma(v.x, nl[r], cur[r][2 * q]);
                            cur[r][2 * q + 1] = f2_fma(v.y, nl[r], cur[r][2 * q + 1]);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; r++)
                if (pos[r] < k0 + d) {  // dead (their second half is in S.u), or no row
#pragma unroll
                    for (int h = 0; h < kBpH / 2; h++) cur[r][h] = f2_dup(__int_as_float(0x7fffffff));
                }
        }
        first = d;
        if (d < hw) break;  // stopped in the first half
    }
    // (oth: columns 0..15, cur: 16..31) the second half of the first half's pivot rows
    if (pw > kBpH) {
#pragma unroll
        for (int r = 0; r < RPT; r++)
            if (pos[r] >= k0 && pos[r] < k0 + first) bp_take_row(cur[r], S.u[pos[r] - k0]);
    }
    const bool stopped = done < pw;
    if (stopped && tid == 0) {
        st[m] = k0 + done + 1;
        if (info != nullptr && info != st) info[m] = k0 + done + 1;
    }
    __syncthreads();  // S.crow and S.u are read before l11 is used below; done is uniform

    // 3. the panel at its final rows; L21 (zero after a stop: the update then changes nothing) and
    //    L11; the rows whose position changed
    auto elem = [&](int r, int c) { return f2_get(c < 16 ? oth[r][c % 16 / 2] : cur[r][c % 16 / 2], c & 1); };
#pragma unroll
    for (int r = 0; r < RPT; r++) {
        if (pos[r] < 0) continue;
        float* row = T + (long long)pos[r] * ldt + k0;
        if (vec) {
#pragma unroll
            for (int q = 0; q < kBpH / 4; q++) {
                reinterpret_cast<ulonglong2*>(row)[q] = make_ulonglong2(oth[r][2 * q], oth[r][2 * q + 1]);
                reinterpret_cast<ulonglong2*>(row + kBpH)[q] = make_ulonglong2(cur[r][2 * q], cur[r][2 * q + 1]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < kBpW; c++)
                if (c < pw) row[c] = elem(r, c);
        }
        if (PIVOT && pos[r] != k0 + tid + r * NT) {
            const int q = atomicAdd(&S.mv_cnt, 1);
            S.mv_src[q] = k0 + tid + r * NT;
            S.mv_dst[q] = pos[r];
        }
        if (!EXACT && ntr > 0 && pos[r] >= k0 + kBpW) {
            float4* dh = reinterpret_cast<float4*>(L21 + (long long)(pos[r] - k0 - kBpW) * kBpW);
            float4* dl = reinterpret_cast<float4*>(L21 + lo + (long long)(pos[r] - k0 - kBpW) * kBpW);
#pragma unroll
            for (int q = 0; q < kBpW / 4; q++) {
                float h[4], lw[4];
#pragma unroll
                for (int e = 0; e < 4; e++) tf32_split(stopped ? 0.0f : elem(r, 4 * q + e), h[e], lw[e]);
                dh[q] = make_float4(h[0], h[1], h[2], h[3]);
                dl[q] = make_float4(lw[0], lw[1], lw[2], lw[3]);
            }
        }
        if (pos[r] < k0 + kBpW) {
#pragma unroll
            for (int c = 0; c < kBpW; c++) S.l11[pos[r] - k0][c] = -elem(r, c);
        }
    }
    __syncthreads();

    // 4. the rest of each moved row (columns 0..k0-1 and k0+pw..n-1) to its destination row,
    //    kMvCols columns a round staged in shared memory by cp.async: a round reads all its values
    //    before any is written (the moves form cycles)
    const int cnt = S.mv_cnt;  // <= 64: each of the panel's interchanges moves two rows
    if (cnt > 0) {
        const int nx = n - pw;  // columns outside the panel
        const int rounds = (nx + kMvCols - 1) / kMvCols;
        auto col_of = [&](int x) { return x < k0 ? x : x + pw; };
        // round rd: columns rd * kMvCols .. of every moved row into buffer rd & 1 (one cp.async group)
        auto fetch = [&](int rd) {
            const int x0 = rd * kMvCols;
            float* b = mvbuf[rd & 1];
            for (int e = tid; e < cnt * (kMvCols / 4); e += NT) {
                const int r = e / (kMvCols / 4), xq = x0 + (e % (kMvCols / 4)) * 4;
                float* d = b + r * kMvCols + (xq - x0);
                const float* srow = T + (long long)S.mv_src[r] * ldt;
                if (vec && xq + 3 < nx) {
                    cp_async16(d, srow + col_of(xq));  // four columns on the same side of the panel
                } else {
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (xq + u < nx) cp_async4(d + u, srow + col_of(xq + u));
                }
            }
            cp_async_commit();
        };
        // two rounds in flight: a round's values are all read (into its buffer) before any of them
        // is written; rounds cover disjoint columns
        fetch(0);
        if (rounds > 1) fetch(1);
        for (int rd = 0; rd < rounds; rd++) {
            if (rd + 1 < rounds)
                cp_async_wait_group<1>();
            else
                cp_async_wait_group<0>();
            __syncthreads();
            const int x0 = rd * kMvCols;
            const float* b = mvbuf[rd & 1];
            for (int e = tid; e < cnt * (kMvCols / 4); e += NT) {
                const int r = e / (kMvCols / 4), xq = x0 + (e % (kMvCols / 4)) * 4;
                const float* sv = b + r * kMvCols + (xq - x0);
                float* drow = T + (long long)S.mv_dst[r] * ldt;
                if (vec && xq + 3 < nx) {
                    *reinterpret_cast<float4*>(drow + col_of(xq)) = *reinterpret_cast<const float4*>(sv);
                } else {
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (xq + u < nx) drow[col_of(xq + u)] = sv[u];
                }
            }
            __syncthreads();
            if (rd + 2 < rounds) fetch(rd + 2);
        }
    }
    if (ntr <= 0) return;  // last panel: no trailing block

    // 5. U12 = L11^-1 * (the pivot rows' trailing entries, now in rows k0..k0+31), one thread per
    //    trailing column, in the reference's order (row i takes columns 0..i-1 in turn): the final U
    //    rows (above the stop column only, EXACT) and the TF32 planes of the update (mixed)
    if (stopped) {
        for (int jj = tid; jj < ntr; jj += NT) {
            if (EXACT) {  // rows above the stop, one at a time
                float* t = T + (long long)k0 * ldt + k0 + kBpW + jj;
                for (int i = 1; i < done; i++) {
                    float x = t[(long long)i * ldt];
                    for (int c = 0; c < i; c++) x = fmaf(S.l11[i][c], t[(long long)c * ldt], x);
                    t[(long long)i * ldt] = x;
                }
            } else {
                for (int q = 0; q < kBpW; q++) U12[(long long)jj * kBpW + q] = U12[lo + (long long)jj * kBpW + q] = 0.0f;
            }
        }
        return;
    }
    for (int jj = tid; jj < ntr; jj += NT) {
        float* t = T + (long long)k0 * ldt + k0 + kBpW + jj;
        float u[kBpW];
#pragma unroll
        for (int i = 0; i < kBpW; i++) u[i] = t[(long long)i * ldt];
#pragma unroll
        for (int i = 1; i < kBpW; i++) {
#pragma unroll
            for (int q = 0; q < (i + 3) / 4; q++) {
                const float4 v = reinterpret_cast<const float4*>(S.l11[i])[q];
                const float l[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (4 * q + e < i) u[i] = fmaf(l[e], u[4 * q + e], u[i]);
            }
        }
#pragma unroll
        for (int i = 1; i < kBpW; i++) t[(long long)i * ldt] = u[i];
        if (!EXACT) {
            float4* dh = reinterpret_cast<float4*>(U12 + (long long)jj * kBpW);
            float4* dl = reinterpret_cast<float4*>(U12 + lo + (long long)jj * kBpW);
#pragma unroll
            for (int q = 0; q < kBpW / 4; q++) {
                float h[4], lw[4];
#pragma unroll
                for (int e = 0; e < 4; e++) tf32_split(u[4 * q + e], h[e], lw[e]);
                dh[q] = make_float4(h[0], h[1], h[2], h[3]);
                dl[q] = make_float4(lw[0], lw[1], lw[2], lw[3]);
            }
        }
    }
}

// Trailing update of the plain factorisation, by rows: T(i, j) -= sum_k T(i, k0 + k) T(k0 + k, j)
// for rows i from r0 = k0 + 32 (or the stop column) and columns j from k0 + 32, K = 32 (or the
// columns before the stop), one fmaf at a time in increasing k -- the reference's sequence of
// rank-1 updates, so the result is bit-identical to it. A CTA of 128 threads computes a 64 x 128
// tile, each thread an 8 x 8 block (rows ty + 8 a, columns 8 tx ..): L (row-major, row stride 36
// floats: the eight row values of a step are conflict-free broadcasts) and U arrive in shared
// memory by cp.async while the thread's C block is loaded into registers, so a tile waits for one
// memory round trip; 144 registers, three CTAs an SM. st[m]: the matrix's info code (the update
// is skipped for a matrix stopped earlier). The grid's row tiles cover n - k0 rows (a stop adds up
// to 31 rows to the block).
constexpr int kRuRows = 64, kRuCols = 128, kRuLd = 36;

__global__ void __launch_bounds__(128, 3)
lu_rows_update_kernel(float* const* __restrict__ LUarr, int n, int ldt, int k0, const int* __restrict__ st,
                      int tiles_m, int tiles_n)
{
    __shared__ __align__(16) float Ls[kRuRows][kRuLd];    // Ls[row][k]
    __shared__ __align__(16) float Us[kBpW][kRuCols];     // Us[k][col]
    const int tiles = tiles_m * tiles_n;
    const long long m = blockIdx.x / tiles;
    const int tile = (int)(blockIdx.x % tiles);
    const int code = st[m];
    int r0 = k0 + kBpW, K = kBpW;
    if (code != 0) {
        if (code - 1 < k0) return;  // stopped in an earlier panel: no more updates
        K = code - 1 - k0;          // stopped in this panel at column k0 + K
        r0 = k0 + K;
        if (K == 0) return;
    }
    const int c0 = k0 + kBpW;
    const int rows = n - r0, cols = n - c0;
    const int tr = (tile % tiles_m) * kRuRows, tc = (tile / tiles_m) * kRuCols;
    if (tr >= rows || tc >= cols) return;
    float* T = LUarr[m];
    const bool vec = (reinterpret_cast<uintptr_t>(T) & 15) == 0 && (ldt & 3) == 0;
    const int tid = threadIdx.x;
    // L: rows r0 + tr + i, columns k0 .. k0 + K - 1; U: rows k0 .. k0 + K - 1, columns c0 + tc + j
    if (vec) {
#pragma unroll
        for (int u = 0; u < kRuRows * kBpW / 4 / 128; u++) {
            const int e = tid + 128 * u, i = e / (kBpW / 4), kq = (e % (kBpW / 4)) * 4;
            const bool ok = tr + i < rows && kq < K;
            cp_async16_zf(smem_u32(&Ls[i][kq]), T + (long long)(ok ? r0 + tr + i : r0) * ldt + k0 + kq, ok ? 16 : 0);
        }
#pragma unroll
        for (int u = 0; u < kRuCols * kBpW / 4 / 128; u++) {
            const int e = tid + 128 * u, k = e / (kRuCols / 4), jq = (e % (kRuCols / 4)) * 4;
            const bool ok = k < K && tc + jq + 3 < cols;
            if (ok || tc + jq >= cols || k >= K) {
                cp_async16_zf(smem_u32(&Us[k][jq]), T + (long long)(k0 + (k < K ? k : 0)) * ldt + c0 + (ok ? tc + jq : 0),
                                 ok ? 16 : 0);
            } else {  // the ragged right edge
#pragma unroll
                for (int q = 0; q < 4; q++)
                    Us[k][jq + q] = tc + jq + q < cols ? T[(long long)(k0 + k) * ldt + c0 + tc + jq + q] : 0.0f;
            }
        }
        cp_async_commit();
    } else {
        for (int e = tid; e < kRuRows * kBpW; e += 128) {
            const int i = e / kBpW, k = e % kBpW;
            Ls[i][k] = (tr + i < rows && k < K) ? T[(long long)(r0 + tr + i) * ldt + k0 + k] : 0.0f;
        }
        for (int e = tid; e < kRuCols * kBpW; e += 128) {
            const int k = e / kRuCols, j = e % kRuCols;
            Us[k][j] = (tc + j < cols && k < K) ? T[(long long)(k0 + k) * ldt + c0 + tc + j] : 0.0f;
        }
    }
    const int tx = tid & 15, ty = tid >> 4;  // 16 x 8 threads
    const int jb = tc + 8 * tx;
    const bool full = vec && jb + 7 < cols;
    float acc[8][8];
#pragma unroll
    for (int a = 0; a < 8; a++) {
        const int i = tr + ty + 8 * a;
        const float* src = T + (long long)(r0 + i) * ldt + c0 + jb;
        if (i >= rows) {
#pragma unroll
            for (int b = 0; b < 8; b++) acc[a][b] = 0.0f;
        } else if (full) {
            const float4 x = reinterpret_cast<const float4*>(src)[0], y = reinterpret_cast<const float4*>(src)[1];
            acc[a][0] = x.x, acc[a][1] = x.y, acc[a][2] = x.z, acc[a][3] = x.w;
            acc[a][4] = y.x, acc[a][5] = y.y, acc[a][6] = y.z, acc[a][7] = y.w;
        } else {
#pragma unroll
            for (int b = 0; b < 8; b++) acc[a][b] = jb + b < cols ? src[b] : 0.0f;
        }
    }
    if (vec) cp_async_wait_all();
    __syncthreads();
    // one step of k: acc -= l * u, as packed f32x2 fmas (each lane an IEEE fma: fma(u, -l, acc)
    // == fmaf(-l, u, acc) bit for bit)
    auto step = [&](int k) {
        float lv[8];
#pragma unroll
        for (int a = 0; a < 8; a++) lv[a] = Ls[ty + 8 * a][k];
        const float4 u0 = *reinterpret_cast<const float4*>(&Us[k][8 * tx]);
        const float4 u1 = *reinterpret_cast<const float4*>(&Us[k][8 * tx + 4]);
        const float2 up[4] = {make_float2(u0.x, u0.y), make_float2(u0.z, u0.w), make_float2(u1.x, u1.y),
                              make_float2(u1.z, u1.w)};
#pragma unroll
        for (int a = 0; a < 8; a++) {
            const float2 nl = make_float2(-lv[a], -lv[a]);
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const float2 r = __ffma2_rn(up[b], nl, make_float2(acc[a][2 * b], acc[a][2 * b + 1]));
                acc[a][2 * b] = r.x;
                acc[a][2 * b + 1] = r.y;
            }
        }
    };
    if (K == kBpW) {
#pragma unroll 4
        for (int k = 0; k < kBpW; k++) step(k);
    } else {
        for (int k = 0; k < K; k++) step(k);
    }
#pragma unroll
    for (int a = 0; a < 8; a++) {
        const int i = tr + ty + 8 * a;
        if (i >= rows) continue;
        float* dst = T + (long long)(r0 + i) * ldt + c0 + jb;
        if (full) {
            reinterpret_cast<float4*>(dst)[0] = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
            reinterpret_cast<float4*>(dst)[1] = make_float4(acc[a][4], acc[a][5], acc[a][6], acc[a][7]);
        } else {
#pragma unroll
            for (int b = 0; b < 8; b++)
                if (jb + b < cols) dst[b] = acc[a][b];
        }
    }
}

// The panel kernel's CTA shape by panel rows: two rows a thread, small CTAs share an SM.
template <bool EXACT, bool PIVOT>
static cudaError_t panel_launch(cudaStream_t st, float* const* T, int n, int ldt, int k0, int* piv, int* info,
                                int* stat, char* scratch, long long l21_off, long long u12_off, long long per_matrix,
                                int batch)
{
    const int mp = n - k0;
    const unsigned g = (unsigned)batch;
    if (mp <= 128)
        lu_panel_kernel<64, 2, EXACT, PIVOT><<<g, 64, 0, st>>>(T, n, ldt, k0, piv, info, stat, scratch, l21_off,
                                                                u12_off, per_matrix);
    else if (mp <= 256)
        lu_panel_kernel<128, 2, EXACT, PIVOT><<<g, 128, 0, st>>>(T, n, ldt, k0, piv, info, stat, scratch, l21_off,
                                                                  u12_off, per_matrix);
    else if (mp <= 512)
        lu_panel_kernel<256, 2, EXACT, PIVOT><<<g, 256, 0, st>>>(T, n, ldt, k0, piv, info, stat, scratch, l21_off,
                                                                  u12_off, per_matrix);
    else
        lu_panel_kernel<512, 2, EXACT, PIVOT><<<g, 512, 0, st>>>(T, n, ldt, k0, piv, info, stat, scratch, l21_off,
                                                                  u12_off, per_matrix);
    return cudaGetLastError();
}

bool getrf_rows_supported(int n, int batch)
{
    if (n <= 128 || n > 1024) return false;
    // the update's grid (batch x its tiles) must fit a 31-bit grid dimension
    const long long max_tiles = (long long)((n + kRuRows - 1) / kRuRows) * ((n - kBpW + kRuCols - 1) / kRuCols);
    return (long long)batch * max_tiles <= 0x7fffffffLL;
}

cudaError_t getrf_rows_launch(cudaStream_t st, float* const* Aarray, int n, int lda, int* piv, int* info, int* stat,
                              int batch)
{
    if (batch <= 0 || !getrf_rows_supported(n, batch)) return cudaErrorInvalidValue;
    cudaError_t err = cudaMemsetAsync(stat, 0, sizeof(int) * (size_t)batch, st);
    if (err == cudaSuccess && info != nullptr) err = cudaMemsetAsync(info, 0, sizeof(int) * (size_t)batch, st);
    if (err == cudaSuccess && piv != nullptr) err = cudaMemsetAsync(piv, 0, sizeof(int) * (size_t)n * batch, st);
    if (err != cudaSuccess) return err;
    const int nt = (n + kTpT - 1) / kTpT;
    const dim3 tgrid((unsigned)batch, (unsigned)(nt * (nt + 1) / 2));
    lu_rows_out_kernel<<<tgrid, 256, 0, st>>>(Aarray, lda, n);  // in place: by columns -> by rows
    for (int k0 = 0; k0 < n; k0 += kBpW) {
        err = piv != nullptr ? panel_launch<true, true>(st, Aarray, n, lda, k0, piv, info, stat, nullptr, 0, 0, 0, batch)
                             : panel_launch<true, false>(st, Aarray, n, lda, k0, nullptr, info, stat, nullptr, 0, 0, 0,
                                                         batch);
        if (err != cudaSuccess) return err;
        if (n - k0 - kBpW > 0) {
            const int tm = (n - k0 + kRuRows - 1) / kRuRows, tn = (n - k0 - kBpW + kRuCols - 1) / kRuCols;
            lu_rows_update_kernel<<<(unsigned)((long long)batch * tm * tn), 128, 0, st>>>(Aarray, n, lda, k0, stat, tm,
                                                                                          tn);
            err = cudaGetLastError();
            if (err != cudaSuccess) return err;
        }
    }
    lu_rows_out_kernel<<<tgrid, 256, 0, st>>>(Aarray, lda, n);  // by rows -> by columns
    return cudaGetLastError();
}

bool getrf_blocked_tc_supported(int n) { return n > 256 && n <= 1024; }

size_t getrf_blocked_tc_scratch_bytes(int n, int batch)
{
    return (size_t)BpScratch(n).per_matrix * (size_t)batch + (size_t)batch * 16 + 512;
}

cudaError_t getrf_blocked_tc_launch(cudaStream_t st, const float* const* Aarray, int lda, float* const* LUarray, int n,
                                    int ldlu, int* piv, int* info, int batch, void* scratch, unsigned* status,
                                    void* tmslots)
{
    if (!getrf_blocked_tc_supported(n) || batch <= 0) return cudaErrorInvalidValue;
    const BpScratch L(n);
    char* base = static_cast<char*>(scratch);
    float** l21p = reinterpret_cast<float**>(base + L.per_matrix * batch);
    float** u12p = l21p + batch;
    cudaError_t err = cudaMemsetAsync(info, 0, sizeof(int) * (size_t)batch, st);
    if (err == cudaSuccess) err = cudaMemsetAsync(piv, 0, sizeof(int) * (size_t)n * batch, st);
    if (err != cudaSuccess) return err;
    const unsigned bgrid = (unsigned)((batch + 255) / 256);
    init_ptr_array_kernel<<<bgrid, 256, 0, st>>>(l21p, reinterpret_cast<float*>(base + L.l21),
                                                 L.per_matrix / 4, batch);
    init_ptr_array_kernel<<<bgrid, 256, 0, st>>>(u12p, reinterpret_cast<float*>(base + L.u12),
                                                 L.per_matrix / 4, batch);
    const int nt = (n + kTpT - 1) / kTpT;
    lu_rows_in_kernel<<<dim3((unsigned)batch, (unsigned)(nt * nt)), 256, 0, st>>>(Aarray, lda, LUarray, ldlu, n);
    for (int k0 = 0; k0 < n; k0 += kBpW) {
        err = panel_launch<false, true>(st, LUarray, n, ldlu, k0, piv, info, info, base, L.l21, L.u12, L.per_matrix,
                                        batch);
        if (err != cudaSuccess) return err;
        const int mt = n - k0 - kBpW;
        if (mt > 0) {
            // by rows T22 -= L21 * U12 is, on the storage, C -= U12^T * L21^T (m x m, K = 32)
            err = gemm_tc_lu_update(st, mt, u12p, l21p, LUarray, (long long)(k0 + kBpW) * (1 + (long long)ldlu), ldlu,
                                    batch, n - kBpW, status, tmslots);
            if (err != cudaSuccess) return err;
        }
    }
    lu_rows_out_kernel<<<dim3((unsigned)batch, (unsigned)(nt * (nt + 1) / 2)), 256, 0, st>>>(LUarray, ldlu, n);
    return cudaGetLastError();
}

}  // namespace opsblas
