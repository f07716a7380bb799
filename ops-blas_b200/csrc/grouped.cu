// aclblasSgetrfGetrsGrouped*: factor and solve many matrices of different orders in one
// persistent launch. No counterpart in the reference (an extension beside the drop-in chain);
// per instance the results are bit-identical to aclblasSgetrfBatched followed by
// aclblasSgetrsBatched (trans N) on the same matrix: every element takes the same operations in the
// same order (the factorisations are the batched kernels' own code, the solves are not).
//
// A plan describes the batch: groups of instances that share n, nrhs, lda and ldb. Creating it
// chooses, per group with n <= 32, the lanes per matrix from a tuning table written by
// autotune_grouped.py (or from the caller), orders the work largest first, and uploads the task lists
// to the device. Each execution is then one launch on the handle's stream (plus the regular batched
// kernels for groups with n > 128). Orders up to 32 alone: grouped_small_kernel (which also follows as a
// second launch when a mixed plan has many of them). Otherwise grouped_lu_kernel, one CTA of twelve
// warps an SM, whose teams take tasks from a device counter per class of orders, largest class first --
//   n > 32: teams of 4, 2 or 1 warps (by the class) factor one matrix in their share of the CTA's
//     shared memory (lu_mid.cuh), solve the right-hand sides from there (mid_solve) and store LU,
//     pivots and info;
//   n <= 32: each warp takes 32/lanes matrices, factors them in registers (small_getrf_core) and
//     solves from the registers (small_solve_core).
// The last CTA to finish resets the counters, so consecutive executions on one stream need no
// host work, and executions of one plan must not overlap in time.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <type_traits>
#include <vector>

#include "internal.h"
#include "lu_core.cuh"
#include "lu_mid.cuh"

namespace opsblas {

constexpr int kGrpThreads = 384;
constexpr int kGrpWarps = kGrpThreads / 32;
constexpr int kGrpMaxN = 128;  // larger orders use the batched kernels

struct GroupDev {
    int n, nrhs, lda, ldb;
    long long piv_off;  // first pivot of the group's first instance
    int first;          // index of the group's first instance in the pointer arrays
    int lanes;          // n <= 32: lanes per matrix (SEG)
    int pad;
};

struct GroupTask {
    int group;
    int first;  // first instance within the group
    int count;  // instances in this task
    int pad;
};

// ------------------------------------------------------------------------------ n > 32 --
// One matrix per team of W warps, factored in the team's shared memory (lu_mid.cuh); the right-hand
// sides are solved from there, one per warp, while the factors go to global memory. bar: W barriers
// of the panels, then the team's own.
template <int NBLK, int W>
__device__ __forceinline__ void grouped_mid(const GroupDev& g, int li, float* const* Aarray, float* const* Barray,
                                            int* piv, int* info, void* region, int warp, int lane, int bar)
{
    constexpr int R = MidSmem<NBLK, W>::R;
    auto& M = *static_cast<MidSmem<NBLK, W>*>(region);
    const int n = g.n;
    const long long inst = (long long)g.first + li;
    float* A = Aarray[inst];
    mid_stage<NBLK, W>(M, A, g.lda, n, warp, lane);
    if (warp == 0 && lane == 0) M.stop = n;
    cp_async_wait_all();
    team_sync<W * 32>(bar + W);
    mid_getrf<NBLK, true, W, 0>(M, n, warp, lane, bar);
    team_sync<W * 32>(bar + W);
    // column c + i W, i < C; those past the last one repeat it
    auto solve = [&](auto count, int c) {
        constexpr int C = decltype(count)::value;
        const int last = (g.nrhs - 1 - c) / W;
        float* bc = Barray[inst] + (long long)c * g.ldb;
        float y[C][R];
#pragma unroll
        for (int t = 0; t < R; t++) {
            const int r = lane + 32 * t < n ? M.rowof[lane + 32 * t] : -1;
#pragma unroll
            for (int i = 0; i < C; i++) y[i][t] = r >= 0 ? bc[r + (long long)(min(i, last) * W) * g.ldb] : 0.0f;
        }
        __syncwarp();  // every lane has read its b before any lane writes x
        mid_solve<NBLK, W, C>(M, n, lane, y);
#pragma unroll
        for (int i = 0; i < C; i++) {
            if (i > last) break;
#pragma unroll
            for (int t = 0; t < R; t++)
                if (lane + 32 * t < n) bc[lane + 32 * t + (long long)(i * W) * g.ldb] = y[i][t];
        }
    };
    if (g.nrhs > 2 * W) {
        for (int c = warp; c < g.nrhs; c += 4 * W) solve(std::integral_constant<int, 4>{}, c);
    } else if (g.nrhs > W) {
        solve(std::integral_constant<int, 2>{}, warp);
    } else if (warp < g.nrhs) {
        solve(std::integral_constant<int, 1>{}, warp);
    }
    mid_store<NBLK, W>(M, A, g.lda, n, piv + g.piv_off + (long long)li * n, warp, lane);
    if (warp == 0 && lane == 0) info[inst] = M.stop < n ? M.stop + 1 : 0;
}

// Classes of orders and how the CTA's twelve warps and its shared memory are dealt out to each: as many
// matrices at a time as the memory (or the sixteen barriers) hold, with the warps a matrix that were
// fastest in the batched kernel at that number of matrices an SM (getrf_mid.cu).
constexpr int kGrpClasses = 6;  // 113..128, 97..112, 81..96, 65..80, 33..64, 1..32
__host__ __device__ constexpr int grp_class(int n)
{
    return n > 112 ? 0 : n > 96 ? 1 : n > 80 ? 2 : n > 64 ? 3 : n > 32 ? 4 : 5;
}
__host__ __device__ constexpr int grp_team_warps(int c) { return c == 0 ? 4 : c < 3 ? 2 : 1; }
__host__ __device__ constexpr int grp_teams(int c)
{
    return c == 0 ? 3 : c == 1 ? 4 : c == 2 ? 5 : c == 3 ? 7 : c == 4 ? 11 : 12;
}
__host__ __device__ constexpr size_t grp_region(int c)
{
    return c == 0 ? sizeof(MidSmem<8, 4>) : c == 1 ? sizeof(MidSmem<7, 2>) : c == 2 ? sizeof(MidSmem<6, 2>)
           : c == 3 ? sizeof(MidSmem<5, 1>) : c == 4 ? sizeof(MidSmem<4, 1>)
                                            : 3 * 32 * sizeof(float);  // small: two row buffers, owners
}
static_assert(grp_teams(0) * grp_region(0) <= 231000 && grp_teams(1) * grp_region(1) <= 231000 &&
              grp_teams(2) * grp_region(2) <= 231000 && grp_teams(3) * grp_region(3) <= 231000 &&
              grp_teams(4) * grp_region(4) <= 231000, "one CTA an SM");

// ----------------------------------------------------------------------------- n <= 32 --
template <int N, int SEG>
__device__ __forceinline__ void grouped_small(const GroupDev& g, const GroupTask& task, float* const* Aarray,
                                              float* const* Barray, int* piv, int* info, float* rowbuf, int* owner,
                                              int lane)
{
    constexpr int NC = (N + 3) / 4;
    const int seg = lane / SEG;
    const int r = lane % SEG;
    const int li = task.first + seg;
    const bool mvalid = seg < task.count;
    const bool rvalid = mvalid && r < N;
    const long long inst = (long long)g.first + li;
    const int lda = g.lda;
    float* A = mvalid ? Aarray[inst] : nullptr;
    float4 a4[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) a4[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (rvalid) {
        const float* Ar = A + r;
#pragma unroll
        for (int j = 0; j < N; j++) qset<N>(a4, j, Ar[(long long)j * lda]);
    }
    int pos, mypiv, inf;
    small_getrf_core<N, true, SEG>(a4, pos, mypiv, inf, rowbuf, seg, r, mvalid, rvalid);
    if (g.nrhs > 0) {
        float* Bm = mvalid ? Barray[inst] : nullptr;
        for (int c = 0; c < g.nrhs; c++) {
            float* bc = rvalid ? Bm + (long long)c * g.ldb : nullptr;
            float y = rvalid ? bc[r] : 0.0f;
            y = small_solve_core<N, SEG>(a4, pos, rvalid, seg, r, owner + seg * SEG, y);
            if (rvalid) bc[pos] = y;
        }
    }
    if (rvalid) {
        float* Ap = A + pos;
#pragma unroll
        for (int j = 0; j < N; j++) Ap[(long long)j * lda] = qget<N>(a4, j);
        piv[g.piv_off + (long long)li * N + r] = mypiv;
        if (r == 0) info[inst] = inf;
    }
}

template <int N>
__device__ __forceinline__ void grouped_small_dispatch(const GroupDev& g, const GroupTask& task,
                                                       float* const* Aarray, float* const* Barray, int* piv,
                                                       int* info, float* rowbuf, int* owner, int lane)
{
    constexpr int NAT = SmallShape<N>::SEG;
    if (NAT == 32 || g.lanes == NAT)
        grouped_small<N, NAT>(g, task, Aarray, Barray, piv, info, rowbuf, owner, lane);
    else
        grouped_small<N, 32>(g, task, Aarray, Barray, piv, info, rowbuf, owner, lane);
}

// Tasks of n <= 32, a warp each. A CTA's warps start with neighbours of the list, which are mostly of one
// order: the code of an order is long and runs once a task, so that an SM whose warps took scattered tasks
// waited for instructions (400 orders of 4 to 32: 46 us; together 20). After that each warp asks for itself.
// FIRST: the CTAs start together, and their first tasks need no counter.
template <int WARPS, bool FIRST>
__device__ __forceinline__ void grouped_small_tasks(const GroupDev* groups, const GroupTask* __restrict__ tasks,
                                                    int count, int* counter, float* const* Aarray,
                                                    float* const* Barray, int* piv, int* info, float* rowbuf, int* owner,
                                                    int* s_task, int wid, int lane)
{
    int t = (int)blockIdx.x * WARPS + wid;
    if (!FIRST) {
        if (threadIdx.x == 0) *s_task = atomicAdd(counter, WARPS);
        __syncthreads();
        t = *s_task + wid;
    }
    while (t < count) {
        const GroupTask task = tasks[t];
        const GroupDev& g = groups[task.group];  // fields read when needed: fewer live registers
        switch (g.n) {
#define OPSBLAS_GROUPED_CASE(NN)                                                                                    \
    case NN:                                                                                                        \
        grouped_small_dispatch<NN>(g, task, Aarray, Barray, piv, info, rowbuf, owner, lane);                        \
        break;
            OPSBLAS_FOR_N_1_32(OPSBLAS_GROUPED_CASE)
#undef OPSBLAS_GROUPED_CASE
            default:
                break;
        }
        __syncwarp();  // the warp's shared memory is read before its next task writes it
        t = lane == 0 ? atomicAdd(counter, 1) + (FIRST ? (int)gridDim.x * WARPS : 0) : 0;
        t = __shfl_sync(0xffffffffu, t, 0);
    }
}

// Tasks of one class of n > 32, taken by the CTA's teams from the class's counter.
template <int C>
__device__ __forceinline__ void grouped_class(const GroupDev* groups, const GroupTask* __restrict__ tasks, int count,
                                              bool only, int* counter, float* const* Aarray, float* const* Barray, int* piv,
                                              int* info, unsigned char* dyn, int* s_task, int wid, int lane)
{
    constexpr int W = grp_team_warps(C);
    const int team = wid / W, warp = wid % W;
    if (team >= grp_teams(C)) return;
    const int bar = 1 + team * (W + 1);
    unsigned char* region = dyn + (size_t)team * grp_region(C);
    // only: there is no other class. Every SM's first team, then its second, and so on, take the first tasks;
    // asked for, they go to the SMs that start first (400 orders of 33 to 64: 67 us, 54). With classes to
    // follow that is as well: the other SMs go on to those meanwhile (400 of 65 to 96: 82 us, 125).
    const int spread = only ? grp_teams(C) * (int)gridDim.x : 0;
    for (bool first = only;; first = false) {
        team_sync<W * 32>(bar + W);  // the previous task's shared memory and task number are done with
        int t = team * (int)gridDim.x + (int)blockIdx.x;
        if (!first && W == 1) {
            t = lane == 0 ? atomicAdd(counter, 1) + spread : 0;
            t = __shfl_sync(0xffffffffu, t, 0);
        } else if (!first) {
            if (warp == 0 && lane == 0) s_task[team] = atomicAdd(counter, 1) + spread;
            team_sync<W * 32>(bar + W);
            t = s_task[team];
        }
        if (t >= count) break;
        const GroupTask task = tasks[t];
        const GroupDev& g = groups[task.group];  // fields read when needed: fewer live registers
        if constexpr (C < 4) {
            grouped_mid<8 - C, W>(g, task.first, Aarray, Barray, piv, info, region, warp, lane, bar);
        } else {
            if (g.n > 48)
                grouped_mid<4, W>(g, task.first, Aarray, Barray, piv, info, region, warp, lane, bar);
            else
                grouped_mid<3, W>(g, task.first, Aarray, Barray, piv, info, region, warp, lane, bar);
        }
    }
}

// One CTA an SM. The classes follow each other, largest orders first; within a class every team works
// on its own. tasks: the classes' lists one after the other, class c at [first[c], first[c + 1]).
// counters: one a class, then the CTAs that are done.
struct GroupLists {
    int first[kGrpClasses + 1];
};

// The last CTA out resets the counters for the next execution.
__device__ __forceinline__ void grouped_last_out(int* counters)
{
    __syncthreads();  // none of the CTA's warps asks for a task any more
    if (threadIdx.x == 0) {
        __threadfence();
        const int f = atomicAdd(&counters[kGrpClasses], 1);
        if (f == (int)gridDim.x - 1) {
            for (int c = 0; c <= kGrpClasses; c++) atomicExch(&counters[c], 0);
        }
    }
}

__global__ void __launch_bounds__(kGrpThreads, 1)
grouped_lu_kernel(const GroupDev* groups, const GroupTask* __restrict__ tasks, const GroupLists lists,
                  int* __restrict__ counters, float* const* Aarray, float* const* Barray, int* piv, int* info)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ int s_task[kGrpWarps];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
#define OPSBLAS_GROUPED_CLASS(C)                                                                                    \
    if (lists.first[C + 1] > lists.first[C]) {                                                                      \
        const int count = lists.first[C + 1] - lists.first[C];                                                      \
        grouped_class<C>(groups, tasks + lists.first[C], count, count == lists.first[kGrpClasses], counters + C,    \
                         Aarray, Barray, piv, info, dyn, s_task, wid, lane);                                        \
        __syncthreads();                                                                                            \
    }
    OPSBLAS_GROUPED_CLASS(0)
    OPSBLAS_GROUPED_CLASS(1)
    OPSBLAS_GROUPED_CLASS(2)
    OPSBLAS_GROUPED_CLASS(3)
    OPSBLAS_GROUPED_CLASS(4)
#undef OPSBLAS_GROUPED_CLASS
    constexpr int S = kGrpClasses - 1;
    if (lists.first[S + 1] > lists.first[S]) {
        float* rowbuf = reinterpret_cast<float*>(dyn + (size_t)wid * grp_region(S));
        grouped_small_tasks<kGrpWarps, false>(groups, tasks + lists.first[S], lists.first[S + 1] - lists.first[S],
                                              counters + S, Aarray, Barray, piv, info, rowbuf,
                                              reinterpret_cast<int*>(rowbuf + 64), s_task, wid, lane);
    }
    grouped_last_out(counters);
}

// A plan of orders up to 32 only: nothing needs the shared memory or the registers of the classes above, and
// sixteen warps an SM in two CTAs hide more latency than twelve (20000 orders of 4 to 32: 123 us, 98).
constexpr int kGrpSmallWarps = 8;

__global__ void __launch_bounds__(kGrpSmallWarps * 32, 2)
grouped_small_kernel(const GroupDev* groups, const GroupTask* __restrict__ tasks, int count, int* __restrict__ counters,
                     float* const* Aarray, float* const* Barray, int* piv, int* info)
{
    __shared__ __align__(16) float rowbuf[kGrpSmallWarps][64];
    __shared__ int owner[kGrpSmallWarps][32];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    grouped_small_tasks<kGrpSmallWarps, true>(groups, tasks, count, counters + kGrpClasses - 1, Aarray, Barray, piv,
                                              info, rowbuf[wid], owner[wid], nullptr, wid, lane);
    grouped_last_out(counters);
}

// ------------------------------------------------------------------------- host side --
struct TuneRow {
    int lo, hi, lanes, warps, rows;
};

// Rows per lane and warps per matrix for n > 32, which callers and tables may name: they have no effect (the
// kernel deals out its warps by the order, grp_class) and are checked and reported for those that name them.
static bool reg_shape_valid(int n, int rows, int warps)
{
    if (n <= 32 || n > 32 * rows) return false;
    return (rows == 2 && (warps == 2 || warps == 4 || warps == 8)) || (rows == 3 && (warps == 4 || warps == 8)) ||
           (rows == 4 && warps == 8);
}

static void reg_default_shape(int n, int& rows, int& warps)
{
    rows = (n + 31) / 32;
    warps = rows == 2 ? 2 : (rows == 3 ? 4 : 8);
}

// Built-in choices, used when no tuning table is found.
static void default_config(int n, int cfg[3])
{
    if (n <= 32) {
        cfg[0] = n <= 4 ? 4 : (n <= 8 ? 8 : (n <= 16 ? 16 : 32));
        cfg[1] = 0;
        cfg[2] = 0;
    } else {
        cfg[0] = 0;
        reg_default_shape(n, cfg[2], cfg[1]);
    }
}

static std::string tuning_path()
{
    const char* env = std::getenv("OPSBLAS_GROUPED_TUNING");
    if (env && *env) return env;
    Dl_info dli;
    if (dladdr(reinterpret_cast<void*>(&default_config), &dli) && dli.dli_fname) {
        std::string p(dli.dli_fname);
        const size_t s = p.rfind('/');
        return (s == std::string::npos ? std::string(".") : p.substr(0, s)) + "/grouped_tuning.txt";
    }
    return "grouped_tuning.txt";
}

// Table rows "n_lo n_hi lanes warps rows"; '#' starts a comment.
static std::vector<TuneRow> load_tuning()
{
    std::vector<TuneRow> rows;
    FILE* f = std::fopen(tuning_path().c_str(), "r");
    if (!f) return rows;
    char line[256];
    while (std::fgets(line, sizeof line, f)) {
        if (line[0] == '#') continue;
        TuneRow r;
        if (std::sscanf(line, "%d %d %d %d %d", &r.lo, &r.hi, &r.lanes, &r.warps, &r.rows) == 5) rows.push_back(r);
    }
    std::fclose(f);
    return rows;
}

// Makes cfg valid for n: lanes in {natural, 32} (n <= 32); an instantiated (rows, warps) shape
// with 32 * rows >= n (n > 32).
static void sanitize_config(int n, int cfg[3])
{
    int def[3];
    default_config(n, def);
    if (n <= 32) {
        if (cfg[0] != def[0] && cfg[0] != 32) cfg[0] = def[0];
        cfg[1] = 0;
        cfg[2] = 0;
    } else {
        cfg[0] = 0;
        if (!reg_shape_valid(n, cfg[2], cfg[1])) {
            cfg[1] = def[1];
            cfg[2] = def[2];
        }
    }
}

struct GroupHost {
    int n, nrhs, lda, ldb, size, first;
    long long piv_off;
    int cfg[3];
};

}  // namespace opsblas

struct _aclblas_grouped_plan {
    int device = 0;
    std::vector<opsblas::GroupHost> groups;
    int total = 0;
    void* dmem = nullptr;
    opsblas::GroupDev* d_groups = nullptr;
    opsblas::GroupTask* d_tasks = nullptr;
    int* d_counters = nullptr;
    opsblas::GroupLists lists = {};
    int grid = 0;
    size_t smem = 0;      // dynamic shared memory per CTA
    bool has_persistent = false;
    bool small_apart = false;  // the tasks of n <= 32 run in grouped_small_kernel, after the others if there are any
    int small_grid = 0, small_first = 0, small_count = 0;  // its CTAs and tasks; grid: grouped_lu_kernel's CTAs
};

using namespace opsblas;

extern "C" aclblasStatus_t aclblasSgetrfGetrsGroupedPlanCreate(aclblasHandle_t handle, int groupCount,
                                                               const int nArray[], const int nrhsArray[],
                                                               const int ldaArray[], const int ldbArray[],
                                                               const int groupSizeArray[], const int* configArray,
                                                               aclblasGroupedPlan_t* plan)
{
    static const char* kApi = "aclblasSgetrfGetrsGroupedPlanCreate";
    if (handle == nullptr) {
        log_error(kApi, "handle is nullptr");
        return ACLBLAS_STATUS_HANDLE_IS_NULLPTR;
    }
    if (plan == nullptr || groupCount < 0) {
        log_error(kApi, "plan must not be nullptr and groupCount must be >= 0");
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    *plan = nullptr;
    if (groupCount > 0 && (!nArray || !nrhsArray || !ldaArray || !ldbArray || !groupSizeArray)) {
        log_error(kApi, "group arrays must not be nullptr");
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    long long total = 0;
    for (int g = 0; g < groupCount; g++) {
        const int n = nArray[g];
        if (n < 0 || nrhsArray[g] < 0 || groupSizeArray[g] < 0 || ldaArray[g] < max1(n) || ldbArray[g] < max1(n)) {
            log_error(kApi, "group %d: n=%d nrhs=%d lda=%d ldb=%d size=%d is invalid", g, n, nrhsArray[g],
                      ldaArray[g], ldbArray[g], groupSizeArray[g]);
            return ACLBLAS_STATUS_INVALID_VALUE;
        }
        total += groupSizeArray[g];
    }
    if (total > 0x7fffffffLL) {
        log_error(kApi, "more than 2^31-1 instances");
        return ACLBLAS_STATUS_INVALID_VALUE;
    }

    auto* p = new _aclblas_grouped_plan();
    p->device = handle->device;
    const std::vector<TuneRow> table = load_tuning();
    long long piv_off = 0;
    int first = 0;
    for (int g = 0; g < groupCount; g++) {
        GroupHost h;
        h.n = nArray[g];
        h.nrhs = nrhsArray[g];
        h.lda = ldaArray[g];
        h.ldb = ldbArray[g];
        h.size = groupSizeArray[g];
        h.first = first;
        h.piv_off = piv_off;
        default_config(h.n, h.cfg);
        for (const TuneRow& r : table)
            if (h.n >= r.lo && h.n <= r.hi) {
                h.cfg[0] = r.lanes;
                h.cfg[1] = r.warps;
                h.cfg[2] = r.rows;
            }
        if (configArray) {
            for (int q = 0; q < 3; q++)
                if (configArray[3 * g + q] > 0) h.cfg[q] = configArray[3 * g + q];
        }
        sanitize_config(h.n, h.cfg);
        first += h.size;
        piv_off += (long long)h.n * h.size;
        p->groups.push_back(h);
    }
    p->total = first;

    // task lists, largest matrices first
    std::vector<int> order(groupCount);
    for (int g = 0; g < groupCount; g++) order[g] = g;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return p->groups[a].n > p->groups[b].n; });
    std::vector<GroupTask> tasks;
    size_t smem = 0;
    int cls = 0;
    for (int g : order) {
        const GroupHost& h = p->groups[g];
        if (h.n == 0 || h.size == 0 || h.n > kGrpMaxN) continue;
        const int c = grp_class(h.n);
        while (cls < c) p->lists.first[++cls] = (int)tasks.size();
        smem = std::max(smem, grp_teams(c) * grp_region(c));
        const int per = h.n > 32 ? 1 : 32 / h.cfg[0];  // matrices a task
        for (int i = 0; i < h.size; i += per) tasks.push_back({g, i, std::min(per, h.size - i), 0});
    }
    while (cls < kGrpClasses) p->lists.first[++cls] = (int)tasks.size();
    p->has_persistent = !tasks.empty();
    // many small tasks repay a launch of their own, which runs sixteen warps an SM in place of twelve; fewer
    // fill the SMs that have finished their larger orders (us, together and apart: orders of 4 to 40 with 8
    // columns, 20000 384 and 349, 100000 1610 and 1476; of 1 to 33, 300000 1456 and 1125)
    const int mids = p->lists.first[kGrpClasses - 1], smalls = (int)tasks.size() - mids;
    p->small_apart = smalls > 0 && (mids == 0 || smalls >= 4 * 2 * kGrpSmallWarps * sm_count());
    p->smem = smem;

    std::vector<GroupDev> gd(std::max(groupCount, 1));
    for (int g = 0; g < groupCount; g++) {
        const GroupHost& h = p->groups[g];
        gd[g] = {h.n, h.nrhs, h.lda, h.ldb, h.piv_off, h.first, h.cfg[0], 0};
    }
    if (p->has_persistent) {
        const size_t bg = gd.size() * sizeof(GroupDev);
        const size_t bt = tasks.size() * sizeof(GroupTask);
        cudaError_t err = cudaMalloc(&p->dmem, bg + bt + 256);
        if (err != cudaSuccess) {
            log_error(kApi, "cannot allocate %zu bytes for the plan", bg + bt + 256);
            delete p;
            return ACLBLAS_STATUS_ALLOC_FAILED;
        }
        char* d = static_cast<char*>(p->dmem);
        p->d_counters = reinterpret_cast<int*>(d);
        p->d_groups = reinterpret_cast<GroupDev*>(d + 256);
        p->d_tasks = reinterpret_cast<GroupTask*>(d + 256 + bg);
        err = cudaMemset(p->d_counters, 0, 256);
        if (err == cudaSuccess) err = cudaMemcpy(p->d_groups, gd.data(), bg, cudaMemcpyHostToDevice);
        if (err == cudaSuccess) err = cudaMemcpy(p->d_tasks, tasks.data(), bt, cudaMemcpyHostToDevice);
        int per_sm = 1, small_per_sm = 1;
        if (err == cudaSuccess && p->small_apart)
            err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&small_per_sm, grouped_small_kernel, kGrpSmallWarps * 32, 0);
        if (err == cudaSuccess && !(p->small_apart && mids == 0)) {
            err = ensure_smem_limit(grouped_lu_kernel, (int)p->smem);
            if (err == cudaSuccess)
                err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, grouped_lu_kernel, kGrpThreads, p->smem);
        }
        if (err != cudaSuccess || per_sm < 1 || small_per_sm < 1) {
            log_error(kApi, "plan set-up failed: %s", cudaGetErrorString(err));
            cudaFree(p->dmem);
            delete p;
            return err != cudaSuccess ? launch_status(kApi, err) : ACLBLAS_STATUS_NOT_SUPPORTED;
        }
        const long long lu_tasks = p->small_apart ? mids : (long long)tasks.size();
        p->grid = (int)std::min<long long>(lu_tasks, sm_count());
        if (p->small_apart) {
            p->small_first = mids;
            p->small_count = smalls;
            p->small_grid = (int)std::min<long long>(((long long)smalls + kGrpSmallWarps - 1) / kGrpSmallWarps,
                                                     (long long)small_per_sm * sm_count());
            p->lists.first[kGrpClasses] = mids;  // grouped_lu_kernel leaves them alone
        }
    }
    *plan = p;
    return ACLBLAS_STATUS_SUCCESS;
}

extern "C" aclblasStatus_t aclblasSgetrfGetrsGroupedPlanGetConfig(aclblasGroupedPlan_t plan, int* configArray)
{
    if (plan == nullptr || configArray == nullptr) return ACLBLAS_STATUS_INVALID_VALUE;
    for (size_t g = 0; g < plan->groups.size(); g++)
        for (int q = 0; q < 3; q++) configArray[3 * g + q] = plan->groups[g].cfg[q];
    return ACLBLAS_STATUS_SUCCESS;
}

extern "C" aclblasStatus_t aclblasSgetrfGetrsGroupedPlanDestroy(aclblasGroupedPlan_t plan)
{
    if (plan == nullptr) return ACLBLAS_STATUS_INVALID_VALUE;
    if (plan->dmem) cudaFree(plan->dmem);
    delete plan;
    return ACLBLAS_STATUS_SUCCESS;
}

extern "C" aclblasStatus_t aclblasSgetrfGetrsGroupedBatched(aclblasHandle_t handle, aclblasGroupedPlan_t plan,
                                                            float* const Aarray[], int* PivotArray, int* infoArray,
                                                            float* const Barray[])
{
    static const char* kApi = "aclblasSgetrfGetrsGroupedBatched";
    if (handle == nullptr) {
        log_error(kApi, "handle is nullptr");
        return ACLBLAS_STATUS_HANDLE_IS_NULLPTR;
    }
    if (plan == nullptr) {
        log_error(kApi, "plan is nullptr");
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (plan->total == 0) return ACLBLAS_STATUS_SUCCESS;
    bool need_b = false;
    for (const GroupHost& h : plan->groups) need_b |= h.nrhs > 0 && h.n > 0 && h.size > 0;
    if (!Aarray || !PivotArray || !infoArray || (need_b && !Barray)) {
        log_error(kApi, "Aarray, PivotArray, infoArray (and Barray when a group has nrhs > 0) must not be nullptr");
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    if (handle->device != plan->device) {
        log_error(kApi, "the plan was made on device %d, the handle is on device %d", plan->device, handle->device);
        return ACLBLAS_STATUS_INVALID_VALUE;
    }
    cudaStream_t st = handle->stream;
    if (plan->has_persistent) {
        if (plan->grid > 0)
            grouped_lu_kernel<<<(unsigned)plan->grid, kGrpThreads, plan->smem, st>>>(
                plan->d_groups, plan->d_tasks, plan->lists, plan->d_counters, Aarray, Barray, PivotArray, infoArray);
        if (plan->small_grid > 0)
            grouped_small_kernel<<<(unsigned)plan->small_grid, kGrpSmallWarps * 32, 0, st>>>(
                plan->d_groups, plan->d_tasks + plan->small_first, plan->small_count, plan->d_counters, Aarray, Barray,
                PivotArray, infoArray);
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return launch_status(kApi, err);
    }
    // groups beyond the persistent kernel's sizes: the regular batched kernels
    for (const GroupHost& h : plan->groups) {
        if (h.n <= kGrpMaxN || h.size == 0) continue;
        aclblasStatus_t s = aclblasSgetrfBatched(handle, h.n, Aarray + h.first, h.lda, PivotArray + h.piv_off,
                                                 infoArray + h.first, h.size);
        if (s != ACLBLAS_STATUS_SUCCESS) return s;
        if (h.nrhs > 0) {
            cudaError_t err = getrs_launch(st, false, h.n, h.nrhs, Aarray + h.first, h.lda, PivotArray + h.piv_off,
                                           Barray + h.first, h.ldb, h.size);
            if (err != cudaSuccess) return launch_status(kApi, err);
        }
    }
    return ACLBLAS_STATUS_SUCCESS;
}
