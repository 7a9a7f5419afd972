// Grouping: stable token -> expert grouping on the GPU (upstream src/grouping.rs:12-111 and the six kernels
// of native/grouping.cu).  Same result contract:
//   ids[u]      distinct expert ids of the window, ascending
//   count[0]    their number
//   members[u]  row * 32 + slot of every row that picked ids[u], ascending rows, then -1 up to maxm;
//               rows u >= count are all -1
// One launch for any window size (upstream: one block for <= 32 rows, five launches up to 8192 rows): CTA e
// owns expert e.  It first marks the used experts from the picks itself (so it knows its place among them without
// a second kernel or a global scan), then compacts the rows that picked e in row order with one block scan per 8192
// rows.  Nothing is ordered by atomics.  A row that names an expert twice counts once, with its first slot, as in
// upstream's row-bitmap.
// A launch is bound by the latency of its steps.  Marking by atomicOr on a bitmap queued a whole window on a few words of
// shared memory, and a scan per 1024 rows was a chain of barriers: 4096 rows x 5 of 65 experts 14.1 -> 6.4 us, 8192 rows 25.0 ->
// 9.0, 17 rows 4.5 -> 4.1, 8192 x 9 of 289 45.8 -> 26.5 (launches back to back).
#include <algorithm>
#include <new>

#include "common.cuh"

namespace gf {
int check_config(const glmflash_config *cfg, size_t cfg_bytes, int max_rows_limit);

constexpr int GROUP_THREADS = 1024, GROUP_STEPS = 8;

__global__ void __launch_bounds__(GROUP_THREADS) grouping_kernel(const int *__restrict__ picks, int rows, int slots, int E1,
                                                                int maxm, int *__restrict__ ids, int *__restrict__ count,
                                                                int *__restrict__ members) {
    __shared__ int used[GROUP_THREADS];           // E1 <= 1024
    __shared__ int sums[GROUP_STEPS * 32], totals[GROUP_STEPS];
    const int e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    used[tid] = 0;
    pdl_wait();                                   // picks may be the previous kernel's output; ids / members its input
    pdl_launch_dependents();
    __syncthreads();
    const int total = rows * slots;
#pragma unroll 4
    for (int i = tid; i < total; i += GROUP_THREADS) {
        const int p = picks[i];
        if (p >= 0 && p < E1) used[p] = 1;        // (every writer stores the same)
    }
    __syncthreads();
    const bool mine = used[e] != 0;
    const int place = __syncthreads_count(used[tid] && tid < e), n_used = __syncthreads_count(used[tid]);
    if (e == 0 && tid == 0) *count = n_used;
    if (mine && tid == 0) ids[place] = e;
    if (!mine && e >= n_used && tid == 0) ids[e] = -1;       // tail of ids: not read by consumers, kept tidy

    if (mine) {
        int *out = members + (size_t)place * maxm;
        int base = 0;
        for (int r0 = 0; r0 < rows; r0 += GROUP_STEPS * GROUP_THREADS) {
            int slot[GROUP_STEPS], before[GROUP_STEPS];
#pragma unroll
            for (int i = 0; i < GROUP_STEPS; ++i) {
                const int r = r0 + i * GROUP_THREADS + tid;
                slot[i] = -1;
                if (r < rows)
                    for (int s = slots - 1; s >= 0; --s)
                        if (picks[r * slots + s] == e) slot[i] = s;     // first matching slot wins
                const uint32_t ball = __ballot_sync(0xffffffffu, slot[i] >= 0);
                before[i] = __popc(ball & ((1u << lane) - 1u));
                if (lane == 0) sums[i * 32 + warp] = __popc(ball);
            }
            __syncthreads();
            if (warp < GROUP_STEPS) {             // a warp scans the 32 sums of one step
                const int v = sums[tid];
                int incl = v;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int up = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += up;
                }
                sums[tid] = incl - v;
                if (lane == 31) totals[warp] = incl;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < GROUP_STEPS; ++i) {
                const int off = base + sums[i * 32 + warp] + before[i];
                if (slot[i] >= 0 && off < maxm) out[off] = (r0 + i * GROUP_THREADS + tid) * 32 + slot[i];
                base += totals[i];
            }
            __syncthreads();
        }
        for (int j = min(base, maxm) + tid; j < maxm; j += GROUP_THREADS) out[j] = -1;
    }
    // rows of `members` beyond the used ones: row e is unused exactly when e >= n_used
    if (e >= n_used)
        for (int j = tid; j < maxm; j += GROUP_THREADS) members[(size_t)e * maxm + j] = -1;
}

int launch_grouping(cudaStream_t s, const int *picks, int rows, int slots, int E1, int maxm, int *ids, int *count,
                    int *members, bool pdl) {
    return launch_k(grouping_kernel, dim3(E1), dim3(GROUP_THREADS), 0, s, pdl, picks, rows, slots, E1, maxm, ids, count,
                    members);
}
}  // namespace gf

using namespace gf;

struct glmflash_grouping {
    glmflash_config cfg;
    void *pool = nullptr;                                    // the one allocation behind the tables
    int *ids = nullptr, *count = nullptr, *members = nullptr;
};

extern "C" int glmflash_grouping_new(const glmflash_config *cfg, size_t cfg_bytes, glmflash_grouping **out) {
    GF_REQUIRE(out != nullptr, "out is null");
    *out = nullptr;
    if (check_config(cfg, cfg_bytes, 8192)) return -1;       // upstream: 1..=8192, src/grouping.rs:30
    glmflash_grouping *g = new (std::nothrow) glmflash_grouping();
    GF_REQUIRE(g != nullptr, "out of host memory");
    g->cfg = *cfg;
    const size_t E1 = cfg->experts + 1;
    Pool pool;
    pool.take(&g->ids, E1 * 4);
    pool.take(&g->count, 4);
    pool.take(&g->members, E1 * cfg->max_rows * 4);
    if (pool.alloc(&g->pool)) {
        glmflash_grouping_free(g);
        return -1;
    }
    cudaMemset(g->ids, 0xff, E1 * 4);
    cudaMemset(g->members, 0xff, E1 * cfg->max_rows * 4);
    *out = g;
    return 0;
}

extern "C" void glmflash_grouping_free(glmflash_grouping *g) {
    if (!g) return;
    cudaFree(g->pool);
    delete g;
}

extern "C" int glmflash_grouping_run(glmflash_grouping *g, void *stream, const int32_t *picks, int rows) {
    GF_REQUIRE(g && picks, "null argument");
    GF_REQUIRE(rows > 0 && rows <= g->cfg.max_rows, "grouping rows exceed scratch");
    return launch_grouping((cudaStream_t)stream, picks, rows, g->cfg.slots, g->cfg.experts + 1, g->cfg.max_rows, g->ids,
                           g->count, g->members, g->cfg.pdl != 0);
}

extern "C" const int32_t *glmflash_grouping_ids(const glmflash_grouping *g) { return g ? g->ids : nullptr; }
extern "C" const int32_t *glmflash_grouping_count(const glmflash_grouping *g) { return g ? g->count : nullptr; }
extern "C" const int32_t *glmflash_grouping_members(const glmflash_grouping *g) { return g ? g->members : nullptr; }
