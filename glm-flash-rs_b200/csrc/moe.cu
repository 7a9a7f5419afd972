// Moe: grouping -> experts -> combine for one window (upstream src/moe.rs:11-182 for one row,
// src/model_verifier.rs:1291-1305 and src/batch.rs:1160-1210 for windows and chunks), plus the rank-ordered
// sum that follows the cross-GPU all-gather (upstream src/model.rs:485-496).
#include <algorithm>
#include <initializer_list>
#include <new>

#include <stdlib.h>

#include "common.cuh"
#include "owners.cuh"
#include "stream.cuh"

namespace gf {
int experts_run_fused(glmflash_experts *e, cudaStream_t s, const glmflash_weights *w, const void *input, int x_stride,
                      const int32_t *picks, const float *route_w, float *out, float *out2, int rows, float *y, int *status);
int *fast_experts_status_word(glmflash_fast_experts *f);
int fast_experts_run(glmflash_fast_experts *f, void *stream, const glmflash_weights *w, const void *input, int x_stride, const int32_t *picks,
                     const int32_t *ids, const int32_t *count, const int32_t *members, int rows, int maxm, int shared_x, bool fine);

// out[r][d] = sum_{s < slots-1, expert computed here} w[r][s] * Y[r*slots+s][d]  (+ Y[shared pair] if computed here)
// fp32, ascending slot order, shared last: the order of the oracle's combine.
__global__ void __launch_bounds__(256) combine_kernel(const float *__restrict__ Y, const int *__restrict__ picks,
                                                      const float *__restrict__ route_w, float *__restrict__ out, int slots,
                                                      int H, int E, int shared_exl3, int e_lo, int e_hi, int srow_lo,
                                                      int srow_hi) {
    // Launched behind the down GEMM only.  That kernel, like the grouping, plan, rotation and gate / up kernels in front of it, runs
    // its own pdl_wait before it triggers, so when this one starts, everything in front of the down GEMM has completed, the
    // router's table and weights among it: they are read ahead of the wait.  Only the pair results Y belong to the kernel in front.
    const int r = blockIdx.y;
    const int d = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    __shared__ float wgt_sh[32];
    __shared__ uint32_t live_sh;
    if (threadIdx.x < 32) {
        const int s = threadIdx.x;
        bool keep = false;
        float w = 0.f;
        if (s < slots) {
            const int e = picks[r * slots + s];
            keep = !(e < 0 || e > E || (e == E ? !shared_exl3 : (e < e_lo || e >= e_hi)));
            if (e == E && srow_hi > srow_lo && (r < srow_lo || r >= srow_hi)) keep = false;   // shared expert: row window
            w = route_w[r * slots + s];
        }
        wgt_sh[s] = w;
        const uint32_t mask = __ballot_sync(0xffffffffu, keep);
        if (s == 0) live_sh = mask;
    }
    __syncthreads();
    const uint32_t live = live_sh;
    pdl_wait();
    pdl_launch_dependents();
    if (d >= H) return;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < slots; ++s) {
        if (!((live >> s) & 1u)) continue;
        const float4 y = *reinterpret_cast<const float4 *>(Y + ((size_t)r * slots + s) * H + d);
        if (s == slots - 1) { acc.x += y.x; acc.y += y.y; acc.z += y.z; acc.w += y.w; }
        else {
            const float w = wgt_sh[s];
            acc.x += w * y.x; acc.y += w * y.y; acc.z += w * y.z; acc.w += w * y.w;
        }
    }
    *reinterpret_cast<float4 *>(out + (size_t)r * H + d) = acc;
}

// Inputs of a window from pinned host memory to the owner's buffers: the input rows in 16-byte words, then the routing table
// and its weights.
__global__ void __launch_bounds__(256) stage_in_kernel(const uint4 *x_host, uint4 *x, int nx, const int *picks_host, int *picks,
                                                       const float *w_host, float *w, int np) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < nx) x[i] = x_host[i];
    else if (i < nx + np) picks[i - nx] = picks_host[i - nx];
    else if (i < nx + 2 * np) w[i - nx - np] = w_host[i - nx - np];
}

__global__ void __launch_bounds__(256) rank_sum_kernel(const float *__restrict__ gathered, int world, size_t n,
                                                       float *__restrict__ out) {
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    float4 acc = *reinterpret_cast<const float4 *>(gathered + i);
    for (int k = 1; k < world; ++k) {
        const float4 v = *reinterpret_cast<const float4 *>(gathered + (size_t)k * n + i);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    *reinterpret_cast<float4 *>(out + i) = acc;
}

int launch_combine(cudaStream_t s, const float *Y, const int *picks, const float *route_w, float *out, int rows,
                   const glmflash_config &c) {
    const dim3 grid((unsigned)((c.hidden / 4 + 255) / 256), (unsigned)rows);
    return launch_k(combine_kernel, grid, dim3(256), 0, s, c.pdl != 0, Y, picks, route_w, out, c.slots, c.hidden, c.experts,
                     c.shared_exl3, c.expert_lo, c.expert_hi, c.shared_row_lo, c.shared_row_hi);
}
}  // namespace gf

using namespace gf;

bool gf::one_launch_selected() {
    const char *env = getenv("GLMFLASH_LAYER_KERNELS");
    return env && env[0] == '1';
}

// Calls up to this many rows go to the streamed kernel on a handle for more than 16.  Windows of up to 16 always do, as on a handle of their
// own: one launch, and the bytes do not depend on the handle (us a layer, streamed | GEMMs: 16 experts of 2048 x 1536, top-6: 1 row 26 | 56, 16
// rows 61 | 83; 384 of 1024 x 1024, top-8: 21 | 56 and 105 | 152; 8 of 2048 x 768, top-8: 25 | 52 and 42 | 53; behind the GEMMs where a row
// takes all of 16 experts: 1024 x 1024, 30 | 48 and 66 | 49).  For longer ones the kernel decodes an expert's weights once per 16 of its rows
// and adds partial sums for every row (the GEMMs: once per 320, for a fixed 35 us of kernels in front and behind, which weigh the more rows
// the smaller an expert is).  us a layer, streamed | GEMMs, and the rows per routed expert where the lines cross:
//   2048 x 1536, 64 experts, top-4: 64 rows 190 | 195, 80: 204 | 204, 128: 253 | 210     5.0     512 x 1024, 16, top-6: 24: 39 | 40, 32: 45 | 40     9.7
//   2304 x 2048, 32, top-4: 44: 160 | 161, 52: 171 | 161     5.6                           1024 x 512, 48, top-5: 100: 65 | 70, 128: 75 | 70     12
//   3072 x 1024, 16, top-2: 40: 71 | 73, 48: 74 | 74     5.8                               1536 x 256, 30, top-2: 96: 42 | 57, 128: 50 | 60     > 8.5
//   1024 x 2048, 24, top-3: 54: 79 | 82, 64: 86 | 82     7.3                               512 x 512, 32, top-3: 60: 34 | 38, 90: 43 | 42     8.2
//   1536 x 768, 100, top-5: 112: 140 | 149, 128: 150 | 150     6.4                         512 x 256, 64, top-8: 40: 34 | 40, 60: 42 | 41     7.2
// Hence 4.5 + 3 * 2^20 / (hidden * inter) rows per routed expert, 8 at most; at most 128 rows, and none above 16 where the exchange areas, which
// grow with the rows, would pass 256 MB.  With many experts the chunk's tables leave no room for the second CTA of an SM, and the GEMMs win earlier
// (4096 x 512, 288 experts, top-8: 18 rows, the last of two CTAs, 200 | 263, 19: 259 | 266, 24: 307 | 292, 40: 417 | 388; 1024 x 1024, 128,
// top-8: 60: 132 | 147, 80: 200 | 152).
static int short_chunk_rows(const glmflash_config &c) {
    const double per_expert = std::min(8., 4.5 + (3 << 20) / ((double)c.hidden * c.inter));
    size_t rows = std::min<size_t>({(size_t)c.max_rows, ST_MAX_ROWS, (size_t)(per_expert * c.experts / (c.slots - 1)), ((size_t)256 << 20) / stream_chunk_row_bytes(c)});
    while (rows > 16 && !stream_chunk_pairs(c, (int)rows)) --rows;
    return (int)std::max<size_t>(rows, 16);
}

struct glmflash_moe {
    glmflash_config cfg;
    glmflash_grouping *grouping = nullptr;
    glmflash_experts *experts = nullptr;            // windows of <= 16 rows
    glmflash_fast_experts *fast = nullptr;          // chunks of > 16 rows
    glmflash_experts *chunk = nullptr;              // beside them: the streamed kernel's buffers for calls of up to chunk_rows rows
    int chunk_rows = 0;
    void *pool = nullptr;                           // the one allocation behind the buffers below
    float *out = nullptr;
    void *in_dev = nullptr;                         // staging for run_host
    int *picks_dev = nullptr;
    float *w_dev = nullptr;
    int phases = 31;                                // profiling aid, see glmflash_moe_set_phases
    bool one_launch = false;                        // windows of <= 16 rows: the one-launch layer kernel (window.cu)
};

extern "C" int glmflash_moe_new(const glmflash_config *cfg, size_t cfg_bytes, glmflash_moe **out) {
    GF_REQUIRE(out != nullptr, "out is null");
    *out = nullptr;
    if (check_config(cfg, cfg_bytes, 8192)) return -1;
    glmflash_moe *m = new (std::nothrow) glmflash_moe();
    GF_REQUIRE(m != nullptr, "out of host memory");
    m->cfg = *cfg;
    int rc;                                         // (the window kernel groups its rows itself)
    if (cfg->max_rows <= 16) rc = glmflash_experts_new(cfg, cfg_bytes, &m->experts);
    else if (!(rc = glmflash_grouping_new(cfg, cfg_bytes, &m->grouping)) && !(rc = glmflash_fast_experts_new(cfg, cfg_bytes, &m->fast))) {
        m->chunk_rows = short_chunk_rows(*cfg);
        glmflash_config cc = *cfg;
        cc.max_rows = m->chunk_rows;
        cc.shared_row_lo = cc.shared_row_hi = 0;
        rc = experts_new(&cc, sizeof(cc), ST_MAX_ROWS, &m->chunk);
        if (!rc)                                    // (the row window counts rows of the chunk, whatever the owner holds)
            m->chunk->cfg.shared_row_lo = cfg->shared_row_lo, m->chunk->cfg.shared_row_hi = cfg->shared_row_hi;
    }
    const size_t rows = cfg->max_rows;
    Pool pool;
    pool.take(&m->out, rows * cfg->hidden * 4);
    pool.take(&m->in_dev, rows * cfg->hidden * 2);
    pool.take(&m->picks_dev, rows * cfg->slots * 4);
    pool.take(&m->w_dev, rows * cfg->slots * 4);
    if (rc || pool.alloc(&m->pool)) {
        glmflash_moe_free(m);
        return -1;
    }
    m->one_launch = one_launch_selected();
    *out = m;
    return 0;
}

extern "C" void glmflash_moe_free(glmflash_moe *m) {
    if (!m) return;
    glmflash_grouping_free(m->grouping);
    glmflash_experts_free(m->experts);
    glmflash_fast_experts_free(m->fast);
    glmflash_experts_free(m->chunk);
    cudaFree(m->pool);
    delete m;
}

extern "C" int glmflash_moe_run(glmflash_moe *m, void *stream, const glmflash_weights *w, const void *input, int x_stride,
                                const int32_t *picks, const float *route_w, int rows) {
    GF_REQUIRE(m && w && input && picks && route_w, "null argument");
    GF_REQUIRE(rows > 0 && rows <= m->cfg.max_rows, "rows outside the scratch bound");
    const float *Y;
    if (m->experts && m->one_launch && m->phases == 31 && experts_window_supported(m->cfg, rows))
        // windows of <= 16 rows: grouping, rotation, both projections, epilogues and the combine in one launch
        return experts_run_window(m->experts, (cudaStream_t)stream, w, input, x_stride, picks, route_w, rows, m->out, nullptr, -1);
    if (m->experts) {
        // one streamed launch: grouping, input rotation, both projections, epilogues and the combine
        return experts_run_fused(m->experts, (cudaStream_t)stream, w, input, x_stride, picks, route_w, m->phases & 16 ? m->out : nullptr, nullptr, rows,
                                 nullptr, nullptr);
    } else if (rows <= m->chunk_rows && (m->phases | 16) == 31) {
        // a window or a short chunk on a handle for more rows: the streamed kernel as well, its pair rows and status word those of
        // the chunk owner
        return experts_run_fused(m->chunk, (cudaStream_t)stream, w, input, x_stride, picks, route_w, m->phases & 16 ? m->out : nullptr, nullptr, rows,
                                 glmflash_fast_experts_output(m->fast), fast_experts_status_word(m->fast));
    } else {
        if ((m->phases & 1) && glmflash_grouping_run(m->grouping, stream, picks, rows)) return -1;
        const int32_t *ids = glmflash_grouping_ids(m->grouping), *count = glmflash_grouping_count(m->grouping),
                      *members = glmflash_grouping_members(m->grouping);
        // calls as short as some that the streamed kernel serves are as exact as there (the tables are of this call: no expert has more members
        // than it has rows)
        if (fast_experts_run(m->fast, stream, w, input, x_stride, picks, ids, count, members, rows, m->cfg.max_rows, w->suh_g == w->suh_u,
                             (m->phases & 1) != 0))
            return -1;
        Y = glmflash_fast_experts_output(m->fast);
    }
    if (!(m->phases & 16)) return 0;
    return launch_combine((cudaStream_t)stream, Y, picks, route_w, m->out, rows, m->cfg);
}

// Expert-parallel form of glmflash_moe_run.  Windows of <= 16 rows: the layer kernel itself pushes each finished block
// of this rank's partial into every peer's receive slot and adds the ranks' slots in rank order (one launch per
// layer and rank); larger windows: the experts of this rank, then the exchange kernel of the owner.
extern "C" int glmflash_moe_run_ep(glmflash_moe *m, glmflash_ep *ep, void *stream, const glmflash_weights *w, const void *input,
                                   int x_stride, const int32_t *picks, const float *route_w, int rows, int shared_here) {
    GF_REQUIRE(m && ep && w && input && picks && route_w, "null argument");
    GF_REQUIRE(rows > 0 && rows <= m->cfg.max_rows, "rows outside the scratch bound");
    if (m->experts && m->one_launch && experts_window_supported(m->cfg, rows)) {
        WinPeers peers;
        float *result = nullptr;
        if (ep_window_peers(ep, &peers, &result)) return -1;
        GF_REQUIRE(peers.max_rows == m->cfg.max_rows, "the layer owner and the exchange owner were built for different row counts");
        return experts_run_window(m->experts, (cudaStream_t)stream, w, input, x_stride, picks, route_w, rows, result,
                                  peers.world > 1 ? &peers : nullptr, shared_here);
    }
    const int shared = shared_here < 0 ? m->cfg.shared_exl3 : shared_here;
    GF_REQUIRE((shared == 2) == (m->cfg.shared_exl3 == 2),
               "the shared expert's owner is decided per window (2) either by both the layer owner and the call, or by neither");
    const int saved = m->phases;
    m->phases &= ~16;                               // experts only: the combine is the exchange kernel's first step
    const int rc = glmflash_moe_run(m, stream, w, input, x_stride, picks, route_w, rows);
    m->phases = saved;
    if (rc) return -1;
    return glmflash_ep_combine(ep, stream, glmflash_moe_pairs(m), picks, route_w, rows, shared);
}

extern "C" int glmflash_moe_set_phases(glmflash_moe *m, int mask) {
    GF_REQUIRE(m != nullptr, "null argument");
    m->phases = mask;
    if (m->experts) return glmflash_experts_set_phases(m->experts, (mask >> 1) & 7);
    return 0;                                      // prefill pipeline: only grouping (1) and combine (16) are selectable here
}

extern "C" float *glmflash_moe_output(const glmflash_moe *m) { return m ? m->out : nullptr; }
extern "C" const int32_t *glmflash_moe_status(const glmflash_moe *m) {
    if (!m) return nullptr;
    return m->experts ? glmflash_experts_status(m->experts) : glmflash_fast_experts_status(m->fast);
}
extern "C" int glmflash_moe_clear_status(glmflash_moe *m, void *stream) {
    GF_REQUIRE(m != nullptr, "null argument");
    return m->experts ? glmflash_experts_clear_status(m->experts, stream) : glmflash_fast_experts_clear_status(m->fast, stream);
}
extern "C" const float *glmflash_moe_pairs(const glmflash_moe *m) {
    if (!m) return nullptr;
    return m->experts ? glmflash_experts_y(m->experts) : glmflash_fast_experts_output(m->fast);
}

// Whether kernels of the current device can read and write these host buffers where they are (pinned memory under unified
// addressing).
static bool device_reads(std::initializer_list<const void *> ptrs) {
    for (const void *p : ptrs) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (at.type != cudaMemoryTypeHost || at.devicePointer != p) return false;
    }
    return true;
}

extern "C" int glmflash_moe_run_host(glmflash_moe *m, void *stream, const glmflash_weights *w, const void *input_host,
                                     int x_stride, const int32_t *picks_host, const float *route_w_host, int rows,
                                     float *out_host) {
    GF_REQUIRE(m && w && input_host && picks_host && route_w_host && out_host, "null argument");
    GF_REQUIRE(rows > 0 && rows <= m->cfg.max_rows, "rows outside the scratch bound");
    GF_REQUIRE(x_stride == m->cfg.hidden, "run_host takes densely packed rows (x_stride == hidden)");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t H = m->cfg.hidden, S = m->cfg.slots;
    if (m->experts && !m->one_launch && m->phases == 31 && device_reads({input_host, picks_host, route_w_host, out_host}) &&
        ((uintptr_t)input_host | (uintptr_t)out_host) % 16 == 0) {
        // Windows of <= 16 rows in pinned memory: one kernel fetches all three inputs over the bus and the layer kernel stores the
        // finished rows to host memory beside the owner's.  Three copies in and one out are four trips through a copy engine,
        // each longer than its few KB take (8 rows: 112 us a call, of which the layer is half).
        const int nx = (int)((size_t)rows * H * 2 / 16), np = (int)(rows * S);
        if (launch_k(stage_in_kernel, dim3((unsigned)((nx + 2 * np + 255) / 256)), dim3(256), 0, s, m->cfg.pdl != 0, (const uint4 *)input_host,
                     (uint4 *)m->in_dev, nx, (const int *)picks_host, m->picks_dev, route_w_host, m->w_dev, np))
            return -1;
        if (experts_run_fused(m->experts, s, w, m->in_dev, x_stride, m->picks_dev, m->w_dev, m->out, out_host, rows, nullptr, nullptr)) return -1;
        GF_CUDA(cudaStreamSynchronize(s));
        return 0;
    }
    GF_CUDA(cudaMemcpyAsync(m->in_dev, input_host, (size_t)rows * H * 2, cudaMemcpyHostToDevice, s));
    GF_CUDA(cudaMemcpyAsync(m->picks_dev, picks_host, (size_t)rows * S * 4, cudaMemcpyHostToDevice, s));
    GF_CUDA(cudaMemcpyAsync(m->w_dev, route_w_host, (size_t)rows * S * 4, cudaMemcpyHostToDevice, s));
    if (glmflash_moe_run(m, stream, w, m->in_dev, x_stride, m->picks_dev, m->w_dev, rows)) return -1;
    GF_CUDA(cudaMemcpyAsync(out_host, m->out, (size_t)rows * H * 4, cudaMemcpyDeviceToHost, s));
    GF_CUDA(cudaStreamSynchronize(s));
    return 0;
}

extern "C" int glmflash_rank_sum(void *stream, const float *gathered, int world, int rows, int hidden, float *out) {
    GF_REQUIRE(gathered && out, "null argument");
    GF_REQUIRE(world >= 1 && rows >= 1 && hidden >= 4 && hidden % 4 == 0, "bad shape");
    const size_t n = (size_t)rows * hidden;
    rank_sum_kernel<<<(unsigned)((n / 4 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(gathered, world, n, out);
    GF_CUDA(cudaGetLastError());
    return 0;
}
