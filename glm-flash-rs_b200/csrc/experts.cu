// ExpertGpu: the decode / verify owner (upstream src/experts.rs:365-563) and the single-linear probe.
#include <algorithm>
#include <new>

#include "gemv.cuh"
#include "owners.cuh"
#include "stream.cuh"

namespace gf {
size_t experts_window_sync_words(const glmflash_config &c);

int check_config(const glmflash_config *cfg, size_t cfg_bytes, int max_rows_limit) {
    GF_REQUIRE(cfg != nullptr, "config is null");
    GF_REQUIRE(cfg_bytes == sizeof(glmflash_config), "config size mismatch (ABI)");
    GF_REQUIRE(cfg->hidden > 0 && cfg->hidden % 256 == 0, "hidden must be a positive multiple of 256");
    GF_REQUIRE(cfg->inter > 0 && cfg->inter % 256 == 0, "inter must be a positive multiple of 256");
    GF_REQUIRE(cfg->experts > 0 && cfg->experts < 1024, "experts must be in 1..1023");
    GF_REQUIRE(cfg->slots >= 2 && cfg->slots <= 32, "slots must be in 2..32");
    GF_REQUIRE(cfg->max_rows >= 1 && cfg->max_rows <= max_rows_limit, "max_rows outside the scratch bound");
    GF_REQUIRE(cfg->expert_lo >= 0 && cfg->expert_hi <= cfg->experts && cfg->expert_lo <= cfg->expert_hi,
               "expert window must satisfy 0 <= lo <= hi <= experts");
    GF_REQUIRE(cfg->limit > 0.f, "limit must be positive");
    GF_REQUIRE(cfg->shared_exl3 >= 0 && cfg->shared_exl3 <= 2, "shared_exl3 must be 0, 1 or 2");
    if (cfg->shared_exl3 == 2) {
        const int W = cfg->expert_hi - cfg->expert_lo;
        GF_REQUIRE(cfg->max_rows <= 16, "shared_exl3 = 2 (owner decided per window) is for handles of <= 16 rows");
        GF_REQUIRE(W > 0 && cfg->expert_lo % W == 0 && (cfg->experts + W - 1) / W <= 32,
                   "shared_exl3 = 2 needs equal contiguous expert windows (expert_lo a multiple of the window size, at most 32 ranks)");
    }
    GF_REQUIRE(cfg->shared_row_lo >= 0 && cfg->shared_row_lo <= cfg->shared_row_hi, "shared-expert row window must satisfy 0 <= lo <= hi");
    GF_REQUIRE(cfg->shared_row_hi == 0 || cfg->max_rows > 16, "a shared-expert row window needs a handle for more than 16 rows");
    int dev_count = 0;
    if (cudaGetDeviceCount(&dev_count) != cudaSuccess || dev_count == 0) return fail("no CUDA device: there is no CPU path");
    return 0;
}

}  // namespace gf

using namespace gf;

// max_rows_limit: 16 for the public owner.  Chunk owners keep one for their windows and short chunks, whose pair rows are the chunk owner's and
// whose down inputs nobody reads afterwards.
int gf::experts_new(const glmflash_config *cfg, size_t cfg_bytes, int max_rows_limit, glmflash_experts **out) {
    GF_REQUIRE(out != nullptr, "out is null");
    *out = nullptr;
    if (check_config(cfg, cfg_bytes, max_rows_limit)) return -1;
    glmflash_experts *e = new (std::nothrow) glmflash_experts();
    GF_REQUIRE(e != nullptr, "out of host memory");
    e->cfg = *cfg;
    const size_t H = cfg->hidden, I = cfg->inter, P = (size_t)cfg->max_rows * cfg->slots;
    Pool pool;
    if (max_rows_limit <= 16) {
        pool.take(&e->xd, P * I * 2);
        pool.take(&e->y, P * H * 4);
    }
    pool.take(&e->status, 4);
    pool.take(&e->ll_z1, stream_z1_words(*cfg) * 8);
    pool.take(&e->ll_z2, stream_z2_words(*cfg) * 8);
    pool.take(&e->ll_xr, stream_xr_words(*cfg) * 8);
    pool.take(&e->ll_xd, stream_xdl_words(*cfg) * 8);
    pool.take(&e->ctrl, CTRL_WORDS * 4);
    if (max_rows_limit <= 16 && one_launch_selected()) {                         // scratch of the alternative layer kernel (window.cu)
        e->sync_words = experts_window_sync_words(*cfg);
        pool.take(&e->z1, (size_t)2 * (H / 128) * P * I * 4);
        pool.take(&e->z2, (size_t)(I / 128) * P * H * 4);
        pool.take(&e->sync, e->sync_words * 4);
    }
    if (pool.alloc(&e->pool)) {
        glmflash_experts_free(e);
        return -1;
    }
    *out = e;
    return 0;
}

extern "C" int glmflash_experts_new(const glmflash_config *cfg, size_t cfg_bytes, glmflash_experts **out) {
    return experts_new(cfg, cfg_bytes, 16, out);              // upstream: 1..=MAX_ROWS (16), src/experts.rs:391-394
}

extern "C" void glmflash_experts_free(glmflash_experts *e) {
    if (!e) return;
    cudaFree(e->pool);
    delete e;
}

// Fills in what both forms of a window share and launches it.
static int run_stream(const glmflash_experts *e, cudaStream_t s, StreamArgs a, const glmflash_weights *w, const void *input, int x_stride, int rows) {
    const glmflash_config &c = e->cfg;
    GF_REQUIRE(((uintptr_t)w->gt | (uintptr_t)w->ut | (uintptr_t)w->dt) % 16 == 0, "trellis tensors must be 16-byte aligned");
    GF_REQUIRE(((uintptr_t)input) % 8 == 0, "input must be 8-byte aligned");
    a.vec = ((uintptr_t)w->suh_g | (uintptr_t)w->suh_u | (uintptr_t)w->suh_d | (uintptr_t)w->svh_g | (uintptr_t)w->svh_u | (uintptr_t)w->svh_d) % 8 == 0;
    a.gt = w->gt; a.ut = w->ut; a.dt = w->dt;
    a.suh_g = (const __half *)w->suh_g; a.suh_u = (const __half *)w->suh_u; a.suh_d = (const __half *)w->suh_d;
    a.svh_g = (const __half *)w->svh_g; a.svh_u = (const __half *)w->svh_u; a.svh_d = (const __half *)w->svh_d;
    a.x = (const __nv_bfloat16 *)input; a.x_stride = x_stride;
    a.z1 = e->ll_z1; a.z2 = e->ll_z2; a.xr = e->ll_xr; a.xdl = e->ll_xd; a.xd = e->xd;
    if (!a.y) a.y = e->y;
    a.ctrl = e->ctrl;
    if (!a.status) a.status = e->status;
    a.H = c.hidden; a.I = c.inter; a.rows = rows; a.slots = c.slots; a.E = c.experts;
    a.e_lo = c.expert_lo; a.e_hi = c.expert_hi; a.shared = c.shared_exl3; a.limit = c.limit;
    a.srow_lo = c.shared_row_lo; a.srow_hi = c.shared_row_hi;
    a.cut1 = stream_cut(c.hidden, rows > 16);
    a.cut2 = stream_cut(c.inter, rows > 16);
    a.umax = stream_umax(c, rows, a.picks == nullptr);
    a.do_g = (e->phases & 2) != 0;
    a.do_d = (e->phases & 4) != 0;
    return launch_stream(s, a, c.pdl != 0);
}

extern "C" int glmflash_experts_run_rows(glmflash_experts *e, void *stream, const glmflash_weights *w, const void *input,
                                         int x_stride, const int32_t *picks, const int32_t *ids, const int32_t *count,
                                         const int32_t *members, int rows, int maxm) {
    GF_REQUIRE(e && w && input && picks && ids && count && members, "null argument");
    const glmflash_config &c = e->cfg;
    GF_REQUIRE(c.shared_exl3 != 2, "shared_exl3 = 2 (owner decided per window) is served by the layer calls, not by run_rows");
    GF_REQUIRE(rows > 0 && rows <= c.max_rows && maxm >= rows && maxm <= c.max_rows, "expert verifier row/member bounds");
    GF_REQUIRE(x_stride >= c.hidden && x_stride % 4 == 0, "x_stride must be >= hidden and a multiple of 4");
    StreamArgs a{};
    a.ids = ids; a.count = count; a.members = members; a.maxm = maxm;
    return run_stream(e, (cudaStream_t)stream, a, w, input, x_stride, rows);
}

// The layer pipeline's form (used by Moe for windows of <= 16 rows): expert and members come from the routing table, and with
// `out` the rows are combined in the same launch.
namespace gf {
int experts_run_fused(glmflash_experts *e, cudaStream_t s, const glmflash_weights *w, const void *input, int x_stride,
                      const int32_t *picks, const float *route_w, float *out, float *out2, int rows, float *y, int *status) {
    const glmflash_config &c = e->cfg;
    GF_REQUIRE(rows > 0 && rows <= c.max_rows, "expert verifier row/member bounds");
    GF_REQUIRE(x_stride >= c.hidden && x_stride % 4 == 0, "x_stride must be >= hidden and a multiple of 4");
    StreamArgs a{};
    a.picks = picks; a.route_w = route_w; a.out = out; a.out2 = out2; a.y = y; a.status = status;
    return run_stream(e, s, a, w, input, x_stride, rows);
}
}  // namespace gf

extern "C" int glmflash_experts_set_phases(glmflash_experts *e, int mask) {
    GF_REQUIRE(e != nullptr, "null argument");
    e->phases = mask;
    return 0;
}

extern "C" float *glmflash_experts_y(const glmflash_experts *e) { return e ? e->y : nullptr; }
extern "C" const uint16_t *glmflash_experts_xd(const glmflash_experts *e) { return e ? (const uint16_t *)e->xd : nullptr; }
extern "C" const int32_t *glmflash_experts_status(const glmflash_experts *e) { return e ? e->status : nullptr; }
extern "C" int glmflash_experts_clear_status(glmflash_experts *e, void *stream) {
    GF_REQUIRE(e != nullptr, "null argument");
    // a give-up may have left arrival counters of the one-launch kernel half way: clear them with the status word
    GF_CUDA(cudaMemsetAsync(e->status, 0, 4, (cudaStream_t)stream));
    if (e->sync) GF_CUDA(cudaMemsetAsync(e->sync, 0, e->sync_words * 4, (cudaStream_t)stream));
    return 0;
}
