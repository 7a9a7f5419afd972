// Launch interface of the streamed layer kernel (stream.cu).
#pragma once
#include "common.cuh"

namespace gf {

// Counters of an owner, 512 bytes apart: every CTA of a launch draws from the first two and reads the last at the same moment,
// and in one line the reads queue behind four hundred atomics (3,000 clocks at the head of every layer).
enum : int { CTRL_UNIT = 0, CTRL_FIN = 128, CTRL_DONE = 256, CTRL_EPOCH = 384, CTRL_WORDS = 512 };

struct StreamArgs {
    const uint32_t *gt, *ut, *dt;                            // trellis banks
    const __half *suh_g, *suh_u, *suh_d, *svh_g, *svh_u, *svh_d;
    const __nv_bfloat16 *x;                                  // layer input [rows][x_stride]
    const int *picks;                                        // routing table [rows][slots], or nullptr with the grouping tables
    const int *ids, *count, *members;                        // (used when picks == nullptr; members [.][maxm])
    const float *route_w;                                    // [rows][slots] for the combine
    unsigned long long *z1, *z2, *xr, *xdl;                  // {value, epoch} words: gate / up and down partials, their inputs
    __half *xd;                                              // plain down inputs [P][I]
    float *y, *out, *out2;                                   // pair results [P][H]; combined rows [rows][H] (out2: a second copy) or nullptr
    unsigned *ctrl;                                          // CTRL_WORDS
    int *status;
    int H, I, rows, x_stride, slots, maxm, E, e_lo, e_hi, shared, srow_lo, srow_hi, umax;
    float limit;
    int vec;                                                 // the scale vectors are 8-byte aligned
    int do_g, do_d;                                          // profiling aid: the phases to run
};

// 8-byte words of the three exchange areas of an owner
inline size_t stream_z1_words(const glmflash_config &c) {
    return (size_t)2 * ((c.hidden + 511) / 512) * c.max_rows * c.slots * c.inter;
}
inline size_t stream_z2_words(const glmflash_config &c) { return (size_t)((c.inter + 511) / 512) * c.max_rows * c.slots * c.hidden; }
inline size_t stream_xr_words(const glmflash_config &c) { return (size_t)c.max_rows * c.slots * c.hidden; }
inline size_t stream_xdl_words(const glmflash_config &c) { return (size_t)c.max_rows * c.slots * c.inter / 2; }

// Most rows of a chunk that the kernel takes (its tables live in shared memory and its exchange areas grow with the rows).
constexpr int ST_MAX_ROWS = 128;
int launch_stream(cudaStream_t s, const StreamArgs &a, bool pdl);

}  // namespace gf
