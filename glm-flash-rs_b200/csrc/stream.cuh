// Launch interface of the streamed layer kernel (stream.cu).
#pragma once
#include "common.cuh"

namespace gf {

// Counters of an owner, 512 bytes apart: every CTA of a launch draws from the first two and reads the last at the same moment,
// and in one line the reads queue behind four hundred atomics (3,000 clocks at the head of every layer).
enum : int { CTRL_UNIT = 0, CTRL_FIN = 128, CTRL_DONE = 256, CTRL_EPOCH = 384, CTRL_WORDS = 512 };

// How k is cut: a partial sum is a chain over `split` k-tiles (the last one may be shorter).
struct StreamCut {
    int split, splits;                                       // k-tiles of a split, number of splits
};
// Windows of up to 16 rows: at most eight splits, 256 k each where that suffices, else the next power of two that divides K, else the
// largest number of equal splits of whole 128-k blocks (K = 2304: six of 384).  A K that has no such split of at most 1024 k (3328) is
// cut into 256 k.  Chunks of more than 16 rows are cut into 512 k: half the exchange, which grows with the rows, and with sixteen
// products an instruction as many roundings a partial as 256 k have with eight.
inline StreamCut stream_cut(int K, bool chunk) {
    const int KT = K / 16;
    StreamCut c{16, 0};
    while (KT / c.split > 8) c.split *= 2;
    if (KT % c.split)
        for (int n = 8; n >= 1; --n)
            if (KT % n == 0 && KT / n % 8 == 0) { c.split = KT / n; break; }
    if (c.split > 64) c.split = 16;
    if (chunk) c.split = 32;
    c.splits = (KT + c.split - 1) / c.split;
    return c;
}

struct StreamArgs {
    const uint32_t *gt, *ut, *dt;                            // trellis banks
    const __half *suh_g, *suh_u, *suh_d, *svh_g, *svh_u, *svh_d;
    const __nv_bfloat16 *x;                                  // layer input [rows][x_stride]
    const int *picks;                                        // routing table [rows][slots], or nullptr with the grouping tables
    const int *ids, *count, *members;                        // (used when picks == nullptr; members [.][maxm])
    const float *route_w;                                    // [rows][slots] for the combine
    unsigned long long *z1, *z2, *xr, *xdl;                  // {value, epoch} words: gate / up and down partials, their inputs
    __half *xd;                                              // plain down inputs [P][I], or nullptr
    float *y, *out, *out2;                                   // pair results [P][H]; combined rows [rows][H] (out2: a second copy) or nullptr
    unsigned *ctrl;                                          // CTRL_WORDS
    int *status;
    int H, I, rows, x_stride, slots, maxm, E, e_lo, e_hi, shared, srow_lo, srow_hi, umax;
    StreamCut cut1, cut2;                                    // of the gate / up and the down matrix
    float limit;
    int vec;                                                 // the scale vectors are 8-byte aligned
    int two;                                                 // two CTAs share an SM (set by launch_stream)
    int do_g, do_d;                                          // profiling aid: the phases to run
};

// 8-byte words of the exchange areas of an owner; its windows of up to 16 rows and its chunks are cut differently
inline size_t stream_split_rows(const glmflash_config &c, int K) {
    const size_t window = (size_t)stream_cut(K, false).splits * (c.max_rows < 16 ? c.max_rows : 16);
    const size_t chunk = c.max_rows > 16 ? (size_t)stream_cut(K, true).splits * c.max_rows : 0;
    return window > chunk ? window : chunk;
}
inline size_t stream_z1_words(const glmflash_config &c) { return 2 * stream_split_rows(c, c.hidden) * c.slots * c.inter; }
inline size_t stream_z2_words(const glmflash_config &c) { return stream_split_rows(c, c.inter) * c.slots * c.hidden; }
// bytes of them that a row of a chunk costs
inline size_t stream_chunk_row_bytes(const glmflash_config &c) {
    return (size_t)8 * c.slots * ((size_t)2 * stream_cut(c.hidden, true).splits * c.inter + (size_t)stream_cut(c.inter, true).splits * c.hidden + c.hidden + c.inter / 2);
}
inline size_t stream_xr_words(const glmflash_config &c) { return (size_t)c.max_rows * c.slots * c.hidden; }
inline size_t stream_xdl_words(const glmflash_config &c) { return (size_t)c.max_rows * c.slots * c.inter / 2; }

// Most rows of a chunk that the kernel takes (its tables live in shared memory and its exchange areas grow with the rows).
constexpr int ST_MAX_ROWS = 128;
// Most entries of the tables: distinct experts that this GPU computes (at most one per pick, and at most its window and the shared
// one; with the grouping's tables the places in ids, skipped ones included), and for chunks one more for every 16 members.
inline int stream_umax(const glmflash_config &c, int rows, bool tables) {
    const int here = tables ? c.experts + 1 : (c.expert_hi - c.expert_lo) + (c.shared_exl3 ? 1 : 0), picks = rows * c.slots;
    const int distinct = picks < here ? picks : here;
    return (distinct > 1 ? distinct : 1) + (rows > 16 ? picks / 16 : 0);
}
bool stream_chunk_pairs(const glmflash_config &c, int rows);
int launch_stream(cudaStream_t s, StreamArgs a, bool pdl);

}  // namespace gf
