// FastExperts: the prefill owner (upstream src/fast_experts.rs:27-208) as two persistent grouped GEMMs on the
// 5th-generation tensor cores (tcgen05.mma, accumulators in tensor memory), sm_100a only.
//
// Replaces upstream's fast_rot_in / fast_expert_plan / fast_gu_shared / fast_gu_separate / fast_down /
// fast_down_large (native/exl3_prefill.cu:402-430,657-889), which decode each 16x16 trellis tile into mma.sync
// fragments in registers.  Here:
//
//   plan      members per distinct expert, chunks of at most 320 or 160 rows (as even as an expert's rows go, long ones first) and the
//             GROUPED row order (rows of an expert contiguous): src_pair[j] = pair index of grouped row j.
//   rot       the input rotation writes Xs[j] = fp16(H(x[row] * suh[e]) / sqrt 128) in grouped order, so the rows of a chunk are
//             a contiguous slab that TMA tensor loads bring into shared memory in the 128-byte-swizzled K-major layout the tensor
//             core reads.
//   gemm      persistent PAIRS of CTAs (74 clusters of two), one CTA per SM, 28 warps.  A work item is (chunk, pair of 128-column
//             blocks).  The decoded weights are the M operand and live in TENSOR MEMORY, the rows are N, only as many as there are
//             (in 32): tcgen05.mma.cta_group::2, M 256 x N <= 256 x K 16 -- each CTA decodes one of the two column blocks and brings half of
//             the rows, and holds its columns' accumulators of all rows.  Roles:
//               warp 0       TMA producer of the rows (half of the chunk's x 128 k per stage)
//               warp 1       first CTA: issues the MMAs of the pair, commits stages and passes to both CTAs.  It waits for one barrier a
//                            stage, on which the rows' bytes and the decode warps of both CTAs count
//               warp 2       allocates / frees tensor memory (512 columns)
//               warp 3       TMA producer of the packed words, a ring of its own
//               warps 4-11   epilogue: 32 rows x 128 columns at a time from tensor memory, transposed through shared memory so that four
//                            lanes hold a row; the 128-point Hadamard transform, scales, limited SwiGLU, down-input rotation;
//                            fp16 Xd rows (gate/up) or fp32 Y rows (down)
//               warps 12-27  decode the trellis tiles (bit-exact codebook) in registers and store them to tensor memory (tcgen05.st):
//                            the places of a word's weights are those that the instruction gives a lane
//             The gate and the up projection of an item are two PASSES over K with their own accumulators: while the up pass
//             runs, the epilogue warps turn the gate accumulators into silu(gate) (kept as bf16 in the places of Xd), and the up pass's
//             epilogue overlaps the next item's gate pass.  Down is one pass per item.
//             Before, the rows were M (256 a tile, filled or not) and the weights went through shared memory: a chunk of 40 rows cost as
//             much as one of 256, an expert of 257 rows twice as much as one of 256.  us gate/up | down, before -> now: 500 rows 197 | 101
//             -> 127 | 66, 4096 rows 350 | 181 -> 277 | 137, eight experts of 64 at 4096 rows 81 | 39 -> 49 | 33 (2048 x 1536, 64 experts,
//             top-4); 8192 rows of 4096 x 512, 288 experts, top-8: 587 | 697 -> 540 | 505.  What bounds it now: instruction issue (0.70 to 0.80 of the
//             cycles while all SMs work: decode, epilogue) and the last round of items (0.82 to 0.87 of the time); short K (512): the
//             epilogue, which a pass of four stages does not cover.
//             Tried: more epilogue warps (three warpgroups of 104 registers 309 against 280 us at 4096 rows; four and eight decode warps for
//             down 157 against 139, 8192 rows 687 against 530), the words' copies prefetched to L2 a pass ahead and deeper rings of rows
//             or words (no change; two stages of words: 190 against 143 at 500 rows), stages of 64 k (158 | 83 at 500 rows: the same steps
//             for half the work), silu(gate) in shared memory (chunks of 256 rows then: 314 | 157 at 4096), down's rows out by bulk copies (640
//             against 530 at 8192 rows).
// Arithmetic: one full-K fp32 accumulation chain per output (as upstream's prefill path, which is likewise not
// bit-equal to its decode path: native/exl3_prefill.cu:20-23), the same transforms and rounding points as
// upstream's epilogue (native/exl3_prefill.cu:596-622 == native/exl3.cu:260-321) with exp / divide in their fast
// forms; short calls of the layer in finer steps (FINE).  Deterministic: static work assignment, no atomics; every pair's result depends only
// on its own row.
// Every wait is bounded; a wait that gives up raises the abort flag, every role leaves its loops, tensor memory
// is freed and the status word reports the failure.
#include <cuda.h>

#include <algorithm>
#include <new>

#include "gemv.cuh"

namespace gf {
int check_config(const glmflash_config *cfg, size_t cfg_bytes, int max_rows_limit);
int *fast_experts_status_word(glmflash_fast_experts *f);
int fast_experts_run(glmflash_fast_experts *f, void *stream, const glmflash_weights *w, const void *input, int x_stride, const int32_t *picks,
                     const int32_t *ids, const int32_t *count, const int32_t *members, int rows, int maxm, int shared_x, bool fine);

constexpr int FG_DEC = 16;                                 // trellis-decode warps
constexpr int FG_THREADS = (12 + FG_DEC) * 32;
constexpr int FG_BN = 128, FG_BK = 128;                    // columns of a CTA, k of a stage
constexpr int FG_CHUNK = 320;                              // most rows of a work item
constexpr int FG_FINE_ROWS = 128;                          // most rows of a call with partial sums (FINE)
constexpr int FG_CHAIN = 512 / FG_BK;                      // stages of one of them
constexpr int FG_BOXES = 8;                                // boxes of rows that one copy takes: 16, 32, .. 128
constexpr int FG_HALF_BYTES = FG_CHUNK / 2 * 128;          // 20 KB: a CTA's rows x 64 k of fp16, half of a stage
constexpr int FG_TILE_BYTES = 2 * FG_HALF_BYTES;
constexpr int FG_WORD_BYTES = 8192;                        // packed words of a stage: 8 k-tiles x 8 n-tiles
constexpr int FG_MAXU = 1024;

// plan layout (int32): [0] 128-row tiles of all experts (informative), [1] total grouped rows, [2] chunks
constexpr int PLAN_INTS = 4;
// ---------------------------------------------------------------------------------------------- plan
// Launched with one block per bank entry: every block recomputes the (tiny) scans, block 0 publishes the plan,
// block b writes the grouped rows of distinct expert b.
__global__ void __launch_bounds__(FG_MAXU) fast_plan_kernel(const int *__restrict__ ids, const int *__restrict__ count,
                                                          const int *__restrict__ members, int maxm, int slots, int E,
                                                          int shared_exl3, int e_lo, int e_hi, int srow_lo, int srow_hi,
                                                          int *__restrict__ plan, int4 *__restrict__ chunks,
                                                          int *__restrict__ src_pair, int *__restrict__ row_expert, int nbp, int workers) {
    __shared__ int cnt_sh[FG_MAXU], row_sh[FG_MAXU], e_sh[FG_MAXU], first_sh[FG_MAXU], order_sh[FG_MAXU];
    __shared__ int wsum[3][32], at_sh, classes_sh[2][12], cost_sh[2];
    const int u = threadIdx.x, lane = u & 31, warp = u >> 5;
    if (u < 24) classes_sh[u / 12][u % 12] = 0;
    pdl_wait();                                             // (every kernel of the chain: nothing is read or written before)
    pdl_launch_dependents();
    const int n = min(count[0], FG_MAXU);
    int cnt = 0, e = -1, first = 0;
    if (u < n) {
        e = ids[u];
        if (!expert_skipped(e, E, shared_exl3, e_lo, e_hi)) {
            const int *m = members + (size_t)u * maxm;
            // the first place in [0, end) whose member is past something that the list does not come back from, else end.  Seven probes a
            // step: a list of 8192 takes five trips through L2 instead of thirteen
            auto first_past = [&](int end, auto past) {
                int lo = 0, hi = end;
                while (lo < hi) {
                    const int step = (hi - lo + 7) >> 3;    // probes at the ends of the first seven of eight parts
                    int below = 0;
#pragma unroll
                    for (int i = 1; i < 8; ++i) below += lo + i * step <= hi && !past(m[min(lo + i * step, hi) - 1]);
                    hi = below < 7 ? min(hi, lo + (below + 1) * step - 1) : hi;
                    lo = lo + below * step;
                }
                return lo;
            };
            cnt = first_past(maxm, [](int code) { return code < 0; });       // members come first, then -1
            if (e == E && srow_hi > srow_lo) {
                // the shared expert is computed here for a window of rows only: members ascend by row (code = row * 32
                // + slot), so the window is a contiguous run of the list
                first = first_past(cnt, [=](int code) { return (code >> 5) >= srow_lo; });
                cnt = first_past(cnt, [=](int code) { return (code >> 5) >= srow_hi; }) - first;
            }
        }
    }
    // Chunks of at most 320 rows, or of 160: twice as many decode the weights twice, but a few long ones (the shared expert's, at 500 rows)
    // hold up their pairs: 135 against 128 us (gate / up), at 4096 rows 284 against 344.  What the gate / up items cost the pairs that
    // have the longest of every turn, in clocks a stage: 1,000 for the decode or 4.4 a row for the MMAs.  Both constants are of 2048 x 1536, and
    // the down items have no say; with each cut forced (42 calls of eight shapes, 1024 x 256 to 2048 x 2048 and 4096 x 512, 8 to 288 experts, 200
    // to 8192 rows) the rule's is within 3 % of the better one, but for 200 to 400 rows of few experts, where it keeps 320 (16 experts of 2304 x
    // 768: 74 us against 66 and 79 | 74; 24 of 1024 x 2048: 91 | 82 and 97 | 92): there the last epilogue of the longest chunk counts as well.
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int cap = FG_CHUNK >> i, n_i = (cnt + cap - 1) / cap;
        if (n_i) atomicAdd(&classes_sh[i][((cnt + n_i - 1) / n_i + 31) >> 5], n_i);
    }
    __syncthreads();
    if (warp < 2) {
        const int *classes = classes_sh[warp];
        int all = 0, cost = 0;
        for (int k = 1; k <= FG_CHUNK / 32; ++k) all += classes[k];
        const int turns = (all * nbp + workers - 1) / workers;
        for (int t = lane; t < turns; t += 32) {
            const int place = t * workers / nbp;            // the turn's first chunk, and its class
            int k = FG_CHUNK / 32 + 1, longer = 0;
#pragma unroll
            for (int c = FG_CHUNK / 32; c >= 1; --c)
                if (longer <= place) { k = c; longer += classes[c]; }
            cost += max(1000, 141 * k);
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) cost += __shfl_xor_sync(0xffffffffu, cost, d);
        if (lane == 0) cost_sh[warp] = cost;
    }
    __syncthreads();
    const int cap = cost_sh[1] < cost_sh[0] ? FG_CHUNK / 2 : FG_CHUNK;
    // as even as they go, in the order of their length (in 32 rows, long ones first), so that the static round robin over the CTA pairs takes
    // about equal ones in a turn and ends with the short ones
    const int tiles = (cnt + 127) / 128, nch = (cnt + cap - 1) / cap, size = nch ? (cnt + nch - 1) / nch : 0;
    const int key = (size + 31) >> 5;
    // block-wide exclusive scan of rows, totals of tiles and chunks
    int r_inc = cnt, t_inc = tiles, c_inc = nch;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, r_inc, d), b = __shfl_up_sync(0xffffffffu, t_inc, d), c = __shfl_up_sync(0xffffffffu, c_inc, d);
        if (lane >= d) { r_inc += a; t_inc += b; c_inc += c; }
    }
    if (lane == 31) { wsum[0][warp] = r_inc; wsum[1][warp] = t_inc; wsum[2][warp] = c_inc; }
    order_sh[u] = key << 16 | nch;
    if (u == 0) at_sh = 0;
    __syncthreads();
    int r_off = 0, r_all = 0, t_all = 0, c_all = 0;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) r_off += wsum[0][w];
        r_all += wsum[0][w]; t_all += wsum[1][w]; c_all += wsum[2][w];
    }
    const int r_ex = r_off + r_inc - cnt;
    cnt_sh[u] = cnt; row_sh[u] = r_ex; e_sh[u] = e; first_sh[u] = first;
    if (u == 0 && blockIdx.x == 0) { plan[0] = t_all; plan[1] = r_all; plan[2] = c_all; }
    // chunks of this block's expert (there are at least as many blocks as experts): behind those of longer ones and of experts in front with as
    // long ones, counted by all threads
    const int b = blockIdx.x;
    if (b < n) {
        const int mine = order_sh[b] >> 16;
        int at = key > mine || (key == mine && u < b) ? nch : 0;
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) at += __shfl_xor_sync(0xffffffffu, at, d);
        if (lane == 0 && at) atomicAdd(&at_sh, at);
    }
    __syncthreads();
    if (u == b && u < n)
        for (int c = 0; c < nch; ++c) chunks[at_sh + c] = make_int4(e, r_ex + c * size, min(size, cnt - c * size), 0);
    for (int uu = blockIdx.x; uu < n; uu += gridDim.x) {
        const int c = cnt_sh[uu], rb = row_sh[uu], ee = e_sh[uu], f0 = first_sh[uu];
        for (int m = u; m < c; m += FG_MAXU) {
            const int code = members[(size_t)uu * maxm + f0 + m];
            src_pair[rb + m] = (code >> 5) * slots + (code & 31);
            row_expert[rb + m] = (code >> 5) << 10 | ee;
        }
    }
}

// ---------------------------------------------------------------------------------------------- rotation
// Four lanes hold a 128-block, 32 values each (columns 32 j + 8 t + i: 16-byte pieces, 64 contiguous bytes a block and instruction), so that five of
// the seven butterflies run in registers, from stride 2 on as packed fp32, and two across lanes.  The butterflies keep their order (stride
// 1..64).  A warp stays with eight blocks of one matrix and walks grouped rows: the sign / scale vector waits in registers as fp32 until the
// expert changes, and the next row's input is on its way meanwhile.
// What bounds it: issue slots and shuffles (about 8 instructions a value) and the trips for the next row; the writes alone take 30 and 90 us
// (6 TB/s).  With 16 values a lane, three butterflies across lanes and the vector read and converted for every row: 67 us at 4096 rows x 2048 x
// 5 pairs x 2 matrices (168 MB written) and 237 us at 8192 x 4096 x 8 x 1 (537 MB); now 53 and 160.  More warps with fewer registers spill
// (71 and 225), several waves of blocks change nothing.
// HALVES: the sign / scale vectors are 2-byte aligned only (the streamed kernel takes such vectors, and so do short calls here).
constexpr int ROT_WARPS = 4;
template <bool HALVES>
__global__ void __launch_bounds__(ROT_WARPS * 32, 4) fast_rot_kernel(const __nv_bfloat16 *__restrict__ x, int x_stride, const int *__restrict__ plan,
                                                                 const int *__restrict__ row_expert, const __half *__restrict__ suh0,
                                                                 const __half *__restrict__ suh1, __half *__restrict__ out0,
                                                                 __half *__restrict__ out1, int K, bool vec) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3, group = lane >> 2;
    const int KB = K >> 7, slices = (KB + 7) >> 3, per_warp = KB < 8 ? 8 / KB : 1;         // rows of a warp (short rows: several)
    const __half *suh = blockIdx.y ? suh1 : suh0;
    const float2 neg1 = make_float2(-1.f, -1.f);
    const int w = blockIdx.x * ROT_WARPS + warp, slice = w % slices, part = w / slices, parts = (int)gridDim.x * ROT_WARPS / slices;
    const int sub = KB < 8 ? group / KB : 0, blk = KB < 8 ? group - sub * KB : slice * 8 + group, k = blk * 128 + 8 * t;
    pdl_wait();
    pdl_launch_dependents();
    __half *out = blockIdx.y ? out1 : out0;
    const int rows = plan[1], size = (rows + parts - 1) / parts, end = min(rows, (part + 1) * size);
    const bool mine = blk < KB && sub < per_warp && part < parts;
    int j = part * size + sub, code = 0, next = 0, e = -1;
    uint4 xv[4];
    auto fetch = [&] {                                                     // row j's input (code: row and expert)
        if (!mine || j >= end) return;
        code = next;
        next = row_expert[min(j + per_warp, end - 1)];
        const __nv_bfloat16 *p = x + (size_t)(code >> 10) * x_stride + k;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (vec) xv[i] = *reinterpret_cast<const uint4 *>(p + 32 * i);
            else {
                const uint2 a = *reinterpret_cast<const uint2 *>(p + 32 * i), b = *reinterpret_cast<const uint2 *>(p + 32 * i + 4);
                xv[i] = make_uint4(a.x, a.y, b.x, b.y);
            }
        }
    };
    if (mine && j < end) next = row_expert[j];
    fetch();
    float2 sv[16];
    for (int first = part * size; first < end && part < parts; first += per_warp) {
        const bool here = mine && j < end;
        if (here && (code & 1023) != e) {
            e = code & 1023;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const __half *q = suh + (size_t)e * K + k + 32 * (i >> 2) + 2 * (i & 3);
                const uint32_t h = HALVES ? __half_as_ushort(__ldg(q)) | (uint32_t)__half_as_ushort(__ldg(q + 1)) << 16 : __ldg(reinterpret_cast<const uint32_t *>(q));
                sv[i] = __half22float2(*reinterpret_cast<const __half2 *>(&h));
            }
        }
        float2 v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {                                     // times the sign / scale vector, stride 1
            const uint32_t b = i & 2 ? (i & 1 ? xv[i >> 2].w : xv[i >> 2].z) : (i & 1 ? xv[i >> 2].y : xv[i >> 2].x);
            const float2 m = __fmul2_rn(make_float2(__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u)), sv[i]);
            v[i] = make_float2(m.x + m.y, m.x - m.y);
        }
        const int row = j;
        j += per_warp;
        fetch();
        auto in_lane = [&](int d) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (!(i & d)) {
                    const float2 a = v[i], b = v[i | d];
                    v[i] = __fadd2_rn(a, b);
                    v[i | d] = __ffma2_rn(b, neg1, a);
                }
        };
        in_lane(1);
        in_lane(2);
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) {                                  // strides 8, 16: lower + upper | lower - upper
            const float sg = t & d ? -1.f : 1.f;
            const float2 s2 = make_float2(sg, sg);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, v[i].x, d), __shfl_xor_sync(0xffffffffu, v[i].y, d));
                v[i] = __ffma2_rn(v[i], s2, o);
            }
        }
        in_lane(4);
        in_lane(8);
        if (here) {
            __half *o = out + (size_t)row * K + k;
            const float2 sc = make_float2(HAD_SCALE, HAD_SCALE);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 r = __fmul2_rn(v[4 * i + q], sc);
                    h[q] = pack_half2(r.x, r.y);
                }
                *reinterpret_cast<uint4 *>(o + 32 * i) = make_uint4(h[0], h[1], h[2], h[3]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------- tcgen05 helpers
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *slot_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]^T over a pair of CTAs, M 256 x N x K 16, fp16 operands, fp32 accumulate: each CTA brings 128
// rows of A (lanes of its tensor memory, two k a column) and N / 2 rows of B, and keeps its 128 rows of D for all N columns
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// sixteen lanes x 32 columns of tensor memory: lane (G, T) of the warp holds columns 4 x + T of rows G (r[2 x]) and G + 8 (r[2 x + 1])
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// arrive on the mbarrier of both CTAs of the pair when every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
// arrive on the mbarrier at the same offset in CTA `cta` of the cluster
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t *bar, uint32_t cta) {
    asm volatile(
        "{\n\t.reg .b32 r;\n\t"
        "mapa.shared::cluster.u32 r, %0, %1;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [r];\n\t}"
        ::"r"(smem_u32(bar)), "r"(cta)
        : "memory");
}
// one thread of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
// 32 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// the same, complete on return
__device__ __forceinline__ void tmem_ld32_now(uint32_t taddr, float *v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart; the tile base is 1024-aligned and
// a K step of 16 halves advances the start address by 32 bytes inside the swizzle atom.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);          // start address
    d |= (uint64_t)1 << 16;                               // leading byte offset (unused with swizzle): 16 B
    d |= (uint64_t)(1024 >> 4) << 32;                     // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                               // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                               // SWIZZLE_128B
    return d;
}
// kind::f16: D fp32, A and B fp16, both K-major, M 256 (the pair's columns of the matrix), N rows
__device__ __forceinline__ uint32_t umma_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(2 * FG_BN >> 4) << 24); }

// Tensor copy of one CTA of a pair whose bytes count on a barrier of either of them (its address in the cluster).
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
// address in the cluster of the barrier at the same offset in CTA `cta`
__device__ __forceinline__ uint32_t mbar_of_cluster(uint64_t *bar, uint32_t cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(bar)), "r"(cta));
    return r;
}

// Wait on an mbarrier phase, giving up when the abort flag is up or after a bounded number of polls.  SLEEP: nanoseconds a poll may
// sleep; every role but the one on the critical path (MMA issue) sleeps, because two dozen polling warps delay it
// by some 200 clocks per wait.
template <uint32_t SLEEP>
__device__ __forceinline__ bool wait_or_abort(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *status, int code) {
    if (mbar_try_wait(bar, parity)) return true;
    for (uint32_t i = 0; i < 4000000u; ++i) {
        if (SLEEP ? mbar_try_wait_hint(bar, parity, SLEEP) : mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        // another CTA of this launch has already given up: leave as well instead of sitting out the limit here too
        if ((i & 15u) == 15u && *reinterpret_cast<volatile int *>(status) != 0) { *abort_flag = 1; return false; }
    }
    *abort_flag = 1;
    atomicExch(status, code);
    return false;
}

// Two values rounded to bf16 (nearest even) by one packed conversion, read back as fp32: per value the bits of bf16r.
__device__ __forceinline__ float2 bf16r2(float x, float y) {
    const __nv_bfloat162 b = __float22bfloat162_rn(make_float2(x, y));
    const uint32_t w = *reinterpret_cast<const uint32_t *>(&b);
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// 128-point Walsh-Hadamard transform of a row that four neighbouring lanes hold: lane t has columns 16 j + 4 t + i at v[4 j + i].  Butterflies
// stride 1..64, (lower + upper, lower - upper): upstream's order (native/exl3.cu:208-219), so every sum associates as there.  Strides 4 and 8
// cross lanes; from stride 2 on two neighbours take the same side and share one packed fp32 instruction of sm_100 (add.f32x2 /
// fma.f32x2; a - b as b * -1 + a, one rounding, the same bits).
__device__ __forceinline__ void fwht128_quad(float (&v)[32], int t) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float a = v[i], b = v[i + 1];
        v[i] = a + b;
        v[i + 1] = a - b;
    }
    const float2 neg1 = make_float2(-1.f, -1.f);
    auto in_lane = [&](int s) {
#pragma unroll
        for (int i = 0; i < 32; i += 2)
            if (!(i & s)) {
                const float2 a = make_float2(v[i], v[i + 1]), b = make_float2(v[i | s], v[(i | s) + 1]);
                const float2 lo = __fadd2_rn(a, b), hi = __ffma2_rn(b, neg1, a);
                v[i] = lo.x; v[i + 1] = lo.y;
                v[i | s] = hi.x; v[(i | s) + 1] = hi.y;
            }
    };
    in_lane(2);
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        const float sg = t & d ? -1.f : 1.f;
        const float2 s2 = make_float2(sg, sg);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, v[i], d), __shfl_xor_sync(0xffffffffu, v[i + 1], d));
            const float2 r = __ffma2_rn(make_float2(v[i], v[i + 1]), s2, o);
            v[i] = r.x; v[i + 1] = r.y;
        }
    }
    in_lane(4);
    in_lane(8);
    in_lane(16);
}

// The same for a whole warp, by the barrier's shared-memory address; the lanes go on together, or not at all.
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, int code) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (__all_sync(0xffffffffu, ok != 0)) return true;
    for (uint32_t i = 0;; ++i) {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity), "r"(500u) : "memory");
        if (__all_sync(0xffffffffu, ok != 0)) return true;
        bool end = *abort_flag != 0;
        if (!end && (i & 15u) == 15u) end = *reinterpret_cast<volatile int *>(status) != 0;
        if (!end && i >= 4000000u) {
            atomicExch(status, code);
            end = true;
        }
        if (__any_sync(0xffffffffu, end)) {
            *abort_flag = 1;
            return false;
        }
    }
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
// Arrival of a warp's first lane, predicated (no branch for the warp): on a barrier of this CTA, or by its address in the cluster.
template <bool CLUSTER>
__device__ __forceinline__ void mbar_arrive_lane0(uint32_t bar, int lane) {
    if (CLUSTER) asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cluster.b64 _, [%0];\n\t}" ::"r"(bar), "r"(lane) : "memory");
    else asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"(lane) : "memory");
}

struct FastGemmArgs {
    const int *plan, *src_pair;
    const int4 *chunks;            // {expert, first grouped row, rows, -}
    const __half *sv0, *sv1, *sd;  // gate/up: svh_g, svh_u, suh_d;  down: svh_d
    __half *xd;                    // gate/up out, grouped rows [rows][N]
    float *y;                      // down out, pair rows [P][N]
    int *status;
    int K, N, shared_x;
    float limit;
};

// One work item of a CTA pair: a chunk of an expert's rows and a pair of 128-column blocks.  Each CTA decodes one of them (2 * nbp + its
// rank) and brings half of the rows.  A role walks its pair's items with the next one's chunk already on the way.
struct Items {
    const int4 *chunks;
    int total, step, NBP, item;
    int4 next;
    int e, row, cnt, n, nbp;                                 // n: rows of the MMAs (cnt rounded up to 32)
    __device__ __forceinline__ Items(const int4 *c, int first, int all, int pairs, int nbps) : chunks(c), total(all), step(pairs), NBP(nbps), item(first - pairs) {
        if (first < total) next = __ldg(chunks + first / NBP);
    }
    __device__ __forceinline__ bool advance() {
        item += step;
        if (item >= total) return false;
        e = next.x; row = next.y; cnt = next.z; n = (next.z + 31) & ~31; nbp = item % NBP;
        if (item + step < total) next = __ldg(chunks + (item + step) / NBP);
        return true;
    }
};

// position in a ring of barriers and the parity of its phase
struct Ring {
    uint32_t slot, parity;
    __device__ __forceinline__ void next(uint32_t depth) {
        if (++slot == depth) { slot = 0; parity ^= 1; }
    }
    template <uint32_t N>
    __device__ __forceinline__ void skip(uint32_t depth) {                  // N < depth
        slot += N;
        if (slot >= depth) { slot -= depth; parity ^= 1; }
    }
};

struct FgMaps {
    CUtensorMap rows[2][FG_BOXES];                           // grouped rows of the gate and up (or the down) input
    CUtensorMap bank[2];                                     // packed words
};

// Tensor memory: columns [0, 192) three stages of decoded weights (64 columns = 128 k), [192, 512) accumulators.  Even passes have theirs
// at the lower end, odd ones at the upper, so that two of up to 160 rows have room side by side; longer ones wait until the epilogue has
// taken out the columns that they share with the last pass, while the decode fills the stages.
constexpr int FG_STAGES = 3, FG_ACOLS = FG_BK / 2, FG_DCOL = FG_STAGES * FG_ACOLS, FG_DCOLS = 512 - FG_DCOL;
static_assert(FG_DCOLS >= FG_CHUNK, "accumulators of a pass");

// FINE: chains of FG_CHAIN stages with accumulators of their own, as many a pass as have room in half of the columns: the stages of a pass
// of n <= 128 rows.
__device__ __forceinline__ int fine_stages(int n) { return (n <= 32 ? 5 : n <= 64 ? 2 : 1) * FG_CHAIN; }
static_assert(5 * 32 <= FG_DCOLS / 2 && FG_FINE_ROWS <= FG_DCOLS / 2, "accumulators of a pass with partial sums");

template <int MATS>
struct FgCfg {
    static constexpr int WSTAGES = 4;                        // packed words
    // Waits go by the parity of a phase: whoever waits for one has to know that the phase before it is over.  The decode warps take every
    // second stage, so the stage in front of theirs in a slot of words has to be one of theirs as well: copies land in any order.  (The MMAs
    // of stages complete in order.)
    static_assert(WSTAGES % 2 == 0, "words of the decode warps");
    static constexpr int SCALES = MATS == 2 ? 3 * 128 : 128, SCALE_BUFS = MATS == 2 ? 1 : 2;   // scale vectors of an item, of one or two items
    static constexpr int TABLE_BYTES = 256 + SCALE_BUFS * SCALES * 4;                        // barriers, scale vectors
    static_assert((2 * FG_STAGES + 2 * WSTAGES + 6 + 1) * 8 <= 256, "barriers");
    static constexpr int TBUF_BYTES = 2 * 32 * 128 * 4;                                      // per epilogue warpgroup a slab of 32 rows
    static constexpr size_t SMEM = 1024 /*align*/ + (size_t)FG_STAGES * FG_TILE_BYTES + (size_t)WSTAGES * FG_WORD_BYTES + TABLE_BYTES + TBUF_BYTES;
};

// Registers per thread: launched with 72 x 896; the producer warpgroup gives to the two epilogue warpgroups (24 + 2 x 160 + 4 x 40 = 504).
constexpr uint32_t FG_SLEEP = 500;
constexpr int FG_REGS_MMA = 24, FG_REGS_EPI = 160, FG_REGS_DEC = 40;

// All 128 threads of an epilogue warpgroup: whether every one of them says yes.
__device__ __forceinline__ bool group_all(int group, bool yes) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.red.and.pred p, %2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r) : "r"((uint32_t)yes), "r"(2 + group) : "memory");
    return r != 0;
}
__device__ __forceinline__ void group_barrier(int group) { asm volatile("barrier.sync %0, 128;" ::"r"(2 + group) : "memory"); }

// FINE: the layer's calls of up to FG_FINE_ROWS rows, whose neighbours the streamed kernel serves, are as exact as there.  A sum is made of
// chains of at most 512 k, added in ascending order, and silu takes the full exponential and divide.  Mean distance of a layer's rows from
// sums in 64 bits with all rounding points in place, one chain and fast forms | FINE | streamed kernel: 2048 x 1536, 64 experts, top-4, 112
// rows 1.34e-4 | 5.6e-5 | 5.5e-5; 1024 x 2048, 24, top-3, 96 rows 9.6e-5 | 6.3e-5 | 6.1e-5; 3072 x 1024, 16, top-2, 112 rows 1.55e-4 | 4.2e-5
// | 4.2e-5; 4096 x 512, 288, top-8, 64 rows 1.73e-4 | 5.2e-5 | 5.1e-5 (600 rows each, standard error 3e-6 to 2e-5).  The chains make the difference:
// they cost up to 2 % (with a wait of the MMAs for the epilogue at each of them 10 %), the silu 2 to 6 % (128 rows of the first shape 206 | 212 us);
// for all calls it would cost 5 % at 4096 rows (590 | 618 us).
template <int MATS, bool FINE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FG_THREADS, 1)
fast_gemm_kernel(const __grid_constant__ FgMaps maps, const FastGemmArgs a) {
    using C = FgCfg<MATS>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);      // 1024-aligned operand tiles
    unsigned char *bring = smem;                                           // [FG_STAGES] rows
    unsigned char *wring = bring + (size_t)FG_STAGES * FG_TILE_BYTES;      // [WSTAGES] packed words
    float *tbuf = reinterpret_cast<float *>(wring + (size_t)C::WSTAGES * FG_WORD_BYTES);             // [2 groups][32 rows][128]
    unsigned char *tables = reinterpret_cast<unsigned char *>(tbuf) + C::TBUF_BYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(tables);                 // [FG_STAGES] (first CTA) rows landed and weights decoded, in both
    uint64_t *done = full + FG_STAGES;                                     // [FG_STAGES] MMAs of the stage completed
    uint64_t *wfull = done + FG_STAGES;                                    // [WSTAGES] packed words landed
    uint64_t *wempty = wfull + C::WSTAGES;                                 // [WSTAGES] read by the stage's decode warps
    uint64_t *tmem_full = wempty + C::WSTAGES;                             // [2] accumulators of a pass complete
    uint64_t *tmem_empty = tmem_full + 2;                                  // [2] (first CTA) accumulators drained, both CTAs' warps
    uint64_t *tmem_early = tmem_empty + 2;                                 // [2] (first CTA) what the next pass overwrites of them drained
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_early + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    float *scales = reinterpret_cast<float *>(tables + 256);               // [SCALE_BUFS][SCALES]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int KT = a.K >> 4, NBP = a.N >> 8, KS = a.K / FG_BK;

    if (tid == 0) {
        for (int s = 0; s < FG_STAGES; ++s) { mbar_init(full + s, 1 + FG_DEC); mbar_init(done + s, 1); }
        for (int s = 0; s < C::WSTAGES; ++s) { mbar_init(wfull + s, 1); mbar_init(wempty + s, FG_DEC / 2); }
        for (int b = 0; b < 2; ++b) { mbar_init(tmem_full + b, 1); mbar_init(tmem_empty + b, 16); mbar_init(tmem_early + b, 16); }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 2) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    cluster_sync();                                                        // the peer's barriers are initialised as well
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents();
    const int total = a.plan[2] * NBP, items = total > pair ? (total - pair + pairs - 1) / pairs : 0;
    // the slot that stage `it` takes is free: stage it - FG_STAGES has been consumed
    auto slot_free = [&](uint32_t it) {
        return it < FG_STAGES || wait_or_abort<FG_SLEEP>(done + it % FG_STAGES, (it / FG_STAGES - 1) & 1, abort_flag, a.status, GF_STATUS_TMA_TIMEOUT);
    };
    // after a give-up: the copies in flight, if any, have landed before the CTA leaves (bounded)
    auto land = [&](uint64_t *bar, uint32_t depth, uint32_t it) {
        for (uint32_t k = it > depth ? it - depth : 0; k < it; ++k) mbar_wait(bar + k % depth, (k / depth) & 1, nullptr, 1000u);
    };

    if (warp < 4) {
        // ------------------------------------------------------------------ warpgroup 0: TMA, MMA issue
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FG_REGS_MMA));
        if (warp == 0 && lane == 0) {
            // (the copies of both CTAs count on the first one's barrier)
            const uint32_t full0 = mbar_of_cluster(full, 0);
            uint32_t it = 0;
            bool ok = true;
            for (Items t(a.chunks, pair, total, pairs, NBP); ok && !*abort_flag && t.advance();) {
                // n / 2 rows of this CTA, those of the second MMA of more than 256 apart
                const int n1 = min(t.n, 256), n2 = t.n - n1, row1 = t.row + rank * (n1 >> 1), row2 = t.row + 256 + rank * (n2 >> 1);
                for (int pm = 0; pm < MATS && ok; ++pm) {
                    const CUtensorMap *map = maps.rows[pm == 1 && !a.shared_x], *map1 = map + (n1 >> 5) - 1, *map2 = map + max((n2 >> 5) - 1, 0);
                    for (int s = 0; s < KS; ++s, ++it) {
                        const uint32_t slot = it % FG_STAGES, bar = full0 + 8 * slot;
                        if (!slot_free(it)) { ok = false; break; }
                        if (rank == 0) mbar_expect_tx(full + slot, (uint32_t)t.n * FG_BK * 2);        // (of both CTAs)
                        unsigned char *dst = bring + slot * FG_TILE_BYTES;
                        tma_load_2d_pair(dst, map1, s * FG_BK, row1, bar);
                        tma_load_2d_pair(dst + FG_HALF_BYTES, map1, s * FG_BK + 64, row1, bar);
                        if (n2) {
                            tma_load_2d_pair(dst + 128 * 128, map2, s * FG_BK, row2, bar);
                            tma_load_2d_pair(dst + 128 * 128 + FG_HALF_BYTES, map2, s * FG_BK + 64, row2, bar);
                        }
                    }
                }
            }
            if (!ok || *abort_flag) land(rank ? done : full, FG_STAGES, it);      // (the second CTA's copies count elsewhere: it stays that long)
        } else if (warp == 1 && rank == 0) {
            // One elected thread of this warp issues every MMA of the pair; the warp runs the loop together, so that the descriptors
            // stay in uniform registers.  Its instruction stream is the critical path of the tensor pipe: ring positions and parities are
            // counted along (with modulo arithmetic a stage took 800 clocks of it beside the busy decode warps, 500 rows) and
            // the shared-memory descriptor is built once and advanced by adding constants (the address field
            // counts 16-byte units, a K step of 16 halves is 32 bytes; of A: eight columns).
            const uint64_t desc_b0 = umma_desc_sw128(smem_u32(bring));
            Ring ring{0, 0};
            uint32_t pc = 0;
            int before = 0;                                          // rows of the pass in front
            bool ok = true;
            for (Items t(a.chunks, pair, total, pairs, NBP); ok && t.advance();) {
                const int n2 = t.n - min(t.n, 256);                  // (one instruction takes 256 rows)
                const uint32_t idesc = umma_idesc(t.n - n2), idesc2 = umma_idesc(n2);
                const int most = FINE ? fine_stages(t.n) : KS, passes = FINE ? MATS * ((KS + most - 1) / most) : MATS;
                int left = KS;                                       // (FINE) stages of the matrix that are left
                for (int pm = 0; pm < passes && ok; ++pm, ++pc) {
                    const int steps = FINE ? min(left, most) : KS;
                    if (FINE && (left -= steps) == 0) left = KS;
                    const uint32_t pb = pc & 1;
                    // the accumulators of the pass before the last one, and where they reach into these, of the last one have been drained
                    ok = __all_sync(0xffffffffu, wait_or_abort<0>(tmem_empty + pb, ((pc >> 1) & 1) ^ 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT) &&
                                                     (before + t.n <= FG_DCOLS || wait_or_abort<0>((t.n <= before ? tmem_early : tmem_empty) + (pb ^ 1), ((pc - 1) >> 1) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT)));
                    if (!ok) break;
                    before = t.n;
                    tc_fence_after();
                    uint32_t d0 = tmem_base + FG_DCOL + (pb ? FINE ? FG_DCOLS / 2 : FG_DCOLS - t.n : 0);
                    for (int s = steps; s; --s) {
                        ok = __all_sync(0xffffffffu, wait_or_abort<0>(full + ring.slot, ring.parity, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT));
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t db = desc_b0 + ring.slot * (FG_TILE_BYTES >> 4);
                        const uint32_t ta = tmem_base + ring.slot * FG_ACOLS, first = FINE ? (steps - s) % FG_CHAIN : s != steps;
                        if (FINE && !first && s != steps) d0 += t.n;
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < FG_BK / 16; ++kk) {
                                const uint64_t dk = db + 2 * (kk & 3) + (kk >> 2) * (FG_HALF_BYTES >> 4);
                                umma_f16(d0, ta + 8 * kk, dk, idesc, kk > 0 ? 1u : first);
                                if (!FINE && n2) umma_f16(d0 + 256, ta + 8 * kk, dk + (128 * 128 >> 4), idesc2, kk > 0 ? 1u : first);
                            }
                            umma_commit(done + ring.slot);          // both CTAs may overwrite the stage once these MMAs have read it
                            if (s == 1) umma_commit(tmem_full + pb);           // the accumulators of this pass are complete
                        }
                        __syncwarp();
                        ring.next(FG_STAGES);
                    }
                }
            }
        } else if (warp == 3 && lane == 0) {
            // packed words of this CTA's column block, a ring of their own a few stages ahead of the decode
            uint32_t it = 0;
            bool ok = true;
            for (Items t(a.chunks, pair, total, pairs, NBP); ok && !*abort_flag && t.advance();) {
                for (int pm = 0; pm < MATS && ok; ++pm)
                    for (int s = 0; s < KS; ++s, ++it) {
                        const uint32_t ws = it % C::WSTAGES;
                        if (!wait_or_abort<FG_SLEEP>(wempty + ws, ((it / C::WSTAGES) & 1) ^ 1, abort_flag, a.status, GF_STATUS_TMA_TIMEOUT)) { ok = false; break; }
                        mbar_expect_tx(wfull + ws, FG_WORD_BYTES);
                        tma_load_3d(wring + ws * FG_WORD_BYTES, &maps.bank[pm], 0, t.e * KT + 8 * s, (2 * t.nbp + rank) * 8, wfull + ws);
                    }
            }
            if (!ok || *abort_flag) land(wfull, C::WSTAGES, it);
        }
    } else if (warp < 12) {
        // ------------------------------------------------------------------ warpgroups 1-2: epilogue
        // The accumulators have the columns of the matrix as lanes and rows as columns.  A warpgroup takes every other slab of 32 rows: a
        // thread reads its lane's 32 rows, the slab is transposed through shared memory, and four neighbouring lanes hold a row
        // (columns 16 j + 4 t + i).
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FG_REGS_EPI));
        const int q = warp & 3, group = (warp - 4) >> 2, m = q * 32 + lane, em = tid - 128;
        const int rr = m >> 2, t4 = (m & 3) * 4;             // row of a slab, first column of a group of 16
        // element (row r, column c) of a slab sits at r * 128 + (c ^ 16 (r & 1)): conflict-free both ways
        float *slab = tbuf + group * 32 * 128;
        uint32_t pc = 0, turn = 0;
        bool ok = true;
        // scale vectors of an item: fetched while the one before it runs, by both warpgroups (the 1 / sqrt(128) of every Hadamard transform is
        // folded into them, the transform is linear: one multiply per element less in each epilogue step)
        Items t(a.chunks, pair, total, pairs, NBP);
        __half sc0, sc1;                                     // (converted when they are used: the loads are not waited for)
        auto fetch = [&](int item, int e) {
            const size_t o = (size_t)e * a.N + (2 * (item % NBP) + rank) * 128 + (em & 127);
            if (em < 128) sc0 = a.sv0[o];
            else if (MATS == 2) { sc0 = a.sv1[o]; sc1 = a.sd[o]; }
        };
        if (pair < total) fetch(pair, t.next.x);
        auto act = [](float g) { return FINE ? silu(g) : __fdividef(g, 1.f + __expf(-g)); };
        // A warpgroup decides together whether a wait has given up: a warp never stands alone at a barrier.  One that has goes on through the
        // items for the barrier of both.
        while (t.advance()) {
            const int nb = 2 * t.nbp + rank;
            float *sc = scales + (C::SCALE_BUFS == 2 ? (turn++ & 1) * C::SCALES : 0);
            if (C::SCALE_BUFS == 1) asm volatile("bar.sync 1, 256;" ::: "memory");           // (the last item's have been read)
            if (em < 128) sc[em] = __half2float(sc0) * HAD_SCALE;
            else if (MATS == 2) { sc[em] = __half2float(sc0) * HAD_SCALE; sc[em + 128] = __half2float(sc1) * HAD_SCALE; }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (!ok) continue;
            if (t.item + t.step < total) fetch(t.item + t.step, t.next.x);
            const int mine = ((t.cnt + 31) / 32 - group + 1) >> 1;       // slabs of this warpgroup: group, group + 2, ..
            float v[3][32];
#pragma unroll 1
            for (int pm = 0, left = KS; pm < MATS; ++pm, ++pc) {
                const uint32_t pb = pc & 1;
                ok = wait_or_abort<FG_SLEEP>(tmem_full + pb, (pc >> 1) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT);
                if (!(ok = group_all(group, ok))) break;
                __syncwarp();                                            // (tcgen05.ld is for the warp as one)
                tc_fence_after();
                // Slabs in the order in which the next pass needs their columns: from the top at even passes, from the bottom at odd ones.  Three
                // are taken out at once, which for up to 256 rows covers what a next pass of no more rows overwrites.
                const uint32_t lanes = tmem_base + ((uint32_t)(q * 32) << 16), col = FG_DCOL + (pb ? FINE ? FG_DCOLS / 2 : FG_DCOLS - t.n : 0);
                auto slab_of = [&](int k) { return 2 * (pb || FINE ? k : max(mine - 1 - k, 0)) + group; };
                auto at = [&](int k) { return lanes + min(col + 32 * slab_of(k), 480u); };     // (past the end: some other slab, no branches)
                auto arrive = [&](uint64_t *bar) {                       // this warp's lanes are in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(bar + pb, 0);
                    __syncwarp();
                };
                if (FINE) {
                    // the next chains of the sums (v[0], v[1]: no more than two slabs); behind the matrix's last ones it goes on below
                    const int chains = (min(left, fine_stages(t.n)) + FG_CHAIN - 1) / FG_CHAIN;
                    int c = 0;
                    if (left == KS) {
                        tmem_ld32(at(0), v[0]);
                        tmem_ld32(at(1), v[1]);
                        tmem_ld_wait();
                        c = 1;
                    }
                    auto add = [&](int k, int c) {
                        tmem_ld32_now(at(k) + c * t.n, v[2]);
#pragma unroll
                        for (int r = 0; r < 32; r += 2) {
                            const float2 sum = __fadd2_rn(make_float2(v[k][r], v[k][r + 1]), make_float2(v[2][r], v[2][r + 1]));
                            v[k][r] = sum.x; v[k][r + 1] = sum.y;
                        }
                    };
#pragma unroll 1
                    for (; c < chains && mine; ++c) {
                        add(0, c);
                        if (mine > 1) add(1, c);
                    }
                    arrive(tmem_early);
                    arrive(tmem_empty);
                    left -= chains * FG_CHAIN;
                    if (left > 0) { --pm; continue; }
                    left = KS;
                } else {
#pragma unroll
                    for (int k = 0; k < 3; ++k) tmem_ld32(at(k), v[k]);
                    tmem_ld_wait();
                    if (t.n <= 256) arrive(tmem_early);
                    if (t.n <= 192) arrive(tmem_empty);
                }
                auto finish = [&](float (&x)[32], int k) {
                    group_barrier(group);                                // (the last slab has been read)
#pragma unroll
                    for (int r = 0; r < 32; ++r) slab[r * 128 + (m ^ (r & 1 ? 16 : 0))] = x[r];
                    const int row = slab_of(k) * 32 + rr;                // of the chunk
                    const bool here = row < t.cnt;
                    __half *o = a.xd + (size_t)(t.row + row) * a.N + nb * 128 + t4;
                    uint2 gate[8];
                    int p = 0;
                    if (MATS == 2 && pm == 1 && here)
#pragma unroll
                        for (int j = 0; j < 8; ++j) gate[j] = *reinterpret_cast<const uint2 *>(o + 16 * j);
                    if (MATS == 1 && here) p = __ldg(a.src_pair + t.row + row);
                    group_barrier(group);
                    const float *even = slab + rr * 128 + t4 + (rr & 1) * 16, *odd = slab + rr * 128 + t4 - (rr & 1) * 16;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 f = *reinterpret_cast<const float4 *>((j & 1 ? odd : even) + 16 * j);
                        x[4 * j] = f.x; x[4 * j + 1] = f.y; x[4 * j + 2] = f.z; x[4 * j + 3] = f.w;
                    }
                    fwht128_quad(x, m & 3);
                    if (MATS == 2 && pm == 0) {
                        // gate: scale, bf16 rounding, clamp, silu (rounded).  The values wait in this thread's places of the row of Xd, which its
                        // up pass overwrites (80 KB of shared memory otherwise)
                        if (here)
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const float4 sg = *reinterpret_cast<const float4 *>(sc + 16 * j + t4);
                                const float2 r0 = bf16r2(x[4 * j] * sg.x, x[4 * j + 1] * sg.y), r1 = bf16r2(x[4 * j + 2] * sg.z, x[4 * j + 3] * sg.w);
                                const float g0 = fminf(r0.x, a.limit), g1 = fminf(r0.y, a.limit), g2 = fminf(r1.x, a.limit), g3 = fminf(r1.y, a.limit);
                                // (one packed conversion rounds both values to bf16 and packs them: .x in the low half)
                                const __nv_bfloat162 s0 = __float22bfloat162_rn(make_float2(act(g0), act(g1)));
                                const __nv_bfloat162 s1 = __float22bfloat162_rn(make_float2(act(g2), act(g3)));
                                *reinterpret_cast<uint2 *>(o + 16 * j) = make_uint2(*reinterpret_cast<const uint32_t *>(&s0), *reinterpret_cast<const uint32_t *>(&s1));
                            }
                    } else if (MATS == 2) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 su = *reinterpret_cast<const float4 *>(sc + 128 + 16 * j + t4), sd = *reinterpret_cast<const float4 *>(sc + 256 + 16 * j + t4);
                            const float2 r0 = bf16r2(x[4 * j] * su.x, x[4 * j + 1] * su.y), r1 = bf16r2(x[4 * j + 2] * su.z, x[4 * j + 3] * su.w);
                            const float u0 = fminf(fmaxf(r0.x, -a.limit), a.limit), u1 = fminf(fmaxf(r0.y, -a.limit), a.limit);
                            const float u2 = fminf(fmaxf(r1.x, -a.limit), a.limit), u3 = fminf(fmaxf(r1.y, -a.limit), a.limit);
                            const float2 p0 = bf16r2(__uint_as_float(gate[j].x << 16) * u0, __uint_as_float(gate[j].x & 0xffff0000u) * u1);
                            const float2 p1 = bf16r2(__uint_as_float(gate[j].y << 16) * u2, __uint_as_float(gate[j].y & 0xffff0000u) * u3);
                            x[4 * j] = p0.x * sd.x; x[4 * j + 1] = p0.y * sd.y; x[4 * j + 2] = p1.x * sd.z; x[4 * j + 3] = p1.y * sd.w;
                        }
                        fwht128_quad(x, m & 3);
                        if (here)
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                *reinterpret_cast<uint2 *>(o + 16 * j) = make_uint2(pack_half2(x[4 * j], x[4 * j + 1]), pack_half2(x[4 * j + 2], x[4 * j + 3]));
                    } else if (here) {
                        // down: y rows are pair rows; 64 contiguous bytes a row and instruction
                        float *y = a.y + (size_t)p * a.N + nb * 128 + t4;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 s4 = *reinterpret_cast<const float4 *>(sc + 16 * j + t4);
                            *reinterpret_cast<float4 *>(y + 16 * j) = make_float4(x[4 * j] * s4.x, x[4 * j + 1] * s4.y, x[4 * j + 2] * s4.z, x[4 * j + 3] * s4.w);
                        }
                    }
                };
                // One copy of the slab's code: unrolled over the three slabs it came from L2 again and again (20 clocks an instruction).
#pragma unroll 1
                for (int k = 0; k < mine; ++k) {
                    finish(v[0], k);
#pragma unroll
                    for (int r = 0; r < 32; ++r) { v[0][r] = v[1][r]; v[1][r] = v[2][r]; }
                    if (!FINE && k == 0 && t.n > 192) {                           // the fourth and the fifth slab, as soon as there is room
                        tmem_ld32_now(at(3), v[2]);
                        if (t.n <= 256) arrive(tmem_empty);
                    }
                    if (!FINE && k == 1 && t.n > 256) {
                        tmem_ld32_now(at(4), v[2]);
                        arrive(tmem_early);
                        arrive(tmem_empty);
                    }
                }
            }
        }
        // the arrivals of the last commits have come in before this CTA ends (the accumulators are complete: these are on their way)
        const uint32_t stages = (uint32_t)(items * MATS * KS);
        for (uint32_t k = stages > FG_STAGES ? stages - FG_STAGES : 0; k < stages && ok; ++k)
            ok = wait_or_abort<FG_SLEEP>(done + k % FG_STAGES, (k / FG_STAGES) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT);
    } else {
        // ------------------------------------------------------------------ warpgroups 3-6: trellis decode
        // A warp takes every second stage and, of it, one of the two n-tiles (16 columns) whose lanes of tensor memory it may write.  A lane
        // reads word number `lane` of a tile and the word in front of it: those are k 2 T, 2 T + 1, 2 T + 8, 2 T + 9 of columns G and G + 8,
        // just the places that tcgen05.st gives it.  The first half of the stage is decoded before the slot is free.
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FG_REGS_DEC));
        // Beside the 320 instructions of a warp's share of a stage (64 weights a lane) the loop had 125 of its own with modulo arithmetic, generic
        // addresses and branches around single arrivals, and this kernel is bound by instruction issue (500 rows: 0.80 of the active
        // cycles): addresses and parities are counted along, arrivals are predicated.
        const int q = warp & 3, half = (warp >> 2) & 1;
        const uint32_t stages = (uint32_t)(items * MATS * KS);
        const uint32_t lanes = tmem_base + ((uint32_t)(q * 32 + half * 16) << 16);
        const uint32_t words0 = smem_u32(wring) + (2 * q + half) * 1024, word = words0 + lane * 4, before = words0 + ((lane + 31) & 31) * 4;
        const uint32_t wfull0 = smem_u32(wfull), wempty0 = smem_u32(wempty), done0 = smem_u32(done), full0 = mbar_of_cluster(full, 0);
        const uint32_t first = (warp - 12) >> 3;
        Ring rw{first, 0}, rs{first, 1};                     // (the first turn of a stage's slot waits for nothing: the phase before the first is over)
        for (uint32_t it = first; it < stages; it += 2) {
            if (!wait_warp(wfull0 + 8 * rw.slot, rw.parity, abort_flag, a.status, GF_STATUS_TMA_TIMEOUT)) break;
            const uint32_t at = rw.slot * FG_WORD_BYTES;
            bool ok = true;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t o[16];
#pragma unroll
                for (int kt = 0; kt < 4; ++kt) {
                    const uint32_t w = lds32(word + at + h * 512 + kt * 128), pw = lds32(before + at + h * 512 + kt * 128);
                    uint32_t hi[4], lo[4];
                    codeword_pair(__funnelshift_r(w, pw, 12), hi[0], lo[0]);                 // k = 2 T:     columns G, G + 8
                    codeword_pair(__funnelshift_r(w, pw, 8), hi[1], lo[1]);                  // k = 2 T + 1
                    codeword_pair(__funnelshift_r(w, pw, 4), hi[2], lo[2]);                  // k = 2 T + 8
                    codeword_pair(w, hi[3], lo[3]);                                          // k = 2 T + 9
                    o[4 * kt] = __byte_perm(weight_dup(hi[0]), weight_dup(hi[1]), 0x5410);
                    o[4 * kt + 1] = __byte_perm(weight_dup(lo[0]), weight_dup(lo[1]), 0x5410);
                    o[4 * kt + 2] = __byte_perm(weight_dup(hi[2]), weight_dup(hi[3]), 0x5410);
                    o[4 * kt + 3] = __byte_perm(weight_dup(lo[2]), weight_dup(lo[3]), 0x5410);
                }
                if (h == 0) {
                    ok = wait_warp(done0 + 8 * rs.slot, rs.parity, abort_flag, a.status, GF_STATUS_TMA_TIMEOUT);
                    if (!ok) break;
                    tc_fence_after();
                }
                tmem_st16(lanes + rs.slot * FG_ACOLS + h * (FG_ACOLS / 2), o);
            }
            if (!ok) break;
            __syncwarp();
            mbar_arrive_lane0<false>(wempty0 + 8 * rw.slot, lane);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            mbar_arrive_lane0<true>(full0 + 8 * rs.slot, lane);
            rw.skip<2>(C::WSTAGES);
            rs.skip<2>(FG_STAGES);
        }
    }

    tc_fence_before();
    // the pair ends together: no arrival or operand read is outstanding (not the aligned form: one lane of warps 0 and 1 worked alone)
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    tc_fence_after();
    if (warp == 2) tmem_dealloc(tmem_base, 512);
}

}  // namespace gf

using namespace gf;

// ---------------------------------------------------------------------------------------------- host side
namespace {
// Blocks of the rotation a matrix: what the SMs hold at once, fewer where a warp would have less than two rows, a whole number of the
// slices of a row.
long rot_blocks(long rows, int K, int mats, int sms) {
    const long slices = (K / 128 + 7) / 8, warps = (rows + 1) / 2 * slices;
    const long blocks = std::min((warps + ROT_WARPS - 1) / ROT_WARPS, 4L * sms / mats);
    return (blocks + slices - 1) / slices * slices;
}
int fail_if(cudaError_t e) { return e == cudaSuccess ? 0 : gf::fail_cuda(e, "cudaFuncSetAttribute"); }

// fp16 matrix [rows][K] row-major; boxes of 16, 32, .. 128 rows x 64 halves (128 bytes), 128-byte swizzle
int make_maps(CUtensorMap (&map)[FG_BOXES], void *base, uint64_t rows, uint64_t K) {
    const uint64_t dims[2] = {K, rows}, strides[1] = {K * 2};
    for (uint32_t i = 0; i < FG_BOXES; ++i) {
        const uint32_t box[2] = {64, 16 * (i + 1)};
        if (gf::encode_map(map + i, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, dims, strides, box, "grouped rows")) return -1;
    }
    return 0;
}
}  // namespace

struct glmflash_fast_experts {
    glmflash_config cfg;
    void *pool = nullptr;                                   // the one allocation behind the buffers below
    __half *xg = nullptr, *xu = nullptr, *xd = nullptr;     // grouped rows
    float *out = nullptr;                                   // pair rows
    int4 *chunks = nullptr;
    int *plan = nullptr, *src_pair = nullptr, *row_expert = nullptr /* row << 10 | expert */, *status = nullptr;
    FgMaps gateup, down;                                    // (the words' maps are filled in for each run)
    int sms = 0;
    int phases = 15;                                        // profiling aid: 1 plan, 2 rotation, 4 gate/up, 8 down
};

extern "C" int glmflash_fast_experts_new(const glmflash_config *cfg, size_t cfg_bytes, glmflash_fast_experts **out) {
    GF_REQUIRE(out != nullptr, "out is null");
    *out = nullptr;
    if (check_config(cfg, cfg_bytes, 8192)) return -1;       // upstream: 1..=8192 rows, src/fast_experts.rs:44-47
    GF_REQUIRE(cfg->experts + 1 <= FG_MAXU, "too many experts for the prefill plan");
    glmflash_fast_experts *f = new (std::nothrow) glmflash_fast_experts();
    GF_REQUIRE(f != nullptr, "out of host memory");
    f->cfg = *cfg;
    const size_t H = cfg->hidden, I = cfg->inter, P = (size_t)cfg->max_rows * cfg->slots;
    int dev = 0;
    cudaDeviceProp prop;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaGetDeviceProperties(&prop, dev) != cudaSuccess) {
        delete f;
        return fail("cannot query the CUDA device");
    }
    f->sms = prop.multiProcessorCount;
    if (prop.major != 10) {
        delete f;
        return fail("the prefill path needs an sm_100 GPU (tcgen05 / tensor memory)");
    }
    Pool pool;
    pool.take(&f->xg, P * H * 2);
    pool.take(&f->xu, P * H * 2);
    pool.take(&f->xd, P * I * 2);
    pool.take(&f->out, P * H * 4);
    pool.take(&f->plan, PLAN_INTS * 4);
    pool.take(&f->chunks, (P / (FG_CHUNK / 2) + cfg->experts + 1) * sizeof(int4));
    pool.take(&f->src_pair, P * 4);
    pool.take(&f->row_expert, P * 4);
    pool.take(&f->status, 16);
    if (pool.alloc(&f->pool) || make_maps(f->gateup.rows[0], f->xg, P, H) || make_maps(f->gateup.rows[1], f->xu, P, H) || make_maps(f->down.rows[0], f->xd, P, I) ||
        fail_if(cudaFuncSetAttribute(fast_gemm_kernel<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FgCfg<2>::SMEM)) ||
        fail_if(cudaFuncSetAttribute(fast_gemm_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FgCfg<1>::SMEM)) ||
        fail_if(cudaFuncSetAttribute(fast_gemm_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FgCfg<2>::SMEM)) ||
        fail_if(cudaFuncSetAttribute(fast_gemm_kernel<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FgCfg<1>::SMEM))) {
        glmflash_fast_experts_free(f);
        return -1;
    }
    *out = f;
    return 0;
}

extern "C" void glmflash_fast_experts_free(glmflash_fast_experts *f) {
    if (!f) return;
    cudaFree(f->pool);
    delete f;
}

// fine: a call of up to FG_FINE_ROWS rows takes partial sums; no expert may have more members than the call has rows
int gf::fast_experts_run(glmflash_fast_experts *f, void *stream, const glmflash_weights *w, const void *input, int x_stride, const int32_t *picks,
                         const int32_t *ids, const int32_t *count, const int32_t *members, int rows, int maxm, int shared_x, bool fine) {
    GF_REQUIRE(f && w && input && picks && ids && count && members, "null argument");
    const glmflash_config &c = f->cfg;
    GF_REQUIRE(rows > 0 && rows <= c.max_rows && maxm >= rows && maxm <= c.max_rows, "expert rows/member stride outside scratch");
    GF_REQUIRE(x_stride >= c.hidden && x_stride % 4 == 0, "x_stride must be >= hidden and a multiple of 4");
    fine = fine && rows <= FG_FINE_ROWS;
    GF_REQUIRE(((uintptr_t)w->gt | (uintptr_t)w->ut | (uintptr_t)w->dt) % 16 == 0, "trellis tensors must be 16-byte aligned");
    const bool aligned = ((uintptr_t)w->suh_g | (uintptr_t)w->suh_u) % 8 == 0;
    GF_REQUIRE((uintptr_t)input % 8 == 0 && (aligned || fine), "input and scale vectors must be 8-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    const int H = c.hidden, I = c.inter;
    const long P = (long)rows * c.slots;
    const bool pdl = c.pdl != 0;                            // a kernel's launch and set-up overlap the tail of the one in front
    if (f->phases & 1)
        if (launch_k(fast_plan_kernel, dim3((unsigned)c.experts + 1), dim3(FG_MAXU), 0, s, pdl, ids, count, members, maxm, c.slots, c.experts,
                     c.shared_exl3, c.expert_lo, c.expert_hi, c.shared_row_lo, c.shared_row_hi, f->plan, f->chunks, f->src_pair, f->row_expert, I / 256, f->sms / 2))
            return -1;
    const int mats = shared_x ? 1 : 2;
    if (f->phases & 2)
        if (launch_k(aligned ? fast_rot_kernel<false> : fast_rot_kernel<true>, dim3((unsigned)rot_blocks(P, H, mats, f->sms), (unsigned)mats), dim3(ROT_WARPS * 32), 0, s, pdl, (const __nv_bfloat16 *)input, x_stride,
                     f->plan, f->row_expert, (const __half *)w->suh_g, (const __half *)w->suh_u, f->xg, f->xu, H,
                     ((uintptr_t)input % 16 == 0 && x_stride % 8 == 0)))
            return -1;
    FastGemmArgs a{};
    a.plan = f->plan; a.chunks = f->chunks; a.src_pair = f->src_pair; a.status = f->status; a.limit = c.limit;
    if (bank_map(&f->gateup.bank[0], w->gt, c.experts + 1, H, I, 8, false) || bank_map(&f->gateup.bank[1], w->ut, c.experts + 1, H, I, 8, false) ||
        bank_map(&f->down.bank[0], w->dt, c.experts + 1, I, H, 8, false))
        return -1;
    a.sv0 = (const __half *)w->svh_g; a.sv1 = (const __half *)w->svh_u; a.sd = (const __half *)w->suh_d;
    a.xd = f->xd; a.y = nullptr; a.K = H; a.N = I; a.shared_x = shared_x ? 1 : 0;
    if ((f->phases & 4) && launch_k(fine ? fast_gemm_kernel<2, true> : fast_gemm_kernel<2, false>, dim3((unsigned)f->sms & ~1u), dim3(FG_THREADS), FgCfg<2>::SMEM, s, pdl, f->gateup, a))
        return -1;
    a.sv0 = (const __half *)w->svh_d; a.sv1 = nullptr; a.sd = nullptr;
    a.xd = nullptr; a.y = f->out; a.K = I; a.N = H; a.shared_x = 1;
    if ((f->phases & 8) && launch_k(fine ? fast_gemm_kernel<1, true> : fast_gemm_kernel<1, false>, dim3((unsigned)f->sms & ~1u), dim3(FG_THREADS), FgCfg<1>::SMEM, s, pdl, f->down, a))
        return -1;
    return 0;
}

extern "C" int glmflash_fast_experts_run(glmflash_fast_experts *f, void *stream, const glmflash_weights *w, const void *input,
                                         int x_stride, const int32_t *picks, const int32_t *ids, const int32_t *count,
                                         const int32_t *members, int rows, int maxm, int shared_x) {
    return fast_experts_run(f, stream, w, input, x_stride, picks, ids, count, members, rows, maxm, shared_x, false);
}

int *gf::fast_experts_status_word(glmflash_fast_experts *f) { return f->status; }

extern "C" int glmflash_fast_experts_set_phases(glmflash_fast_experts *f, int mask) {
    GF_REQUIRE(f != nullptr, "null argument");
    f->phases = mask;
    return 0;
}
extern "C" float *glmflash_fast_experts_output(const glmflash_fast_experts *f) { return f ? f->out : nullptr; }
extern "C" const uint16_t *glmflash_fast_experts_xd(const glmflash_fast_experts *f) { return f ? (const uint16_t *)f->xd : nullptr; }
extern "C" const int32_t *glmflash_fast_experts_row_pairs(const glmflash_fast_experts *f) { return f ? f->src_pair : nullptr; }
extern "C" const int32_t *glmflash_fast_experts_plan(const glmflash_fast_experts *f) { return f ? f->plan : nullptr; }
extern "C" const int32_t *glmflash_fast_experts_status(const glmflash_fast_experts *f) { return f ? f->status : nullptr; }
extern "C" int glmflash_fast_experts_clear_status(glmflash_fast_experts *f, void *stream) {
    GF_REQUIRE(f != nullptr, "null argument");
    GF_CUDA(cudaMemsetAsync(f->status, 0, 4, (cudaStream_t)stream));
    return 0;
}
