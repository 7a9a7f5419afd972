// FastExperts: the prefill owner (upstream src/fast_experts.rs:27-208) as two persistent grouped GEMMs on the
// 5th-generation tensor cores (tcgen05.mma, accumulators in tensor memory), sm_100a only.
//
// Replaces upstream's fast_rot_in / fast_expert_plan / fast_gu_shared / fast_gu_separate / fast_down /
// fast_down_large (native/exl3_prefill.cu:402-430,657-889), which decode each 16x16 trellis tile into mma.sync
// fragments in registers.  Here:
//
//   plan      members per distinct expert, chunks of at most 256 rows (as even as an expert's rows go, long ones first) and the
//             GROUPED row order (rows of an expert contiguous): src_pair[j] = pair index of grouped row j.
//   rot       the input rotation writes Xs[j] = fp16(H(x[row] * suh[e]) / sqrt 128) in grouped order, so the A operand of a chunk is
//             a contiguous slab that TMA tensor loads bring into shared memory in the 128-byte-swizzled K-major layout the tensor
//             core reads.
//   gemm      persistent PAIRS of CTAs (74 clusters of two), one CTA per SM, 28 warps.  A work item is (chunk, pair of 128-column
//             blocks): tcgen05.mma.cta_group::2, M 256 x N 256 x K 16 -- each CTA brings half of the rows and decodes ONE of the two
//             column blocks, and keeps its rows' accumulators for both.  Roles:
//               warp 0       TMA producer of the row tiles (128 rows x 64 k per stage)
//               warp 1       first CTA: issues the MMAs of the pair, commits stages and passes to both CTAs; second CTA: relays
//                            "my half of the stage is there" to the first
//               warp 2       allocates / frees tensor memory (512 columns)
//               warp 3       TMA producer of the packed words, a ring of its own
//               warps 4-11   epilogue, one accumulator row per thread (column block 0: warps 4-7, block 1: warps 8-11):
//                            tcgen05.ld 128 fp32, the 128-point Hadamard transform in the thread's registers, scales, limited
//                            SwiGLU, down-input rotation; fp16 Xd rows (gate/up) or fp32 Y rows (down)
//               warps 12-27  decode the trellis tiles (bit-exact codebook) in registers and, when the slot is free, store them to
//                            the swizzled K-major tile
//             The gate and the up projection of an item are two PASSES over K with their own accumulators (256 columns each):
//             while the up pass runs, the epilogue warps turn the gate accumulators into silu(gate) (kept as bf16 in shared
//             memory), and the up pass's epilogue overlaps the next item's gate pass, so tensor memory is double-buffered by
//             construction.  Down is one pass per item, alternating the two accumulator halves.
//             What bounds it: with one CTA per tile pair (M 128 x N 128 instructions) the operand reads of the MMAs alone filled
//             shared memory (128 bytes a clock); the pair halves them.  What is left is the loop from a stage's release to its
//             next use (decode store, relay, issue, commit) and the decode itself: 4096 tokens, gate/up 407 -> 358 us, of which
//             249 us remain without decode and epilogue arithmetic.
// Arithmetic: one full-K fp32 accumulation chain per output (as upstream's prefill path, which is likewise not
// bit-equal to its decode path: native/exl3_prefill.cu:20-23), the same transforms and rounding points as
// upstream's epilogue (native/exl3_prefill.cu:596-622 == native/exl3.cu:260-321) with exp / divide in their fast
// forms.  Deterministic: static work assignment, no atomics; every pair's result depends only on its own row.
// Every wait is bounded; a wait that gives up raises the abort flag, every role leaves its loops, tensor memory
// is freed and the status word reports the failure.
#include <cuda.h>

#include <algorithm>
#include <new>

#include "gemv.cuh"

namespace gf {
int check_config(const glmflash_config *cfg, size_t cfg_bytes, int max_rows_limit);
int *fast_experts_status_word(glmflash_fast_experts *f);

constexpr int FG_DEC = 16;                                 // trellis-decode warps: n-tile by n-tile, round robin
constexpr int FG_THREADS = (12 + FG_DEC) * 32;
constexpr int FG_BM = 128, FG_BN = 128, FG_BK = 64;        // rows and columns of a CTA's operand tiles, k of a stage
constexpr int FG_TILE_BYTES = FG_BM * FG_BK * 2;           // 16 KB: one 128 x 64 fp16 operand tile
constexpr int FG_WORD_BYTES = 4096;                        // packed words of a stage: 4 k-tiles x 8 n-tiles
constexpr int FG_CHUNK = 2 * FG_BM;                        // rows of a work item: 128 per CTA of the pair
constexpr int FG_MAXU = 1024;

// plan layout (int32): [0] total 128-row tiles, [1] total grouped rows, [2] chunks
constexpr int PLAN_INTS = 4;
// ---------------------------------------------------------------------------------------------- plan
// Launched with one block per bank entry: every block recomputes the (tiny) scans, block 0 publishes the plan,
// block b writes the grouped rows of distinct expert b.
__global__ void __launch_bounds__(FG_MAXU) fast_plan_kernel(const int *__restrict__ ids, const int *__restrict__ count,
                                                          const int *__restrict__ members, int maxm, int slots, int E,
                                                          int shared_exl3, int e_lo, int e_hi, int srow_lo, int srow_hi,
                                                          int *__restrict__ plan, int4 *__restrict__ chunks,
                                                          int *__restrict__ src_pair, int *__restrict__ row_expert) {
    __shared__ int cnt_sh[FG_MAXU], row_sh[FG_MAXU], e_sh[FG_MAXU], first_sh[FG_MAXU];
    __shared__ int wsum[4][32];
    const int u = threadIdx.x, lane = u & 31, warp = u >> 5;
    pdl_wait();                                             // (every kernel of the chain: nothing is read or written before)
    pdl_launch_dependents();
    const int n = min(count[0], FG_MAXU);
    int cnt = 0, e = -1, first = 0;
    if (u < n) {
        e = ids[u];
        if (!expert_skipped(e, E, shared_exl3, e_lo, e_hi)) {
            const int *m = members + (size_t)u * maxm;
            int lo = 0, hi = maxm;                          // members come first: the count is the first -1
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (m[mid] >= 0) lo = mid + 1; else hi = mid;
            }
            cnt = lo;
            if (e == E && srow_hi > srow_lo) {
                // the shared expert is computed here for a window of rows only: members ascend by row (code = row * 32
                // + slot), so the window is a contiguous run of the list
                auto lower = [&](int row) {                 // first member whose row is >= `row`
                    int a = 0, b = cnt;
                    while (a < b) {
                        const int mid = (a + b) >> 1;
                        if ((m[mid] >> 5) < row) a = mid + 1; else b = mid;
                    }
                    return a;
                };
                first = lower(srow_lo);
                cnt = lower(srow_hi) - first;
            }
        }
    }
    // chunks of at most 256 rows, as even as they go; those of more than 128 rows come first in the list, so that the static
    // round robin over the CTA pairs ends with the short ones
    const int tiles = (cnt + FG_BM - 1) / FG_BM, nch = (cnt + FG_CHUNK - 1) / FG_CHUNK, size = nch ? (cnt + nch - 1) / nch : 0;
    const int pairs = size > FG_BM ? nch : 0, single = nch - pairs;
    // block-wide exclusive scans of long chunks, short chunks, rows (and the tile total)
    int p_inc = pairs, s_inc = single, r_inc = cnt, t_inc = tiles;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, p_inc, d), b = __shfl_up_sync(0xffffffffu, s_inc, d),
                  c = __shfl_up_sync(0xffffffffu, r_inc, d), t = __shfl_up_sync(0xffffffffu, t_inc, d);
        if (lane >= d) { p_inc += a; s_inc += b; r_inc += c; t_inc += t; }
    }
    if (lane == 31) { wsum[0][warp] = p_inc; wsum[1][warp] = s_inc; wsum[2][warp] = r_inc; wsum[3][warp] = t_inc; }
    __syncthreads();
    int p_off = 0, s_off = 0, r_off = 0, p_all = 0, s_all = 0, r_all = 0, t_all = 0;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) { p_off += wsum[0][w]; s_off += wsum[1][w]; r_off += wsum[2][w]; }
        p_all += wsum[0][w]; s_all += wsum[1][w]; r_all += wsum[2][w]; t_all += wsum[3][w];
    }
    const int p_ex = p_off + p_inc - pairs, s_ex = s_off + s_inc - single, r_ex = r_off + r_inc - cnt;
    cnt_sh[u] = cnt; row_sh[u] = r_ex; e_sh[u] = e; first_sh[u] = first;
    if (u == 0 && blockIdx.x == 0) { plan[0] = t_all; plan[1] = r_all; plan[2] = p_all + s_all; }
    if (u < n && u % (int)gridDim.x == (int)blockIdx.x)
        for (int c = 0; c < nch; ++c)
            chunks[(pairs ? p_ex : p_all + s_ex) + c] = make_int4(e, r_ex + c * size, min(size, cnt - c * size), 0);
    __syncthreads();
    for (int uu = blockIdx.x; uu < n; uu += gridDim.x) {
        const int c = cnt_sh[uu], rb = row_sh[uu], ee = e_sh[uu], f0 = first_sh[uu];
        for (int m = u; m < c; m += FG_MAXU) {
            const int code = members[(size_t)uu * maxm + f0 + m];
            src_pair[rb + m] = (code >> 5) * slots + (code & 31);
            row_expert[rb + m] = ee;
        }
    }
}

// ---------------------------------------------------------------------------------------------- rotation
// A warp takes 512 values of a grouped row: 8 lanes per 128-block, 16 values per lane, so that four of the seven butterflies run in
// registers (from stride 2 on as packed fp32) and three across lanes.  The butterflies keep their order (stride 1..64), so the
// sums are those of a warp per block.  With four values per lane and five butterflies across lanes the kernel issued 29
// instructions a value and took 83 us at 4096 rows x 2048 x 5 pairs x 2 matrices (168 MB written).
__global__ void __launch_bounds__(256) fast_rot_kernel(const __nv_bfloat16 *__restrict__ x, int x_stride,
                                                       const int *__restrict__ plan, const int *__restrict__ src_pair,
                                                       const int *__restrict__ row_expert, const __half *__restrict__ suh0,
                                                       const __half *__restrict__ suh1, __half *__restrict__ out0,
                                                       __half *__restrict__ out1, int K, int slots, int mats, bool vec) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KB = K >> 7, parts = (KB + 3) >> 2;
    pdl_wait();
    pdl_launch_dependents();
    const long items = (long)plan[1] * parts;
    const float2 neg1 = make_float2(-1.f, -1.f);
    for (long it = (long)blockIdx.x * 8 + warp; it < items; it += (long)gridDim.x * 8) {
        const int j = (int)(it / parts), blk = (int)(it % parts) * 4 + (lane >> 3);
        if (blk >= KB) continue;                                           // (whole groups of eight lanes)
        const unsigned group = 0xffu << (lane & 24);
        const int e = row_expert[j], row = src_pair[j] / slots, k = blk * 128 + (lane & 7) * 16;
        const __nv_bfloat16 *xp = x + (size_t)row * x_stride + k;
        uint32_t xw[8];
        if (vec) {
            const uint4 a = *reinterpret_cast<const uint4 *>(xp), b = *reinterpret_cast<const uint4 *>(xp + 8);
            xw[0] = a.x; xw[1] = a.y; xw[2] = a.z; xw[3] = a.w; xw[4] = b.x; xw[5] = b.y; xw[6] = b.z; xw[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint2 a = *reinterpret_cast<const uint2 *>(xp + 4 * i);
                xw[2 * i] = a.x; xw[2 * i + 1] = a.y;
            }
        }
#pragma unroll 1
        for (int mat = 0; mat < mats; ++mat) {
            const __half *sp = (mat ? suh1 : suh0) + (size_t)e * K + k;
            uint32_t sw[8];
            if (vec) {
                const uint4 a = __ldg(reinterpret_cast<const uint4 *>(sp)), b = __ldg(reinterpret_cast<const uint4 *>(sp + 8));
                sw[0] = a.x; sw[1] = a.y; sw[2] = a.z; sw[3] = a.w; sw[4] = b.x; sw[5] = b.y; sw[6] = b.z; sw[7] = b.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint2 a = __ldg(reinterpret_cast<const uint2 *>(sp + 4 * i));
                    sw[2 * i] = a.x; sw[2 * i + 1] = a.y;
                }
            }
            float2 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {                                   // times the sign / scale vector, stride 1
                const float2 s = __half22float2(*reinterpret_cast<const __half2 *>(&sw[i]));
                const float a = __uint_as_float(xw[i] << 16) * s.x, b = __uint_as_float(xw[i] & 0xffff0000u) * s.y;
                v[i] = make_float2(a + b, a - b);
            }
#pragma unroll
            for (int d = 1; d < 8; d <<= 1)                                // strides 2, 4, 8
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (!(i & d)) {
                        const float2 a = v[i], b = v[i | d];
                        v[i] = __fadd2_rn(a, b);
                        v[i | d] = __ffma2_rn(b, neg1, a);
                    }
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) {                              // strides 16, 32, 64: lower + upper | lower - upper
                const float sg = lane & d ? -1.f : 1.f;
                const float2 s2 = make_float2(sg, sg);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 o = make_float2(__shfl_xor_sync(group, v[i].x, d), __shfl_xor_sync(group, v[i].y, d));
                    v[i] = __ffma2_rn(v[i], s2, o);
                }
            }
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = pack_half2(v[i].x * HAD_SCALE, v[i].y * HAD_SCALE);
            uint4 *dst = reinterpret_cast<uint4 *>((mat ? out1 : out0) + (size_t)j * K + k);
            dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
            dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
    }
}

// ---------------------------------------------------------------------------------------------- tcgen05 helpers
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *slot_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]^T over a pair of CTAs, M 256 x N 256 x K 16, fp16 operands, fp32 accumulate: each CTA
// brings 128 rows of A and 128 rows (columns of D) of B at the same shared-memory offsets and keeps its 128 rows of D
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
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
// kind::f16: D fp32, A and B fp16, both K-major, N 256, M 256 (the pair's)
constexpr uint32_t UMMA_IDESC = (1u << 4) | ((uint32_t)(2 * FG_BN >> 3) << 17) | ((uint32_t)(2 * FG_BM >> 4) << 24);

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// Wait on an mbarrier phase, giving up when the abort flag is up or after a bounded number of polls.  SLEEP: nanoseconds a poll may
// sleep; every role but the two on the critical path (MMA issue, relay) sleeps, because two dozen polling warps delay those two
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

// In-register 128-point Walsh-Hadamard transform, butterflies stride 1..64, (lower + upper, lower - upper):
// upstream's order (native/exl3.cu:208-219), so every sum associates as there.
// Two values rounded to bf16 (nearest even) by one packed conversion, read back as fp32: per value the bits of bf16r.
__device__ __forceinline__ float2 bf16r2(float x, float y) {
    const __nv_bfloat162 b = __float22bfloat162_rn(make_float2(x, y));
    const uint32_t w = *reinterpret_cast<const uint32_t *>(&b);
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// From stride 2 on, the two neighbours (i, i + 1) take the same side of their butterflies, so a pair goes through one
// packed fp32 instruction of sm_100 (add.f32x2 / fma.f32x2; a - b as b * -1 + a, one rounding, the same bits): half
// the issue slots of the transform, which matters because this kernel is bound by instruction issue.
__device__ __forceinline__ void fwht128_regs(float (&v)[128]) {
#pragma unroll
    for (int i = 0; i < 128; i += 2) {
        const float a = v[i], b = v[i + 1];
        v[i] = a + b;
        v[i + 1] = a - b;
    }
    const float2 neg1 = make_float2(-1.f, -1.f);
#pragma unroll
    for (int s = 2; s < 128; s <<= 1)
#pragma unroll
        for (int i = 0; i < 128; i += 2)
            if (!(i & s)) {
                const float2 a = make_float2(v[i], v[i + 1]), b = make_float2(v[i | s], v[(i | s) + 1]);
                const float2 lo = __fadd2_rn(a, b), hi = __ffma2_rn(b, neg1, a);
                v[i] = lo.x; v[i + 1] = lo.y;
                v[i | s] = hi.x; v[(i | s) + 1] = hi.y;
            }
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

// One work item of a CTA pair: a chunk of an expert's rows and a pair of 128-column blocks.  This CTA brings `cnt` of the rows
// (starting at grouped row `row`) and decodes column block 2 * nbp + its rank.
struct ItemInfo {
    int e, row, cnt, nbp;
};
__device__ __forceinline__ ItemInfo item_info(int item, int NBP, const int4 *chunks, int rank) {
    const int4 c = __ldg(chunks + item / NBP);
    const int h = (c.z + 1) >> 1;                            // rows of the first CTA; both take about half
    return ItemInfo{c.x, c.y + (rank ? h : 0), rank ? c.z - h : h, item % NBP};
}

template <int MATS>
struct FgCfg {
    static constexpr int ASTAGES = MATS == 2 ? 4 : 6;        // rows
    static constexpr int BSTAGES = 4;                        // decoded weights: written from registers as soon as the slot is free
    static constexpr int WSTAGES = MATS == 2 ? 5 : 6;        // packed words
    static constexpr int DONE = 8;                           // ring of stage-completed barriers (more than any ring above)
    static constexpr int GBUF_BYTES = MATS == 2 ? 64 * 256 * 4 : 0;                          // silu(gate) as bf16 pairs
    static constexpr int TABLE_BYTES = 512 + 2 * 3 * 128 * 4;                                // barriers, scale vectors
    static constexpr int TBUF_BYTES = MATS == 1 ? 8 * 2 * 32 * 16 * 4 : 0;    // down: per epilogue warp two tiles of 32 rows x 16 floats
    static constexpr size_t SMEM = 1024 /*align*/ + (size_t)(ASTAGES + BSTAGES) * FG_TILE_BYTES + (size_t)WSTAGES * FG_WORD_BYTES +
                                   GBUF_BYTES + TABLE_BYTES + TBUF_BYTES;
};

// Registers per thread: launched with 72 x 896; the producer warpgroup and the decode warpgroups give theirs to the two epilogue
// warpgroups (24 + 2 x 152 + 4 x 40 = 488 of 504).
constexpr uint32_t FG_SLEEP = 500;
constexpr int FG_REGS_MMA = 24, FG_REGS_EPI = 152, FG_REGS_DEC = 40;

template <int MATS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FG_THREADS, 1)
fast_gemm_kernel(const __grid_constant__ CUtensorMap mapA0, const __grid_constant__ CUtensorMap mapA1, const __grid_constant__ CUtensorMap mapT0,
                 const __grid_constant__ CUtensorMap mapT1, const FastGemmArgs a) {
    using C = FgCfg<MATS>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);      // 1024-aligned operand tiles
    unsigned char *aring = smem, *bring = aring + (size_t)C::ASTAGES * FG_TILE_BYTES;
    unsigned char *wring = bring + (size_t)C::BSTAGES * FG_TILE_BYTES;     // [WSTAGES] packed words, 128-byte swizzle
    uint32_t *gbuf = reinterpret_cast<uint32_t *>(wring + (size_t)C::WSTAGES * FG_WORD_BYTES);       // [64][256]
    unsigned char *tables = wring + (size_t)C::WSTAGES * FG_WORD_BYTES + C::GBUF_BYTES;
    uint64_t *afull = reinterpret_cast<uint64_t *>(tables);                // [ASTAGES] rows landed
    uint64_t *bfull = afull + C::ASTAGES;                                  // [BSTAGES] decoded (+ in the first CTA: the second CTA's half)
    uint64_t *done = bfull + C::BSTAGES;                                   // [DONE] MMAs of stage i completed: done[i % DONE]
    uint64_t *wfull = done + C::DONE;                                   // [WSTAGES] packed words landed
    uint64_t *wempty = wfull + C::WSTAGES;                                 // [WSTAGES] read by the stage's decode warps
    uint64_t *tmem_full = wempty + C::WSTAGES;                             // [2] accumulators of a pass complete
    uint64_t *tmem_empty = tmem_full + 2;                                  // [2] (first CTA) accumulators drained, both CTAs' warps
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    float *scales = reinterpret_cast<float *>(tables + 512);               // [2 column blocks][3][128]
    float *tbuf = reinterpret_cast<float *>(tables + C::TABLE_BYTES);      // [8 warps][2][32 rows][16] (down only)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int KT = a.K >> 4, NBP = a.N >> 8, KS = a.K / FG_BK;

    if (tid == 0) {
        for (int s = 0; s < C::ASTAGES; ++s) mbar_init(afull + s, 1);
        for (int s = 0; s < C::BSTAGES; ++s) mbar_init(bfull + s, 8 + (rank == 0));
        for (int s = 0; s < C::DONE; ++s) mbar_init(done + s, 1);
        for (int s = 0; s < C::WSTAGES; ++s) { mbar_init(wfull + s, 1); mbar_init(wempty + s, 8); }
        for (int b = 0; b < 2; ++b) { mbar_init(tmem_full + b, 1); mbar_init(tmem_empty + b, 16); }
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
    // the slot that stage `it` of a ring of `depth` stages takes is free: stage it - depth has been consumed
    auto slot_free = [&](uint32_t it, uint32_t depth) {
        if (it < depth) return true;
        const uint32_t j = it - depth;
        return wait_or_abort<FG_SLEEP>(done + j % C::DONE, (j / C::DONE) & 1, abort_flag, a.status, GF_STATUS_TMA_TIMEOUT);
    };

    if (warp < 4) {
        // ------------------------------------------------------------------ warpgroup 0: TMA, MMA issue, relay
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FG_REGS_MMA));
        if (warp == 0 && lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int item = pair; item < total && ok && !*abort_flag; item += pairs) {
                const ItemInfo t = item_info(item, NBP, a.chunks, rank);
                for (int pm = 0; pm < MATS && ok; ++pm) {
                    const CUtensorMap *map = (pm == 1 && !a.shared_x) ? &mapA1 : &mapA0;
                    for (int s = 0; s < KS; ++s, ++it) {
                        const uint32_t slot = it % C::ASTAGES;
                        if (!slot_free(it, C::ASTAGES)) { ok = false; break; }
                        if (t.cnt == 0) { mbar_arrive(afull + slot); continue; }       // (a chunk of one row: the peer has it)
                        mbar_expect_tx(afull + slot, FG_TILE_BYTES);
                        tma_load_2d(aring + (size_t)slot * FG_TILE_BYTES, map, s * FG_BK, t.row, afull + slot);
                    }
                }
            }
        } else if (warp == 1 && rank == 0) {
            // One elected thread of this warp issues every MMA of the pair; the warp runs the loop together, so that the descriptors
            // stay in uniform registers.  Its instruction stream is the critical path of the tensor pipe, so the
            // shared-memory descriptors are built once (stage 0) and advanced by adding constants: the address field
            // counts 16-byte units, a stage is a tile apart, a K step of 16 halves is 32 bytes.
            const uint64_t desc_a0 = umma_desc_sw128(smem_u32(aring)), desc_b0 = umma_desc_sw128(smem_u32(bring));
            uint32_t it = 0, pc = 0;
            bool ok = true;
            for (int item = pair; item < total && ok; item += pairs) {
                for (int pm = 0; pm < MATS && ok; ++pm, ++pc) {
                    const uint32_t pb = pc & 1;
                    ok = __all_sync(0xffffffffu, wait_or_abort<0>(tmem_empty + pb, ((pc >> 1) & 1) ^ 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t d0 = tmem_base + pb * 256;
                    for (int s = 0; s < KS; ++s, ++it) {
                        const uint32_t sa = it % C::ASTAGES, sb = it % C::BSTAGES;
                        ok = __all_sync(0xffffffffu, wait_or_abort<0>(afull + sa, (it / C::ASTAGES) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT) &&
                                                         wait_or_abort<0>(bfull + sb, (it / C::BSTAGES) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT));
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t da = desc_a0 + (uint64_t)(sa * (FG_TILE_BYTES >> 4)), db = desc_b0 + (uint64_t)(sb * (FG_TILE_BYTES >> 4));
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < FG_BK / 16; ++kk) umma_f16(d0, da + 2 * kk, db + 2 * kk, UMMA_IDESC, kk > 0 || s > 0 ? 1u : 0u);
                            umma_commit(done + it % C::DONE);       // both CTAs may overwrite the stage once these MMAs have read it
                            if (s == KS - 1) umma_commit(tmem_full + pb);      // the accumulators of this pass are complete
                        }
                        __syncwarp();
                    }
                }
            }
        } else if (warp == 3 && lane == 0) {
            // packed words of this CTA's column block, a ring of their own a few stages ahead of the decode
            uint32_t it = 0;
            bool ok = true;
            for (int item = pair; item < total && ok && !*abort_flag; item += pairs) {
                const ItemInfo t = item_info(item, NBP, a.chunks, rank);
                for (int pm = 0; pm < MATS && ok; ++pm)
                    for (int s = 0; s < KS; ++s, ++it) {
                        const uint32_t ws = it % C::WSTAGES;
                        if (!wait_or_abort<FG_SLEEP>(wempty + ws, ((it / C::WSTAGES) & 1) ^ 1, abort_flag, a.status, GF_STATUS_TMA_TIMEOUT)) { ok = false; break; }
                        mbar_expect_tx(wfull + ws, FG_WORD_BYTES);
                        tma_load_3d(wring + ws * FG_WORD_BYTES, pm ? &mapT1 : &mapT0, 0, t.e * KT + 4 * s, (2 * t.nbp + rank) * 8, wfull + ws);
                    }
            }
        } else if (warp == 1 && lane == 0) {
            // second CTA: tell the issuing thread that this CTA's half of a stage is there
            uint32_t it = 0;
            bool ok = true;
            for (int item = pair; item < total && ok && !*abort_flag; item += pairs)
                for (int s = 0; s < MATS * KS && ok; ++s, ++it) {
                    const uint32_t sa = it % C::ASTAGES, sb = it % C::BSTAGES;
                    ok = wait_or_abort<0>(afull + sa, (it / C::ASTAGES) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT) &&
                         wait_or_abort<0>(bfull + sb, (it / C::BSTAGES) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT);
                    if (ok) mbar_arrive_cluster(bfull + sb, 0);
                }
        }
    } else if (warp < 12) {
        // ------------------------------------------------------------------ warpgroups 1-2: epilogue (column block 0 | 1)
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FG_REGS_EPI));
        const int q = warp & 3, cb = (warp - 4) >> 2;        // TMEM lane quadrant, column block of the item
        const int m = q * 32 + lane, em = cb * 128 + m;      // row of this CTA, thread of the epilogue (0..255)
        const float *sc = scales + cb * 384;
        uint32_t pc = 0;
        bool ok = true;
        // A warp whose wait gave up (or that sees the abort flag) does not leave this loop: it walks the remaining items
        // arriving at the two barriers only, so that a sibling which passed the same wait at the last moment never
        // stands alone at a barrier of eight warps.
        for (int item = pair; item < total; item += pairs) {
            const ItemInfo t = item_info(item, NBP, a.chunks, rank);
            const int nb = 2 * t.nbp + cb;
            // scale vectors of (expert, column block): written by the block's 128 threads, read by them
            asm volatile("bar.sync 1, 256;");
            if (ok && *abort_flag) ok = false;
            if (ok) {
                const size_t o = (size_t)t.e * a.N + nb * 128 + m;
                // the 1 / sqrt(128) of every Hadamard transform is folded into the scale vectors here (the transform is
                // linear), which takes one multiply per element out of each epilogue step
                float *w = scales + cb * 384 + m;
                w[0] = __half2float(a.sv0[o]) * HAD_SCALE;
                if (MATS == 2) { w[128] = __half2float(a.sv1[o]) * HAD_SCALE; w[256] = __half2float(a.sd[o]) * HAD_SCALE; }
            }
            asm volatile("bar.sync 1, 256;");
            if (!ok) continue;
            float v[128];
            for (int pm = 0; pm < MATS; ++pm, ++pc) {
                const uint32_t pb = pc & 1;
                if (!wait_or_abort<FG_SLEEP>(tmem_full + pb, (pc >> 1) & 1, abort_flag, a.status, GF_STATUS_MMA_TIMEOUT)) { ok = false; break; }
                tc_fence_after();
                const bool has = t.cnt > q * 32;             // (uniform: rows of this warp)
                if (has) {
                    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + pb * 256 + cb * FG_BN;
#pragma unroll
                    for (int c = 0; c < 4; ++c) tmem_ld32(taddr + c * 32, v + c * 32);
                    tmem_ld_wait();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(tmem_empty + pb, 0);  // this warp's rows are in registers
                if (!has) continue;
                fwht128_regs(v);
                const float2 *sc2 = reinterpret_cast<const float2 *>(sc);
                if (MATS == 2 && pm == 0) {
                    // gate: scale, bf16 rounding, clamp, silu (rounded) -> two bf16 per word, this thread's column of gbuf
#pragma unroll
                    for (int i = 0; i < 64; ++i) {
                        const float2 sg = sc2[i];
                        const float2 gr = bf16r2(v[2 * i] * sg.x, v[2 * i + 1] * sg.y);
                        const float g0 = fminf(gr.x, a.limit), g1 = fminf(gr.y, a.limit);
                        // (one packed conversion rounds both values to bf16 and packs them: .x in the low half)
                        const __nv_bfloat162 sp = __float22bfloat162_rn(make_float2(__fdividef(g0, 1.f + __expf(-g0)),
                                                                                   __fdividef(g1, 1.f + __expf(-g1))));
                        gbuf[i * 256 + em] = *reinterpret_cast<const uint32_t *>(&sp);
                    }
                } else if (MATS == 2) {
#pragma unroll
                    for (int i = 0; i < 64; ++i) {
                        const uint32_t gp = gbuf[i * 256 + em];
                        const float2 su = sc2[64 + i], sd2 = sc2[128 + i];
                        const float2 ur = bf16r2(v[2 * i] * su.x, v[2 * i + 1] * su.y);
                        const float u0 = fminf(fmaxf(ur.x, -a.limit), a.limit), u1 = fminf(fmaxf(ur.y, -a.limit), a.limit);
                        const float2 pr = bf16r2(__uint_as_float(gp << 16) * u0, __uint_as_float(gp & 0xffff0000u) * u1);
                        v[2 * i] = pr.x * sd2.x;
                        v[2 * i + 1] = pr.y * sd2.y;
                    }
                    fwht128_regs(v);
                    if (m < t.cnt) {
                        uint4 *o = reinterpret_cast<uint4 *>(a.xd + (size_t)(t.row + m) * a.N + nb * 128);
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            __half2 h[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j)       // one packed conversion per pair (the same rounding per value)
                                h[j] = __float22half2_rn(make_float2(v[8 * c + 2 * j], v[8 * c + 2 * j + 1]));
                            o[c] = make_uint4(*reinterpret_cast<uint32_t *>(&h[0]), *reinterpret_cast<uint32_t *>(&h[1]),
                                              *reinterpret_cast<uint32_t *>(&h[2]), *reinterpret_cast<uint32_t *>(&h[3]));
                        }
                    }
                } else {
                    // down: y rows are pair rows, scattered by src_pair.  A thread owns one row, so direct stores would
                    // put 32 rows x 16 bytes into every store instruction (half-filled sectors).  The rows go through
                    // per-warp shared-memory tiles, 16 columns at a time, and leave as 8 rows x 64 contiguous bytes per
                    // instruction.  Chunk c of row r sits at chunk c ^ ((r >> 1) & 3): conflict-free both ways.  Two tiles in
                    // turn, so that a block of columns is written while the one before is on its way out: with one, the 16
                    // steps ran one after the other, 16,000 of an item's 20,000 epilogue clocks (4096 tokens: 200 -> 191 us).
                    const int p = m < t.cnt ? a.src_pair[t.row + m] : -1;
                    float *wbuf = tbuf + (warp - 4) * 1024;
                    int pr[4];                               // pair rows that this lane writes
#pragma unroll
                    for (int i = 0; i < 4; ++i) pr[i] = __shfl_sync(0xffffffffu, p, (lane >> 2) + 8 * i);
                    auto put = [&](int ch) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const int col = ch * 16 + 4 * c;
                            const float4 s4 = *reinterpret_cast<const float4 *>(sc + col);
                            *reinterpret_cast<float4 *>(wbuf + (ch & 1) * 512 + lane * 16 + ((c ^ ((lane >> 1) & 3)) << 2)) =
                                make_float4(v[col] * s4.x, v[col + 1] * s4.y, v[col + 2] * s4.z, v[col + 3] * s4.w);
                        }
                    };
                    put(0);
#pragma unroll
                    for (int ch = 0; ch < 8; ++ch) {
                        __syncwarp();
                        float4 val[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int rr = (lane >> 2) + 8 * i;
                            val[i] = *reinterpret_cast<const float4 *>(wbuf + (ch & 1) * 512 + rr * 16 + (((lane & 3) ^ ((rr >> 1) & 3)) << 2));
                        }
                        if (ch < 7) put(ch + 1);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (pr[i] >= 0)
                                *reinterpret_cast<float4 *>(a.y + (size_t)pr[i] * a.N + nb * 128 + ch * 16 + 4 * (lane & 3)) = val[i];
                    }
                    __syncwarp();                            // (the next item's first tile overwrites one that is read here)
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ warpgroups 3-6: trellis decode of B
        // An n-tile of a stage at a time, round robin over the warps.  A lane reads 16 bytes (four words: all 16 k of columns G and
        // G + 8) of k-tile T of the stage, decodes them in registers and, once the slot is free, stores them as four 16-byte pieces
        // of the K-major tile, conflict-free under its swizzle: the decode is not part of the loop from a slot's release to the
        // next MMA.
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FG_REGS_DEC));
        const int G = lane >> 2, T = lane & 3;
        // byte offsets in the n-tile of the B tile: rows G and + 8; 16-byte pieces 2 T and 2 T + 1, piece c of row r at c ^ (r & 7)
        const uint32_t off0 = G * 128 + ((2 * T) ^ G) * 16, off1 = G * 128 + ((2 * T + 1) ^ G) * 16;
        const uint32_t tiles_all = (uint32_t)(items * MATS * KS) * 8;
        for (uint32_t c = warp - 12; c < tiles_all; c += FG_DEC) {
            const uint32_t it = c >> 3, nt = c & 7, sb = it % C::BSTAGES, ws = it % C::WSTAGES;
            // (the vote also brings the lanes together again: they may have left the wait apart)
            if (!__all_sync(0xffffffffu, wait_or_abort<FG_SLEEP>(wfull + ws, (it / C::WSTAGES) & 1, abort_flag, a.status, GF_STATUS_TMA_TIMEOUT))) break;
            // the lane's four words and the word in front of them (circular): row (n-tile, k-tile) of 128 bytes, piece c of row r at
            // c ^ (r & 7)
            const uint32_t row = nt * 4 + T;
            const unsigned char *wp = wring + ws * FG_WORD_BYTES + row * 128;
            const uint4 wv = *reinterpret_cast<const uint4 *>(wp + ((G ^ (row & 7)) << 4));
            const uint32_t before = *reinterpret_cast<const uint32_t *>(wp + ((((G + 7) & 7) ^ (row & 7)) << 4) + 12);
            const uint32_t w[4] = {wv.x, wv.y, wv.z, wv.w};
            uint32_t o[4][4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t pw = t == 0 ? before : w[t - 1];
                uint32_t hi[4], lo[4];
                codeword_pair(__funnelshift_r(w[t], pw, 12), hi[0], lo[0]);                  // k = 2t:     columns G, G + 8
                codeword_pair(__funnelshift_r(w[t], pw, 8), hi[1], lo[1]);                   // k = 2t + 1
                codeword_pair(__funnelshift_r(w[t], pw, 4), hi[2], lo[2]);                   // k = 2t + 8
                codeword_pair(w[t], hi[3], lo[3]);                                           // k = 2t + 9
                o[0][t] = __byte_perm(weight_dup(hi[0]), weight_dup(hi[1]), 0x5410);
                o[1][t] = __byte_perm(weight_dup(hi[2]), weight_dup(hi[3]), 0x5410);
                o[2][t] = __byte_perm(weight_dup(lo[0]), weight_dup(lo[1]), 0x5410);
                o[3][t] = __byte_perm(weight_dup(lo[2]), weight_dup(lo[3]), 0x5410);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(wempty + ws);
            if (!__all_sync(0xffffffffu, slot_free(it, C::BSTAGES))) break;
            unsigned char *bt = bring + (size_t)sb * FG_TILE_BYTES + nt * 2048;
            *reinterpret_cast<uint4 *>(bt + off0) = make_uint4(o[0][0], o[0][1], o[0][2], o[0][3]);
            *reinterpret_cast<uint4 *>(bt + off1) = make_uint4(o[1][0], o[1][1], o[1][2], o[1][3]);
            *reinterpret_cast<uint4 *>(bt + off0 + 1024) = make_uint4(o[2][0], o[2][1], o[2][2], o[2][3]);
            *reinterpret_cast<uint4 *>(bt + off1 + 1024) = make_uint4(o[3][0], o[3][1], o[3][2], o[3][3]);
            fence_async_smem();                              // generic-proxy stores -> visible to the tensor core
            __syncwarp();
            if (lane == 0) mbar_arrive(bfull + sb);
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
int fail_if(cudaError_t e) { return e == cudaSuccess ? 0 : gf::fail_cuda(e, "cudaFuncSetAttribute"); }

// fp16 matrix [rows][K] row-major; box = 128 rows x 64 halves (128 bytes), 128-byte swizzle
int make_map(CUtensorMap *map, void *base, uint64_t rows, uint64_t K) {
    const uint64_t dims[2] = {K, rows}, strides[1] = {K * 2};
    const uint32_t box[2] = {FG_BK, FG_BM};
    return gf::encode_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, dims, strides, box, "grouped rows");
}
}  // namespace

struct glmflash_fast_experts {
    glmflash_config cfg;
    void *pool = nullptr;                                   // the one allocation behind the buffers below
    __half *xg = nullptr, *xu = nullptr, *xd = nullptr;     // grouped rows
    float *out = nullptr;                                   // pair rows
    int4 *chunks = nullptr;
    int *plan = nullptr, *src_pair = nullptr, *row_expert = nullptr, *status = nullptr;
    CUtensorMap map_xg, map_xu, map_xd;
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
    pool.take(&f->chunks, (P / FG_CHUNK + cfg->experts + 1) * sizeof(int4));
    pool.take(&f->src_pair, P * 4);
    pool.take(&f->row_expert, P * 4);
    pool.take(&f->status, 16);
    if (pool.alloc(&f->pool) || make_map(&f->map_xg, f->xg, P, H) ||
        make_map(&f->map_xu, f->xu, P, H) || make_map(&f->map_xd, f->xd, P, I) ||
        fail_if(cudaFuncSetAttribute(fast_gemm_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FgCfg<2>::SMEM)) ||
        fail_if(cudaFuncSetAttribute(fast_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FgCfg<1>::SMEM))) {
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

extern "C" int glmflash_fast_experts_run(glmflash_fast_experts *f, void *stream, const glmflash_weights *w, const void *input,
                                         int x_stride, const int32_t *picks, const int32_t *ids, const int32_t *count,
                                         const int32_t *members, int rows, int maxm, int shared_x) {
    GF_REQUIRE(f && w && input && picks && ids && count && members, "null argument");
    const glmflash_config &c = f->cfg;
    GF_REQUIRE(rows > 0 && rows <= c.max_rows && maxm >= rows && maxm <= c.max_rows, "expert rows/member stride outside scratch");
    GF_REQUIRE(x_stride >= c.hidden && x_stride % 4 == 0, "x_stride must be >= hidden and a multiple of 4");
    GF_REQUIRE(((uintptr_t)w->gt | (uintptr_t)w->ut | (uintptr_t)w->dt) % 16 == 0, "trellis tensors must be 16-byte aligned");
    GF_REQUIRE(((uintptr_t)input | (uintptr_t)w->suh_g | (uintptr_t)w->suh_u) % 8 == 0, "input and scale vectors must be 8-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    const int H = c.hidden, I = c.inter;
    const long P = (long)rows * c.slots;
    const bool pdl = c.pdl != 0;                            // a kernel's launch and set-up overlap the tail of the one in front
    if (f->phases & 1)
        if (launch_k(fast_plan_kernel, dim3((unsigned)c.experts + 1), dim3(FG_MAXU), 0, s, pdl, ids, count, members, maxm, c.slots, c.experts,
                     c.shared_exl3, c.expert_lo, c.expert_hi, c.shared_row_lo, c.shared_row_hi, f->plan, f->chunks, f->src_pair, f->row_expert))
            return -1;
    const int mats = shared_x ? 1 : 2;
    if (f->phases & 2)
        if (launch_k(fast_rot_kernel, dim3((unsigned)std::min<long>((P * ((H + 511) / 512) + 7) / 8, 32L * f->sms)), dim3(256), 0, s, pdl,
            (const __nv_bfloat16 *)input, x_stride, f->plan, f->src_pair, f->row_expert, (const __half *)w->suh_g, (const __half *)w->suh_u, f->xg,
            f->xu, H, c.slots, mats, (((uintptr_t)input | (uintptr_t)w->suh_g | (uintptr_t)w->suh_u) % 16 == 0 && x_stride % 8 == 0)))
            return -1;
    FastGemmArgs a{};
    a.plan = f->plan; a.chunks = f->chunks; a.src_pair = f->src_pair; a.status = f->status; a.limit = c.limit;
    CUtensorMap mg, mu, md;
    if (bank_map(&mg, w->gt, c.experts + 1, H, I, 4) || bank_map(&mu, w->ut, c.experts + 1, H, I, 4) || bank_map(&md, w->dt, c.experts + 1, I, H, 4))
        return -1;
    a.sv0 = (const __half *)w->svh_g; a.sv1 = (const __half *)w->svh_u; a.sd = (const __half *)w->suh_d;
    a.xd = f->xd; a.y = nullptr; a.K = H; a.N = I; a.shared_x = shared_x ? 1 : 0;
    if ((f->phases & 4) && launch_k(fast_gemm_kernel<2>, dim3((unsigned)f->sms & ~1u), dim3(FG_THREADS), FgCfg<2>::SMEM, s, pdl, f->map_xg, f->map_xu, mg, mu, a))
        return -1;
    a.sv0 = (const __half *)w->svh_d; a.sv1 = nullptr; a.sd = nullptr;
    a.xd = nullptr; a.y = f->out; a.K = I; a.N = H; a.shared_x = 1;
    if ((f->phases & 8) && launch_k(fast_gemm_kernel<1>, dim3((unsigned)f->sms & ~1u), dim3(FG_THREADS), FgCfg<1>::SMEM, s, pdl, f->map_xd, f->map_xd, md, md, a))
        return -1;
    return 0;
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
