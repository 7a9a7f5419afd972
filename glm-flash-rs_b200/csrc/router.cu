// Router next to the expert path: logits = x . Wr^T and the sigmoid top-k that produces the routing table the expert
// kernels consume.  Upstream runs precompiled kernels here (_router_part, _router_sum, _topk: call sites src/moe.rs:77-111,
// src/window_ops.rs:159-199) whose source is not published, so the semantics are the benchmark's definition:
//   score = sigmoid(logit); the top-k scores of a row, ties to the lower expert id, in descending order;
//   weight = score / sum of the chosen scores; the row's last slot is the shared expert (id E) with weight 1.
// Selection is done on the logits (sigmoid is monotonic), so it does not depend on the precision of expf.
#include "common.cuh"

namespace gf {

// logits[r][e] = sum_k x[r][k] * wr[e][k] and, with picks, the top-k of every row, in one launch for any number of rows.
//
// CTA = 16 MT rows (of a cluster of CTAs that cut K between them when there are few rows); 8 warps cut the CTA's K; a warp runs
// mma.m16n8k16 (bf16, fp32 accumulation) on 64 experts at a time.  The k slots of a fragment may be any eight k as long as both
// operands agree, so a lane loads 16 contiguous bytes of a row (k = 8 t .. 8 t + 7 of a 32-k step) and uses them as the fragments
// of two instructions: no shared memory, no shuffles in front of the tensor cores.  The warps' and CTAs' sums are added in a
// fixed order.  Few rows are bound by latency: one memory round trip for the whole matrix (a cluster of 8 CTAs = 64 warps, one
// 32-k step each at K = 2048), one exchange through distributed shared memory.  Many rows are bound by reading the router matrix
// from L2 once per CTA (256 KB at 64 experts).  One warp per (row, expert) with scalar multiply-adds, and a CTA per row in the
// small form, took 133 us at 4096 rows and 9 us at one.
constexpr int RT_NE = 64, RT_ST = RT_NE + 4;                 // experts per round; floats per row of a partial

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Top-k of one row by one warp: lane l holds the logits of experts l, l + 32, ...; k rounds of a warp arg-max (value
// descending, id ascending), the winner is struck out.  E <= 1024.  `row` may point to shared or global memory.
__device__ __forceinline__ void topk_row(const float *row, int E, int topk, int *picks, float *weights, int lane) {
    constexpr int PER = 32;                          // 1024 / 32
    float v[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = lane + 32 * j;
        v[j] = e < E ? row[e] : -INFINITY;
    }
    float sum = 0.f, mine = 0.f;                     // lane j keeps the score of the j-th choice
    for (int t = 0; t < topk; ++t) {
        float best = -INFINITY;
        int bid = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int e = lane + 32 * j;
            if (32 * j >= E) break;                                         // (uniform)
            if (e < E && (v[j] > best || (v[j] == best && e < bid))) { best = v[j]; bid = e; }
        }
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, m);
            const int oi = __shfl_xor_sync(0xffffffffu, bid, m);
            if (ob > best || (ob == best && oi < bid)) { best = ob; bid = oi; }
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (32 * j >= E) break;
            if (lane + 32 * j == bid) v[j] = -INFINITY;                     // struck out (its owner lane only)
        }
        const float score = 1.f / (1.f + expf(-best));
        sum += score;
        if (lane == t) { mine = score; picks[t] = bid; }
    }
    if (lane < topk) weights[lane] = mine / sum;
    if (lane == 0) { picks[topk] = E; weights[topk] = 1.f; }
}

// The same by LANES lanes of a warp, which takes 32 / LANES rows side by side: lane l of the row's has experts l, l + LANES, ...; E <= 8 LANES,
// topk <= LANES.  All lanes of the warp call; rows that are not `live` are read nowhere and stored nowhere.  The choices are
// those of topk_row (the same order of values and ids).  Four rows of a tile one after another in every warp took a third of the router's time:
// 4096 rows of 64 experts 15.9 -> 11.1 us, 8192 rows 22.0 -> 16.2.
template <int LANES>
__device__ __forceinline__ void topk_rows(const float *row, bool live, int E, int topk, int *picks, float *weights, int lane) {
    const int l = lane & (LANES - 1);
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = live && l + LANES * j < E ? row[l + LANES * j] : -INFINITY;
    float sum = 0.f, mine = 0.f;
    for (int t = 0; t < topk; ++t) {
        float best = -INFINITY;
        int bid = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = l + LANES * j;
            if (e < E && (v[j] > best || (v[j] == best && e < bid))) { best = v[j]; bid = e; }
        }
#pragma unroll
        for (int m = LANES / 2; m >= 1; m >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, m);
            const int oi = __shfl_xor_sync(0xffffffffu, bid, m);
            if (ob > best || (ob == best && oi < bid)) { best = ob; bid = oi; }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (l + LANES * j == bid) v[j] = -INFINITY;
        const float score = 1.f / (1.f + expf(-best));
        sum += score;
        if (l == t) {
            mine = score;
            if (live) picks[t] = bid;
        }
    }
    if (!live) return;
    if (l < topk) weights[l] = mine / sum;
    if (l == 0) { picks[topk] = E; weights[topk] = 1.f; }
}

__global__ void __launch_bounds__(256) topk_kernel(const float *__restrict__ logits, int rows, int E, int topk,
                                                   int *__restrict__ picks, float *__restrict__ weights) {
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 8 + warp;
    if (r >= rows) return;
    topk_row(logits + (size_t)r * E, E, topk, picks + (size_t)r * (topk + 1), weights + (size_t)r * (topk + 1), lane);
}

template <int MT>
__global__ void __launch_bounds__(256) route_kernel(const __nv_bfloat16 *__restrict__ x, int x_stride,
                                                    const __nv_bfloat16 *__restrict__ wr, int rows, int H, int E, int topk,
                                                    float *__restrict__ logits, int *__restrict__ picks, float *__restrict__ weights) {
    extern __shared__ __align__(16) float part[];                          // [8 warps][16 MT][RT_ST], then the CTA's sums [16 MT][RT_ST]
    float *red = part + 8 * 16 * MT * RT_ST;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    uint32_t cr, cn;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(cr));
    asm("mov.u32 %0, %cluster_nctarank;" : "=r"(cn));
    const int r0 = (int)(blockIdx.x / cn) * 16 * MT, steps = (H + 31) >> 5, first = (int)cr * 8 + warp, stride = (int)cn * 8;
    if (first < steps && first * 32 + 8 * t < H)                           // the router matrix is a constant: hint its first lines into L2
        for (int n = 0; n < RT_NE / 8; ++n)
            if (8 * n + g < E) asm volatile("prefetch.global.L2 [%0];" ::"l"(wr + (size_t)(8 * n + g) * H + first * 32 + 8 * t));
    pdl_wait();
    pdl_launch_dependents();
    for (int e0 = 0; e0 < E; e0 += RT_NE) {
        float acc[MT][RT_NE / 8][4];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < RT_NE / 8; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[m][n][c] = 0.f;
        auto fetch = [&](int s, uint4 (&av)[MT][2], uint4 (&bv)[RT_NE / 8]) {
            const int k = s * 32 + 8 * t;
            const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = r0 + 16 * m + 8 * h + g;
                    av[m][h] = r < rows && k < H ? __ldg(reinterpret_cast<const uint4 *>(x + (size_t)r * x_stride + k)) : zero;
                }
#pragma unroll
            for (int n = 0; n < RT_NE / 8; ++n)
                bv[n] = e0 + 8 * n + g < E && k < H ? __ldg(reinterpret_cast<const uint4 *>(wr + (size_t)(e0 + 8 * n + g) * H + k)) : zero;
        };
        auto multiply = [&](const uint4 (&av)[MT][2], const uint4 (&bv)[RT_NE / 8]) {
#pragma unroll
            for (int n = 0; n < RT_NE / 8; ++n)
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    mma_bf16(acc[m][n], av[m][0].x, av[m][1].x, av[m][0].y, av[m][1].y, bv[n].x, bv[n].y);
                    mma_bf16(acc[m][n], av[m][0].z, av[m][1].z, av[m][0].w, av[m][1].w, bv[n].z, bv[n].w);
                }
        };
        // Sixteen rows a CTA: the next step's operands are on their way meanwhile (1000 rows 15.5 -> 9.9 us, one row 6.2 -> 5.5).  With 32 the
        // second set of registers costs more than it gives (4096 rows 11.2 -> 12.8, 8192 16.5 -> 24.7: one CTA an SM).
        if constexpr (MT == 1) {
            uint4 av[2][MT][2], bv[2][RT_NE / 8];
            if (first < steps) fetch(first, av[0], bv[0]);
            for (int s = first; s < steps; s += 2 * stride) {
                if (s + stride < steps) fetch(s + stride, av[1], bv[1]);
                multiply(av[0], bv[0]);
                if (s + stride >= steps) break;
                if (s + 2 * stride < steps) fetch(s + 2 * stride, av[0], bv[0]);
                multiply(av[1], bv[1]);
            }
        } else {
            for (int s = first; s < steps; s += stride) {
                uint4 av[MT][2], bv[RT_NE / 8];
                fetch(s, av, bv);
                multiply(av, bv);
            }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < RT_NE / 8; ++n) {
                float *p = part + (size_t)(warp * 16 * MT + 16 * m + g) * RT_ST + 8 * n + 2 * t;
                *reinterpret_cast<float2 *>(p) = make_float2(acc[m][n][0], acc[m][n][1]);
                *reinterpret_cast<float2 *>(p + 8 * RT_ST) = make_float2(acc[m][n][2], acc[m][n][3]);
            }
        __syncthreads();
        for (int i = tid; i < 16 * MT * RT_NE; i += 256) {
            const int r = i / RT_NE, c = i % RT_NE;
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) v += part[(size_t)(w * 16 * MT + r) * RT_ST + c];
            red[r * RT_ST + c] = v;
            if (cn == 1 && r0 + r < rows && e0 + c < E) logits[(size_t)(r0 + r) * E + e0 + c] = v;
        }
        if (cn > 1) {                                                      // row r of the tile is finished by CTA r % cn
            cluster_sync();
            for (int i = tid; i < 16 * MT * RT_NE; i += 256) {
                const int r = i / RT_NE, c = i % RT_NE;
                if (r % (int)cn != (int)cr || r0 + r >= rows || e0 + c >= E) continue;
                float v = 0.f;
                for (uint32_t q = 0; q < cn; ++q) v += cluster_map(red, q)[r * RT_ST + c];
                logits[(size_t)(r0 + r) * E + e0 + c] = v;
                part[r * RT_ST + c] = v;                                   // (this CTA has read its warps' sums)
            }
            // peers may still be reading this CTA's sums
            if (e0 + RT_NE < E) cluster_sync();
            else asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        } else {
            __syncthreads();
        }
    }
    if (picks) {
        __syncthreads();
        // the logits of up to 64 experts are still in shared memory: one trip to L2 less in front of the selection
        const float *row = E > RT_NE ? logits + (size_t)r0 * E : cn > 1 ? part : red;
        const int row_stride = E > RT_NE ? E : RT_ST;
        if (E <= 64 && topk <= 8) {
            for (int i = warp * 4; i * (int)cn < 16 * MT; i += 32) {
                const int r = (int)cr + (int)cn * (i + (lane >> 3));
                topk_rows<8>(row + (size_t)r * row_stride, r < 16 * MT && r0 + r < rows, E, topk, picks + (size_t)(r0 + r) * (topk + 1),
                             weights + (size_t)(r0 + r) * (topk + 1), lane);
            }
        } else if (MT == 1 && E <= 128 && topk <= 16) {        // (in the other kernel the code alone costs 4 %)
            for (int i = warp * 2; i * (int)cn < 16 * MT; i += 16) {
                const int r = (int)cr + (int)cn * (i + (lane >> 4));
                topk_rows<16>(row + (size_t)r * row_stride, r < 16 * MT && r0 + r < rows, E, topk, picks + (size_t)(r0 + r) * (topk + 1),
                              weights + (size_t)(r0 + r) * (topk + 1), lane);
            }
        } else {
            for (int r = (int)cr + (int)cn * warp; r < 16 * MT; r += (int)cn * 8)
                if (r0 + r < rows)
                    topk_row(row + (size_t)r * row_stride, E, topk, picks + (size_t)(r0 + r) * (topk + 1), weights + (size_t)(r0 + r) * (topk + 1), lane);
        }
    }
    if (cn > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

static int launch_route(cudaStream_t s, const uint16_t *x, int x_stride, const uint16_t *wr, int rows, int H, int E, int topk, float *logits,
                        int *picks, float *weights, bool pdl) {
    static int sms[64] = {};                       // (threads that come here together set the same)
    int dev = 0;
    GF_CUDA(cudaGetDevice(&dev));
    GF_REQUIRE(dev >= 0 && dev < 64, "device ordinal out of range");
    if (!sms[dev]) {
        int n = 0;
        GF_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
        GF_CUDA(cudaFuncSetAttribute(route_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 9 * 32 * RT_ST * (int)sizeof(float)));
        sms[dev] = n;
    }
    // Rows per CTA: 32 once 16 would give more CTAs than there are SMs (the matrix is read once per CTA).  Clusters of 8 along K
    // while the rows fill less than an eighth of the GPU.
    const bool wide = rows > 16 * sms[dev];
    const int tiles = wide ? (rows + 31) / 32 : (rows + 15) / 16, cn = tiles * 8 <= sms[dev] && H >= 512 ? 8 : 1;
    const size_t smem = (size_t)9 * (wide ? 32 : 16) * RT_ST * sizeof(float);
    const dim3 grid((unsigned)(tiles * cn)), block(256), cluster((unsigned)cn);
    const __nv_bfloat16 *xb = (const __nv_bfloat16 *)x, *wb = (const __nv_bfloat16 *)wr;
    return wide ? launch_kc(route_kernel<2>, grid, block, cluster, smem, s, pdl, xb, x_stride, wb, rows, H, E, topk, logits, picks, weights)
                : launch_kc(route_kernel<1>, grid, block, cluster, smem, s, pdl, xb, x_stride, wb, rows, H, E, topk, logits, picks, weights);
}
}  // namespace gf

using namespace gf;

extern "C" int glmflash_router_logits(void *stream, const uint16_t *x, int x_stride, const uint16_t *wr, int rows, int hidden,
                                      int experts, float *logits, int pdl) {
    GF_REQUIRE(x && wr && logits, "null argument");
    GF_REQUIRE(rows > 0 && hidden > 0 && hidden % 8 == 0 && experts > 0, "rows, experts positive; hidden a multiple of 8");
    GF_REQUIRE(x_stride >= hidden && x_stride % 8 == 0, "x_stride must be >= hidden and a multiple of 8");
    GF_REQUIRE(((uintptr_t)x | (uintptr_t)wr) % 16 == 0, "x and the router matrix must be 16-byte aligned");
    return launch_route((cudaStream_t)stream, x, x_stride, wr, rows, hidden, experts, 0, logits, nullptr, nullptr, pdl != 0);
}

extern "C" int glmflash_topk(void *stream, const float *logits, int rows, int experts, int topk, int32_t *picks, float *weights,
                             int pdl) {
    GF_REQUIRE(logits && picks && weights, "null argument");
    GF_REQUIRE(rows > 0 && experts > 0 && experts <= 1024, "experts must be in 1..1024");
    GF_REQUIRE(topk >= 1 && topk <= 31 && topk <= experts, "topk must be in 1..31 and at most the number of experts");
    return launch_k(topk_kernel, dim3((unsigned)((rows + 7) / 8)), dim3(256), 0, (cudaStream_t)stream, pdl != 0, logits, rows,
                    experts, topk, picks, weights);
}

extern "C" int glmflash_route(void *stream, const uint16_t *x, int x_stride, const uint16_t *wr, int rows, int hidden,
                              int experts, int topk, float *logits, int32_t *picks, float *weights, int pdl) {
    GF_REQUIRE(x && wr && logits && picks && weights, "null argument");
    GF_REQUIRE(rows > 0 && hidden > 0 && hidden % 8 == 0 && experts > 0 && experts <= 1024,
               "rows positive; hidden a multiple of 8; experts in 1..1024");
    GF_REQUIRE(topk >= 1 && topk <= 31 && topk <= experts, "topk must be in 1..31 and at most the number of experts");
    GF_REQUIRE(x_stride >= hidden && x_stride % 8 == 0, "x_stride must be >= hidden and a multiple of 8");
    GF_REQUIRE(((uintptr_t)x | (uintptr_t)wr) % 16 == 0, "x and the router matrix must be 16-byte aligned");
    return launch_route((cudaStream_t)stream, x, x_stride, wr, rows, hidden, experts, topk, logits, picks, weights, pdl != 0);
}
