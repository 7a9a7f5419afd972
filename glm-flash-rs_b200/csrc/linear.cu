// The single EXL3 linear (upstream src/experts.rs:100-135 for one matrix): y = fp16(H(fp16(H(x * suh) / sqrt 128) . W) / sqrt 128 * svh)
// for 1..16 fp16 rows, in one launch.
//
// A cluster of up to 8 CTAs owns 128 columns and cuts K into stages of 256; a CTA requests all of its stages at once, rotates
// its part of the input while they travel, decodes (gemv.cuh) and leaves its partial in shared memory; after a cluster barrier
// row m is finished by CTA m % cluster, which adds the partials in ascending order.  A call is bound by its latencies (launch,
// one memory round trip, 1,900 clocks of decode per stage, the exchange): 2048 x 1536 has 96 CTAs of one stage.  The form with a
// table kernel and a rotation kernel in front and scratch in global memory took three launches.
#include <algorithm>

#include "gemv.cuh"

namespace gf {

constexpr int LIN_THREADS = 256, LIN_PST = 132;
inline size_t lin_smem_bytes(int sets, int stages) {
    return 1024 + (size_t)stages * ST_WBYTES + (size_t)stages * sets * 8 * ST_XROW + (size_t)sets * 8 * LIN_PST * 4 + 256;
}

template <int SETS>
__global__ void __launch_bounds__(LIN_THREADS) linear_kernel(const __grid_constant__ CUtensorMap map, const __half *__restrict__ x, int rows,
                                                             const __half *__restrict__ suh, const __half *__restrict__ svh, int K, int N,
                                                             __half *__restrict__ y, int max_stages, bool vec) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int XBYTES = SETS * 8 * ST_XROW;
    unsigned char *words = smem, *xbuf = words + (size_t)max_stages * ST_WBYTES;
    float *part = reinterpret_cast<float *>(xbuf + (size_t)max_stages * XBYTES);       // [SETS * 8][LIN_PST]
    uint64_t *bars = reinterpret_cast<uint64_t *>(part + SETS * 8 * LIN_PST);                      // one per stage
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nb = blockIdx.x, cn = gridDim.y, cr = blockIdx.y;
    const int all = K >> 8, stages = (all - cr + cn - 1) / cn;                                     // stage i of this CTA: cr + i * cn
    if (tid == 0) {
        for (int i = 0; i < stages; ++i) {
            mbar_init(bars + i, 1);
            mbar_expect_tx(bars + i, ST_WBYTES);
        }
        mbar_fence_init();
        for (int i = 0; i < stages; ++i) tma_load_3d(words + (size_t)i * ST_WBYTES, &map, 0, (cr + i * cn) * 16, nb * 8, bars + i);
    }
    const uint2 sv = ldg_half4(svh + nb * 128 + 4 * lane, vec);
    // rotation: a warp per (row, stage, 128-block)
    for (int q = warp; q < rows * stages * 2; q += LIN_THREADS / 32) {
        const int blk = q & 1, i = (q >> 1) % stages, r = (q >> 1) / stages, k = (cr + i * cn) * 256 + blk * 128 + 4 * lane;
        const uint2 xv = ldg_half4(x + (size_t)r * K + k, vec), hv = ldg_half4(suh + k, vec);
        const float2 x01 = __half22float2(*reinterpret_cast<const __half2 *>(&xv.x)), x23 = __half22float2(*reinterpret_cast<const __half2 *>(&xv.y));
        const float2 s01 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.x)), s23 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.y));
        float v[4] = {x01.x * s01.x, x01.y * s01.y, x23.x * s23.x, x23.y * s23.y};
        fwht128(v, lane);
        *reinterpret_cast<uint2 *>(xbuf + (size_t)i * XBYTES + r * ST_XROW + blk * 256 + 8 * lane) =
            make_uint2(pack_half2(v[0] * HAD_SCALE, v[1] * HAD_SCALE), pack_half2(v[2] * HAD_SCALE, v[3] * HAD_SCALE));
    }
    __syncthreads();
    float acc[SETS][4];
#pragma unroll
    for (int s = 0; s < SETS; ++s)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[s][c] = 0.f;
    for (int i = 0; i < stages; ++i)
        if (__all_sync(0xffffffffu, mbar_wait(bars + i, 0)))                                 // (bounded; a copy that never lands leaves the sum short)
            st_decode<SETS, true>(words + (size_t)i * ST_WBYTES, xbuf + (size_t)i * XBYTES, warp, lane, acc);
    const int G = lane >> 2, T = lane & 3;
#pragma unroll
    for (int s = 0; s < SETS; ++s) {
        float *pp = part + (s * 8 + 2 * T) * LIN_PST + warp * 16 + G;
        pp[0] = acc[s][0];
        pp[LIN_PST] = acc[s][1];
        pp[8] = acc[s][2];
        pp[LIN_PST + 8] = acc[s][3];
    }
    cluster_sync();
    for (int m = cr + cn * warp; m < rows; m += cn * (LIN_THREADS / 32)) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        float4 q[8];
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (c < cn) q[c] = *reinterpret_cast<const float4 *>(cluster_map(part, c) + m * LIN_PST + 4 * lane);
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (c < cn) { v[0] += q[c].x; v[1] += q[c].y; v[2] += q[c].z; v[3] += q[c].w; }
        fwht128(v, lane);
        const float2 c01 = __half22float2(*reinterpret_cast<const __half2 *>(&sv.x)), c23 = __half22float2(*reinterpret_cast<const __half2 *>(&sv.y));
        *reinterpret_cast<uint2 *>(y + (size_t)m * N + nb * 128 + 4 * lane) =
            make_uint2(pack_half2(v[0] * HAD_SCALE * c01.x, v[1] * HAD_SCALE * c01.y), pack_half2(v[2] * HAD_SCALE * c23.x, v[3] * HAD_SCALE * c23.y));
    }
    cluster_sync();                                                       // peers may still be reading this CTA's partials
}

static int launch_linear(cudaStream_t s, const uint16_t *x, int rows, const uint32_t *words, const uint16_t *suh, const uint16_t *svh, int K, int N,
                         uint16_t *y) {
    const int sets = rows > 8 ? 2 : 1, cn = std::min(8, K / 256), stages = (K / 256 + cn - 1) / cn;
    const size_t smem = lin_smem_bytes(sets, stages);
    GF_REQUIRE(smem <= 227 * 1024, "K is too large for the single linear's shared-memory staging");
    static size_t configured[64][2] = {};
    int dev = 0;
    GF_CUDA(cudaGetDevice(&dev));
    size_t &have = configured[dev & 63][sets - 1];
    if (have < smem) {
        GF_CUDA(cudaFuncSetAttribute(sets == 2 ? linear_kernel<2> : linear_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        have = smem;
    }
    CUtensorMap map;
    if (bank_map(&map, words, 1, K, N)) return -1;
    const bool vec = ((uintptr_t)x | (uintptr_t)suh | (uintptr_t)svh) % 8 == 0;
    const dim3 grid((unsigned)(N / 128), (unsigned)cn), block(LIN_THREADS), cluster(1, (unsigned)cn, 1);
    const __half *xh = (const __half *)x, *suhh = (const __half *)suh, *svhh = (const __half *)svh;
    return sets == 2 ? launch_kc(linear_kernel<2>, grid, block, cluster, smem, s, false, map, xh, rows, suhh, svhh, K, N, (__half *)y, stages, vec)
                     : launch_kc(linear_kernel<1>, grid, block, cluster, smem, s, false, map, xh, rows, suhh, svhh, K, N, (__half *)y, stages, vec);
}

}  // namespace gf

using namespace gf;

// Scratch that callers provide: the call needs none any more, the size and the alignment it asks for are unchanged.
namespace {
size_t linear_scratch(int K) {
    const auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    return up((size_t)16 * K * 2) + up((size_t)(2 + 16) * 4 + 4);
}
}  // namespace

extern "C" size_t glmflash_exl3_linear_scratch_bytes(int K, int N) {
    if (K <= 0 || N <= 0 || K % 256 || N % 128) return 0;
    return linear_scratch(K);
}

extern "C" int glmflash_exl3_linear(void *stream, const uint16_t *x, int rows, const uint32_t *words, const uint16_t *suh,
                                    const uint16_t *svh, int K, int N, uint16_t *y, void *scratch) {
    GF_REQUIRE(x && words && suh && svh && y && scratch, "null argument");
    GF_REQUIRE(K > 0 && K % 256 == 0 && N > 0 && N % 128 == 0, "K must be a multiple of 256 and N of 128");
    GF_REQUIRE(rows >= 1 && rows <= 16, "rows must be in 1..16");
    GF_REQUIRE(((uintptr_t)words) % 16 == 0 && ((uintptr_t)scratch) % 256 == 0, "words 16-byte, scratch 256-byte aligned");
    return launch_linear((cudaStream_t)stream, x, rows, words, suh, svh, K, N, y);
}

// ---- the single EXL3 linear for callers that must not allocate ------------------------------------------------
// The same computation under the limits of the built-in scratch that this call once had (upstream's Rust `Device` hands out
// every byte of device memory at start-up and keeps the request path free of allocator calls).  The kernel needs no scratch any
// more; K and the advertised size stay what they were.
namespace {
constexpr int STATIC_LINEAR_MAX_K = 4096;
constexpr size_t STATIC_LINEAR_BYTES = 135168;            // 132 KiB >= linear_scratch(4096)
}  // namespace

extern "C" size_t glmflash_exl3_linear_static_max_bytes(void) { return STATIC_LINEAR_BYTES; }

extern "C" int glmflash_exl3_linear_static(void *stream, const uint16_t *x, int rows, const uint32_t *words,
                                           const uint16_t *suh, const uint16_t *svh, int K, int N, uint16_t *y) {
    GF_REQUIRE(K > 0 && K % 256 == 0 && N > 0 && N % 128 == 0, "K must be a multiple of 256 and N of 128");
    GF_REQUIRE(K <= STATIC_LINEAR_MAX_K,
               "shape exceeds the built-in scratch (K <= 4096): use glmflash_exl3_linear with caller scratch");
    GF_REQUIRE(linear_scratch(K) <= STATIC_LINEAR_BYTES, "shape exceeds the built-in scratch");
    GF_REQUIRE(x && words && suh && svh && y, "null argument");
    GF_REQUIRE(rows >= 1 && rows <= 16, "rows must be in 1..16");
    GF_REQUIRE(((uintptr_t)words) % 16 == 0, "words must be 16-byte aligned");
    return launch_linear((cudaStream_t)stream, x, rows, words, suh, svh, K, N, y);
}
