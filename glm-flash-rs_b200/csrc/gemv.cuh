// Grouped EXL3 GEMV for up to sixteen rows, sm_100a: the helpers every trellis kernel shares, and the stage decode -- how 256 k of
// one matrix and 128 columns of packed words get into shared memory (one TMA tensor copy) and how eight warps turn them into
// products.  Used by the streamed layer kernel (stream.cu: upstream's exl3_grouped_8_4 / exl3_load_nc_8_1, native/exl3.cu:59-170,
// native/expert_loads.cu:130-285) and the single linear (linear.cu).
//
//   * a lane reads 16 bytes (4 words of one tile) with one LDS.128: that is 32 weights, all 16 k of two columns (G, G + 8), so
//     only one shuffle per 32 weights is needed for the word that precedes the chunk.  The four lanes of a quad read the same
//     16-byte slot of four consecutive k-tiles.
//   * states are cut with funnel shifts in pairs (state_j << 16 | state_{j+4}), multiplied by the codebook constant, masked, and the
//     two fp16 halves of a codeword are added by one HADD2: exactly upstream's fp16 weight (bit-exact decode).
//   * pairs of weights are packed into the A operand of mma.m16n8k8 or m16n8k16 (rows = 16 output columns); the k slots of the
//     instruction are whatever k the lane holds, and the B operand (members, eight per set) is read to match.  fp32 accumulation; a
//     member's column depends on its own activations only.
// An instruction adds its products to the accumulator and rounds, so their number is part of a sum's bits.  Windows of up to 16 rows add
// eight (m16n8k8 has the bits of m16n8k16 over every weight duplicated, a doubled K whose other half is zero, which their kernels
// once ran); the single linear and chunks of more rows add sixteen: half as many roundings, up to 2 % faster (a chunk of 40 rows
// 174 -> 171 us).  A loop of nothing else runs 19.1 weights per clock and SM with sixteen, 17.4 with every weight duplicated.
#pragma once
#include "common.cuh"
#include "tensor_map.cuh"

namespace gf {

// Barrier of two warps (64 threads); ids 1..4, compile-time so that only those are reserved per CTA.
__device__ __forceinline__ void pair_barrier(int pw) {
    switch (pw) {
        case 0: asm volatile("bar.sync 1, 64;" ::: "memory"); break;
        case 1: asm volatile("bar.sync 2, 64;" ::: "memory"); break;
        case 2: asm volatile("bar.sync 3, 64;" ::: "memory"); break;
        default: asm volatile("bar.sync 4, 64;" ::: "memory"); break;
    }
}

__device__ __forceinline__ bool expert_skipped(int e, int E, int shared_exl3, int e_lo, int e_hi) {
    // the window [e_lo, e_hi) selects routed experts; the shared expert (id E) is governed by shared_exl3 alone
    return e < 0 || e > E || (e == E ? !shared_exl3 : (e < e_lo || e >= e_hi));
}

// (w, w) from a masked codeword: one half-precision add of its two halves.
__device__ __forceinline__ uint32_t weight_dup(uint32_t x) {
    const __half2 v = *reinterpret_cast<const __half2 *>(&x);
    const __half2 r = __hadd2(__low2half2(v), __high2half2(v));
    return *reinterpret_cast<const uint32_t *>(&r);
}

constexpr int ST_WBYTES = 16 * 1024;                         // [8 n-tiles][16 k-tiles][128 bytes], 128-byte swizzle
constexpr int ST_XROW = 512 + 16;                            // bytes per staged activation row (256 fp16): conflict-free LDS.128

// Four fp16 constants; vec: the vector is 8-byte aligned (uniform over a launch; views of larger tensors may not be).
__device__ __forceinline__ uint2 ldg_half4(const __half *p, bool vec) {
    if (vec) return __ldg(reinterpret_cast<const uint2 *>(p));
    const unsigned short *u = reinterpret_cast<const unsigned short *>(p);
    return make_uint2(__ldg(u) | (uint32_t)__ldg(u + 1) << 16, __ldg(u + 2) | (uint32_t)__ldg(u + 3) << 16);
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __float22half2_rn(make_float2(a, b));
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// A trellis bank [experts][K / 16][N / 16][32 words] seen as (word of a tile, k-tile of any expert, n-tile): the box of a stage is
// 32 words x `ktiles` k-tiles x 8 n-tiles, [n-tile][k-tile] rows of 128 bytes in shared memory (swizzled for lanes that read 16 bytes of
// four rows at a time; kernels whose warps read a row at a time take them as they are).
inline int bank_map(CUtensorMap *map, const uint32_t *bank, int experts, int K, int N, uint32_t ktiles = 16, bool swizzle = true) {
    const uint64_t dims[3] = {32, (uint64_t)experts * (K / 16), (uint64_t)(N / 16)}, strides[2] = {(uint64_t)(N / 16) * 128, 128};
    const uint32_t box[3] = {32, ktiles, 8};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint32_t *>(bank), dims, strides, box, "trellis bank", swizzle);
}

// ---- decode: one stage (256 k of one matrix and 128 columns) by eight warps ------------------------------------------
// words: the stage; x: the members' activations of its 256 k; warp = n-tile.  acc[s] += columns G, G + 8 of members 8 s + 2 T, + 1.
// ROUNDS: 2, or 1 for a stage of 128 k.  WIDE: sixteen products an instruction instead of eight.
template <int SETS, bool WIDE, int ROUNDS = 2>
__device__ __forceinline__ void st_decode(const unsigned char *words, const unsigned char *x, int warp, int lane, float (&acc)[SETS][4]) {
    const int G = lane >> 2, T = lane & 3;
    // row (n-tile, k-tile) of 128 bytes; its 16-byte chunk c sits at c ^ (k-tile & 7): k-tiles T and 4 + T of a pair of groups
    const unsigned char *wrow = words + warp * (ROUNDS * 1024) + T * 128;
    const int sw[2] = {(G ^ T) * 16, (4 * 128) + (G ^ (4 + T)) * 16};
    const unsigned char *xrow = x + G * ST_XROW + T * 32;
    // two groups of four k-tiles per round: the decode chains of two words are in flight side by side.  (One set: both rounds in line, one row
    // 22.6 -> 22.5 us a layer, 8 rows 53.8 -> 53.4; with two sets that is 2 % slower, 16 rows 78.9 -> 81.5.)
#pragma unroll(SETS == 1 ? 2 : 1)
    for (int r = 0; r < ROUNDS; ++r, wrow += 8 * 128, xrow += 256) {
        uint4 wv[2];
        uint32_t before[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            wv[q] = *reinterpret_cast<const uint4 *>(wrow + sw[q]);
            before[q] = __shfl_sync(0xffffffffu, wv[q].w, (lane + 28) & 31);      // the word in front of this lane's four (circular)
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t b0[SETS][4], b1[SETS][4];       // activations 16 T + 2 t, + 1 and 16 T + 8 + 2 t, + 1 of the group
#pragma unroll
            for (int s = 0; s < SETS; ++s) {
                const uint4 lo = *reinterpret_cast<const uint4 *>(xrow + s * 8 * ST_XROW + q * 128);
                const uint4 hi = *reinterpret_cast<const uint4 *>(xrow + s * 8 * ST_XROW + q * 128 + 16);
                b0[s][0] = lo.x; b0[s][1] = lo.y; b0[s][2] = lo.z; b0[s][3] = lo.w;
                b1[s][0] = hi.x; b1[s][1] = hi.y; b1[s][2] = hi.z; b1[s][3] = hi.w;
            }
            const uint32_t w[4] = {wv[q].x, wv[q].y, wv[q].z, wv[q].w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t pw = t == 0 ? before[q] : w[t - 1];
                uint32_t af[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t hi[2], lo[2];
                    codeword_pair(__funnelshift_r(w[t], pw, h ? 4 : 12), hi[0], lo[0]);         // k = 2t + 8h:     columns G, G + 8
                    codeword_pair(h ? w[t] : __funnelshift_r(w[t], pw, 8), hi[1], lo[1]);       // k = 2t + 8h + 1
                    af[2 * h] = __byte_perm(weight_dup(hi[0]), weight_dup(hi[1]), 0x5410);
                    af[2 * h + 1] = __byte_perm(weight_dup(lo[0]), weight_dup(lo[1]), 0x5410);
                    if (!WIDE)
#pragma unroll
                        for (int s = 0; s < SETS; ++s) mma1688(acc[s], af[2 * h], af[2 * h + 1], h ? b1[s][t] : b0[s][t]);
                }
                if (WIDE)
#pragma unroll
                    for (int s = 0; s < SETS; ++s) mma16816(acc[s], af, b0[s][t], b1[s][t]);
            }
        }
    }
}

}  // namespace gf
