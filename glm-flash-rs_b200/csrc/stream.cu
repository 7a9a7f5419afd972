// The MoE layer for windows of 1..16 rows (decode and speculative verify) and for chunks of up to 128 as ONE launch: a
// persistent, warp-specialised kernel that streams the packed words of the chosen experts through shared memory and never
// lets the decode warps wait for a phase of the layer.
//
// Replaces upstream's rot_in / exl3_grouped_8_4 / gateup_epilogue / down_epilogue / combine sequence (native/exl3.cu:59-321,
// native/expert_loads.cu:130-285, src/moe.rs:101-181).  Same operands, member and pair conventions and rounding points.
//
// Work is cut into units of one partial sum: (distinct expert, matrix, split of k, 128-column block), the gate / up units of all experts
// first, the down units after them.  A split is 256 k at K <= 2048 (stream_cut), one or more stages of 16 k-tiles x 8 n-tiles
// (16 KB, 32,768 weights).  A CTA (512 threads, 768 with two teams of decode warps) has four roles:
//   warps 0-7   decode: warp = n-tile.  A lane reads 16 bytes (4 words of one tile: all 16 k of columns G and G + 8) with
//               one LDS.128, cuts the states in pairs with funnel shifts, forms the weights exactly as upstream does (fp16
//               sum of the codeword halves) and packs them into A operands of mma.m16n8k8 (chunks: k16); members are the N dimension
//               (8 per set, two sets for 9..16 rows), fp32 accumulation over the split.
//               Two teams (one CTA an SM, units of one stage) take the stages in turn.
//   then three  X: put the members' activations of a stage's k range into shared memory as soon as they are there: rotated layer
//               inputs (gate / up) or the finished rows of the gate / up phase (down).
//   one warp    feeds a four-stage ring, ONE tensor copy per stage (box 128 B x 16 k-tiles x 8 n-tiles, 128-byte swizzle).  Sixteen
//               bulk copies of the 1-KB rows held the issuing warp for 2,900 clocks a stage, longer than its decode takes.
//   four warps  finish: rotate the layer input (fp16(H(x * suh) / sqrt 128), once per pair and matrix), then add the splits of
//               an output block, ascending, and run the epilogue (Hadamard, scales, limited SwiGLU, down-input
//               rotation; for the down phase Hadamard, output scale and the weighted sum over the row's slots,
//               ascending, shared expert last).
// Partial sums and finished rows travel through L2 as 8-byte words {value, launch epoch}: the reader polls the data itself
// until it carries the epoch, so a hand-over costs one L2 round trip instead of fence + counter + load, and nothing has
// to be cleared between launches.
//
// Units and finish jobs are drawn from two counters, in order, by CTAs that are running.  A gate / up unit waits for nothing,
// and everything that a later unit or job waits for has been drawn by a CTA that runs: the launch makes progress with any
// number of resident CTAs, next to any other kernel (no co-residency is assumed).
//
// The sums of a window of up to 16 rows have a fixed order that does not depend on it: eight products an instruction, the k-tiles of a
// split in order, the splits ascending.  A row has the bits of its 1-row call, and of the cluster kernels that this one replaced.  With sixteen products
// an instruction, 512 k a split and half as many partials, the sums were as far from 64-bit ones (6.3e-7 against 6.2e-7 of a down
// row at K = 1536; 47 layers of one token 1142 us against 1101 now), but other bits: now and then a bf16 rounding behind them fell the
// other way, and a one-row layer moved by up to 1e-3.
//
// What bounds it: the decode instructions, about 5 a weight; a loop that does nothing else sustains 17.6 weights per clock and SM with 8
// warps (two chunks in flight per warp) and 18.7 with 16, so an SM has 16 decode warps where it can: two CTAs, or one with two teams
// (launch_stream).  The earlier form (clusters of short-lived CTAs, three launches per layer) spent half of its time on the
// phases around the decode.  Units of 512 k leave some SMs with twice the work of others at one row: 24.4 us a layer, 23.4 with 256 k.
#include <algorithm>

#include "gemv.cuh"
#include "owners.cuh"
#include "stream.cuh"

namespace gf {

constexpr int ST_STAGES = 4, ST_XW = 3;
// Warps of a CTA: eight decode warps a team, the X warps, the producer, four finish warps.
template <int TEAMS>
struct StWarps {
    static constexpr int DEC = 8 * TEAMS, PROD = DEC + ST_XW, FIN = PROD + 1, THREADS = (FIN + 4) * 32;
};
constexpr size_t ST_MAX_SMEM = 227 * 1024 - 4352;            // dynamic part (4,240 bytes are static)
constexpr size_t ST_HALF_SM = 116 * 1024;                    // two such CTAs do not fit an SM
constexpr size_t ST_TWO_SMEM = 228 * 1024 / 2 - 1024 - 4352; // dynamic part of one of two (each has 1 KB of the system's as well)
constexpr uint32_t ST_POLLS = 1u << 21;                      // polls of a global word before a wait gives up (about a second)

enum : int { UNIT_G = 0, UNIT_D = 1, UNIT_END = 2 };       // low byte of a descriptor, matrix in bit 8
enum : int { DESC_LAST = 1 << 9, DESC_CONT = 1 << 10, DESC_K = 12 };   // the stage ends its split; goes on with one; its first 128 k (from bit 12 on)

// ---- {value, epoch} words -------------------------------------------------------------------------------------------
__device__ __forceinline__ void ll_store2(unsigned long long *p, uint32_t v0, uint32_t v1, uint32_t epoch) {
    const unsigned long long e = (unsigned long long)epoch << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(e | v0), "l"(e | v1) : "memory");
}
__device__ __forceinline__ void ll_load4(const unsigned long long *p, unsigned long long (&w)[4]) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w[0]), "=l"(w[1]) : "l"(p) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w[2]), "=l"(w[3]) : "l"(p + 2) : "memory");
}
__device__ __forceinline__ bool ll_ready(const unsigned long long (&w)[4], uint32_t epoch) {
    return (uint32_t)(w[0] >> 32) == epoch && (uint32_t)(w[1] >> 32) == epoch && (uint32_t)(w[2] >> 32) == epoch &&
           (uint32_t)(w[3] >> 32) == epoch;
}

// t / d for 0 <= t < 2^21 with inv = 1 / d (approximate): the half keeps the product away from the integers.  An integer
// division costs about 130 clocks of latency, and drawing a unit takes six of them.
__device__ __forceinline__ float fast_inv(int d) { return __fdividef(1.f, (float)d); }
__device__ __forceinline__ int fast_div(int t, float inv) { return (int)(((float)t + 0.5f) * inv); }

// Shared state of a CTA: give-ups are sticky, every wait of the CTA then ends at once.
struct StCta {
    volatile int *abort_flag;
    int *status;
    __device__ __forceinline__ void give_up(int code) const {
        *abort_flag = 1;
        atomicExch(status, code);
    }
    // Poll bookkeeping of a wait on global memory: false when it has to end.
    __device__ __forceinline__ bool again(uint32_t &n) const {
        if (*abort_flag) return false;
        if ((++n & 255u) == 0u) {
            if (*reinterpret_cast<volatile int *>(status) != 0) { *abort_flag = 1; return false; }
            if (n >= ST_POLLS) { give_up(GF_STATUS_TMA_TIMEOUT); return false; }
        }
        return true;
    }
    __device__ __forceinline__ bool wait(uint64_t *bar, uint32_t parity) const {
        if (mbar_try_wait(bar, parity)) return true;
        for (uint32_t i = 0; i < 4000000u; ++i) {
            if (mbar_try_wait_hint(bar, parity, 1000u)) return true;
            if (*abort_flag) return false;
            if ((i & 255u) == 255u && *reinterpret_cast<volatile int *>(status) != 0) { *abort_flag = 1; return false; }
        }
        give_up(GF_STATUS_TMA_TIMEOUT);
        return false;
    }
    // The same for a whole warp, by the barrier's shared-memory address; the lanes go on together, or not at all.
    __device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity) const {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (__all_sync(0xffffffffu, ok != 0)) return true;
        for (uint32_t i = 0;; ++i) {
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok) : "r"(bar), "r"(parity), "r"(1000u) : "memory");
            if (__all_sync(0xffffffffu, ok != 0)) return true;
            bool end = *abort_flag != 0;
            if (!end && (i & 255u) == 255u && *reinterpret_cast<volatile int *>(status) != 0) {
                *abort_flag = 1;
                end = true;
            }
            if (!end && i >= 4000000u) {
                give_up(GF_STATUS_TMA_TIMEOUT);
                end = true;
            }
            if (__any_sync(0xffffffffu, end)) return false;
        }
    }
};
// Arrival of a warp's first lane on a barrier of this CTA, predicated (no branch for the warp).
__device__ __forceinline__ void arrive_lane0(uint32_t bar, int lane) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"(lane) : "memory");
}

// Four words of this lane, polled until they carry the epoch (uniform result for the warp).
__device__ __forceinline__ bool ll_wait4(const StCta &c, const unsigned long long *p, uint32_t epoch, unsigned long long (&w)[4]) {
    ll_load4(p, w);
    uint32_t n = 0;
    while (!__all_sync(0xffffffffu, ll_ready(w, epoch))) {
        if (!__all_sync(0xffffffffu, c.again(n))) return false;
        __nanosleep(20);
        ll_load4(p, w);
    }
    return true;
}

// v += the partials [lo, hi) of four columns of a pair, ascending, DEPTH requested at a time and polled until all carry the epoch.
// last_only: between the attempts only the last of them is polled; it is mostly the last to come.  With two CTAs an SM polls of all
// four cost the decode warps issue slots (8 rows 60.3 -> 59.5 us a layer); with one the extra round trip costs more (47 layers of
// one token 1113 -> 1144 us).
template <int DEPTH>
__device__ __forceinline__ bool sum_splits(bool last_only, const StCta &c, const unsigned long long *z, size_t split_stride, int lo, int hi, uint32_t epoch,
                                           float (&v)[4]) {
    z += (size_t)lo * split_stride;
#pragma unroll 1
    for (; lo < hi; lo += DEPTH, z += DEPTH * split_stride) {
        unsigned long long w[DEPTH][4];
        uint32_t n = 0;
#pragma unroll 1
        for (;;) {
            // (past the end the last split is read again: no branches between the loads)
            bool ok = true;
            const unsigned long long *zi = z;
#pragma unroll
            for (int i = 0; i < DEPTH; ++i) {
                ll_load4(zi, w[i]);
                if (lo + i + 1 < hi) zi += split_stride;
            }
#pragma unroll
            for (int i = 0; i < DEPTH; ++i) ok = ok && ll_ready(w[i], epoch);
            if (__all_sync(0xffffffffu, ok)) break;
            if (!__all_sync(0xffffffffu, c.again(n))) return false;
            __nanosleep(20);
            unsigned long long last[4];
            if (last_only && !ll_wait4(c, z + (size_t)(min(hi - lo, DEPTH) - 1) * split_stride, epoch, last)) return false;
        }
#pragma unroll
        for (int i = 0; i < DEPTH; ++i)
            if (lo + i < hi)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += __uint_as_float((uint32_t)w[i][j]);
    }
    return true;
}

// A decode lane holds columns G and G + 8 of an n-tile and stores them side by side, so that one instruction takes both: word 2 G + h of
// a tile is column G + 8 h.  A reading lane takes four consecutive words (z_word) and swaps two of them with its partner, which
// leaves it columns 4 lane .. 4 lane + 3.
__device__ __forceinline__ int z_word(int lane) { return (lane >> 2) * 16 + (lane & 1) * 8 + (lane & 2) * 2; }
__device__ __forceinline__ void z_columns(float (&v)[4], int lane) {
    const bool up = lane & 2;
    const float a = __shfl_xor_sync(0xffffffffu, up ? v[0] : v[1], 2), b = __shfl_xor_sync(0xffffffffu, up ? v[2] : v[3], 2);
    const float c = up ? v[1] : v[0], d = up ? v[3] : v[2];
    v[0] = up ? a : c; v[1] = up ? b : d; v[2] = up ? c : a; v[3] = up ? d : b;
}

// ---- shared memory of a CTA ------------------------------------------------------------------------------------------
// [stages] words | [stages] activations | barriers, descriptors | tables of the window
struct StTables {
    int *e, *mask, *pref;                // [umax] expert id, row mask (bit = row of the window); [umax + 1] finish-job prefix
    uint16_t *pair;                      // [umax][16] pair index of member m
    short *state;                        // [P] expert of a pair computed here, -1 not computed, -2 a repeated pick of its row
    // more than 16 rows only
    int *base;                           // [E + 1] number of an expert's first entry above
    uint32_t *rows_of;                   // [E + 1][words] rows that picked the expert, a bit each
    int words;
};
constexpr int ST_META = 512;             // barriers and descriptors
inline size_t st_smem_bytes(int sets, int umax, int rows, int P, int E) {
    const size_t tables = (size_t)(3 * umax + 1) * 4 + (size_t)umax * 32 + (size_t)P * 2 + 64 +
                          (rows > 16 ? (size_t)(E + 1) * 4 * (1 + (rows + 31) / 32) : 0);
    return (size_t)ST_STAGES * (ST_WBYTES + sets * 8 * ST_XROW) + ST_META + (tables + 127) / 128 * 128 +
           1024 /*align*/;
}

// Whether pair (row, expert e) is another GPU's: expert window, shared expert's switch (sh) and its row window.
__device__ __forceinline__ bool st_skipped(const StreamArgs &a, int row, int e, int sh) {
    return expert_skipped(e, a.E, sh, a.e_lo, a.e_hi) || (e == a.E && a.srow_hi > a.srow_lo && (row < a.srow_lo || row >= a.srow_hi));
}

// Distinct experts of the window that this GPU computes (ascending), their members (ascending rows) and the prefix of
// their members (one finish job per member and column block).  All threads of the CTA; the caller's barrier publishes the
// tables.  This is the head of every layer's critical path.  `used` (32 words) and tb.mask are zero on entry; row, slot: of
// pick number threadIdx.x.  Returns the number of experts.
template <int TEAMS>
__device__ __forceinline__ int st_build_tables(const StreamArgs &a, const StTables &tb, uint32_t *used, int row, int slot) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (a.picks && a.rows == 1 && a.shared != 2) {
        // one row: every warp finds the order of the picks itself and writes the same tables (no block barrier)
        constexpr int NONE = 0x7fffffff;
        const int e = lane < a.slots ? __ldcg(a.picks + lane) : NONE;
        int key = e == NONE || st_skipped(a, 0, e, a.shared) ? NONE : e;
        int less = 0;
        bool dup = false;
        for (int j = 0; j < a.slots; ++j) {
            const int v = __shfl_sync(0xffffffffu, key, j);
            less += v < key;
            dup |= v == key && j < lane && key != NONE;
        }
        if (__any_sync(0xffffffffu, dup)) {                      // a repeated pick counts once: rank among the first ones
            const int first = dup ? NONE : key;
            less = 0;
            for (int j = 0; j < a.slots; ++j) less += __shfl_sync(0xffffffffu, first, j) < key;
        }
        const bool here = key != NONE && !dup;
        if (here) {
            tb.e[less] = e;
            tb.mask[less] = 1;
            tb.pair[less * 16] = (uint16_t)lane;
        }
        if (lane < a.slots) tb.state[lane] = here ? (short)e : key == NONE ? (short)-1 : (short)-2;
        const int U = __popc(__ballot_sync(0xffffffffu, here));
        if (lane < U) tb.pref[lane] = lane;
        if (lane == 0) tb.pref[U] = U;
        __syncwarp();
        return U;
    }
    const int P = a.rows * a.slots;                              // <= 512: one per thread
    // key: the expert id (routing table) or the place in ids (grouping tables)
    int key = -1, e = -1, n_ids = 0;
    if (a.picks) {
        if (tid < P) {
            e = __ldcg(a.picks + tid);
            tb.state[tid] = (short)e;
            // ids above E name nothing; the shared expert counts for the rows of its window only (no row: it is not in the bitmap)
            if (e >= 0 && e <= a.E && !(e == a.E && st_skipped(a, row, e, 1))) {
                key = e;
                atomicOr(&used[key >> 5], 1u << (key & 31));
            }
        }
    } else {
        n_ids = min(__ldcg(a.count), a.umax);
        if (tid < P) tb.state[tid] = -1;
        if (tid < n_ids) {
            e = __ldcg(a.ids + tid);
            if (!expert_skipped(e, a.E, a.shared, a.e_lo, a.e_hi)) {
                key = tid;
                atomicOr(&used[key >> 5], 1u << (key & 31));
            }
        }
    }
    __syncthreads();
    // experts that another GPU computes do not count: the expert window, and the shared expert by the config's switch or,
    // when its owner is decided per window, by shared_owner_rank
    int sh = a.shared;
    if (a.picks && sh == 2) sh = shared_owner_rank(used, a.E, a.e_hi - a.e_lo, lane) == a.e_lo / (a.e_hi - a.e_lo);
    if (a.picks && key >= 0 && expert_skipped(key, a.E, sh, a.e_lo, a.e_hi)) key = -1;
    const int words = a.picks ? (a.E >> 5) + 1 : (n_ids + 31) >> 5;
    int U = 0, u = 0;
    const bool all = !a.picks || (sh && a.e_lo == 0 && a.e_hi == a.E);   // every id of the bitmap is computed here
#pragma unroll 4
    for (int w = 0; w < words; ++w) {
        uint32_t bits = used[w];
        if (!all) {
            const int lo = min(max(a.e_lo - 32 * w, 0), 32), hi = min(max(a.e_hi - 32 * w, 0), 32);
            uint32_t keep = hi > lo ? (0xffffffffu >> (32 - (hi - lo))) << lo : 0u;
            if (sh && (a.E >> 5) == w) keep |= 1u << (a.E & 31);
            bits &= keep;
        }
        U += __popc(bits);
        if (w < (key >> 5)) u += __popc(bits);
        else if (w == (key >> 5)) u += __popc(bits & ((1u << (key & 31)) - 1u));
    }
    U = min(U, a.umax);
    if (key < 0 || u >= U) u = -1;
    bool dup = false;
    if (u >= 0) tb.e[u] = e;
    if (a.picks) {
        if (u >= 0) {                                            // a pick that repeats an earlier slot of its row does not count
            for (int q = 1; q <= slot; ++q) dup |= tb.state[tid - q] == (short)e;
            if (!dup) atomicOr(&tb.mask[u], 1 << row);
        }
    } else if (u >= 0) {                                         // members come first; a member is row * 32 + slot
        uint32_t bits = 0u;
        for (int m = 0; m < min(a.maxm, 16); ++m) {
            const int code = __ldcg(a.members + (size_t)tid * a.maxm + m);
            if (code < 0) break;
            const int p = (code >> 5) * a.slots + (code & 31);
            tb.pair[u * 16 + m] = (uint16_t)p;
            tb.state[p] = (short)e;
            bits |= 1u << m;
        }
        tb.mask[u] = (int)bits;
    }
    __syncthreads();
    if (a.picks) {
        if (u >= 0 && !dup) tb.pair[u * 16 + __popc(tb.mask[u] & ((1u << row) - 1u))] = (uint16_t)tid;
        if (tid < P) tb.state[tid] = u < 0 ? (short)-1 : dup ? (short)-2 : (short)e;
    }
    if (warp == StWarps<TEAMS>::FIN) {
        int run = 0;
        for (int u0 = 0; u0 < U; u0 += 32) {
            const int c = u0 + lane < U ? __popc(tb.mask[u0 + lane]) : 0;
            int incl = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += up;
            }
            if (u0 + lane < U) tb.pref[u0 + lane] = run + incl - c;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) tb.pref[U] = run;
    }
    return U;
}

// The same for chunks of more than 16 rows (routing table only): an expert with more than 16 members gets an entry for every 16
// of them, for which its weights are decoded again.  Every CTA has to come to the same tables.  tb.rows_of is zero on entry.
template <int TEAMS>
__device__ __forceinline__ int st_build_tables_many(const StreamArgs &a, const StTables &tb) {
    constexpr int THREADS = StWarps<TEAMS>::THREADS;
    __shared__ int total;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, P = a.rows * a.slots, W = tb.words;
    const float inv_slots = fast_inv(a.slots);
    auto members = [&](int e) {
        int n = 0;
        for (int w = 0; w < W; ++w) n += __popc(tb.rows_of[e * W + w]);
        return n;
    };
    for (int i = tid; i < P; i += THREADS) {
        const int e = __ldcg(a.picks + i);
        tb.state[i] = e < 0 || e > a.E ? (short)-1 : (short)e;
    }
    __syncthreads();
    auto first_of_row = [&](int i, int row, int e) {             // a pick that repeats an earlier slot of its row does not count
        bool dup = false;
        for (int q = row * a.slots; q < i; ++q) dup |= tb.state[q] == (short)e;
        return !dup;
    };
    auto skipped = [&](int row, int e) { return st_skipped(a, row, e, a.shared); };
    for (int i = tid; i < P; i += THREADS) {
        const int e = tb.state[i], row = fast_div(i, inv_slots);
        if (!skipped(row, e) && first_of_row(i, row, e)) atomicOr(&tb.rows_of[e * W + (row >> 5)], 1u << (row & 31));
    }
    __syncthreads();
    if (warp == 0) {
        int run = 0;
        for (int e0 = 0; e0 <= a.E; e0 += 32) {
            const int g = e0 + lane <= a.E ? (members(e0 + lane) + 15) >> 4 : 0;
            int incl = g;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += up;
            }
            if (e0 + lane <= a.E) tb.base[e0 + lane] = run + incl - g;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) total = run;
    }
    __syncthreads();
    for (int i = tid; i < P; i += THREADS) {
        const int e = tb.state[i], row = fast_div(i, inv_slots);
        // (marking a pick changes nothing for the row's others: the first one of an expert keeps its id)
        if (skipped(row, e)) { tb.state[i] = -1; continue; }
        if (!first_of_row(i, row, e)) { tb.state[i] = -2; continue; }
        int pos = __popc(tb.rows_of[e * W + (row >> 5)] & ((1u << (row & 31)) - 1u));
        for (int w = 0; w < (row >> 5); ++w) pos += __popc(tb.rows_of[e * W + w]);
        const int v = tb.base[e] + (pos >> 4);
        tb.pair[v * 16 + (pos & 15)] = (uint16_t)i;
        if ((pos & 15) == 0) {
            tb.e[v] = e;
            tb.mask[v] = (1 << min(16, members(e) - pos)) - 1;
        }
    }
    __syncthreads();
    const int U = total;
    if (warp == StWarps<TEAMS>::FIN) {
        int run = 0;
        for (int u0 = 0; u0 < U; u0 += 32) {
            const int c = u0 + lane < U ? __popc(tb.mask[u0 + lane]) : 0;
            int incl = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += up;
            }
            if (u0 + lane < U) tb.pref[u0 + lane] = run + incl - c;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) tb.pref[U] = run;
    }
    return U;
}

// Register split over the warpgroups.  One team: decode and decode keep the 64 of the launch, X + producer give 16 to finish (64 + 64 + 48 +
// 80); decode at 56 registers took 60.5 instead of 58.1 at 8 rows.  Two teams: launched with 80, all give to finish (4 x 64 + 48 + 176).
template <bool INC, int N>
__device__ __forceinline__ void st_regs() {
    if (INC) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// TEAMS: groups of eight decode warps that take the stages in turn.  Two: one CTA an SM with all its registers, for windows whose units
// are one stage each.
template <int SETS, bool MANY, int ROUNDS, int TEAMS>
__global__ void __launch_bounds__(StWarps<TEAMS>::THREADS, TEAMS == 1 ? 2 : 1)
stream_kernel(const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_d,
              const __grid_constant__ StreamArgs a) {
    constexpr int ST_DEC = StWarps<TEAMS>::DEC, ST_PROD = StWarps<TEAMS>::PROD, ST_FIN = StWarps<TEAMS>::FIN, ST_THREADS = StWarps<TEAMS>::THREADS;
    constexpr int DEPTH = TEAMS == 2 ? 8 : 4;                         // partials that a finish warp has on the way: its registers
    static_assert(ST_STAGES % TEAMS == 0, "a team keeps its slots of the ring");
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);          // the swizzle atom is 1024 bytes
    constexpr int XBYTES = SETS * 8 * ST_XROW, SKT = 8 * ROUNDS, SBYTES = SKT * 1024;          // k-tiles and bytes of a stage
    unsigned char *words = smem, *xbuf = smem + ST_STAGES * ST_WBYTES;
    unsigned char *meta = xbuf + ST_STAGES * XBYTES;
    uint64_t *ready = reinterpret_cast<uint64_t *>(meta);             // stage described
    uint64_t *wfull = ready + ST_STAGES;                              // its words landed
    uint64_t *xfull = wfull + ST_STAGES;                              // its activations staged
    uint64_t *empty = xfull + ST_STAGES;                              // consumed
    int4 *desc = reinterpret_cast<int4 *>(meta + 256);                // {kind | matrix << 8 | flags | k, expert number, first word of the partials, -}
    int *job_sh = reinterpret_cast<int *>(desc + ST_STAGES);          // [2]
    StTables tb;
    tb.e = reinterpret_cast<int *>(meta + ST_META);
    tb.mask = tb.e + a.umax;
    tb.pref = tb.mask + a.umax;
    tb.pair = reinterpret_cast<uint16_t *>(tb.pref + a.umax + 1);
    tb.state = reinterpret_cast<short *>(tb.pair + a.umax * 16);
    tb.base = reinterpret_cast<int *>(tb.state + ((a.rows * a.slots + 1) & ~1));
    tb.rows_of = reinterpret_cast<uint32_t *>(tb.base + a.E + 1);
    tb.words = (a.rows + 31) >> 5;
    __shared__ int abort_sh, first_sh;
    __shared__ uint32_t used_sh[32];
    __shared__ __align__(16) float fin_sh[8][128];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int H = a.H, I = a.I, P = a.rows * a.slots;
    const int SK1 = a.cut1.splits, SK2 = a.cut2.splits, NB1 = I >> 7, NB2 = H >> 7;
    const StCta cta{&abort_sh, a.status};
    if (tid == 0) {
        for (int s = 0; s < ST_STAGES; ++s) {
            mbar_init(ready + s, 1);
            mbar_init(wfull + s, 1);
            mbar_init(xfull + s, ST_XW);
            mbar_init(empty + s, 8);
        }
        abort_sh = 0;
        mbar_fence_init();
    }
    if (tid < 32) used_sh[tid] = 0u;
    for (int i = tid; i < a.umax; i += ST_THREADS) tb.mask[i] = 0;
    if (MANY)
        for (int i = tid; i < (a.E + 1) * tb.words; i += ST_THREADS) tb.rows_of[i] = 0u;
    __syncthreads();
    // The arguments of a launch and the tables' inputs are cold everywhere: touch the argument lines (constant-cache misses cost a
    // thousand clocks each where they are met one after another) and hint the inputs into L2 while the kernel before drains.
    // (a plain indexed read of the parameter: a volatile one would not be a parameter-space access)
    if (tid < (int)(sizeof(StreamArgs) / 4)) asm volatile("" ::"r"(reinterpret_cast<const int *>(&a)[tid]));
    if (tid >= 256 && tid < 259) asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)(tid == 256 ? &map_g : tid == 257 ? &map_u : &map_d)) : "memory");
    if (tid < P && tid % 32 == 0 && a.picks) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.picks + tid));
    const int row = tid / a.slots, slot = tid - row * a.slots;        // of routing-table entry number tid
    pdl_launch_dependents();                        // before the wait: the next kernel may start while the one in front of this still runs
    pdl_wait();
    // the first draws of the producer and the finish group travel while the tables are built
    int drawn = 0;
    if (tid == ST_PROD * 32) drawn = (int)atomicAdd(a.ctrl + CTRL_UNIT, 1u);
    if (tid == ST_FIN * 32) drawn = (int)atomicAdd(a.ctrl + CTRL_FIN, 1u);
    const uint32_t epoch = next_epoch(__ldcg(a.ctrl + CTRL_EPOCH));   // words of earlier launches carry others
    const int U = MANY ? st_build_tables_many<TEAMS>(a, tb) : st_build_tables<TEAMS>(a, tb, used_sh, row, slot);
    if (tid == ST_FIN * 32) first_sh = drawn;
    __syncthreads();
    const int units_g = a.do_g ? U * 2 * SK1 * NB1 : 0, units = units_g + (a.do_d ? U * SK2 * NB2 : 0);

    // ---- rotated layer inputs, once per (member, matrix, 128-block): fp16(H(x * suh) / sqrt 128) (upstream rot_in_kernel,
    //      native/exl3.cu:224-241).  They are the first jobs of the finish queue, cut so that every CTA gets about one, and the
    //      first job of a CTA is done by all of its warps but the producer: nothing else can start before.
    const int HB = H >> 7, rots = a.do_g ? tb.pref[U] * 2 * HB : 0;
    const int rot_job = max(1, fast_div(rots + (int)gridDim.x - 1, fast_inv((int)gridDim.x))), jobs_r = fast_div(rots + rot_job - 1, fast_inv(rot_job));
    const float inv_hb = fast_inv(HB), inv_slots = fast_inv(a.slots);
    auto member_expert = [&](int q) {                                 // expert number of member q of all experts' lists
        int lo = 0, hi = U;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (tb.pref[mid] <= q) lo = mid; else hi = mid;
        }
        return lo;
    };
    auto rotate = [&](int r) {                                        // one warp
        const int rq = fast_div(r, inv_hb), k = (r - rq * HB) * 128 + 4 * lane, q = rq >> 1, mat = rq & 1;
        const int u = member_expert(q), p = tb.pair[u * 16 + q - tb.pref[u]];
        const uint2 sv = ldg_half4((mat ? a.suh_u : a.suh_g) + (size_t)tb.e[u] * H + k, a.vec);
        const uint2 xv = __ldcg(reinterpret_cast<const uint2 *>(a.x + (size_t)fast_div(p, inv_slots) * a.x_stride + k));
        const __nv_bfloat162 x01 = *reinterpret_cast<const __nv_bfloat162 *>(&xv.x), x23 = *reinterpret_cast<const __nv_bfloat162 *>(&xv.y);
        const __half2 s01 = *reinterpret_cast<const __half2 *>(&sv.x), s23 = *reinterpret_cast<const __half2 *>(&sv.y);
        float v[4] = {__bfloat162float(x01.x) * __low2float(s01), __bfloat162float(x01.y) * __high2float(s01),
                      __bfloat162float(x23.x) * __low2float(s23), __bfloat162float(x23.y) * __high2float(s23)};
        fwht128(v, lane);
        ll_store2(a.xr + ((size_t)(mat * P + p) * H + k) / 2, pack_half2(v[0] * HAD_SCALE, v[1] * HAD_SCALE), pack_half2(v[2] * HAD_SCALE, v[3] * HAD_SCALE), epoch);
    };
    if (warp != ST_PROD) {
        const int first = first_sh, w = warp - (warp > ST_PROD);
        if (first < jobs_r)
            for (int r = first * rot_job + w; r < min(rots, (first + 1) * rot_job); r += ST_THREADS / 32 - 1) rotate(r);
    }

    if (warp < ST_DEC) {
        // ---------------------------------------------------------------------------------------------- decode
        if (TEAMS == 2) st_regs<false, 64>();
        const int G = lane >> 2, T = lane & 3, tile = warp & 7;
        const uint32_t wfull0 = smem_u32(wfull), xfull0 = smem_u32(xfull), empty0 = smem_u32(empty);
        float acc[SETS][4];                                           // over a split
        for (uint32_t it = warp >> 3;; it += TEAMS) {
            const int s = it % ST_STAGES, phase = (it / ST_STAGES) & 1;
            if (!cta.wait_warp(wfull0 + 8 * s, phase)) break;
            const int4 d = desc[s];
            const int kind = d.x & 0xff;
            if (kind == UNIT_END) break;
            const int nmem = __popc(tb.mask[d.y]);
            const uint32_t p01 = *reinterpret_cast<const uint32_t *>(tb.pair + d.y * 16 + 2 * T);
            const uint32_t p23 = SETS == 2 ? *reinterpret_cast<const uint32_t *>(tb.pair + d.y * 16 + 8 + 2 * T) : 0u;
            if (!cta.wait_warp(xfull0 + 8 * s, phase)) break;
            if (!(d.x & DESC_CONT))
#pragma unroll
                for (int q = 0; q < SETS; ++q)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[q][j] = 0.f;
            const unsigned char *ws = words + s * SBYTES, *xs = xbuf + s * XBYTES;
            // (few experts of a window or chunk have more than eight members; with the second set's operand loads in every
            // unit, eleven rows of the 4096 x 512 layer took 115 us instead of 107 and a chunk of 40 192 instead of 180)
            if (SETS == 1 || nmem <= 8) st_decode<1, MANY, ROUNDS>(ws, xs, tile, lane, reinterpret_cast<float (&)[1][4]>(acc));
            else st_decode<SETS, MANY, ROUNDS>(ws, xs, tile, lane, acc);
            __syncwarp();
            arrive_lane0(empty0 + 8 * s, lane);
            if (!(d.x & DESC_LAST)) continue;
            const int N = kind == UNIT_G ? I : H;
            unsigned long long *z = (kind == UNIT_G ? a.z1 : a.z2) + (unsigned)d.z + tile * 16 + 2 * G;
#pragma unroll
            for (int q = 0; q < SETS; ++q) {
                const uint32_t pp = q ? p23 : p01;
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (q * 8 + 2 * T + j < nmem)
                        ll_store2(z + (size_t)(j ? pp >> 16 : pp & 0xffffu) * N, __float_as_uint(acc[q][j]), __float_as_uint(acc[q][2 + j]), epoch);
            }
        }
    } else if (warp < ST_PROD) {
        st_regs<false, 48>();
        // ---------------------------------------------------------------------------------------------- activations
        const int xw = warp - ST_DEC;
        const uint32_t ready0 = smem_u32(ready), xfull0 = smem_u32(xfull);
        for (uint32_t it = 0;; ++it) {
            const int s = it % ST_STAGES;
            if (!cta.wait_warp(ready0 + 8 * s, (it / ST_STAGES) & 1)) break;
            const int4 d = desc[s];
            const int kind = d.x & 0xff;
            if (kind == UNIT_END) break;
            const int nmem = __popc(tb.mask[d.y]), K = kind == UNIT_G ? H : I;
            const uint16_t *pair = tb.pair + d.y * 16;
            // a warp per member, the loads of two in flight; 128 k are half a warp's, whose other half reads and writes the same again
            const int part = ROUNDS == 2 ? lane : lane & 15;
            const unsigned long long *src = (kind == UNIT_G ? a.xr + (size_t)((d.x >> 8) & 1) * P * (H / 2) : a.xdl) + (d.x >> DESC_K) * 64 + 4 * part;
            unsigned char *xs = xbuf + s * XBYTES + 16 * part;
            const bool poll = kind == UNIT_G || a.do_g;               // (the down phase alone takes what the last run left)
            bool ok = true;
            // (the warps start in turn: most experts have a member or two; 8 rows 59.5 -> 59.1 us a layer with the polls above)
            for (int t0 = (xw + ST_XW - (int)(it % ST_XW)) % ST_XW; t0 < nmem; t0 += 2 * ST_XW) {
                unsigned long long w[2][4];
                int m[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    m[i] = min(t0 + i * ST_XW, nmem - 1);             // past the end: the last one again
                    ll_load4(src + (size_t)pair[m[i]] * (K / 2), w[i]);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (poll && !__all_sync(0xffffffffu, ll_ready(w[i], epoch))) ok = ok && ll_wait4(cta, src + (size_t)pair[m[i]] * (K / 2), epoch, w[i]);
                    *reinterpret_cast<uint4 *>(xs + m[i] * ST_XROW) = make_uint4((uint32_t)w[i][0], (uint32_t)w[i][1], (uint32_t)w[i][2], (uint32_t)w[i][3]);
                }
            }
            __syncwarp();
            if (!ok) break;
            arrive_lane0(xfull0 + 8 * s, lane);
        }
    } else if (warp >= ST_FIN) {
        st_regs<true, TEAMS == 2 ? 176 : 80>();
        // ---------------------------------------------------------------------------------------------- finish
        const int fw = warp - ST_FIN, ft = tid - ST_FIN * 32;
        const int jobs_g = jobs_r + (a.do_g ? tb.pref[U] * NB1 : 0), jobs = jobs_g + (a.do_d ? a.rows * NB2 : 0);
        const float inv_nb1 = fast_inv(NB1), inv_nb2 = fast_inv(NB2);
        if (ft == 0 && drawn < jobs_r) drawn = (int)atomicAdd(a.ctrl + CTRL_FIN, 1u);      // the first job was a rotation: done above
        for (uint32_t it = 0;; ++it) {
            // one thread publishes the group's job and draws the one behind a gate / up job; a group that has given up ends together here
            if (ft == 0) {
                job_sh[it & 1] = abort_sh ? 0x7fffffff : drawn;
                if (drawn < (a.two ? jobs_g : jobs)) drawn = (int)atomicAdd(a.ctrl + CTRL_FIN, 1u);
            }
            asm volatile("bar.sync 5, 128;" ::: "memory");
            const int j = job_sh[it & 1];
            if (j >= jobs) break;
            if (j < jobs_r) {
                for (int r = j * rot_job + fw; r < min(rots, (j + 1) * rot_job); r += 4) rotate(r);
            } else if (j < jobs_g) {
                // gate / up of one member: warp 2 adds the up matrix's partials, transforms them and hands the clamped values over; warp
                // 0 does the same for gate, applies SwiGLU, rotates and stores.
                const int q = fast_div(j - jobs_r, inv_nb1), nb = j - jobs_r - q * NB1, lo = member_expert(q);
                const int role = fw >> 1, half = fw & 1;
                const int p = tb.pair[lo * 16 + q - tb.pref[lo]], col = nb * 128 + 4 * lane;
                const size_t so = (size_t)tb.e[lo] * I + col;
                const uint2 sv = ldg_half4((role ? a.svh_u : a.svh_g) + so, a.vec);
                const uint2 sd = ldg_half4(a.suh_d + so, a.vec);
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                const unsigned long long *z = a.z1 + ((size_t)role * SK1 * P + p) * I + nb * 128 + z_word(lane);
                if (a.two) {
                    // With two CTAs an SM eight finish warps are always waiting, and their polls cost the decode warps issue slots: only
                    // warp 3 polls, for the partial that is drawn last (16 rows: 695 -> 671 us over 8 layers; with one CTA the extra
                    // round trip costs more, 47 layers of one row 1128 -> 1141 us).
                    unsigned long long last[4];
                    if (fw == 3) ll_wait4(cta, z + (size_t)(SK1 - 1) * P * I, epoch, last);
                    asm volatile("bar.sync 5, 128;" ::: "memory");
                }
                if (!half) {
                    sum_splits<DEPTH>(a.two, cta, z, (size_t)P * I, 0, SK1, epoch, v);
                    z_columns(v, lane);
                    fwht128(v, lane);
                    const float2 c01 = __half22float2(*reinterpret_cast<const __half2 *>(&sv.x)), c23 = __half22float2(*reinterpret_cast<const __half2 *>(&sv.y));
                    const float r[4] = {bf16r(v[0] * HAD_SCALE * c01.x), bf16r(v[1] * HAD_SCALE * c01.y), bf16r(v[2] * HAD_SCALE * c23.x),
                                        bf16r(v[3] * HAD_SCALE * c23.y)};
                    if (role == 1) {
                        *reinterpret_cast<float4 *>(&fin_sh[2][4 * lane]) =
                            make_float4(fminf(fmaxf(r[0], -a.limit), a.limit), fminf(fmaxf(r[1], -a.limit), a.limit),
                                        fminf(fmaxf(r[2], -a.limit), a.limit), fminf(fmaxf(r[3], -a.limit), a.limit));
                        pair_barrier(2);
                    } else {
                        float sg[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float g = fminf(r[i], a.limit);
                            sg[i] = bf16r(silu(g));
                        }
                        pair_barrier(2);
                        const float4 uu = *reinterpret_cast<const float4 *>(&fin_sh[2][4 * lane]);
                        const float2 d01 = __half22float2(*reinterpret_cast<const __half2 *>(&sd.x)), d23 = __half22float2(*reinterpret_cast<const __half2 *>(&sd.y));
                        float o4[4] = {bf16r(sg[0] * uu.x) * d01.x, bf16r(sg[1] * uu.y) * d01.y, bf16r(sg[2] * uu.z) * d23.x, bf16r(sg[3] * uu.w) * d23.y};
                        fwht128(o4, lane);
                        const uint32_t w0 = pack_half2(o4[0] * HAD_SCALE, o4[1] * HAD_SCALE), w1 = pack_half2(o4[2] * HAD_SCALE, o4[3] * HAD_SCALE);
                        if (!abort_sh) {
                            ll_store2(a.xdl + ((size_t)p * I + col) / 2, w0, w1, epoch);
                            if (a.xd) *reinterpret_cast<uint2 *>(a.xd + (size_t)p * I + col) = make_uint2(w0, w1);
                        }
                    }
                }
                // (the group's barrier at the top of the loop separates the uses of fin_sh of one job from the next: a warp
                // writes its row of the next job only after every warp of the group has passed it)
            } else {
                // down: the slots of a row eight at a time, two per warp, then the weighted sum, ascending slots
                const int row = fast_div(j - jobs_g, inv_nb2), nb = j - jobs_g - row * NB2, col = nb * 128 + 4 * lane;
                float acc = 0.f;
                // (a routing weight a lane, on its way while the sums are: one after another behind them they were 3,000 clocks at the end of a layer)
                const float wgt = a.out && lane < a.slots ? __ldcg(a.route_w + row * a.slots + lane) : 0.f;
                for (int s0 = 0; s0 < a.slots; s0 += 8) {
                    int e[2];
                    float v[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                    uint2 sv[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int s = s0 + 4 * i + fw, p = row * a.slots + s;
                        e[i] = s < a.slots ? tb.state[p] : -1;
                        if (e[i] >= 0) sv[i] = ldg_half4(a.svh_d + (size_t)e[i] * H + col, a.vec);
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        if (e[i] >= 0)
                            sum_splits<DEPTH>(a.two, cta, a.z2 + (size_t)(row * a.slots + s0 + 4 * i + fw) * H + nb * 128 + z_word(lane), (size_t)P * H, 0, SK2, epoch, v[i]);
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        if (e[i] >= 0) {
                            z_columns(v[i], lane);
                            fwht128(v[i], lane);
                        }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float *y = a.y + (size_t)(row * a.slots + s0 + 4 * i + fw) * H + col;
                        if (e[i] >= 0) {
                            const float2 c01 = __half22float2(*reinterpret_cast<const __half2 *>(&sv[i].x)), c23 = __half22float2(*reinterpret_cast<const __half2 *>(&sv[i].y));
                            const float4 o = make_float4(v[i][0] * HAD_SCALE * c01.x, v[i][1] * HAD_SCALE * c01.y, v[i][2] * HAD_SCALE * c23.x,
                                                         v[i][3] * HAD_SCALE * c23.y);
                            *reinterpret_cast<float4 *>(y) = o;
                            *reinterpret_cast<float4 *>(&fin_sh[4 * i + fw][4 * lane]) = o;
                        } else if (e[i] == -2) {                  // a repeated pick: its pair row is not computed here
                            *reinterpret_cast<float4 *>(&fin_sh[4 * i + fw][4 * lane]) = *reinterpret_cast<const float4 *>(y);
                        }
                    }
                    // A down job's successor is drawn behind its sums: one that waited behind a waiting job was done after it, with other CTAs
                    // idle (16 rows: 7,000 clocks at the end of a layer, 8 layers 625 -> 590 us; one row has a job for one CTA in nine, and
                    // loses 6 us of 1,050 by the late draw).
                    if (a.two && ft == 0 && s0 + 8 >= a.slots) drawn = (int)atomicAdd(a.ctrl + CTRL_FIN, 1u);
                    if (a.out) {
                        asm volatile("bar.sync 5, 128;" ::: "memory");
                        for (int i = 0; i < min(8, a.slots - s0); ++i) {
                            const float w = __shfl_sync(0xffffffffu, wgt, s0 + i);
                            if (tb.state[row * a.slots + s0 + i] != -1) {
                                const float y = fin_sh[i][ft];
                                acc = s0 + i == a.slots - 1 ? acc + y : fmaf(w, y, acc);       // (one rounding, however the branch is compiled)
                            }
                        }
                        asm volatile("bar.sync 5, 128;" ::: "memory");
                    }
                }
                if (a.out) a.out[(size_t)row * H + nb * 128 + ft] = acc;
                if (a.out2) a.out2[(size_t)row * H + nb * 128 + ft] = acc;
            }
        }
    } else {
        // ---------------------------------------------------------------------------------------------- producer
        st_regs<false, 48>();
        uint32_t it = 0;
        bool ok = true;
        const float inv_nb1 = fast_inv(NB1), inv_nb2 = fast_inv(NB2), inv_sk1 = fast_inv(SK1), inv_sk2 = fast_inv(SK2);
        const int split1 = a.cut1.split, split2 = a.cut2.split;
        while (ok) {
            // A unit is drawn only when there is room for it (the draw and the copy take 3,000 clocks, the stages in front of it
            // 6,000 and more): units drawn earlier would only arrive late at whoever waits for their sums.
            int s = it % ST_STAGES;
            ok = __all_sync(0xffffffffu, cta.wait(empty + s, ((it / ST_STAGES) & 1) ^ 1));
            if (!ok) break;
            if (it && lane == 0) drawn = (int)atomicAdd(a.ctrl + CTRL_UNIT, 1u);
            int t = __shfl_sync(0xffffffffu, drawn, 0);
            if (t >= units) {
                for (int team = 0; team < TEAMS && ok; ++team) {      // one end for each
                    if (team) {
                        s = ++it % ST_STAGES;
                        ok = __all_sync(0xffffffffu, cta.wait(empty + s, ((it / ST_STAGES) & 1) ^ 1));
                        if (!ok) break;
                    }
                    if (lane == 0) {
                        desc[s] = make_int4(UNIT_END, 0, 0, 0);
                        mbar_arrive(ready + s);
                        mbar_arrive(wfull + s);
                    }
                    __syncwarp();
                }
                break;
            }
            const bool g = t < units_g;
            if (!g) t -= units_g;
            const int q = fast_div(t, g ? inv_nb1 : inv_nb2), nb = t - q * (g ? NB1 : NB2);
            t = fast_div(q, g ? inv_sk1 : inv_sk2);
            const int split = q - t * (g ? SK1 : SK2), mat = g ? t & 1 : 0, u = g ? t >> 1 : t, head = (g ? UNIT_G : UNIT_D) | mat << 8;
            const CUtensorMap *map = g ? (mat ? &map_u : &map_g) : &map_d;
            const int KT = (g ? H : I) >> 4, len = g ? split1 : split2, row = tb.e[u] * KT, first = split * len, last = min(KT, first + len);
            const unsigned z = (unsigned)(mat * SK1 + split) * (unsigned)(P * (g ? I : H)) + (unsigned)(nb * 128);
            for (int kt = first;;) {
                const bool end = kt + SKT == last;
                if (lane == 0) {
                    desc[s] = make_int4(head | (kt != first ? DESC_CONT : 0) | (end ? DESC_LAST : 0) | (kt >> 3) << DESC_K, u, (int)z, 0);
                    mbar_arrive(ready + s);
                    mbar_expect_tx(wfull + s, SBYTES);
                    tma_load_3d(words + s * SBYTES, map, 0, row + kt, nb * 8, wfull + s);
                }
                ++it;
                kt += SKT;
                if (end) break;
                s = it % ST_STAGES;
                ok = __all_sync(0xffffffffu, cta.wait(empty + s, ((it / ST_STAGES) & 1) ^ 1));
                if (!ok) break;
            }
        }
        // after a give-up copies may be in flight: they have landed before the CTA leaves (bounded)
        if (abort_sh && lane == 0)
            for (uint32_t k = it > ST_STAGES ? it - ST_STAGES : 0; k < it; ++k) mbar_wait(wfull + k % ST_STAGES, (k / ST_STAGES) & 1);
    }
    __syncthreads();
    if (tid == 0) {
        // the last CTA of the launch puts the counters back and advances the epoch; a later launch of the stream reads them
        if (atomicAdd(a.ctrl + CTRL_DONE, 1u) == gridDim.x - 1) {
            a.ctrl[CTRL_UNIT] = 0u;
            a.ctrl[CTRL_FIN] = 0u;
            a.ctrl[CTRL_DONE] = 0u;
            a.ctrl[CTRL_EPOCH] = epoch;
        }
    }
}

// Whether two CTAs of a chunk of these rows share an SM: with many experts the tables of the window take the room.
bool stream_chunk_pairs(const glmflash_config &c, int rows) {
    return st_smem_bytes(2, stream_umax(c, rows, false), rows, rows * c.slots, c.experts) <= ST_TWO_SMEM;
}

int launch_stream(cudaStream_t s, StreamArgs a, bool pdl) {
    static int sms[64] = {};
    static bool configured[64][7] = {};
    int dev = 0;
    GF_CUDA(cudaGetDevice(&dev));
    GF_REQUIRE(dev >= 0 && dev < 64, "device ordinal out of range");
    if (!sms[dev]) GF_CUDA(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev));
    // Stages of 128 k where a split is not a whole number of 256 k (K = 2304): the stage is a constant of the kernel.
    const bool fine = a.cut1.split % 16 || a.cut2.split % 16;
    const int sets = a.rows > 8 ? 2 : 1;
    size_t smem = st_smem_bytes(sets, a.umax, a.rows, a.rows * a.slots, a.E);
    GF_REQUIRE(smem <= ST_MAX_SMEM, "routing table too large for the window kernel");
    // CTAs per SM.  One has shorter chains for few units (one token: 23.8 us a layer, 28.6 with two); two fill the decode pipes (16
    // rows: 80 against 95 us).  The lines cross at about nine units of 512 k per SM, counted with one expert per pick of this GPU's
    // window (us with one | two; 2048 x 1536, 2 rows, 9.7 units: 34.2 | 33.2; 3 rows, 14.6: 42.1 | 38.9; 2304 x 768, 2 rows, 6.5: 26.0 |
    // 26.4; 1024 x 2048, 3 rows, 7.8: 24.9 | 26.7).
    const long pairs = (long)a.rows * (((long)(a.slots - 1) * (a.e_hi - a.e_lo) + a.E - 1) / a.E + (a.shared ? 1 : 0));
    const long units = std::min<long>(pairs, a.umax) * (2L * ((a.H + 511) / 512) * (a.I / 128) + (long)((a.I + 511) / 512) * (a.H / 128));
    const int per_sm = units >= 9L * sms[dev] ? 2 : 1;
    a.two = per_sm == 2;
    // Two teams of decode warps (sixteen) where one CTA has an SM and every unit is one stage of 256 k (a unit of more would have to stay
    // with its team): eight warps form 15 weights a clock beside the other roles, sixteen 18 (47 layers of one row 1105 -> 1050 us, 8 with
    // their router 257 -> 245).
    const bool teams = per_sm == 1 && a.rows <= 16 && a.cut1.split == 16 && a.cut2.split == 16;
    // (chunks have a kernel of their own: with their tables as a branch, windows of 11 rows were 1 % slower)
    const int which = a.rows > 16 ? 4 : teams ? 4 + sets : sets - 1 + 2 * fine;
    const auto kernel = which == 0   ? stream_kernel<1, false, 2, 1>
                        : which == 1 ? stream_kernel<2, false, 2, 1>
                        : which == 2 ? stream_kernel<1, false, 1, 1>
                        : which == 3 ? stream_kernel<2, false, 1, 1>
                        : which == 4 ? stream_kernel<2, true, 2, 1>
                        : which == 5 ? stream_kernel<1, false, 2, 2>
                                     : stream_kernel<2, false, 2, 2>;
    const dim3 grid((unsigned)(sms[dev] * per_sm)), block(teams ? StWarps<2>::THREADS : StWarps<1>::THREADS);
    // One CTA per SM asks for more than half of the shared memory: next to a few CTAs of another kernel (the router of the next
    // layer) the second CTA of an emptier SM was placed before the first of a busier one (8 layers of one token with their
    // router 293 -> 266 us; 47 without 1140 -> 1144, whose next layer now sets up after this one).
    if (per_sm == 1) smem = std::max<size_t>(smem, ST_HALF_SM);
    if (!configured[dev][which]) {                 // (a bound, not a request; threads that come here together set the same)
        GF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ST_MAX_SMEM));
        configured[dev][which] = true;
    }
    CUtensorMap mg, mu, md;
    const uint32_t kt = fine ? 8 : 16;
    if (bank_map(&mg, a.gt, a.E + 1, a.H, a.I, kt) || bank_map(&mu, a.ut, a.E + 1, a.H, a.I, kt) || bank_map(&md, a.dt, a.E + 1, a.I, a.H, kt)) return -1;
    return launch_k(kernel, grid, block, smem, s, pdl, mg, mu, md, a);
}

}  // namespace gf
