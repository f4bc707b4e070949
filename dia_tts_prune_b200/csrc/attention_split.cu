// attention_split.cu - softmax attention of many query rows on the 5th-generation tensor cores, with fp32 operands split into
// two fp16 terms (sm_100a).
//
// A CTA owns 128 (token, head) rows: up to 128 / PK consecutive tokens times PK query heads that read the same key/value head, so
// that a tile of keys serves all of them.  It walks its keys 64 at a time:
//   3 warps   fetch key and value tiles into a ring of shared-memory slots.  A launch in front has scaled them by powers of two and split
//             x = hi + lo into fp16 ([key / 8][channel / 8] blocks of 8 x 16 bytes: the layout is the K-major operand of the scores and the
//             MN-major operand of the value product), so that one lane copies a tile.  Keys beyond the room for them are split here, in an instance of its own
//   1 warp    issues tcgen05.mma: scores S = Q K^T (M = 128, N = 64; lo hi, hi lo, then hi hi, so that the small terms are
//             added first) per group of at most 128 channels, and the value product of a tile before (weights as the
//             operand in tensor memory)
//   8 warps   two groups of four take turns: one thread weighs all 64 keys of its row of a tile - scores from tensor memory (the channel groups
//             are summed here, in fp32), cap, bias, mask, online softmax in base 2, weights split and written to tensor memory.  All a row's two
//             threads tell each other of a tile is the maximum (which the group that has the next tile needs when it has its scores), the
//             weights' scale and two of their four sums.  Both add the value product of every tile to fp32 registers, half of the channels each
// The accumulator of a tensor-core product loses up to one unit in the last place at every step, towards zero (measured: 2e-6
// over K = 2048).  So no accumulator lives longer than one tile and one channel group, and sums over tiles are fp32 additions
// in registers: measured against 64 bits the output is closer than the fp32 FMA kernels' (relative 2-norm, 300 rows, two heads of 128,
// capped: 2.4e-7 against 2.9e-7; 1500 rows, 4 heads of 128: 2.7e-7 against 4.1e-7).
//
// Scaling: every query row, key row and value row is brought to a largest magnitude of [2^14, 2^15) by a power of two of its own
// before the split.  A query's and a key's are undone on the score; a value's joins the weight, and the weights of a row and a tile
// of keys, times their values' magnitudes, are brought to the same range before they are split.  So an element down to 2^-17 of its
// row's largest keeps its 22 bits (a smaller one is off by at most 2^-39 of the largest: a channel that is 2^17 times below the others of
// its tokens has fewer), and nothing of a token that a row does not see, or of another row, enters its result: the bits do not depend on
// what shares the launch.
//
// Bound: the latencies of the row warps' chains.  Per 64 keys and 128 rows 3 x 128 x 64 x (dk + dv) multiply-adds on the tensor pipe (128 + 128: 1150 cycles of
// the scores, whose operands take all of shared memory's bandwidth, and 770) stand against about 5000 cycles.  A row's 64 scores take a thread some 1500
// instructions; with two such warps a scheduler issues on 40 % of the cycles (windowed rows; 31 % over latent rows and for Dia's prompts), and the tensor pipe is
// busy for 24 % (27, 20).  What warps wait for instead, in the same order: instruction fetches 29, 8 and 27 % of their stalls (the code of a tile's turn is some
// 35 KB with the cap; loops are rolled where a roll is possible), loads from tensor memory and of spilled registers 18, 49 and 25 %, fixed latencies 24, 20 and
// 20 %.  Four threads per row that exchanged a tile's maxima and largest weights, 16 keys each, took 8000 cycles.  Times (us, four or two threads per row / now):
// windowed 4096 rows, 16 heads of 128 over 4, window 1024, capped 238 / 205; the same rows over latent rows of 256 + 32 408 / 368; mixed scores, prompts of 1500,
// 333 and 215 rows, 8 heads of 128 over 2 116 / 90; float32 model of 978 rows, four layers 216 / 191; Dia, 861 frames, 36 attentions 3024 / 1624 and 213 for the
// split keys, which every row tile used to split for itself; 9 decoding sequences over 1134 latent rows 281 / 128.
// Every wait is bounded: a wait that runs out makes the CTA write NaN, note it in a word that the host reads, and end; the next launch
// on the device returns an error.
#include <algorithm>
#include <mutex>

#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "attention_split.h"
#include "common.cuh"
#include "gemm_tcgen05.h"

namespace dia {

namespace {

constexpr int kRows = 128, kKeys = 64, kGroupW = 128;        // query rows of a CTA, keys of a tile, channels of a stage
constexpr int kRowWarps = 8, kFetchWarps = 3, kSplitThreads = 32 * (kRowWarps + 1 + kFetchWarps);
constexpr int kMaxSlots = 6, kMaxKStages = 4;
constexpr int kSmemMost = 232448;                             // all of it dynamic
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kSplitGrid = 148 * 16;                           // CTAs of the launch that splits them
constexpr unsigned kSpinMost = 4000000u;

struct Geometry {
    int pk_shift;                            // log2 of the heads of a CTA's rows
    int n_kst, n_vst;                        // channel groups of a key, of a value
    int wk0, wk_last;                        // their padded widths (multiples of 16): all but the last, the last
    int wv0, wv_last;
    int v0_layout, v_last_layout;            // widths in which the value groups lie in a slot (a latent's value group is its key group)
    int shared_kv;                           // the value is the head of the key row: value group i is key group i
    int slot_bytes, n_slots, q_bytes;
    int s_bufs, p_bufs, o_bufs;              // tiles of scores, of weights and of value products in tensor memory (1 or 2 of each)
    int k_sets;                              // scales of a key: one, with mixed scores one per kv head
    int depth;                               // tiles whose scales are in shared memory
    int rings;                               // tiles whose rows' numbers are (2 or 4)
    int four;                                // a denominator per 16 keys (see split_attention_kernel)
    // the split keys and values in SplitAttention::work: SlotTiles per slot, then inverse scales [tile][set][key], then the tiles.  A
    // tile's parts: key groups (per kv head where the launch reads one head at a time), then value groups; its sets of scales: the keys
    // of each kv head, then the values of each (shared_kv: the keys' only)
    int parts, k_parts, sets, cap_tiles;
    int page_shift;                          // log2 of the page size (-1: it is no power of two)
    int* ran_out;                            // the device's word (null: none)
    unsigned tile_bytes, scale_off, tile_off;
};
// where the tiles of a slot's sequence lie: tile j / 64 of its keys is tile base + j / 64 of the room for first <= j / 64 < end; its
// tile 0 is tile `zero` (-1: only by the range)
struct SlotTiles { int base, first, end, zero; };

__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity) {
#pragma unroll 1
    for (unsigned i = 0; i < kSpinMost; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// one look that does not wait
__device__ __forceinline__ bool has_passed(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
// the same for a converged warp, with one answer for all lanes (so that what follows is uniform: see elect_one_sync)
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity) {
#pragma unroll 1
    for (unsigned i = 0; i < kSpinMost; ++i)
        if (__any_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return false;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// operands without swizzle: blocks of 8 rows x 16 bytes; lead / stride: bytes between blocks along the contraction / the rows
// (K-major) or along the contraction / the channels (MN-major)
__device__ __forceinline__ uint64_t block_desc(uint32_t addr, uint32_t lead, uint32_t stride) {
    const uint32_t lo = ((addr & 0x3FFFFu) >> 4) | ((lead >> 4) << 16);
    const uint32_t hi = (stride >> 4) | (1u << 14);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void commit_to(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_smem_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tmem_loaded() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_load32(uint32_t addr, float (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
          "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]),
          "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]),
          "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t addr, float* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
          "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_load8(uint32_t addr, float (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(addr)
                 : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_load_pairs(uint32_t addr, f2* p) {       // 2 N columns
    static_assert(N == 8 || N == 16, "columns of a load");
    float v[2 * N];
    if constexpr (N == 16) tmem_load32(addr, v);
    else tmem_load16(addr, v);
    tmem_loaded();
#pragma unroll
    for (int e = 0; e < N; ++e) p[e] = pack2(v[2 * e], v[2 * e + 1]);
}
// tanh x = x + x^3 q(x^2) for |x| <= kTanhRange: q interpolates (tanh x / x - 1) / x^2 at six Chebyshev nodes (relative error of the
// result 3e-10 before rounding).  A tile's scores mostly lie there, and it takes a fifth of the library call's instructions
// (a tile of capped scores: 2100 -> 800 cycles)
constexpr float kTanhRange = 0.6f;
__device__ __forceinline__ f2 tanh_near_zero(f2 x) {
    const f2 u = mul2(x, x);
    f2 q = twice(2.3707656405e-3f);
    q = fma2(q, u, twice(-8.41007080153e-3f));
    q = fma2(q, u, twice(2.17883219971e-2f));
    q = fma2(q, u, twice(-5.39615517813e-2f));
    q = fma2(q, u, twice(1.33333128669e-1f));
    q = fma2(q, u, twice(-3.33333332312e-1f));
    return fma2(mul2(x, u), q, x);
}
// v[i] *= f[i], N pairs (16-byte aligned; the same addresses for all lanes)
template <int N>
__device__ __forceinline__ void scale_by(f2* v, const float* f) {
#pragma unroll
    for (int e = 0; e < N; e += 2) {
        const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(f + 2 * e);
        v[e] = mul2(v[e], k.x);
        v[e + 1] = mul2(v[e + 1], k.y);
    }
}
__device__ __forceinline__ void tmem_store8(uint32_t addr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

// (x, y) = hi + lo, both rounded to fp16
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void split2(f2 v, uint32_t& hi, uint32_t& lo) {
    float x, y;
    unpack2(v, x, y);
    split2(x, y, hi, lo);
}
// (lo, hi) = the terms of eight values times f: the same as split2 of each, two at a time
__device__ __forceinline__ void split8(const ulonglong2& a, const ulonglong2& b, f2 f, uint4& hi, uint4& lo) {
    const f2 v[4] = {mul2(a.x, f), mul2(a.y, f), mul2(b.x, f), mul2(b.y, f)};
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float x, y;
        unpack2(v[i], x, y);
        const __half2 t = __floats2half2_rn(x, y);
        const float2 u = __half22float2(t);
        unpack2(add2(v[i], pack2(-u.x, -u.y)), x, y);
        const __half2 r = __floats2half2_rn(x, y);
        h[i] = *reinterpret_cast<const uint32_t*>(&t);
        l[i] = *reinterpret_cast<const uint32_t*>(&r);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}
// the power of two that brings a largest magnitude m to [2^14, 2^15), and its inverse (m = 0: 2^114; both stay normal numbers)
__device__ __forceinline__ float scale_of(float m, float& inverse) {
    const int e = max((int)(__float_as_uint(m) >> 23) - 127, -100);
    inverse = __uint_as_float((uint32_t)(e + 113) << 23);
    return __uint_as_float((uint32_t)(min(141 - e, 254)) << 23);
}
constexpr float kFloatMost = 3.402823466e38f;
__device__ __forceinline__ float max_nan(float a, float b) {  // (fmaxf drops a NaN)
    float m;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
    return m;
}
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float m;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}
__device__ __forceinline__ float warp_max_nan(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max_nan(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float max_abs4(float m, const float4& v) {
    return max_nan(max_nan(max_nan(max_nan(m, fabsf(v.x)), fabsf(v.y)), fabsf(v.z)), fabsf(v.w));
}
// lanes 8 apart hold the channels of one row
__device__ __forceinline__ float row_max(float v) {
    v = max_nan(v, __shfl_xor_sync(0xffffffffu, v, 8));
    return max_nan(v, __shfl_xor_sync(0xffffffffu, v, 16));
}
// A row with an infinity or a NaN cannot be split: its terms are zeros (true), and its inverse scale is NaN, which makes the scores, or the
// weights, of those that see it NaN and nobody else's; they are computed once more by plain_row.
__device__ __forceinline__ bool scale_row(float m, float& scale, float& inverse) {
    scale = scale_of(m, inverse);
    const bool bad = !(m <= kFloatMost);
    if (bad) inverse = CUDART_NAN_F;
    return bad;
}
__device__ __forceinline__ int first_key_of(int i, int window, int chunk) {
    const int w = window > 0 ? max(0, i - window + 1) : 0;
    return chunk > 0 ? max(w, i - i % chunk) : w;
}

// how many keys of a slot some row sees (rows_per_slot > 0)
__host__ __device__ __forceinline__ int range_keys(const SplitAttention& p, int slot) {
    const int n = p.mode == 2 && p.n_valid[slot] < p.n_keys ? p.n_valid[slot] : p.n_keys;
    return p.mode == 0 && p.rows_per_slot < n ? p.rows_per_slot : n;
}

__device__ __forceinline__ size_t part_offset(const Geometry& geo, int part) {
    const unsigned k_head = kKeys * 4u * ((geo.n_kst - 1) * geo.wk0 + geo.wk_last), v_head = kKeys * 4u * ((geo.n_vst - 1) * geo.wv0 + geo.wv_last);
    if (part < geo.k_parts) return (size_t)(part / geo.n_kst) * k_head + (size_t)(part % geo.n_kst) * geo.wk0 * kKeys * 4;
    part -= geo.k_parts;
    return (size_t)(geo.k_parts / geo.n_kst) * k_head + (size_t)(part / geo.n_vst) * v_head + (size_t)(part % geo.n_vst) * geo.wv0 * kKeys * 4;
}

// Splits the keys and values that the step's rows see, once for all row tiles: without it each of the M rep / 128 row tiles of a
// key/value head converts every tile it walks, and that conversion (two thirds of the instructions) bounds the kernel below.
// A CTA per (tile of the room, part), but kSplitGrid of them at most, which take further tiles in turn and look up whose they are each time: a room for
// many sequences has far more tiles than a short step fills.  Tiles are dealt to the sequences in order.  Warp w takes keys 8 w .. of the tile.
__global__ void __launch_bounds__(256)
split_keys_kernel(const __grid_constant__ SplitAttention p, const __grid_constant__ Geometry geo) {
    __shared__ int s_first, s_seq, s_run;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = blockIdx.y;
    for (int tile = blockIdx.x; tile < geo.cap_tiles; tile += gridDim.x) {
        const bool writes_plan = tile == 0 && part == 0;
        SlotTiles* plan = reinterpret_cast<SlotTiles*>(p.work);
        // ---- which sequence's tile is this? ----
        __syncthreads();                                          // (the last tile's answer has been read)
        if (tid == 0) { s_seq = -1; s_run = 0; }
        __syncthreads();
        if (p.rows_per_slot > 0 && tid == 0) {                // every slot's keys from 0 on
            int begin = 0;
            for (int slot = 0; slot * p.rows_per_slot < p.M; ++slot) {
                const int n = (range_keys(p, slot) + kKeys - 1) / kKeys;
                if (writes_plan) plan[slot] = SlotTiles{begin, 0, min(n, geo.cap_tiles - begin), -1};
                if (tile >= begin && tile < begin + n) s_seq = slot, s_first = tile - begin;
                begin += n;
            }
        }
        if (p.rows_per_slot > 0) __syncthreads();
        for (int s0 = 0; s0 < p.n_seq; s0 += 32) {                // warp 0: 32 sequences at a time, running sum of their tiles
            if (warp == 0) {
                const int s = s0 + lane;
                int first = 0, n = 0, slot = 0, extra = 0, end = 0;
                if (s < p.n_seq) {
                    slot = p.seq_slot[s];
                    const int r = p.seq_row0[s], pos = p.row_pos[r];
                    first = first_key_of(pos, p.window, p.chunk) / kKeys;
                    end = (pos + p.seq_count[s] + kKeys - 1) / kKeys;
                    extra = p.window > 0 && p.keep_first > 0 && first > 0 ? 1 : 0;    // tile 0 holds the kept keys (of at most 64)
                    n = end - first + extra;
                }
                int sum = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += v;
                }
                const int begin = s_run + sum - n;
                if (writes_plan && s < p.n_seq) {
                    SlotTiles t;
                    t.zero = extra && begin < geo.cap_tiles ? begin : -1;
                    t.base = begin + extra - first;
                    t.first = first;
                    t.end = min(end, geo.cap_tiles - t.base);
                    plan[slot] = t;
                }
                if (s < p.n_seq && tile >= begin && tile < begin + n) {
                    s_seq = s;
                    s_first = extra && tile == begin ? 0 : first + tile - begin - extra;
                }
                __syncwarp();
                if (lane == 31) s_run += sum;
                __syncwarp();
            }
            __syncthreads();
            if (s_seq >= 0 && !writes_plan) break;                // (the same for all threads: read behind the barrier)
            __syncthreads();
        }
        if (s_seq < 0) return;                                // (nor does any later tile belong to one)
        const bool ranged = p.rows_per_slot > 0;
        const int seq = s_seq, slot = ranged ? seq : p.seq_slot[seq], k_end = ranged ? range_keys(p, slot) : p.row_pos[p.seq_row0[seq]] + p.seq_count[seq],
                  j0 = s_first * kKeys;
        // ---- which rows and channels? ----
        const bool is_v = part >= geo.k_parts;
        const int q = is_v ? part - geo.k_parts : part, per = is_v ? geo.n_vst : geo.n_kst, gg = q / per, st = q % per;
        const bool talk = p.talk != nullptr && !is_v;             // (a key group is a whole kv head there)
        const int g = talk ? st : gg, c0 = talk ? 0 : st * kGroupW;
        const int w = talk ? p.kdim : min(kGroupW, (is_v ? p.vdim : p.kdim) - c0), wp = is_v ? (st == per - 1 ? geo.wv_last : geo.wv0) : (st == per - 1 ? geo.wk_last : geo.wk0);
        const int width = is_v ? p.vrow : p.kdim, kin = lane & 7, cq = lane >> 3, j = j0 + warp * 8 + kin, blocks = wp >> 3;
        const bool in = j < k_end;
        const float* src = is_v ? p.vcache : p.kcache;
        if (in) {
            const int page = p.table ? p.table[(size_t)slot * p.max_pages + j / p.page_size] : slot;
            src += (((size_t)page * p.kv_heads + g) * p.page_size + (p.table ? j % p.page_size : j)) * width;
        }
        float4 v[8];
        float m = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = 8 * (cq + 4 * i);
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            v[2 * i] = in && c < w ? *reinterpret_cast<const float4*>(src + c0 + c) : z;
            v[2 * i + 1] = in && c + 4 < w ? *reinterpret_cast<const float4*>(src + c0 + c + 4) : z;
        }
        // the scale is that of the whole row (a latent's value is a part of its key row)
        const int row_w = is_v ? p.vdim : p.kdim;
#pragma unroll
        for (int i = 0; i < 8; ++i) m = max_abs4(m, v[i]);
        if (w < row_w && in)
            for (int c = 4 * cq; c < row_w; c += 16) m = max_abs4(m, *reinterpret_cast<const float4*>(src + c));
        float sc, inverse;
        if (scale_row(row_max(m), sc, inverse)) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        unsigned char* work = reinterpret_cast<unsigned char*>(p.work);
        const int set = is_v ? p.kv_heads + gg : talk ? st : gg;
        if (cq == 0 && (talk || st == 0))
            reinterpret_cast<float*>(work + geo.scale_off)[((size_t)tile * geo.sets + set) * kKeys + warp * 8 + kin] = inverse;
        unsigned char* base = work + geo.tile_off + (size_t)tile * geo.tile_bytes + part_offset(geo, part);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c8 = cq + 4 * i;
            if (c8 >= blocks) continue;
            uint32_t hi[4], lo[4];
            split2(v[2 * i].x * sc, v[2 * i].y * sc, hi[0], lo[0]);
            split2(v[2 * i].z * sc, v[2 * i].w * sc, hi[1], lo[1]);
            split2(v[2 * i + 1].x * sc, v[2 * i + 1].y * sc, hi[2], lo[2]);
            split2(v[2 * i + 1].z * sc, v[2 * i + 1].w * sc, hi[3], lo[3]);
            unsigned char* dst = base + (warp * blocks + c8) * 128 + kin * 16;
            *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(dst + kKeys * wp * 2) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
}

// The key tiles of a CTA in the order in which every role walks them.  A segment is a maximal run of the CTA's tokens with one
// slot and consecutive positions (and, by row mode 1, on one side of n); its keys are the kept first positions in front of its
// window range (phase 0), then the range from its first token's first key on (phase 1).  Tiles start on multiples of 64 (keys in
// front of a token's first key are masked), so that a tile split in advance serves every row tile.
struct Walk {
    const int* s_slot; const int* s_pos;
    const uint32_t* breaks;                                   // bit i: token i does not continue token i - 1's segment
    int n, seg_a, seg_b, phase, j0, k_end, lo;
    __device__ Walk(const int* slots, const int* pos, const uint32_t* brk, int n_tok)
        : s_slot(slots), s_pos(pos), breaks(brk), n(n_tok), seg_a(0), seg_b(0), phase(1), j0(0), k_end(0), lo(0) {}
    // true: tile [j0, min(j0 + 64, k_end)) of the segment's sequence
    __device__ bool next(const SplitAttention& p) {
        if (j0 < k_end) j0 += kKeys;                          // (the tile that was walked last)
        for (;;) {
            if (j0 < k_end) return true;
            if (phase == 0) {
                phase = 1;
                j0 = lo;
                k_end = s_pos[seg_b - 1] + 1;
                if (p.rows_per_slot > 0) k_end = min(k_end, p.n_keys);
                continue;
            }
            seg_a = seg_b;
            if (seg_a >= n) return false;
            const int slot = s_slot[seg_a];
            const int nv = p.rows_per_slot > 0 ? p.n_valid[slot] : 0;
            seg_b = n;
            for (int wd = (seg_a + 1) >> 5; wd < 4; ++wd) {
                uint32_t m = breaks[wd];
                if (wd == (seg_a + 1) >> 5) m &= 0xffffffffu << ((seg_a + 1) & 31);
                if (m) { seg_b = min(n, wd * 32 + __ffs(m) - 1); break; }
            }
            if (p.rows_per_slot > 0 && p.mode != 0) {
                const bool tail = p.mode == 1 && s_pos[seg_a] >= nv;
                phase = 1;
                lo = tail ? nv : 0;
                j0 = lo & ~(kKeys - 1);
                k_end = tail ? p.n_keys : min(nv, p.n_keys);
                continue;
            }
            lo = first_key_of(s_pos[seg_a], p.window, p.chunk) & ~(kKeys - 1);
            phase = 0;
            j0 = 0;
            k_end = p.window > 0 ? min(p.keep_first, lo) : 0;
        }
    }
};

// Row r (position pos of a slot's sequence), head h, in plain fp32, for a row whose sum is NaN: one that sees an infinity or a NaN, or has one
// in its query.  As the row kernels have it: a key that is not seen does not enter, an infinity or a NaN counts in the channels where it is.
// One warp; channels c0 .. c0 + n - 1 (at most 128) to dst, in front of the gate.
__device__ __noinline__ void plain_row(const SplitAttention& p, int r, int slot, int pos, int h, int c0, int n, float* dst) {
    const int lane = threadIdx.x & 31, rep = p.heads / p.kv_heads;
    const bool ranged = p.rows_per_slot > 0;
    const int nv = ranged ? p.n_valid[slot] : 0;
    int lo = 0, end = pos + 1, kept = 0;
    if (ranged && p.mode != 0) {
        const bool tail = p.mode == 1 && pos >= nv;
        lo = tail ? nv : 0;
        end = tail ? p.n_keys : min(nv, p.n_keys);
    } else {
        lo = first_key_of(pos, p.window, p.chunk);
        kept = p.window > 0 ? min(p.keep_first, lo) : 0;
        if (ranged) end = min(end, p.n_keys);
    }
    auto row_at = [&](int j, int g) {
        const int page = p.table ? p.table[(size_t)slot * p.max_pages + j / p.page_size] : slot;
        return ((size_t)page * p.kv_heads + g) * p.page_size + (p.table ? j % p.page_size : j);
    };
    auto dot = [&](int head, int j) {
        const float* q = p.q + (size_t)r * p.ldq + (size_t)head * p.qdim;
        const float* k = p.kcache + row_at(j, head / rep) * p.kdim;
        float s = 0.f;
        for (int c = 0; c < p.kdim; ++c) s = fmaf(q[c], k[c], s);
        return s;
    };
    float m = p.sink ? p.sink[h] : -CUDART_INF_F, l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int part = 0; part < 2; ++part) {
        const int a = part == 0 ? 0 : lo, b = part == 0 ? kept : end;
        for (int j0 = a; j0 < b; j0 += 32) {
            const int j = j0 + lane;
            float s = -CUDART_INF_F;
            if (j < b) {
                if (p.talk) {
                    s = 0.f;
                    for (int t = 0; t < p.heads; ++t) s = fmaf(p.talk[(size_t)h * p.heads + t], dot(t, j), s);
                    s *= p.scale;
                } else {
                    s = dot(h, j) * (p.scale * (p.temp ? p.temp[h] : 1.f));
                }
                if (p.cap > 0.f) s = p.cap * tanhf(s / p.cap);
                if (p.slopes) s -= p.slopes[h] * (float)(pos - j);
            }
            const float m_new = max_nan(m, warp_max_nan(s));
            const bool none = m_new == -CUDART_INF_F;
            const float e = j < b && !none ? expf(s - m_new) : 0.f, corr = none ? 1.f : expf(m - m_new);
            l = l * corr + warp_sum(e);
            m = m_new;
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] *= corr;
            for (int i = 0; i < min(32, b - j0); ++i) {
                const float w = __shfl_sync(0xffffffffu, e, i);
                const float* v = p.vcache + row_at(j0 + i, h / rep) * p.vrow + c0;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (lane + 32 * u < n) o[u] = fmaf(w, v[lane + 32 * u], o[u]);
            }
        }
    }
    if (p.sink) l += expf(p.sink[h] - m);
    float f = l > 0.f ? p.out_scale / l : 0.f;
    if (p.head_gate) f *= p.head_gate[(size_t)r * p.ldg + h];
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (lane + 32 * u < n) dst[lane + 32 * u] = o[u] * f;
}

// NVS: channel groups of a value (1: up to 128 channels, 2: up to 256).  FOUR: a row has a running denominator per 16 keys of a tile (one in all where
// the widest rows leave no shared memory for what its two threads tell each other of them)
// SELF: not all keys have to be split in advance.
template <int NVS, bool FOUR, bool SELF>
__global__ void __launch_bounds__(kSplitThreads, 1)
split_attention_kernel(const __grid_constant__ SplitAttention p, const __grid_constant__ Geometry geo) {
    constexpr int DVH = 64 * NVS;                             // output channels of a thread
    // The block is launched with 168 registers a thread.  A row's thread holds 64 scores and its sums; the others' share is what the issuing warp needs
    // for its operands (with 24 registers an instruction of the value product took 170 cycles to issue, 77 with these)
    constexpr int kRowRegs = NVS == 1 ? 208 : 216, kOtherRegs = NVS == 1 ? 88 : 72;
    static_assert(32 * kRowWarps * kRowRegs + 128 * kOtherRegs <= 168 * kSplitThreads, "registers of the block");
    constexpr int RW = kRowWarps, LW = NVS == 1 ? 16 : 8;     // row warps, pairs of columns in flight
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* ring = smem;
    unsigned char* qs = ring + (size_t)geo.n_slots * geo.slot_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(qs + geo.q_bytes);
    uint64_t* empty = full + geo.n_slots;
    // of the even and of the odd tiles each: the two groups of row warps take turns, and a barrier of either's own is never two phases ahead
    uint64_t* s_full = empty + geo.n_slots;                    // scores of a tile are there / have been read
    uint64_t* s_empty = s_full + 2;
    uint64_t* p_ready = s_empty + 2;                          // weights of a tile are there / its value product is done / has been added
    uint64_t* pv_done = p_ready + 2;
    uint64_t* o_empty = pv_done + 2;
    uint64_t* m_ready = o_empty + 2;                          // [4] the maxima of 32 rows up to a tile are there
    uint64_t* q_ready = m_ready + 4;
    uint64_t* v_ready = q_ready + 1;                          // [depth] the scales of a tile's values are there
    const int n_bars = 2 * geo.n_slots + 15 + (geo.shared_kv ? 0 : geo.depth);
    float* m_x = reinterpret_cast<float*>(full + ((n_bars + 1) & ~1)); // [2][128] maxima up to an even and an odd tile
    // Denominators.  Of a row's two threads the even tiles' has those of a tile's first 32 keys, the other those of the last (not FOUR: the even tiles' has the one)
    float* sum_x = m_x + 2 * kRows;                           // [rings][128][2] sums of a tile that the other group's thread has (not FOUR: [rings / 2][128] of the odd tiles)
    float* q_inv = sum_x + (FOUR ? 2 * (geo.rings - 1) * kRows : 0);  // [128] (an odd tile's sums are stored there when both groups have read it)
    __nv_bfloat16* wi_x = reinterpret_cast<__nv_bfloat16*>(sum_x + (FOUR ? 2 * geo.rings : geo.rings / 2) * kRows); // [rings][128] inverse scales of the weights: powers of two
    float* k_inv = reinterpret_cast<float*>(wi_x + geo.rings * kRows); // [depth][k_sets][64] inverse scales of the keys
    float* v_inv = geo.shared_kv ? k_inv : k_inv + geo.depth * geo.k_sets * kKeys;      // [depth][64] of the values
    int4* s_tile = reinterpret_cast<int4*>(v_inv + geo.depth * kKeys); // [depth] a tile's first key, its tokens (first | end << 16), end of its keys, lo (see Walk)
    uint32_t* s_breaks = reinterpret_cast<uint32_t*>(s_tile + geo.depth);      // [4]
    uint32_t* s_tmem = s_breaks + 4;
    int* s_rows = reinterpret_cast<int*>(s_tmem + 1);         // [2] the row tile; then [0]: its tiles of keys
    int* s_slot = s_rows + 3;                                 // [tokens]
    const int TT = kRows >> geo.pk_shift;
    int* s_pos = s_slot + TT;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int PK = 1 << geo.pk_shift;
    const int h_tiles = p.heads >> geo.pk_shift, row_tile = (int)(gridDim.x / h_tiles) - 1 - (int)(blockIdx.x / h_tiles);
    const int h0 = (int)(blockIdx.x % h_tiles) * PK, rep = p.heads / p.kv_heads, g = h0 / rep;
    // later tokens see more keys: their tiles start first.  With the step's sequences at hand a tile holds rows of one of them (a
    // tile with the rows of 24 decoding sequences walked the keys of all 24 one after the other)
    int r0 = row_tile * TT, n_tok = min(TT, p.M - r0);
    if (p.n_seq > 1) {
        if (tid == 0) s_rows[1] = 0;
        __syncthreads();
        if (warp == 0) {
            const int want = row_tile;
            int run = 0;
            for (int s0 = 0; s0 < p.n_seq; s0 += 32) {
                const int count = s0 + lane < p.n_seq ? p.seq_count[s0 + lane] : 0, n = (count + TT - 1) / TT;
                int sum = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += v;
                }
                const int begin = run + sum - n;
                if (want >= begin && want < begin + n) {
                    s_rows[0] = p.seq_row0[s0 + lane] + (want - begin) * TT;
                    s_rows[1] = min(TT, count - (want - begin) * TT);
                }
                run += __shfl_sync(0xffffffffu, sum, 31);
                if (run > want) break;
            }
        }
        __syncthreads();
        r0 = s_rows[0];
        n_tok = s_rows[1];
        if (n_tok == 0) return;                               // (the grid is an upper bound)
    }

    if (tid == 0) {
        for (int i = 0; i < geo.n_slots; ++i) { mbar_init(&full[i], kFetchWarps); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_empty[i], 4);
            mbar_init(&p_ready[i], 4);
            mbar_init(&pv_done[i], 1);
            mbar_init(&o_empty[i], RW);
        }
        for (int i = 0; i < 4; ++i) mbar_init(&m_ready[i], 1);
        mbar_init(q_ready, RW);
        if (!geo.shared_kv)
            for (int i = 0; i < geo.depth; ++i) mbar_init(&v_ready[i], kFetchWarps);
        fence_mbar_init();
    }
    if (warp == RW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(s_tmem)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid < kRows) {
        const int i = tid, r = r0 + i;
        const bool in = i < n_tok, ranged = p.rows_per_slot > 0;
        int slot = -1, pos = -1;
        bool starts = true;
        if (in) {
            slot = ranged ? r / p.rows_per_slot : p.row_slot[r];
            pos = ranged ? r % p.rows_per_slot : p.row_pos[r];
            if (i > 0) {
                starts = ranged ? pos == 0 : p.row_slot[r - 1] != slot || p.row_pos[r - 1] + 1 != pos;
                if (ranged && p.mode == 1) starts = starts || pos == p.n_valid[slot];
            }
        }
        if (i < TT) { s_slot[i] = slot; s_pos[i] = pos; }
        const uint32_t m = __ballot_sync(0xffffffffu, starts);
        if (lane == 0) s_breaks[warp] = m;
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *s_tmem;
    const uint32_t t_s = tmem, t_p = tmem + 64u * geo.n_kst * geo.s_bufs, t_o = t_p + 64u * geo.p_bufs;    // scores | weights (hi, lo) | value products

    if (warp < RW) {
        // ================= softmax: rows 32 (warp % 4) + lane; warps 0 .. 3 take the even tiles, 4 .. 7 the odd ones =================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
        // ---- the query tile: largest magnitude, then both terms.  Row r of the tile is head h0 + r % PK of token r / PK; a warp takes
        // eight rows at a time, a lane eight channels of one.  (The first keys are on their way meanwhile: with the tile made by all
        // warps in front of the roles, its loops unrolled, a launch of one key tile took 17 us, now 14: cold instruction fetches) ----
        constexpr int RG = kRows / (8 * RW);                  // groups of 8 RW rows
        const int qrow = warp * 8 + (lane & 7), qch = lane >> 3;
        auto q_load = [&](int st, float4 (&v)[RG][4][2]) {    // this lane's channels of channel group st (mixed scores: of kv head st)
            const int width = p.talk ? p.kdim : min(kGroupW, p.kdim - st * kGroupW);      // (a multiple of 4)
            auto add = [&](const float* src, int t, bool first) {
#pragma unroll
                for (int rg = 0; rg < RG; ++rg) {
                    const int row = qrow + 8 * RW * rg, i = row >> geo.pk_shift, h = h0 + (row & (PK - 1));
                    const float* at = src + (size_t)(r0 + i) * p.ldq + (p.talk ? 0 : (size_t)h * p.qdim);
                    const int left = i < n_tok ? width - 8 * qch : 0;
                    const float w = p.talk ? p.talk[h * p.heads + st * rep + t] : 1.f;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (32 * k + 4 * e < left) x = *reinterpret_cast<const float4*>(at + 32 * k + 4 * e);
                            float4& y = v[rg][k][e];
                            if (first) y = p.talk ? make_float4(w * x.x, w * x.y, w * x.z, w * x.w) : x;
                            else y = make_float4(fmaf(w, x.x, y.x), fmaf(w, x.y, y.y), fmaf(w, x.z, y.z), fmaf(w, x.w, y.w));
                        }
                }
            };
            if (!p.talk) {
                add(p.q + st * kGroupW + 8 * qch, 0, true);
                return;
            }
            // the mixed score is linear in the queries: mix those instead
            const float* src = p.q + (size_t)st * rep * p.qdim + 8 * qch;
            add(src, 0, true);
#pragma unroll 1
            for (int t = 1; t < rep; ++t) add(src + (size_t)t * p.qdim, t, false);
        };
        auto q_largest = [&](const float4 (&v)[RG][4][2], float (&m)[RG]) {
#pragma unroll
            for (int rg = 0; rg < RG; ++rg)
#pragma unroll
                for (int k = 0; k < 4; ++k) m[rg] = max_abs4(max_abs4(m[rg], v[rg][k][0]), v[rg][k][1]);
        };
        float scale[RG], m_row[RG] = {};
        bool bad[RG];
        auto q_scales = [&] {                                 // from the four lanes that hold a row
#pragma unroll
            for (int rg = 0; rg < RG; ++rg) {
                float inverse;
                bad[rg] = scale_row(row_max(m_row[rg]), scale[rg], inverse);
                if (lane < 8) q_inv[qrow + 8 * RW * rg] = inverse;
            }
        };
        auto q_store = [&](int st, const float4 (&v)[RG][4][2]) {
            const int w = st == geo.n_kst - 1 ? geo.wk_last : geo.wk0;
            unsigned char* const group = qs + (size_t)st * geo.wk0 * kRows * 4;
#pragma unroll
            for (int rg = 0; rg < RG; ++rg) {
                const int row = qrow + 8 * RW * rg;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int c8 = qch + 4 * k;
                    if (8 * c8 >= w) continue;
                    const float f = scale[rg];
                    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f), a = bad[rg] ? z : v[rg][k][0], b = bad[rg] ? z : v[rg][k][1];
                    uint32_t hi[4], lo[4];
                    split2(a.x * f, a.y * f, hi[0], lo[0]);
                    split2(a.z * f, a.w * f, hi[1], lo[1]);
                    split2(b.x * f, b.y * f, hi[2], lo[2]);
                    split2(b.z * f, b.w * f, hi[3], lo[3]);
                    unsigned char* dst = group + (size_t)(((row >> 3) * (w >> 3) + c8) * 128 + (row & 7) * 16);
                    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4*>(dst + (size_t)w * kRows * 2) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
            }
        };
        float4 qv[RG][4][2];
        // (one group of channels stays in registers, more are read twice)
#pragma unroll 1
        for (int st = 0; st < geo.n_kst; ++st) {
            q_load(st, qv);
            q_largest(qv, m_row);
        }
        q_scales();
#pragma unroll 1
        for (int st = 0; st < geo.n_kst; ++st) {
            if (geo.n_kst > 1) q_load(st, qv);
            q_store(st, qv);
        }
        fence_smem_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_ready);
        asm volatile("bar.sync 1, %0;" ::"n"(32 * RW + 32) : "memory");     // (all queries are stored, the rows' scales and the number of tiles are there)
        const int qt = warp & 3, hf = warp >> 2, row = qt * 32 + lane, tok = row >> geo.pk_shift, h = h0 + (row & (PK - 1));
        const uint32_t lanes = (uint32_t)(qt * 32) << 16;
        const int my_pos = s_pos[tok];
        const int my_lo = first_key_of(max(my_pos, 0), p.window, p.chunk), kept = p.window > 0 ? p.keep_first : 0;
        const bool ranged = p.rows_per_slot > 0 && p.mode != 0;
        // scores and maxima are in units of log 2 (a capped score from its cap on): the largest score's weight is exactly 1 at any magnitude
        const float cap = p.cap;
        const float mult = q_inv[row] * p.scale * (p.temp ? p.temp[h] : 1.f) * (cap > 0.f ? 1.f : kLog2e);
        const float slope = p.slopes ? p.slopes[h] * kLog2e : 0.f;
        // channels of this thread: c0 .. + n_mine, at t_mine in tensor memory
        const int share = NVS == 1 ? geo.wv0 / 2 : DVH, n_mine = NVS == 1 || hf == 0 ? min(share, geo.wv0) : geo.wv_last, c0 = hf * share;
        const uint32_t t_mine = t_o + c0 + lanes;
        f2 O[DVH / 2];
#pragma unroll
        for (int c = 0; c < DVH / 2; ++c) O[c] = 0;
        float m_run = -CUDART_INF_F;
        float2 l2 = make_float2(0.f, 0.f);
        float m_own = 0.f, wi_own = 0.f;                      // of the tile of this group that has not been added yet
        float2 sum_own = make_float2(0.f, 0.f);
        bool ok = true;
        // O <- corr O + the value product of tile t, up to which the maximum is m; this thread's denominators likewise.
        // The numbers of the other group's tile were stored in front of the weights that have been multiplied.
        auto add_values = [&](unsigned t, float m, float wi, float2 sum) {
            if (!wait_for(&pv_done[t & 1u], (t >> 1) & 1u)) return false;
            fence_after();
            if ((int)(t & 1u) != hf) {
                const unsigned at = (t & (geo.rings - 1u)) * kRows + row;
                wi = __bfloat162float(wi_x[at]);
                if (FOUR) sum = reinterpret_cast<const float2*>(sum_x)[at];
                else if (hf == 0) sum.x = sum_x[((t >> 1) & (geo.rings / 2 - 1u)) * kRows + row];
            }
            const float corr = m_run == -CUDART_INF_F ? 0.f : ex2(m_run - m);      // (m is no less)
            const f2 vi2 = twice(wi), c2 = twice(corr);
            l2 = make_float2(fmaf(l2.x, corr, sum.x), fmaf(l2.y, corr, sum.y));
            m_run = m;
            const uint32_t from = t_mine + (geo.o_bufs == 2 ? (t & 1u) * 128u : 0u);
#pragma unroll
            for (int c = 0; c < DVH; c += 2 * LW) {
                if (c < n_mine) {                             // (columns beyond n_mine hold whatever they held; they are not stored)
                    f2 v[LW];
                    tmem_load_pairs<LW>(from + c, v);
#pragma unroll
                    for (int e = 0; e < LW; ++e) O[c / 2 + e] = fma2(v[e], vi2, mul2(O[c / 2 + e], c2));
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_empty[t & 1u]);
            return true;
        };
        const unsigned n_tiles = (unsigned)s_rows[0];
        unsigned my_at = hf, my_round = 0;                    // t % depth, t / depth % 2 (depth is at least 2)
        // In turn t a group weighs tile t, if there is one.  Its own tile t - 2 it adds when it has the maximum of tile t (the product of its last
        // weights has had the time of the loads and the maximum), the other group's tile t - 1 behind.  Wide values leave no registers for sums and
        // scores at a time: both groups' last tiles are added in front.
        constexpr bool MID = NVS == 1;
        float m_other = 0.f;
#pragma unroll 1
        for (unsigned t = hf; ok && t < n_tiles + (MID ? 2 : 3); t += 2) {
            ok = false;                                       // (until this turn is done)
            if (!MID) {
                bool added = true;
#pragma unroll 1
                for (unsigned u = t - 3; added && u != t - 1; ++u)         // (below zero: none)
                    if (u < n_tiles) added = add_values(u, u == t - 2 ? m_own : m_other, wi_own, sum_own);
                if (!added) break;
            }
            float m_old = -CUDART_INF_F;
            if (t < n_tiles) {
                if (!wait_for(&s_full[hf], (t >> 1) & 1u)) break;
                fence_after();
                const int4 tile = s_tile[my_at];
                f2 s[kKeys / 2];
                const float* ki = k_inv + my_at * geo.k_sets * kKeys;
                const uint32_t from = t_s + lanes + (geo.s_bufs == 2 ? (t & 1u) * 64u * geo.n_kst : 0u);
#pragma unroll
                for (int c = 0; c < kKeys; c += 2 * LW) {
                    tmem_load_pairs<LW>(from + c, s + c / 2);
                    if (geo.k_sets > 1) scale_by<LW>(s + c / 2, ki + c);
#pragma unroll 1
                    for (int st = 1; st < geo.n_kst; ++st) {
                        f2 v[LW];
                        tmem_load_pairs<LW>(from + st * 64 + c, v);
                        if (geo.k_sets > 1) scale_by<LW>(v, ki + st * kKeys + c);
#pragma unroll
                        for (int e = 0; e < LW; ++e) s[c / 2 + e] = add2(s[c / 2 + e], v[e]);
                    }
                    if (geo.k_sets == 1) scale_by<LW>(s + c / 2, ki + c);
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_empty[hf]);
                const f2 mult2 = twice(mult);
#pragma unroll
                for (int e = 0; e < kKeys / 2; ++e) s[e] = mul2(s[e], mult2);
                // ---- cap, distance bias, visibility ----
                const int k0 = tile.x;
                if (cap > 0.f) {
                    const f2 ic = twice(1.0f / cap), cc = twice(cap * kLog2e);
                    float big[2] = {0.f, 0.f};
#pragma unroll
                    for (int e = 0; e < kKeys / 2; ++e) {
                        s[e] = mul2(s[e], ic);
                        float x, y;
                        unpack2(s[e], x, y);
                        big[e & 1] = fmaxf(big[e & 1], fmaxf(fabsf(x), fabsf(y)));
                    }
                    // Each score takes the form that its own magnitude asks for; whether all of them are near zero decides the speed only.  The other
                    // form is a rolled loop over the scores in tensor memory, where this tile's weights will be (a launch that has a cap has two
                    // sets of them): a call or an array in local memory here made every tile's scores pass through local memory (64 capped scores
                    // 6700 cycles, 2900 without it)
                    if (__all_sync(0xffffffffu, fmaxf(big[0], big[1]) <= kTanhRange)) {
#pragma unroll
                        for (int e = 0; e < kKeys / 2; ++e) s[e] = tanh_near_zero(s[e]);
                    } else {
                        if (t >= 2 && !wait_for(&pv_done[hf], ((t - 2) >> 1) & 1u)) break;     // (the weights of the tile two before are read)
                        fence_after();
                        const uint32_t at_p = t_p + lanes + (geo.p_bufs == 2 ? (t & 1u) * 64u : 0u);
#pragma unroll
                        for (int c = 0; c < kKeys / 8; ++c) {
                            uint32_t x[8];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                x[2 * e] = (uint32_t)s[c * 4 + e];
                                x[2 * e + 1] = (uint32_t)(s[c * 4 + e] >> 32);
                            }
                            tmem_store8(at_p + c * 8, x);
                        }
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll 1
                        for (int c = 0; c < kKeys; c += 8) {
                            float x[8];
                            uint32_t y[8];
                            tmem_load8(at_p + c, x);
                            tmem_loaded();
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                float near, same;
                                unpack2(tanh_near_zero(pack2(x[e], x[e])), near, same);
                                y[e] = __float_as_uint(fabsf(x[e]) <= kTanhRange ? near : tanhf(x[e]));
                            }
                            tmem_store8(at_p + c, y);
                            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        }
#pragma unroll
                        for (int c = 0; c < kKeys; c += 2 * LW) tmem_load_pairs<LW>(at_p + c, s + c / 2);
                    }
#pragma unroll
                    for (int e = 0; e < kKeys / 2; ++e) s[e] = mul2(s[e], cc);
                }
                if (p.slopes) {
                    const float base = (float)(my_pos - k0);
                    const f2 ns = twice(-slope), down = twice(-2.f);
                    f2 gap = pack2(base, base - 1.f);
#pragma unroll
                    for (int e = 0; e < kKeys / 2; ++e) {
                        s[e] = fma2(ns, gap, s[e]);
                        gap = add2(gap, down);                    // (whole numbers)
                    }
                }
                // the keys that the row sees, a bit each
                uint32_t see[2];
                {
                    const bool live = tok >= (tile.y & 0xffff) && tok < tile.y >> 16;
                    const int end = live ? min(tile.z, ranged ? 0x7fffffff : my_pos + 1) - k0 : 0, from = (ranged ? tile.w : my_lo) - k0, keep = kept - k0;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        auto below = [&](int n) { n -= 32 * i; return n >= 32 ? 0xffffffffu : n <= 0 ? 0u : (1u << n) - 1u; };
                        see[i] = below(end) & (~below(from) | below(keep));
                    }
                }
                const bool all_seen = __all_sync(0xffffffffu, (see[0] & see[1]) == 0xffffffffu);
                auto hide = [&](float x) {                        // x in the place of every key that the row does not see
#pragma unroll
                    for (int e = 0; e < kKeys / 2; ++e) {
                        float a, b;
                        unpack2(s[e], a, b);
                        a = see[e / 16] >> (2 * e % 32) & 1u ? a : x;
                        b = see[e / 16] >> (2 * e % 32 + 1) & 1u ? b : x;
                        s[e] = pack2(a, b);
                    }
                };
                auto largest = [&] {                              // (four chains)
                    float v[4];
#pragma unroll
                    for (int e = 0; e < kKeys / 2; ++e) {
                        float a, b;
                        unpack2(s[e], a, b);
                        v[e & 3] = e < 4 ? max_nan(a, b) : max3_nan(v[e & 3], a, b);
                    }
                    return max_nan(max_nan(v[0], v[1]), max_nan(v[2], v[3]));
                };
                if (!all_seen) hide(-CUDART_INF_F);
                const float mx = largest();
                // the maximum up to the tile before comes from the other group, which has its scores already
                if (t > 0) {
                    if (!wait_for(&m_ready[qt], (t - 1) & 1u)) break;
                    m_old = m_x[(hf ^ 1) * kRows + row];
                }
                const float m_new = max_nan(m_old, mx);
                m_x[hf * kRows + row] = m_new;
                __syncwarp();
                if (lane == 0) mbar_arrive(&m_ready[qt]);
                if (MID && t >= 2 && !add_values(t - 2, m_own, wi_own, sum_own)) break;
                m_own = m_new;
                const float base = m_new == -CUDART_INF_F ? 0.f : m_new;
                const f2 nb = twice(-base);
                float sum[4];                                     // a sum per 16 keys
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    f2 a = 0;
#pragma unroll
                    for (int e = 8 * c; e < 8 * c + 8; ++e) {
                        float x, y;
                        unpack2(add2(s[e], nb), x, y);
                        s[e] = pack2(ex2(x), ex2(y));
                        a = add2(a, s[e]);
                    }
                    float x, y;
                    unpack2(a, x, y);
                    sum[c] = x + y;
                }
                // weight x its value's magnitude, and the largest of them that this row has in the tile
                if (!geo.shared_kv && !wait_for(&v_ready[my_at], my_round)) break;
                scale_by<kKeys / 2>(s, v_inv + my_at * kKeys);
                float wm = largest();
                if (__any_sync(0xffffffffu, wm != wm)) {          // a value that cannot be split, 0 x NaN where it is not seen
                    hide(0.f);
                    wm = largest();
                    if (wm != wm) sum[0] = CUDART_NAN_F;
                }
                const f2 ws = twice(scale_of(wm, wi_own));
                // the weights' columns are free once the value product that read them is done (of two sets: it has been added by now)
                if (geo.p_bufs == 1 && t > 0) {
                    if (!wait_for(&pv_done[(t - 1) & 1u], ((t - 1) >> 1) & 1u)) break;
                    fence_after();
                }
                // (the other group has read the place: the tile `rings` before, or with one set and one product two before, has been added)
                const unsigned place = (t & (geo.rings - 1u)) * kRows + row;
                wi_x[place] = __float2bfloat16(wi_own);
                if constexpr (FOUR) {
                    reinterpret_cast<float2*>(sum_x)[place] = hf == 0 ? make_float2(sum[2], sum[3]) : make_float2(sum[0], sum[1]);
                    sum_own = hf == 0 ? make_float2(sum[0], sum[1]) : make_float2(sum[2], sum[3]);
                } else {
                    sum_own.x = (sum[0] + sum[1]) + (sum[2] + sum[3]);
                    if (hf == 1) sum_x[((t >> 1) & (geo.rings / 2 - 1u)) * kRows + row] = sum_own.x;
                }
                const uint32_t to = t_p + lanes + (geo.p_bufs == 2 ? (t & 1u) * 64u : 0u);
#pragma unroll
                for (int c = 0; c < kKeys / 16; ++c) {
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) split2(mul2(s[c * 8 + e], ws), hi[e], lo[e]);
                    tmem_store8(to + c * 8, hi);
                    tmem_store8(to + 32 + c * 8, lo);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[hf]);
            } else {
                if (MID && t >= 2 && !add_values(t - 2, m_own, wi_own, sum_own)) break;
                if (t == n_tiles && t > 0) {                  // (the other group has the last tile)
                    if (!wait_for(&m_ready[qt], (t - 1) & 1u)) break;
                    m_old = m_x[(hf ^ 1) * kRows + row];
                }
            }
            m_other = m_old;
            ok = !MID || t == 0 || t > n_tiles || add_values(t - 1, m_old, 0.f, make_float2(0.f, 0.f));
            my_at += 2;
            if (my_at >= (unsigned)geo.depth) my_at -= geo.depth, my_round ^= 1u;
        }
        asm volatile("bar.sync 2, %0;" ::"n"(32 * RW) : "memory");           // (the last tiles' sums have been read)
        if (FOUR) reinterpret_cast<float2*>(sum_x)[hf * kRows + row] = l2;
        else if (hf == 0) sum_x[row] = l2.x;
        asm volatile("bar.sync 2, %0;" ::"n"(32 * RW) : "memory");
        float l = sum_x[row];
        if (FOUR) {
            const float2 a = reinterpret_cast<const float2*>(sum_x)[row], b = reinterpret_cast<const float2*>(sum_x)[kRows + row];
            l = ((a.x + a.y) + b.x) + b.y;
        }
        // ---- the sink's own term, normalise, store ----
        if (p.sink) l += ex2(fmaf(p.sink[h], kLog2e, m_run == -CUDART_INF_F ? 0.f : -m_run));
        // through shared memory (the ring and the queries are read; 32 rows of this warp's channels): whole lines reach the output, and
        // one rolled loop serves every kind of output.  (Stored from the registers, row by row, 5500 cycles of a CTA, mostly fetching
        // the unrolled code; 3500 now)
        float f = tok < n_tok && l > 0.f ? p.out_scale / l : 0.f;
        if (p.head_gate && tok < n_tok) f *= p.head_gate[(size_t)(r0 + tok) * p.ldg + h];
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0 && geo.ran_out) {
            *reinterpret_cast<volatile int*>(geo.ran_out) = 1;
            __threadfence_system();
        }
        const int ldst = share + 4;
        float* stage = reinterpret_cast<float*>(smem) + (size_t)warp * 32 * ldst;
#pragma unroll
        for (int c = 0; c < DVH; c += 4)
            if (c < n_mine) *reinterpret_cast<ulonglong2*>(stage + lane * ldst + c) = make_ulonglong2(mul2(O[c / 2], twice(f)), mul2(O[c / 2 + 1], twice(f)));
        __syncwarp();
        const int w4 = max(0, min(n_mine, p.vdim - c0)) >> 2; // (vdim is a multiple of 4)
        for (unsigned again = __ballot_sync(0xffffffffu, ok && tok < n_tok && l != l && w4 > 0); again; again &= again - 1) {
            const int r = __ffs(again) - 1, rw = qt * 32 + r, tk = rw >> geo.pk_shift;
            plain_row(p, r0 + tk, s_slot[tk], s_pos[tk], h0 + (rw & (PK - 1)), c0, 4 * w4, stage + r * ldst);
        }
        __syncwarp();
        int sr = 0, sc = lane;                                // row and group of 4 channels of this lane's turn
        while (w4 > 0 && sc >= w4) { sc -= w4; ++sr; }
#pragma unroll 2
        for (int it = 0; it < w4; ++it) {
            const int rw = qt * 32 + sr, tk = rw >> geo.pk_shift, c = 4 * sc;
            if (tk < n_tok) {
                const size_t head = (size_t)(h0 + (rw & (PK - 1))) * p.vdim + c0 + c, at = (size_t)(r0 + tk) * p.ldo + head;
                float4 o = *reinterpret_cast<const float4*>(stage + sr * ldst + c);
                if (!ok) o = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F);
                if (p.gate) {
                    const float4 z = *reinterpret_cast<const float4*>(p.gate + (size_t)(r0 + tk) * p.ldg + head);
                    o.x *= 1.0f / (1.0f + expf(-z.x)); o.y *= 1.0f / (1.0f + expf(-z.y));
                    o.z *= 1.0f / (1.0f + expf(-z.z)); o.w *= 1.0f / (1.0f + expf(-z.w));
                }
                if (p.out) *reinterpret_cast<float4*>(p.out + at) = o;
                if (p.out_bf16) {
                    const __nv_bfloat162 a = __floats2bfloat162_rn(o.x, o.y), b = __floats2bfloat162_rn(o.z, o.w);
                    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out_bf16) + at) =
                        make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
                }
            }
            sc += 32;
            while (sc >= w4) { sc -= w4; ++sr; }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        if (warp > RW) {
            // ================= keys and values =================
            const int lw = warp - RW - 1, kin = lane & 7, cq = lane >> 3;
            unsigned slot = 0, phase = 0;                         // the ring's next place, rounds % 2
            bool ok = true;
            const unsigned char* const work = reinterpret_cast<const unsigned char*>(p.work);
            const size_t k_first = part_offset(geo, p.talk ? 0 : g * geo.n_kst), v_first = geo.shared_kv ? k_first : part_offset(geo, geo.k_parts + g * geo.n_vst);
            const unsigned k_step = kKeys * 4u * geo.wk0, v_step = kKeys * 4u * (geo.shared_kv ? geo.wk0 : geo.wv0);
            auto copy = [&](void* dst, const unsigned char* src, unsigned bytes, uint64_t* bar) {
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes),
                             "r"(smem_u32(bar))
                             : "memory");
            };
            int4 about{};                                         // what the row warps are told of the newest tile
            struct Tile { int split, slot, j0, k_end; };          // split: the tile of the room that holds these keys (-1: none)
            auto part_width = [&](bool is_v, int part) {
                const int last = (is_v ? geo.n_vst : geo.n_kst) - 1;
                return is_v ? (part == last ? geo.v_last_layout : geo.v0_layout) : (part == last ? geo.wk_last : geo.wk0);
            };
            auto row_at = [&](int of, int j) -> unsigned long long {      // (in kv head 0)
                if (!p.table) return (unsigned long long)of * p.kv_heads * p.page_size + j;
                const unsigned at = geo.page_shift >= 0 ? (unsigned)j >> geo.page_shift : (unsigned)j / (unsigned)p.page_size;
                const unsigned page = p.table[(size_t)of * p.max_pages + at];
                return (unsigned long long)page * ((unsigned)p.kv_heads * (unsigned)p.page_size) + ((unsigned)j - at * (unsigned)p.page_size);
            };
            // SELF: a part that is not split yet comes as it is, into the bytes that its terms will have: the first four of a lane's eight channels where their high terms will be, the
            // others where the low ones will be.  The lane that asked for them splits them there while the next part is on its way.
            constexpr int kEights = (kKeys / 8 + kFetchWarps - 1) / kFetchWarps;      // this warp's keys: eights lw, lw + 3, lw + 6 of a tile, a lane a part of one
            int raw = -1, raw_part = 0;                       // the place and the group of the part that is to be split (-1: none)
            unsigned raw_at = 0;
            bool raw_v = false;
            float raw_more[kEights] = {};                     // largest magnitudes of the keys' channels beyond the part
            auto split_raw = [&](bool behind) {               // behind: another part has been asked for since
                if (behind) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                const bool shared = raw_v && geo.shared_kv;   // (a shared row's scale is its key's)
                const int wp = part_width(raw_v, raw_part), blocks = wp >> 3;
                // (keys of several groups of channels have one scale, which the first group takes)
                const bool own = raw_v ? raw_part == 0 && !shared : raw_part == 0 || geo.k_sets > 1;
                float* const inv = raw_v && !shared ? v_inv + raw_at * kKeys : k_inv + (raw_at * geo.k_sets + (geo.k_sets > 1 ? raw_part : 0)) * kKeys;
                __syncwarp();
#pragma unroll 1
                for (int e = lw; e < kKeys / 8; e += kFetchWarps) {
                    unsigned char* const dst = ring + (size_t)raw * geo.slot_bytes + (e * blocks + cq) * 128 + kin * 16;
                    unsigned char* const low = dst + kKeys * wp * 2;
                    ulonglong2 v[8];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool has = cq + 4 * i < blocks;
                        v[2 * i] = has ? *reinterpret_cast<const ulonglong2*>(dst + i * 512) : make_ulonglong2(0, 0);
                        v[2 * i + 1] = has ? *reinterpret_cast<const ulonglong2*>(low + i * 512) : make_ulonglong2(0, 0);
                    }
                    float sc, inverse;
                    bool bad;
                    if (own) {
                        float m = e < kFetchWarps ? raw_more[0] : e < 2 * kFetchWarps ? raw_more[1] : raw_more[2], m2 = 0.f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float a, b, c, d;
                            unpack2(v[i].x, a, b);
                            unpack2(v[i].y, c, d);
                            m = max3_nan(m, fabsf(a), fabsf(b));
                            m2 = max3_nan(m2, fabsf(c), fabsf(d));
                        }
                        bad = scale_row(row_max(max_nan(m, m2)), sc, inverse);
                        if (lane < 8) inv[e * 8 + lane] = inverse;
                    } else {
                        inverse = inv[e * 8 + kin];
                        bad = inverse != inverse;
                        sc = __uint_as_float((254u << 23) - __float_as_uint(inverse));      // (powers of two)
                    }
                    if (bad) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] = make_ulonglong2(0, 0);
                        sc = 0.f;
                    }
                    const f2 sc2 = twice(sc);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 hi, lo;
                        split8(v[2 * i], v[2 * i + 1], sc2, hi, lo);
                        if (cq + 4 * i < blocks) {
                            *reinterpret_cast<uint4*>(dst + i * 512) = hi;
                            *reinterpret_cast<uint4*>(low + i * 512) = lo;
                        }
                    }
                }
                fence_smem_async();
                __syncwarp();
                if (lane == 0 && raw_v && own) mbar_arrive(&v_ready[raw_at]);
                if (lane == 0) mbar_arrive(&full[raw]);
                raw = -1;
            };
            // the ring's next part: key group `part` of the tile at place at_t of the numbers' rings, or value group `part` of it
            auto fetch = [&](const Tile& z, unsigned at_t, bool is_v, int part) {
                const int wp = part_width(is_v, part);
                // (a part that is split already may bring scales to the place of those that the raw one asks for)
                if constexpr (SELF)
                    if (raw >= 0 && (z.split >= 0 || !__all_sync(0xffffffffu, has_passed(&empty[slot], phase ^ 1u)))) split_raw(false);
                if (z.split >= 0) {                               // split already: with its first key group a tile's scales come along
                    if (lane == 0) {
                        ok = wait_for(&empty[slot], phase ^ 1u);
                        if (lw == 0) {
                            const unsigned bytes = kKeys * wp * 4;
                            const bool scales = !is_v && part == 0;
                            if (scales) s_tile[at_t] = about;
                            mbar_arrive_expect_tx(&full[slot], bytes + (scales ? kKeys * 4u * geo.k_sets : 0u));
                            copy(ring + (size_t)slot * geo.slot_bytes, work + geo.tile_off + (size_t)z.split * geo.tile_bytes + (is_v ? v_first + part * v_step : k_first + part * k_step),
                                 bytes, &full[slot]);
                            if (scales) {
                                const unsigned char* src = work + geo.scale_off + (size_t)z.split * geo.sets * kKeys * 4;
                                copy(k_inv + at_t * geo.k_sets * kKeys, src + (geo.k_sets > 1 ? 0 : g) * kKeys * 4, kKeys * 4u * geo.k_sets, &full[slot]);
                                if (!geo.shared_kv) {
                                    mbar_arrive_expect_tx(&v_ready[at_t], kKeys * 4u);
                                    copy(v_inv + at_t * kKeys, src + (p.kv_heads + g) * kKeys * 4, kKeys * 4u, &v_ready[at_t]);
                                }
                            }
                        } else {
                            if (!is_v && part == 0 && !geo.shared_kv) mbar_arrive(&v_ready[at_t]);
                            mbar_arrive(&full[slot]);
                        }
                    }
                    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                    return;
                }
                if constexpr (SELF) {
                    const int blocks = wp >> 3;
                    const bool shared = is_v && geo.shared_kv;
                    const float* const cache = is_v ? p.vcache : p.kcache;
                    const int width = is_v ? p.vrow : p.kdim, row_w = is_v && !shared ? p.vdim : p.kdim, c0 = p.talk && !is_v ? 0 : part * kGroupW;
                    const int gg = p.talk && !is_v ? part : g, w = min(kGroupW, row_w - c0);
                    const float* src[kEights];                    // this lane's first channels of its keys (of the cache's first row in the place of keys that are not there)
                    bool in[kEights];
                    const bool one_page = !p.table || geo.page_shift >= 6;      // (a tile starts at a multiple of 64 keys)
                    const unsigned long long row0 = one_page ? row_at(z.slot, z.j0) : 0;
                    const float* const head = cache + ((size_t)gg * p.page_size) * width + (c0 + 8 * cq);
#pragma unroll
                    for (int u = 0; u < kEights; ++u) {
                        const int e = (lw + u * kFetchWarps) * 8 + kin;
                        in[u] = lw + u * kFetchWarps < kKeys / 8 && z.j0 + e < z.k_end;
                        src[u] = in[u] ? head + (one_page ? row0 + e : row_at(z.slot, z.j0 + e)) * (unsigned)width : cache + (c0 + 8 * cq);
                    }
                    ok = __all_sync(0xffffffffu, wait_for(&empty[slot], phase ^ 1u));
                    if (!ok) return;
                    if (lw == 0 && !is_v && part == 0 && lane == 0) s_tile[at_t] = about;
                    const uint32_t place = smem_u32(ring) + slot * geo.slot_bytes + kin * 16 + (lw * blocks + cq) * 128, low = kKeys * wp * 2;
                    auto copy16 = [&](uint32_t dst, const float* from, int bytes) {
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(from), "r"(bytes) : "memory");
                    };
                    const bool whole = z.j0 + kKeys <= z.k_end && w == wp;
#pragma unroll
                    for (int u = 0; u < kEights; ++u) {
                        if (lw + u * kFetchWarps >= kKeys / 8) continue;
                        const uint32_t dst = place + u * kFetchWarps * blocks * 128;
                        if (whole) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (cq + 4 * i >= blocks) continue;
                                copy16(dst + i * 512, src[u] + 32 * i, 16);
                                copy16(dst + low + i * 512, src[u] + 32 * i + 4, 16);
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (cq + 4 * i >= blocks) continue;
                                const int left = in[u] ? w - 8 * cq - 32 * i : 0;      // (no channel is read that is not there)
                                copy16(dst + i * 512, left > 0 ? src[u] + 32 * i : cache, left > 0 ? 16 : 0);
                                copy16(dst + low + i * 512, left > 4 ? src[u] + 32 * i + 4 : cache, left > 4 ? 16 : 0);
                            }
                        }
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    if (raw >= 0) split_raw(true);
#pragma unroll
                    for (int u = 0; u < kEights; ++u) raw_more[u] = 0.f;
                    if (part == 0 && !shared && w < row_w) {
#pragma unroll 3
                        for (int c = w + 4 * cq; c < row_w; c += 16) {
#pragma unroll
                            for (int u = 0; u < kEights; ++u)
                                if (in[u]) raw_more[u] = max_abs4(raw_more[u], *reinterpret_cast<const float4*>(src[u] + (c - 8 * cq)));
                        }
                    }
                    raw = (int)slot;
                    raw_part = part;
                    raw_at = at_t;
                    raw_v = is_v;
                } else {
                    // The launch saw to it that all keys are split in advance, or was told so.  If not, eight at a time and rolled: this instance is all about code
                    // that is short (with the other form in it, or with neither, a latent layer of 4096 rows takes 636 us, not 620: the row warps' code is fetched
                    // from other places)
                    const bool shared = is_v && geo.shared_kv;        // (a shared row's scale is its key's)
                    const float* const cache = is_v ? p.vcache : p.kcache;
                    const int width = is_v ? p.vrow : p.kdim, row_w = is_v && !shared ? p.vdim : p.kdim, c0 = p.talk && !is_v ? 0 : part * kGroupW;
                    const int gg = p.talk && !is_v ? part : g, w = min(kGroupW, row_w - c0);
                    float* const inv = is_v ? (part == 0 && !shared ? v_inv + at_t * kKeys : nullptr)
                                            : part == 0 || geo.k_sets > 1 ? k_inv + (at_t * geo.k_sets + (geo.k_sets > 1 ? part : 0)) * kKeys : nullptr;
#pragma unroll 1
                    for (int e = lw; e < kKeys / 8; e += kFetchWarps) {
                        const int j = z.j0 + e * 8 + kin;
                        const bool in = j < z.k_end;
                        const float* src = cache;
                        if (in) {
                            const int page = p.table ? p.table[(size_t)z.slot * p.max_pages + j / p.page_size] : z.slot;
                            src += (((size_t)page * p.kv_heads + gg) * p.page_size + (p.table ? j % p.page_size : j)) * width;
                        }
                        float m = 0.f, sc, inverse;
#pragma unroll 1
                        for (int c = 4 * cq; in && c < row_w; c += 16) m = max_abs4(m, *reinterpret_cast<const float4*>(src + c));
                        const bool bad = scale_row(row_max(m), sc, inverse);
                        // (a value's scales have their place before the ring has one: see geometry_of)
                        if (e == lw && !is_v && !wait_for(&empty[slot], phase ^ 1u)) { ok = false; return; }
                        if (inv && lane < 8) inv[e * 8 + lane] = inverse;
                        if (e == 0 && !is_v && part == 0 && lane == 0) s_tile[at_t] = about;
                        if (e == lw && is_v && !wait_for(&empty[slot], phase ^ 1u)) { ok = false; return; }
                        const int blocks = wp >> 3;
                        unsigned char* dst = ring + (size_t)slot * geo.slot_bytes + e * blocks * 128 + kin * 16;
#pragma unroll 1
                        for (int c8 = cq; c8 < blocks; c8 += 4) {
                            const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
                            const float4 a = in && !bad && 8 * c8 < w ? *reinterpret_cast<const float4*>(src + c0 + 8 * c8) : none;
                            const float4 b = in && !bad && 8 * c8 + 4 < w ? *reinterpret_cast<const float4*>(src + c0 + 8 * c8 + 4) : none;
                            uint32_t hi[4], lo[4];
                            split2(a.x * sc, a.y * sc, hi[0], lo[0]);
                            split2(a.z * sc, a.w * sc, hi[1], lo[1]);
                            split2(b.x * sc, b.y * sc, hi[2], lo[2]);
                            split2(b.z * sc, b.w * sc, hi[3], lo[3]);
                            *reinterpret_cast<uint4*>(dst + c8 * 128) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                            *reinterpret_cast<uint4*>(dst + c8 * 128 + kKeys * wp * 2) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                        }
                    }
                    fence_smem_async();
                    __syncwarp();
                    if (lane == 0 && is_v && inv) mbar_arrive(&v_ready[at_t]);
                    if (lane == 0) mbar_arrive(&full[slot]);
                }
            };
            // the keys of a tile, then the values of the tile s_bufs before: the order in which they are multiplied
            Tile z0{}, z1{}, z2{};                                // the newest first
            unsigned at0 = 0, at1 = 0, at2 = 0;                   // their places
            int known = -1, left = geo.s_bufs, n = 0;             // the sequence whose tiles in the room are known; turns that are left without keys; tiles so far
            SlotTiles room{};
            bool more = true;
            Walk w(s_slot, s_pos, s_breaks, n_tok);
#pragma unroll 1
            while (ok) {
                more = more && w.next(p);
                if (!more && left-- == 0) break;                  // (the last turns have values only)
                z2 = z1; at2 = at1;
                z1 = z0; at1 = at0;
                if (more) {
                    if (n > 0 && ++at0 == (unsigned)geo.depth) at0 = 0;
                    z0.slot = s_slot[w.seg_a];
                    z0.j0 = w.j0;
                    z0.k_end = w.k_end;
                    about = make_int4(w.j0, w.seg_a | w.seg_b << 16, w.k_end, w.lo);
                    z0.split = -1;
                    if (work) {
                        if (z0.slot != known) room = reinterpret_cast<const SlotTiles*>(work)[known = z0.slot];
                        const int j = w.j0 / kKeys;
                        z0.split = j >= room.first && j < room.end ? room.base + j : j == 0 ? room.zero : -1;
                    }
                }
                ++n;
                const bool values = n > geo.s_bufs;               // of the tile s_bufs turns before
                const int nk = more ? geo.n_kst : 0, parts = nk + (values ? geo.n_vst : 0);
#pragma unroll 1
                for (int i = 0; i < parts && ok; ++i) {
                    const bool is_v = i >= nk, two = geo.s_bufs == 2;
                    fetch(!is_v ? z0 : two ? z2 : z1, !is_v ? at0 : two ? at2 : at1, is_v, is_v ? i - nk : i);
                    if (++slot == (unsigned)geo.n_slots) slot = 0, phase ^= 1u;
                }
            }
            if constexpr (SELF) {
                if (ok && raw >= 0) split_raw(false);
                asm volatile("cp.async.wait_group 0;" ::: "memory");  // (a wait may have run out)
            }
        } else {
            // ================= the MMA issuer: the whole warp counts tiles, one elected lane issues =================
            // The number of tiles and the address in tensor memory are broadcast, so that everything below is known to be the same for the
            // whole warp and the instructions' operands stay in uniform registers.  (In a loop that walked the tiles itself an instruction
            // took 100 cycles to issue for the scores and 160 for the values: 4300 cycles of a tile.)
            int n_tiles = 0;
            for (Walk w(s_slot, s_pos, s_breaks, n_tok); w.next(p);) ++n_tiles;
            n_tiles = __shfl_sync(0xffffffffu, n_tiles, 0);
            if (lane == 0) s_rows[0] = n_tiles;
            asm volatile("bar.arrive 1, %0;" ::"n"(32 * RW + 32) : "memory");
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint32_t t_s = tm, t_p = tm + 64u * geo.n_kst * geo.s_bufs, t_o = t_p + 64u * geo.p_bufs;
            const uint32_t idesc_s = (1u << 4) | ((uint32_t)(kKeys >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
            const uint32_t q_addr = smem_u32(qs), ring_addr = smem_u32(ring);
            unsigned at = 0;
            bool ok = true;
            auto values = [&](unsigned t) {                   // value product of tile t
                if (!wait_warp(&p_ready[t & 1u], (t >> 1) & 1u)) { ok = false; return; }
                const unsigned before = t - geo.o_bufs;       // the tile whose product lay there
                if (t >= (unsigned)geo.o_bufs && !wait_warp(&o_empty[before & 1u], (before >> 1) & 1u)) { ok = false; return; }
                const uint32_t weights = t_p + (geo.p_bufs == 2 ? (t & 1u) * 64u : 0u);
#pragma unroll 1
                for (int vs = 0; vs < NVS; ++vs) {
                    const unsigned slot = at % geo.n_slots;
                    if (!wait_warp(&full[slot], (at / geo.n_slots) & 1u)) { ok = false; return; }
                    fence_after();
                    const uint32_t wn = vs == geo.n_vst - 1 ? geo.wv_last : geo.wv0, wp = vs == geo.n_vst - 1 ? geo.v_last_layout : geo.v0_layout;
                    const uint32_t idesc = (1u << 4) | (1u << 16) | ((wn >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
                    const uint32_t va = ring_addr + slot * geo.slot_bytes;
                    const uint64_t vh = block_desc(va, wp * 16u, 128u), vl = block_desc(va + kKeys * wp * 2u, wp * 16u, 128u);
                    const uint32_t step = 2u * wp;            // 16 keys, in descriptor units of 16 bytes
                    const uint32_t d = t_o + 128u * (geo.o_bufs == 2 ? t & 1u : (unsigned)vs);
                    if (elect_one_sync()) {
#pragma unroll 1
                        for (uint32_t e = 0; e < 3; ++e) {        // lo hi, hi lo, hi hi
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) mma_ts(d, weights + (e == 0 ? 32u : 0u) + 8u * k, (e == 1 ? vl : vh) + k * step, idesc, (e | k) != 0);
                        }
                        commit_to(&empty[slot]);
                        if (vs == NVS - 1) commit_to(&pv_done[t & 1u]);
                    }
                    __syncwarp();
                    ++at;
                }
            };
            ok = wait_warp(q_ready, 0);
#pragma unroll 1
            for (unsigned t = 0; ok && t < (unsigned)(n_tiles + geo.s_bufs); ++t) {
                const unsigned before = t - geo.s_bufs;       // the tile whose scores lay there, and whose values are next
                const int groups = t < (unsigned)n_tiles ? geo.n_kst : 0;
                if (groups > 0 && t >= (unsigned)geo.s_bufs && !wait_warp(&s_empty[before & 1u], (before >> 1) & 1u)) { ok = false; break; }
#pragma unroll 1
                for (int st = 0; st < groups; ++st) {
                    const unsigned slot = at % geo.n_slots;
                    if (!wait_warp(&full[slot], (at / geo.n_slots) & 1u)) { ok = false; break; }
                    fence_after();
                    const uint32_t wp = st == geo.n_kst - 1 ? geo.wk_last : geo.wk0;
                    const uint32_t ka = ring_addr + slot * geo.slot_bytes, qa = q_addr + st * geo.wk0 * kRows * 4u;
                    const uint64_t kh = block_desc(ka, 128u, wp * 16u), kl = block_desc(ka + kKeys * wp * 2u, 128u, wp * 16u);
                    const uint64_t qh = block_desc(qa, 128u, wp * 16u), ql = block_desc(qa + kRows * wp * 2u, 128u, wp * 16u);
                    const uint32_t d = t_s + (geo.s_bufs == 2 ? (t & 1u) * 64u * geo.n_kst : 0u) + 64u * st;
                    if (elect_one_sync()) {
                        const uint32_t n = wp >> 4;           // 16 channels per instruction: 2 blocks, 16 descriptor units
#pragma unroll 1
                        for (uint32_t e = 0; e < 3; ++e) {
                            const uint64_t qe = e == 0 ? ql : qh, ke = e == 1 ? kl : kh;
#pragma unroll
                            for (uint32_t k = 0; k < kGroupW / 16; ++k)
                                if (k < n) mma_ss(d, qe + 16u * k, ke + 16u * k, idesc_s, (e | k) != 0);
                        }
                        commit_to(&empty[slot]);
                        if (st == geo.n_kst - 1) commit_to(&s_full[t & 1u]);
                    }
                    __syncwarp();
                    ++at;
                }
                if (t >= (unsigned)geo.s_bufs && ok && before < (unsigned)n_tiles) values(before);
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == RW) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

bool geometry_of(const SplitAttention& a, Geometry& g, size_t& smem) {
    if (a.heads <= 0 || a.kv_heads <= 0 || a.heads % a.kv_heads || a.kdim <= 0 || a.vdim <= 0) return false;
    auto mul4 = [](int v) { return v % 4 == 0; };
    auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (!mul4(a.ldq) || !mul4(a.qdim) || !mul4(a.kdim) || !mul4(a.vdim) || !mul4(a.vrow) || !mul4(a.ldo) || !aligned(a.q) || !aligned(a.kcache) ||
        !aligned(a.vcache) || !aligned(a.out) || (reinterpret_cast<uintptr_t>(a.out_bf16) & 7) || (a.gate && (!mul4(a.ldg) || !aligned(a.gate))))
        return false;
    if (a.qdim != a.kdim || a.vdim > 256 || (a.talk && a.kdim > kGroupW)) return false;
    if (a.rows_per_slot > 0 && (long long)a.rows_per_slot * 16 < a.M) return false;
    auto pad16 = [](int v) { return (v + 15) & ~15; };
    const int rep = a.heads / a.kv_heads;
    g.page_shift = -1;
    if (a.page_size > 0 && (a.page_size & (a.page_size - 1)) == 0)
        for (g.page_shift = 0; 1 << g.page_shift < a.page_size;) ++g.page_shift;
    g.pk_shift = 0;
    while (g.pk_shift < 7 && rep % (2 << g.pk_shift) == 0) ++g.pk_shift;
    if (a.talk) {
        g.n_kst = a.kv_heads;
        g.wk0 = g.wk_last = pad16(a.kdim);
    } else {
        g.n_kst = (a.kdim + kGroupW - 1) / kGroupW;
        g.wk0 = pad16(std::min(a.kdim, kGroupW));
        g.wk_last = pad16(a.kdim - (g.n_kst - 1) * kGroupW);
    }
    g.n_vst = (a.vdim + kGroupW - 1) / kGroupW;
    g.wv0 = pad16(std::min(a.vdim, kGroupW));
    g.wv_last = pad16(a.vdim - (g.n_vst - 1) * kGroupW);
    if (g.n_kst > kMaxKStages || 64 * g.n_kst + 64 + 128 * g.n_vst > 512) return false;      // columns of tensor memory
    g.shared_kv = a.kcache == a.vcache && a.kv_heads == 1 && !a.talk && a.vrow == a.kdim && a.vdim <= a.kdim;
    g.v0_layout = g.wv0;
    g.v_last_layout = g.wv_last;
    if (g.shared_kv) {                                        // value group i lies in key group i
        g.v0_layout = g.n_kst == 1 ? g.wk_last : g.wk0;
        g.v_last_layout = g.n_vst == g.n_kst ? g.wk_last : g.wk0;
    }
    const int k_heads = a.talk ? 1 : a.kv_heads;              // (a mixed score's key groups are all kv heads)
    g.k_parts = k_heads * g.n_kst;
    g.parts = g.k_parts + (g.shared_kv ? 0 : a.kv_heads * g.n_vst);
    g.k_sets = a.talk ? a.kv_heads : 1;
    g.sets = a.kv_heads * (g.shared_kv ? 1 : 2);
    g.tile_bytes = kKeys * 4u * (k_heads * ((g.n_kst - 1) * g.wk0 + g.wk_last) + (g.shared_kv ? 0 : a.kv_heads * ((g.n_vst - 1) * g.wv0 + g.wv_last)));
    g.cap_tiles = 0;
    if (a.work && aligned(a.work) && (a.rows_per_slot > 0 ? !a.table && a.n_seq == 0 : a.table && a.n_seq > 0)) {
        g.scale_off = (unsigned)a.n_slots * sizeof(SlotTiles);
        const size_t per = g.tile_bytes + 4u * kKeys * g.sets, fixed = g.scale_off + 128;
        if (a.work_bytes > fixed) g.cap_tiles = (int)std::min<size_t>((a.work_bytes - fixed) / per, 65535);
        g.tile_off = (unsigned)((g.scale_off + 4u * kKeys * g.sets * (unsigned)g.cap_tiles + 127u) & ~127u);
    }
    // Two of each where tensor memory has the columns.  Two sets of weights first: the groups of row warps do not wait for each other's value
    // product then.  (Wide values have one product of 256 columns, and keys that lie one tile ahead.)
    static constexpr int kBufs[][3] = {{2, 2, 2}, {1, 2, 2}, {1, 1, 2}, {1, 2, 1}, {1, 1, 1}};
    bool fits = false;
    for (const auto& b : kBufs) {
        if (g.n_vst == 2 && (b[0] == 2 || b[2] == 2)) continue;
        if (a.cap > 0.f && b[1] == 1) continue;               // (capped scores pass through the weights' columns)
        g.s_bufs = b[0]; g.p_bufs = b[1]; g.o_bufs = b[2];
        fits = 64 * g.n_kst * b[0] + 64 * b[1] + 128 * g.n_vst * b[2] <= 512;
        if (fits) break;
    }
    if (!fits) return false;
    g.slot_bytes = kKeys * std::max(g.wk0, std::max(g.wv0, g.v0_layout)) * 4;
    g.q_bytes = ((g.n_kst - 1) * g.wk0 + g.wk_last) * kRows * 4;
    // A tile's scales are written when its first key group has its slot: the stage n_slots places before is done.  They lie depth tiles
    // apart so that this stage is no earlier than the first value group of the tile whose scales were there (a value group is multiplied
    // after the rows have used all scales of its tile).  In order, a tile is n_kst key groups and, behind those of the s_bufs tiles next, n_vst
    // value groups.
    const int per_tile = g.n_kst + g.n_vst;
    auto depth_of = [&](int slots) { return g.s_bufs + (slots + g.n_kst + per_tile - 1) / per_tile; };
    // A tile's numbers are stored when its weights are: with one set of weights and one product the tile before has been multiplied by then,
    // the one before that added.
    g.rings = g.p_bufs == 1 && g.o_bufs == 1 ? 2 : 4;
    auto control_of = [&](int slots) {
        const int depth = depth_of(slots), bars = 2 * slots + 15 + (g.shared_kv ? 0 : depth);
        return ((bars + 1) & ~1) * 8 + kRows * (2 * 4 + (g.four ? g.rings * 8 : g.rings * 2) + g.rings * 2) + depth * (kKeys * (g.k_sets + (g.shared_kv ? 0 : 1)) * 4 + 16) + 32 + 2 * (kRows >> g.pk_shift) * 4;
    };
    g.four = 1;
    auto most_slots = [&] {
        for (g.n_slots = kMaxSlots; g.n_slots >= 2; --g.n_slots)
            if (g.n_slots * g.slot_bytes + g.q_bytes + control_of(g.n_slots) <= kSmemMost) return true;
        return false;
    };
    if (!most_slots()) {
        g.four = 0;
        if (g.n_vst == 1 || !most_slots()) return false;      // (only keys of 305 channels and more over values of 129 and more come here)
    }
    g.depth = depth_of(g.n_slots);
    const int control = control_of(g.n_slots);
    // the output is staged in the ring and the queries: 8 warps of 32 rows, 4 floats between the rows
    const int staged = kRows * 2 * ((g.n_vst == 1 ? g.wv0 / 2 : 128) + 4) * 4;
    g.q_bytes = std::max(g.q_bytes, staged - g.n_slots * g.slot_bytes);
    smem = (size_t)g.n_slots * g.slot_bytes + g.q_bytes + control;
    return smem <= (size_t)kSmemMost;
}

template <int NVS, bool FOUR, bool SELF>
cudaError_t launch_inst(const SplitAttention& a, const Geometry& g, size_t smem, cudaStream_t st) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = ask_smem<split_attention_kernel<NVS, FOUR, SELF>>(device, kSmemMost);
    if (e != cudaSuccess) return e;
    const int tt = kRows >> g.pk_shift, tiles = a.n_seq > 1 ? a.M / tt + a.n_seq : (a.M + tt - 1) / tt;
    if (a.work) {
        split_keys_kernel<<<dim3(std::min(g.cap_tiles, std::max(1, kSplitGrid / g.parts)), g.parts), 256, 0, st>>>(a, g);
        ++extra_launches();
    }
    split_attention_kernel<NVS, FOUR, SELF><<<(a.heads >> g.pk_shift) * tiles, kSplitThreads, smem, st>>>(a, g);
    return cudaGetLastError();
}

template <bool SELF>
cudaError_t launch_any(const SplitAttention& a, const Geometry& g, size_t smem, cudaStream_t st) {
    if (g.n_vst == 2) return g.four ? launch_inst<2, true, SELF>(a, g, smem, st) : launch_inst<2, false, SELF>(a, g, smem, st);
    return launch_inst<1, true, SELF>(a, g, smem, st);
}

}  // namespace

// A word of `device` in mapped host memory, which a kernel sets when one of its waits has run out (null: there is none yet, and a stream
// that is being captured is no place to make one)
int* split_attention_ran_out(int device, cudaStream_t st) {
    static std::mutex lock;
    static int* words[64] = {};
    if (device < 0 || device >= 64) return nullptr;
    const std::lock_guard<std::mutex> hold(lock);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (!words[device]) {
        int* w = nullptr;
        if (cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone &&
            cudaHostAlloc(reinterpret_cast<void**>(&w), sizeof(int), cudaHostAllocMapped) == cudaSuccess) {
            *w = 0;
            words[device] = w;
        } else {
            (void)cudaGetLastError();
        }
    }
    return words[device];
}

bool take_ran_out(int device, cudaStream_t st) {
    int* const word = split_attention_ran_out(device, st);
    if (!word || !*reinterpret_cast<volatile int*>(word)) return false;
    *reinterpret_cast<volatile int*>(word) = 0;
    return true;
}

bool split_attention_ok(const SplitAttention& a) {
    Geometry g;
    size_t smem;
    return geometry_of(a, g, smem);
}

int split_attention_keys(const SplitAttention& a, int slot) { return range_keys(a, slot); }

size_t split_attention_work_bytes(const SplitAttention& a, int keys) {
    Geometry g;
    size_t smem;
    if (!geometry_of(a, g, smem)) return 0;
    return (size_t)a.n_slots * sizeof(SlotTiles) + 256 + (size_t)((keys + kKeys - 1) / kKeys) * (g.tile_bytes + 4u * kKeys * g.sets);
}

cudaError_t launch_split_attention(const SplitAttention& a, cudaStream_t st) {
    Geometry g;
    size_t smem;
    if (a.M <= 0 || !geometry_of(a, g, smem)) return cudaErrorNotSupported;
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    g.ran_out = split_attention_ran_out(device, st);          // (mapped and unified: one address on both sides)
    if (take_ran_out(device, st)) return cudaErrorLaunchTimeout;
    SplitAttention with = a;
    if (g.cap_tiles <= 0) with.work = nullptr;
    // whether the room holds every key: a slot's range here, what the caller says for sequences (of kept keys in front of a window it has one tile)
    long long tiles = a.n_tiles > 0 && (a.window <= 0 || a.keep_first <= kKeys) ? a.n_tiles : (long long)1 << 40;
    if (a.rows_per_slot > 0) {
        tiles = 0;
        for (int slot = 0; slot * a.rows_per_slot < a.M; ++slot) tiles += (std::max(range_keys(a, slot), 0) + kKeys - 1) / kKeys;
    }
    return with.work && tiles <= g.cap_tiles ? launch_any<false>(with, g, smem, st) : launch_any<true>(with, g, smem, st);
}

}  // namespace dia
