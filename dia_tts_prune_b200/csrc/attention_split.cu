// attention_split.cu - softmax attention of many query rows on the 5th-generation tensor cores, with fp32 operands split into
// two fp16 terms (sm_100a).
//
// A CTA owns 128 (token, head) rows: up to 128 / PK consecutive tokens times PK query heads that read the same key/value head, so
// that a tile of keys serves all of them.  It walks its keys 64 at a time:
//   4 warps         fetch key and value rows from the pages, scale them by a power of two, split x = hi + lo into fp16 and put both
//                   into a ring of shared-memory slots ([key / 8][channel / 8] blocks of 8 x 16 bytes: the layout is the K-major
//                   operand of the scores and the MN-major operand of the value product)
//   1 warp          issues tcgen05.mma: scores S = Q K^T (M = 128, N = 64; lo hi, hi lo, then hi hi, so that the small terms are
//                   added first) per group of at most 128 channels, and the value product of the tile before (weights as the
//                   operand in tensor memory)
//   8 or 16 warps   two or four threads per row, 32 or 16 keys each: scores from tensor memory (the channel groups are summed here, in fp32),
//                   cap, bias, mask, online softmax in base 2, weights split and written to tensor memory; then the value
//                   product of the tile before is added to the row's fp32 registers
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
// what shares the launch.  Cost, against one scale per tile of rows, keys and values: 4096 rows, 16 heads of 128 over 4, window 1024
// 237 -> 264 us; mixed scores, three prompts of 2048 rows, 8 heads of 128 over 2, 127 -> 146, of which the factors per key and per
// value 5 us each; 16 keys that share a factor (scales in steps of 2^8) take as long.
//
// Bound: the instructions of the row warps and their latencies.  Per 64 keys and 128 rows 3 x 128 x 64 x (dk + dv) multiply-adds on the tensor
// pipe (1536 cycles at 128 + 128) stand against about 8000 cycles of a tile with its share of the CTA's start and end, on 47 % of which a scheduler
// issues (four row warps on each; with two row warps 8800 and 34 %; profiles/split_kernels_ncu.txt).
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
template <int RT>
constexpr int kSplitThreads = 32 * (4 * RT + 8);
constexpr int kMaxSlots = 6, kMaxDepth = 5, kMaxKStages = 4;
constexpr int kSmemMost = 232448;                             // all of it dynamic
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kSplitOnceRows = 512;                           // rows of a kv head (M rep) from which keys with values of up to 128 channels are split in advance
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
    int o_bufs;                              // accumulators of the value product (2 where tensor memory has the columns)
    int k_sets;                              // scales of a key: one, with mixed scores one per kv head
    int depth;                               // tiles whose scales are in shared memory
    // the split keys and values in SplitAttention::work: SlotTiles per slot, then inverse scales [tile][set][key], then the tiles.  A
    // tile's parts: key groups (per kv head where the launch reads one head at a time), then value groups; its sets of scales: the keys
    // of each kv head, then the values of each (shared_kv: the keys' only)
    int parts, k_parts, sets, cap_tiles;
    int* ran_out;                            // the device's word (null: none)
    unsigned tile_bytes, scale_off, tile_off;
};
// where the tiles of a slot's sequence lie: tile j / 64 of its keys is tile base + j / 64 of the room for first <= j / 64 < end; its
// tile 0 is tile `zero` (-1: only by the range)
struct SlotTiles { int base, first, end, zero; };

__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity) {
    for (unsigned i = 0; i < kSpinMost; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// the same for a converged warp, with one answer for all lanes (so that what follows is uniform: see elect_one_sync)
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity) {
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
__device__ __forceinline__ void tmem_load8(uint32_t addr, float* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
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
template <int N>
__device__ __forceinline__ void tmem_load_n(uint32_t addr, float (&v)[N]) {
    if constexpr (N == 32) tmem_load32(addr, v);
    else if constexpr (N == 16) tmem_load16(addr, v);
    else tmem_load8(addr, v);
}
// two fp32 operations in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// tanh x = x + x^3 q(x^2) for |x| <= kTanhRange: q interpolates (tanh x / x - 1) / x^2 at six Chebyshev nodes (relative error of the
// result 3e-10 before rounding).  A tile's scores mostly lie there, and it takes a fifth of the library call's instructions
// (a tile of capped scores: 2100 -> 800 cycles)
constexpr float kTanhRange = 0.6f;
__device__ __forceinline__ float2 tanh_near_zero(float2 x) {
    const float2 u = mul2(x, x);
    float2 q = make_float2(2.3707656405e-3f, 2.3707656405e-3f);
    q = fma2(q, u, make_float2(-8.41007080153e-3f, -8.41007080153e-3f));
    q = fma2(q, u, make_float2(2.17883219971e-2f, 2.17883219971e-2f));
    q = fma2(q, u, make_float2(-5.39615517813e-2f, -5.39615517813e-2f));
    q = fma2(q, u, make_float2(1.33333128669e-1f, 1.33333128669e-1f));
    q = fma2(q, u, make_float2(-3.33333332312e-1f, -3.33333332312e-1f));
    return fma2(mul2(x, u), q, x);
}
// v[i] *= f[i] (16-byte aligned; the same addresses for all lanes)
template <int N>
__device__ __forceinline__ void scale_by(float* v, const float* f) {
#pragma unroll
    for (int e = 0; e < N; e += 4) {
        const float4 k = *reinterpret_cast<const float4*>(f + e);
        const float2 a = mul2(make_float2(v[e], v[e + 1]), make_float2(k.x, k.y)), b = mul2(make_float2(v[e + 2], v[e + 3]), make_float2(k.z, k.w));
        v[e] = a.x; v[e + 1] = a.y; v[e + 2] = b.x; v[e + 3] = b.y;
    }
}
__device__ __forceinline__ void tmem_loaded() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
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

__device__ __forceinline__ size_t part_offset(const Geometry& geo, int part) {
    const unsigned k_head = kKeys * 4u * ((geo.n_kst - 1) * geo.wk0 + geo.wk_last), v_head = kKeys * 4u * ((geo.n_vst - 1) * geo.wv0 + geo.wv_last);
    if (part < geo.k_parts) return (size_t)(part / geo.n_kst) * k_head + (size_t)(part % geo.n_kst) * geo.wk0 * kKeys * 4;
    part -= geo.k_parts;
    return (size_t)(geo.k_parts / geo.n_kst) * k_head + (size_t)(part / geo.n_vst) * v_head + (size_t)(part % geo.n_vst) * geo.wv0 * kKeys * 4;
}

// Splits the keys and values that the step's rows see, once for all row tiles: without it each of the M rep / 128 row tiles of a
// key/value head converts every tile it walks, and that conversion (two thirds of the instructions) bounds the kernel below.
// A CTA per (tile of the room, part), and two rounds of them at most: a room for many sequences has far more tiles than a short step
// fills.  Tiles are dealt to the sequences in order.  Warp w takes keys 8 w .. of the tile.
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
        const int seq = s_seq, slot = p.seq_slot[seq], pos0 = p.row_pos[p.seq_row0[seq]], k_end = pos0 + p.seq_count[seq], j0 = s_first * kKeys;
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
            const int page = p.table[(size_t)slot * p.max_pages + j / p.page_size];
            src += (((size_t)page * p.kv_heads + g) * p.page_size + j % p.page_size) * width;
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

// NVS: channel groups of a value (1: up to 128 channels, 2: up to 256).  RT: threads of a row; each takes 64 / RT keys of a tile and an equal
// share of the output channels
template <int NVS, int RT>
__global__ void __launch_bounds__(kSplitThreads<RT>, 1)
split_attention_kernel(const __grid_constant__ SplitAttention p, const __grid_constant__ Geometry geo) {
    constexpr int DVH = 128 * NVS / RT;                       // output channels of a thread
    constexpr int KP = kKeys / RT, RW = 4 * RT;               // keys of a thread, row warps
    // The block is launched with 128 registers a thread (RT = 4: 80).  (Wide values with two threads per row, 4096 rows, 16 heads over latent
    // rows of 256 + 32, window 1024: 184 and 112 452 us, 192 and 96 443, 200 and 80 421.  What the fetching warps spill is used for
    // keys that are not split in advance only.)
    constexpr int kLaunchRegs = RT == 4 ? 80 : 128;
    constexpr int kRowRegs = RT == 4 ? (NVS == 1 ? 96 : 104) : (NVS == 1 ? 176 : 200), kFetchRegs = RT == 4 ? (NVS == 1 ? 64 : 32) : (NVS == 1 ? 128 : 80);
    static_assert(32 * RW * kRowRegs + 128 * kFetchRegs + 128 * 32 <= kLaunchRegs * kSplitThreads<RT>, "registers of the block");
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* ring = smem;
    unsigned char* qs = ring + (size_t)geo.n_slots * geo.slot_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(qs + geo.q_bytes);
    uint64_t* empty = full + kMaxSlots;
    uint64_t* s_full = empty + kMaxSlots;                     // scores of a tile are there / have been read
    uint64_t* s_empty = s_full + 1;
    uint64_t* p_ready = s_empty + 1;                          // weights of a tile are there / its value product is done
    uint64_t* pv_done = p_ready + 1;
    uint64_t* q_ready = pv_done + 1;
    uint64_t* pair = q_ready + 1;                             // [4] the warps that share rows
    uint64_t* v_ready = pair + 4;                             // [depth] the scales of a tile's values are there
    float* k_inv = reinterpret_cast<float*>(v_ready + kMaxDepth);      // [depth][k_sets][64] inverse scales of the keys
    float* v_inv = geo.shared_kv ? k_inv : k_inv + geo.depth * geo.k_sets * kKeys;      // [depth][64] of the values
    float* row_x = v_inv + geo.depth * kKeys;                 // [2][RT][128] what the threads of a row tell each other
    uint32_t* s_breaks = reinterpret_cast<uint32_t*>(row_x + 2 * RT * kRows);      // [4]
    uint32_t* s_tmem = s_breaks + 4;
    int* s_rows = reinterpret_cast<int*>(s_tmem + 1);         // [2]
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
        for (int i = 0; i < kMaxSlots; ++i) { mbar_init(&full[i], 4); mbar_init(&empty[i], 1); }
        mbar_init(s_full, 1);
        mbar_init(s_empty, RW);
        mbar_init(p_ready, RW);
        mbar_init(pv_done, 1);
        mbar_init(q_ready, RW);
        for (int i = 0; i < 4; ++i) mbar_init(&pair[i], RT);
        for (int i = 0; i < kMaxDepth; ++i) mbar_init(&v_ready[i], 4);
        fence_mbar_init();
    }
    if (warp == RW + 4) {
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
    const uint32_t t_s = tmem, t_p = tmem + 64u * geo.n_kst, t_o = t_p + 64u;    // scores | weights (hi, lo) | value product

    if (warp < RW) {
        // ================= softmax: rows 32 (warp % 4) + lane, keys KP (warp / 4) .. of a tile =================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
        // ---- the query tile: largest magnitude, then both terms.  Row r of the tile is head h0 + r % PK of token r / PK; a warp takes
        // eight rows at a time, a lane eight channels of one.  (The first keys are on their way meanwhile: with the tile made by all
        // warps in front of the roles, its loops unrolled, a launch of one key tile took 17 us, now 14: cold instruction fetches) ----
        const int chunks = ((geo.n_kst - 1) * geo.wk0 + geo.wk_last) >> 3, wkb = geo.wk0 >> 3;
        auto q_values = [&](int row, int ch, float (&v)[8]) { // channels 8 ch .. of the padded row
            const int i = row >> geo.pk_shift, h = h0 + (row & (PK - 1)), st = geo.n_kst == 1 ? 0 : ch / wkb, c = 8 * (ch - st * wkb);
            const int width = p.talk ? p.kdim : min(kGroupW, p.kdim - st * kGroupW);
            const bool in = i < n_tok && ch < chunks, one = in && c < width, both = in && c + 4 < width;    // (widths are multiples of 4)
            const float* src = p.q + (size_t)(r0 + i) * p.ldq + c;
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!p.talk) {
                src += (size_t)h * p.qdim + st * kGroupW;
                const float4 a = one ? *reinterpret_cast<const float4*>(src) : z, b = both ? *reinterpret_cast<const float4*>(src + 4) : z;
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
                v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
                return;
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0.f;
            if (!one) return;
            src += (size_t)st * rep * p.qdim;
            const float* mix = p.talk + h * p.heads + st * rep;
#pragma unroll 4
            for (int t = 0; t < rep; ++t) {                   // the mixed score is linear in the queries: mix those instead
                const float w = mix[t];
                const float4 a = *reinterpret_cast<const float4*>(src + (size_t)t * p.qdim);
                const float4 b = both ? *reinterpret_cast<const float4*>(src + (size_t)t * p.qdim + 4) : z;
                v[0] = fmaf(w, a.x, v[0]); v[1] = fmaf(w, a.y, v[1]); v[2] = fmaf(w, a.z, v[2]); v[3] = fmaf(w, a.w, v[3]);
                v[4] = fmaf(w, b.x, v[4]); v[5] = fmaf(w, b.y, v[5]); v[6] = fmaf(w, b.z, v[6]); v[7] = fmaf(w, b.w, v[7]);
            }
        };
        float* const q_inv = row_x + RT * kRows;              // [128] (read by a row's threads before they exchange anything there)
        auto q_scale = [&](float m, int row, bool& bad) {     // a row's scale from the four lanes that hold it
            float scale, inverse;
            bad = scale_row(row_max(m), scale, inverse);
            if (lane < 8) q_inv[row] = inverse;
            return scale;
        };
        auto q_store = [&](int row, int ch, float scale, bool bad, const float (&v)[8]) {
            if (ch >= chunks) return;
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split2(bad ? 0.f : v[2 * e] * scale, bad ? 0.f : v[2 * e + 1] * scale, hi[e], lo[e]);
            const int st = geo.n_kst == 1 ? 0 : ch / wkb, w = st == geo.n_kst - 1 ? geo.wk_last : geo.wk0, c8 = ch - st * wkb;
            unsigned char* dst = qs + (size_t)st * geo.wk0 * kRows * 4 + (size_t)(((row >> 3) * (w >> 3) + c8) * 128 + (row & 7) * 16);
            *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(dst + (size_t)w * kRows * 2) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        };
        constexpr int RG = 4 / RT;                            // groups of 8 RW rows
        const int qrow = warp * 8 + (lane & 7), qch = lane >> 3;
        if (!p.talk && geo.n_kst == 1) {                      // all of it fits the registers
            float4 v[4 * RG][2];
#pragma unroll
            for (int rg = 0; rg < RG; ++rg) {
                const int row = qrow + 8 * RW * rg, i = row >> geo.pk_shift;
                const float* src = p.q + (size_t)(r0 + i) * p.ldq + (size_t)(h0 + (row & (PK - 1))) * p.qdim + 8 * qch;
                const int left = i < n_tok ? p.kdim - 8 * qch : 0;
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        v[rg * 4 + k][e] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (32 * k + 4 * e < left) v[rg * 4 + k][e] = *reinterpret_cast<const float4*>(src + 32 * k + 4 * e);
                    }
            }
#pragma unroll
            for (int rg = 0; rg < RG; ++rg) {
                float m = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) m = max_abs4(max_abs4(m, v[rg * 4 + i][0]), v[rg * 4 + i][1]);
                bool bad;
                const float scale = q_scale(m, qrow + 8 * RW * rg, bad);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 a = v[rg * 4 + i][0], b = v[rg * 4 + i][1];
                    const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                    q_store(qrow + 8 * RW * rg, qch + 4 * i, scale, bad, x);
                }
            }
        } else {
            for (int rg = 0; rg < RG; ++rg) {
                float m = 0.f, scale = 0.f;
                bool bad = false;
                for (int pass = 0; pass < 2; ++pass) {
                    for (int ch = qch; ch < chunks; ch += 16) {
                        float v[4][8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) q_values(qrow + 8 * RW * rg, ch + 4 * i, v[i]);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (pass == 0) {
#pragma unroll
                                for (int e = 0; e < 8; ++e) m = max_nan(m, fabsf(v[i][e]));
                            } else {
                                q_store(qrow + 8 * RW * rg, ch + 4 * i, scale, bad, v[i]);
                            }
                        }
                    }
                    if (pass == 0) scale = q_scale(m, qrow + 8 * RW * rg, bad);
                }
            }
        }
        fence_smem_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_ready);
        asm volatile("bar.sync 1, %0;" ::"n"(32 * RW) : "memory");          // (all queries are stored, and the rows' scales are there)
        const int qt = warp & 3, hf = warp >> 2, row = qt * 32 + lane, tok = row >> geo.pk_shift, h = h0 + (row & (PK - 1));
        const uint32_t lanes = (uint32_t)(qt * 32) << 16;
        const int my_pos = s_pos[tok];
        const int my_lo = first_key_of(max(my_pos, 0), p.window, p.chunk), kept = p.window > 0 ? p.keep_first : 0;
        const bool ranged = p.rows_per_slot > 0 && p.mode != 0;
        // scores and maxima are in units of log 2 (a capped score from its cap on): the largest score's weight is exactly 1 at any magnitude
        const float cap = p.cap, inv_cap = cap > 0.f ? 1.0f / cap : 0.f;
        const float mult = q_inv[row] * p.scale * (p.temp ? p.temp[h] : 1.f) * (cap > 0.f ? 1.f : kLog2e);
        const float slope = p.slopes ? p.slopes[h] * kLog2e : 0.f;
        // channels of this thread: c0 .. + n_mine, at t_mine in tensor memory
        const int share = NVS == 1 ? (geo.wv0 + 8 * RT - 1) / (8 * RT) * 8 : DVH, part = NVS == 1 ? hf : hf % (RT / 2), group = NVS == 1 ? 0 : hf / (RT / 2);
        const int n_mine = max(0, min(share, (group ? geo.wv_last : geo.wv0) - part * share)), c0 = group * 128 + part * share;
        const uint32_t t_mine = t_o + c0 + lanes;
        float O[DVH];
#pragma unroll
        for (int c = 0; c < DVH; ++c) O[c] = 0.f;
        constexpr int LP = KP / 16;                           // denominators: a sum per 16 keys of a tile, the same with any threads per row
        float m_run = -CUDART_INF_F, l_run[LP] = {}, corr_prev = 1.f, wi_prev = 0.f;
        bool ok = true;
        constexpr int OW = NVS == 1 && RT == 2 ? 32 : 16;     // columns in flight
        auto add_values = [&](unsigned t, float corr, float vi) {      // O <- corr O + vi * value product of tile t (which is done)
            const bool same = __all_sync(0xffffffffu, corr == 1.f);
            const uint32_t from = t_mine + (geo.o_bufs == 2 ? (t & 1u) * 128u : 0u);
            const float2 vi2 = make_float2(vi, vi), c2 = make_float2(corr, corr);
#pragma unroll
            for (int c = 0; c < DVH; c += OW) {
                if (c < n_mine) {                             // (columns beyond n_mine hold whatever they held; they are not stored)
                    float v[OW];
                    if constexpr (OW == 32) tmem_load32(from + c, v);
                    else { tmem_load8(from + c, v); tmem_load8(from + c + 8, v + 8); }
                    tmem_loaded();
#pragma unroll
                    for (int e = 0; e < OW; e += 2) {
                        float2 o = make_float2(O[c + e], O[c + e + 1]);
                        if (!same) o = mul2(o, c2);
                        o = fma2(make_float2(v[e], v[e + 1]), vi2, o);
                        O[c + e] = o.x;
                        O[c + e + 1] = o.y;
                    }
                }
            }
        };
        unsigned t = 0, at_t = 0, round = 0;                  // t % depth, t / depth % 2
        Walk w(s_slot, s_pos, s_breaks, n_tok);
        for (; w.next(p); ++t) {
            if (!wait_for(s_full, t & 1u)) { ok = false; break; }
            fence_after();
            float s[KP];
            const float* ki = k_inv + at_t * geo.k_sets * kKeys + hf * KP;
            constexpr int SW = NVS == 1 ? KP : 8;             // scores in flight (a wide value leaves fewer registers)
#pragma unroll
            for (int c = 0; c < KP; c += SW) {
                float v[SW];
                tmem_load_n<SW>(t_s + lanes + hf * KP + c, v);
                tmem_loaded();
#pragma unroll
                for (int e = 0; e < SW; ++e) s[c + e] = v[e];
                if (geo.k_sets > 1) scale_by<SW>(s + c, ki + c);
                for (int st = 1; st < geo.n_kst; ++st) {
                    tmem_load_n<SW>(t_s + lanes + st * 64 + hf * KP + c, v);
                    tmem_loaded();
                    if (geo.k_sets > 1) scale_by<SW>(v, ki + st * kKeys + c);
#pragma unroll
                    for (int e = 0; e < SW; ++e) s[c + e] += v[e];
                }
                if (geo.k_sets == 1) scale_by<SW>(s + c, ki + c);
            }
            const float2 mult2 = make_float2(mult, mult);
#pragma unroll
            for (int e = 0; e < KP; e += 2) {
                const float2 x = mul2(make_float2(s[e], s[e + 1]), mult2);
                s[e] = x.x;
                s[e + 1] = x.y;
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_empty);
            // ---- cap, distance bias, visibility ----
            const int k0 = w.j0 + hf * KP;
            if (cap > 0.f) {
                const float2 ic = make_float2(inv_cap, inv_cap);
#pragma unroll
                for (int e = 0; e < KP; e += 2) {
                    const float2 x = mul2(make_float2(s[e], s[e + 1]), ic);
                    s[e] = x.x;
                    s[e + 1] = x.y;
                }
                float big = 0.f;
#pragma unroll
                for (int e = 0; e < KP; ++e) big = fmaxf(big, fabsf(s[e]));
                // each score takes the form that its own magnitude asks for; whether all of them are near zero decides the speed only
                const float2 cc = make_float2(cap * kLog2e, cap * kLog2e);
                const bool near = __all_sync(0xffffffffu, big <= kTanhRange);
                if (NVS == 1 && near) {                       // (wide values: one copy of the code, whose registers are few)
#pragma unroll
                    for (int e = 0; e < KP; e += 2) {
                        const float2 r = mul2(tanh_near_zero(make_float2(s[e], s[e + 1])), cc);
                        s[e] = r.x;
                        s[e + 1] = r.y;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < KP; e += 2) {
                        float2 r = tanh_near_zero(make_float2(s[e], s[e + 1]));
                        if (NVS == 1 || !near) {
                            if (!(fabsf(s[e]) <= kTanhRange)) r.x = tanhf(s[e]);
                            if (!(fabsf(s[e + 1]) <= kTanhRange)) r.y = tanhf(s[e + 1]);
                        }
                        r = mul2(r, cc);
                        s[e] = r.x;
                        s[e + 1] = r.y;
                    }
                }
            }
            if (p.slopes) {
                const float base = (float)(my_pos - k0);
                const float2 ns = make_float2(-slope, -slope);
#pragma unroll
                for (int e = 0; e < KP; e += 2) {
                    const float2 r = fma2(ns, make_float2(base - (float)e, base - (float)(e + 1)), make_float2(s[e], s[e + 1]));
                    s[e] = r.x;
                    s[e + 1] = r.y;
                }
            }
            auto hide = [&](float x) {                        // x in the place of every key that the row does not see
                const bool live = tok >= w.seg_a && tok < w.seg_b;
                const int last = live ? min(w.k_end - 1, ranged ? 0x7fffffff : my_pos) : -1, first = ranged ? w.lo : my_lo;
                if (__all_sync(0xffffffffu, k0 + KP - 1 <= last && (k0 >= first || k0 + KP - 1 < kept))) return;
#pragma unroll
                for (int e = 0; e < KP; ++e) {
                    const int j = k0 + e;
                    if (!(j <= last && (j >= first || j < kept))) s[e] = x;
                }
            };
            hide(-CUDART_INF_F);
            float mx = s[0];
#pragma unroll
            for (int e = 1; e < KP; ++e) mx = max_nan(mx, s[e]);
            // (two exchanges a tile in two places: whoever writes one has seen the other threads leave the one before)
            row_x[hf * kRows + row] = mx;
            __syncwarp();
            if (lane == 0) mbar_arrive(&pair[qt]);
            if (!wait_for(&pair[qt], 0)) { ok = false; break; }
#pragma unroll
            for (int i = 1; i < RT; ++i) mx = max_nan(mx, row_x[(hf ^ i) * kRows + row]);
            const float m_new = max_nan(m_run, mx);
            const float base = m_new == -CUDART_INF_F ? 0.f : m_new, corr = m_run == -CUDART_INF_F ? 0.f : ex2(m_run - base);
            const float2 nb = make_float2(-base, -base);
#pragma unroll
            for (int c = 0; c < LP; ++c) {
                float2 sum = make_float2(0.f, 0.f);
#pragma unroll
                for (int e = 16 * c; e < 16 * c + 16; e += 2) {
                    const float2 a = add2(make_float2(s[e], s[e + 1]), nb);
                    s[e] = ex2(a.x);
                    s[e + 1] = ex2(a.y);
                    sum = add2(sum, make_float2(s[e], s[e + 1]));
                }
                l_run[c] = fmaf(l_run[c], corr, sum.x + sum.y);
            }
            m_run = m_new;
            // weight x its value's magnitude, and the largest of them that this row has in the tile
            if (!geo.shared_kv && !wait_for(&v_ready[at_t], round)) { ok = false; break; }
            scale_by<KP>(s, v_inv + at_t * kKeys + hf * KP);
            auto largest = [&] {
                float v = s[0];
#pragma unroll
                for (int e = 1; e < KP; ++e) v = max_nan(v, s[e]);
                return v;
            };
            float wm = largest();
            if (__any_sync(0xffffffffu, wm != wm)) {          // a value that cannot be split, 0 x NaN where it is not seen
                hide(0.f);
                wm = largest();
                if (wm != wm) l_run[0] = CUDART_NAN_F;
            }
            row_x[(RT + hf) * kRows + row] = wm;
            __syncwarp();
            if (lane == 0) mbar_arrive(&pair[qt]);
            // (meanwhile) the value product of the tile before is done: the weights' columns are free, and its sum can be taken
            if (t > 0) {
                if (!wait_for(pv_done, (t - 1) & 1u)) { ok = false; break; }
                fence_after();
            }
            if (!wait_for(&pair[qt], 1)) { ok = false; break; }
            float wi;
#pragma unroll
            for (int i = 1; i < RT; ++i) wm = fmaxf(wm, row_x[(RT + (hf ^ i)) * kRows + row]);
            const float wscale = scale_of(wm, wi);
            const float2 ws = make_float2(wscale, wscale);
#pragma unroll
            for (int c = 0; c < KP / 16; ++c) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 q = mul2(make_float2(s[c * 16 + 2 * e], s[c * 16 + 2 * e + 1]), ws);
                    split2(q.x, q.y, hi[e], lo[e]);
                }
                tmem_store8(t_p + lanes + hf * (KP / 2) + c * 8, hi);
                tmem_store8(t_p + lanes + 32 + hf * (KP / 2) + c * 8, lo);
            }
            // with two accumulators the next value product may start before the last one has been added
            if (t > 0 && geo.o_bufs == 1) add_values(t - 1, corr_prev, wi_prev);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
            if (t > 0 && geo.o_bufs == 2) add_values(t - 1, corr_prev, wi_prev);
            corr_prev = corr;
            wi_prev = wi;
            if (++at_t == (unsigned)geo.depth) at_t = 0, round ^= 1u;
        }
        if (ok && t > 0) {
            ok = wait_for(pv_done, (t - 1) & 1u);
            fence_after();
            add_values(t - 1, corr_prev, wi_prev);
        }
        // ---- the threads' denominators, the sink's own term, normalise, store ----
        // (with two threads they fill the place of the second exchange too: every thread has left it before the last value product)
#pragma unroll
        for (int c = 0; c < LP; ++c) row_x[(hf * LP + c) * kRows + row] = l_run[c];
        __syncwarp();
        if (lane == 0) mbar_arrive(&pair[qt]);
        ok = ok && wait_for(&pair[qt], 0);
        float l = 0.f;
#pragma unroll
        for (int i = 0; i < RT * LP; ++i) l += row_x[i * kRows + row];
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
            if (c < n_mine) *reinterpret_cast<float4*>(stage + lane * ldst + c) = make_float4(O[c] * f, O[c + 1] * f, O[c + 2] * f, O[c + 3] * f);
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
    } else if (warp < RW + 4) {
        // ================= keys and values: warp lw takes keys 16 lw .. + 15 of a tile, a lane one key of either eight =================
        if constexpr (kFetchRegs < kLaunchRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFetchRegs));
        const int lw = warp - RW, kin = lane & 7, cq = lane >> 3;
        unsigned at = 0;                                      // ring position
        bool ok = true;
        size_t cur[2] = {~(size_t)0, ~(size_t)0}, prev[2];    // row of the two keys in the pages of kv head 0 (~0: none)
        const SlotTiles* const plan = reinterpret_cast<const SlotTiles*>(p.work);
        auto split_tile = [&](int slot, int j0) -> int {      // the tile of the room that holds these keys (-1: none)
            if (!plan) return -1;
            const SlotTiles s = plan[slot];
            const int j = j0 / kKeys;
            return j >= s.first && j < s.end ? s.base + j : j == 0 ? s.zero : -1;
        };
        // a part that is split already; with scales, the tile's come along: warp 1 brings its keys' and warp 2 its values' (whose tile is t)
        auto copied = [&](int tile, int part, unsigned bytes, bool scales, unsigned t) {
            const unsigned slot = at % geo.n_slots;
            if (lane == 0) ok = wait_for(&empty[slot], ((at / geo.n_slots) & 1u) ^ 1u);
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) return;
            const unsigned char* work = reinterpret_cast<const unsigned char*>(p.work);
            if (lw == 0 && lane == 0) {
                mbar_arrive_expect_tx(&full[slot], bytes);
                const size_t off = (size_t)tile * geo.tile_bytes + part_offset(geo, part);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 smem_u32(ring + (size_t)slot * geo.slot_bytes)),
                             "l"(work + geo.tile_off + off), "r"(bytes), "r"(smem_u32(&full[slot]))
                             : "memory");
            }
            if (scales) {
                const float* src = reinterpret_cast<const float*>(work + geo.scale_off) + (size_t)tile * geo.sets * kKeys + 2 * lane;
                const unsigned at_t = t % geo.depth;
                if (lw == 1)
                    for (int i = 0; i < geo.k_sets; ++i)
                        *reinterpret_cast<float2*>(k_inv + (at_t * geo.k_sets + i) * kKeys + 2 * lane) =
                            *reinterpret_cast<const float2*>(src + (geo.k_sets > 1 ? i : g) * kKeys);
                if (lw == 2 && !geo.shared_kv)
                    *reinterpret_cast<float2*>(v_inv + at_t * kKeys + 2 * lane) = *reinterpret_cast<const float2*>(src + (p.kv_heads + g) * kKeys);
                __syncwarp();
                if (lane == 0 && !geo.shared_kv) mbar_arrive(&v_ready[at_t]);
            }
            if (lw != 0 && lane == 0) mbar_arrive(&full[slot]);
            ++at;
        };
        auto row_of = [&](const float* cache, int width, int gg, size_t row) {
            return cache + (row != ~(size_t)0 ? (row + (size_t)gg * p.page_size) * width : 0);
        };
        // channels [c0, c0 + w) of rows of `width` floats, of which [0, row_w) set the scale.  m_row: the rows' largest magnitudes - taken
        // (first) or as taken by the first group; inv: where the scales go (null: they are there); ready: told when they are
        auto stage = [&](const float* cache, int width, int row_w, int c0, int w, int wp, int gg, const size_t (&rows)[2], float (&m_row)[2],
                         bool first, float* inv, uint64_t* ready) {
            // groups of eight keys at a time: 16 float4 of two do not fit 64 or 80 registers (us, wide values, two / one: nine sequences over
            // 1134 keys that the room for split keys does not hold 320 / 241, 4096 rows over latent rows of 256 + 32 440 / 405)
            constexpr int KG = RT == 4 || NVS == 2 ? 1 : 2;
            const unsigned slot = at % geo.n_slots;
#pragma unroll 1
            for (int half = 0; half < 2; half += KG) {
                float4 v[8 * KG];
#pragma unroll
                for (int u = 0; u < KG; ++u) {
                    const size_t at_row = half + u ? rows[1] : rows[0];
                    const bool in = at_row != ~(size_t)0;
                    const float* src = row_of(cache, width, gg, at_row) + c0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int c = 8 * (cq + 4 * i);
                        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                        v[u * 8 + 2 * i] = in && c < w ? *reinterpret_cast<const float4*>(src + c) : z;
                        v[u * 8 + 2 * i + 1] = in && c + 4 < w ? *reinterpret_cast<const float4*>(src + c + 4) : z;
                    }
                }
                float sc[KG], inverse[KG];
#pragma unroll
                for (int u = 0; u < KG; ++u) {
                    float m = half + u ? m_row[1] : m_row[0];
                    if (first) {
                        const size_t at_row = half + u ? rows[1] : rows[0];
                        m = 0.f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) m = max_abs4(m, v[u * 8 + i]);
                        if (w < row_w && at_row != ~(size_t)0)
                            for (int c = w + 4 * cq; c < row_w; c += 16) m = max_abs4(m, *reinterpret_cast<const float4*>(row_of(cache, width, gg, at_row) + c));
                        m = row_max(m);
                        if (half + u) m_row[1] = m;
                        else m_row[0] = m;
                    }
                    if (scale_row(m, sc[u], inverse[u])) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[u * 8 + i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
                auto put_scales = [&] {
                    if (inv && lane < 8) {
#pragma unroll
                        for (int u = 0; u < KG; ++u) inv[lw * 16 + (half + u) * 8 + lane] = inverse[u];
                    }
                };
                if (ready) {                                  // (their place is free by then: see geometry_of)
                    put_scales();
                    __syncwarp();
                    if (half + KG == 2 && lane == 0) mbar_arrive(ready);
                }
                if (half == 0 && !wait_for(&empty[slot], ((at / geo.n_slots) & 1u) ^ 1u)) { ok = false; return; }
                if (!ready) put_scales();
                unsigned char* base = ring + (size_t)slot * geo.slot_bytes;
                const int blocks = wp >> 3;
#pragma unroll
                for (int u = 0; u < KG; ++u)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int c8 = cq + 4 * i;
                        if (c8 < blocks) {
                            const float4 a = v[u * 8 + 2 * i], b = v[u * 8 + 2 * i + 1];
                            uint32_t hi[4], lo[4];
                            split2(a.x * sc[u], a.y * sc[u], hi[0], lo[0]);
                            split2(a.z * sc[u], a.w * sc[u], hi[1], lo[1]);
                            split2(b.x * sc[u], b.y * sc[u], hi[2], lo[2]);
                            split2(b.z * sc[u], b.w * sc[u], hi[3], lo[3]);
                            unsigned char* dst = base + ((lw * 2 + half + u) * blocks + c8) * 128 + kin * 16;
                            *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                            *reinterpret_cast<uint4*>(dst + kKeys * wp * 2) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                        }
                    }
            }
            fence_smem_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[slot]);
            ++at;
        };
        // the value groups of tile t; a shared row's scale is its key's, m_key
        auto values = [&](unsigned t, const size_t (&rows)[2], int tile, const float (&m_key)[2]) {
            float m_row[2] = {m_key[0], m_key[1]};
            for (int vs = 0; vs < NVS && ok; ++vs) {
                const int wl = vs == geo.n_vst - 1 ? geo.v_last_layout : geo.v0_layout;
                const bool owns = vs == 0 && !geo.shared_kv;
                if (tile >= 0)
                    copied(tile, geo.shared_kv ? vs : geo.k_parts + g * geo.n_vst + vs, kKeys * wl * 4, false, t);
                else
                    stage(p.vcache, p.vrow, p.vdim, vs * kGroupW, min(kGroupW, (geo.shared_kv ? p.kdim : p.vdim) - vs * kGroupW), wl, g, rows, m_row, owns,
                          owns ? v_inv + (t % geo.depth) * kKeys : nullptr, owns ? &v_ready[t % geo.depth] : nullptr);
            }
        };
        int tile = -1, prev_tile = -1;
        float m_key[2] = {0.f, 0.f}, m_prev[2];
        unsigned t = 0;
        Walk w(s_slot, s_pos, s_breaks, n_tok);
        for (; ok && w.next(p); ++t) {
            const int slot = s_slot[w.seg_a];
            prev_tile = tile;
            tile = split_tile(slot, w.j0);
#pragma unroll
            for (int kg = 0; kg < 2; ++kg) {
                const int j = w.j0 + lw * 16 + kg * 8 + kin;
                prev[kg] = cur[kg];
                cur[kg] = ~(size_t)0;
                if (tile < 0 && j < w.k_end) {
                    const int page = p.table ? p.table[(size_t)slot * p.max_pages + j / p.page_size] : slot;
                    cur[kg] = (size_t)page * p.kv_heads * p.page_size + (p.table ? j % p.page_size : j);
                }
            }
            m_prev[0] = m_key[0];
            m_prev[1] = m_key[1];
            for (int st = 0; st < geo.n_kst && ok; ++st) {
                const int wp = st == geo.n_kst - 1 ? geo.wk_last : geo.wk0;
                const bool first = st == 0 || geo.k_sets > 1;
                if (tile >= 0)
                    copied(tile, p.talk ? st : g * geo.n_kst + st, kKeys * wp * 4, st == 0, t);
                else
                    stage(p.kcache, p.kdim, p.kdim, p.talk ? 0 : st * kGroupW, p.talk ? p.kdim : min(kGroupW, p.kdim - st * kGroupW), wp, p.talk ? st : g,
                          cur, m_key, first, first ? k_inv + ((t % geo.depth) * geo.k_sets + (geo.k_sets > 1 ? st : 0)) * kKeys : nullptr, nullptr);
            }
            if (t > 0 && ok) values(t - 1, prev, prev_tile, m_prev);
        }
        if (t > 0 && ok) values(t - 1, cur, tile, m_key);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == RW + 4) {
            // ================= the MMA issuer: the whole warp walks, one elected lane issues =================
            const uint32_t idesc_s = (1u << 4) | ((uint32_t)(kKeys >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
            const uint32_t q_addr = smem_u32(qs), ring_addr = smem_u32(ring);
            unsigned at = 0;
            bool ok = true;
            auto values = [&](unsigned t) {                   // value product of tile t
                if (!wait_warp(p_ready, t & 1u)) { ok = false; return; }
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
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) mma_ts(d, t_p + 32u + 8u * k, vh + k * step, idesc, k != 0);
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) mma_ts(d, t_p + 8u * k, vl + k * step, idesc, 1u);
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) mma_ts(d, t_p + 8u * k, vh + k * step, idesc, 1u);
                        commit_to(&empty[slot]);
                        if (vs == NVS - 1) commit_to(pv_done);
                    }
                    __syncwarp();
                    ++at;
                }
            };
            unsigned t = 0;
            Walk w(s_slot, s_pos, s_breaks, n_tok);
            ok = wait_warp(q_ready, 0);
            for (; ok && w.next(p); ++t) {
                if (t > 0 && !wait_warp(s_empty, (t - 1) & 1u)) { ok = false; break; }
                for (int st = 0; st < geo.n_kst; ++st) {
                    const unsigned slot = at % geo.n_slots;
                    if (!wait_warp(&full[slot], (at / geo.n_slots) & 1u)) { ok = false; break; }
                    fence_after();
                    const uint32_t wp = st == geo.n_kst - 1 ? geo.wk_last : geo.wk0;
                    const uint32_t ka = ring_addr + slot * geo.slot_bytes, qa = q_addr + st * geo.wk0 * kRows * 4u;
                    const uint64_t kh = block_desc(ka, 128u, wp * 16u), kl = block_desc(ka + kKeys * wp * 2u, 128u, wp * 16u);
                    const uint64_t qh = block_desc(qa, 128u, wp * 16u), ql = block_desc(qa + kRows * wp * 2u, 128u, wp * 16u);
                    const uint32_t d = t_s + 64u * st;
                    if (elect_one_sync()) {
                        const uint32_t n = wp >> 4;           // 16 channels per instruction: 2 blocks, 16 descriptor units
                        for (uint32_t k = 0; k < n; ++k) mma_ss(d, ql + 16u * k, kh + 16u * k, idesc_s, k != 0);
                        for (uint32_t k = 0; k < n; ++k) mma_ss(d, qh + 16u * k, kl + 16u * k, idesc_s, 1u);
                        for (uint32_t k = 0; k < n; ++k) mma_ss(d, qh + 16u * k, kh + 16u * k, idesc_s, 1u);
                        commit_to(&empty[slot]);
                        if (st == geo.n_kst - 1) commit_to(s_full);
                    }
                    __syncwarp();
                    ++at;
                }
                if (t > 0 && ok) values(t - 1);
            }
            if (t > 0 && ok) values(t - 1);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == RW + 4) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// with rt threads per row
bool geometry_of(const SplitAttention& a, Geometry& g, size_t& smem, int rt) {
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
    if (a.work && a.table && a.rows_per_slot <= 0 && a.n_seq > 0 && aligned(a.work)) {
        g.scale_off = (unsigned)a.n_slots * sizeof(SlotTiles);
        const size_t per = g.tile_bytes + 4u * kKeys * g.sets, fixed = g.scale_off + 128;
        if (a.work_bytes > fixed) g.cap_tiles = (int)std::min<size_t>((a.work_bytes - fixed) / per, 65535);
        g.tile_off = (unsigned)((g.scale_off + 4u * kKeys * g.sets * (unsigned)g.cap_tiles + 127u) & ~127u);
    }
    g.o_bufs = g.n_vst == 1 && 64 * g.n_kst + 64 + 256 <= 512 ? 2 : 1;
    g.slot_bytes = kKeys * std::max(g.wk0, std::max(g.wv0, g.v0_layout)) * 4;
    g.q_bytes = ((g.n_kst - 1) * g.wk0 + g.wk_last) * kRows * 4;
    // A tile's scales are written when its first key group has its slot: the stage n_slots places before is done.  They lie depth tiles
    // apart so that this stage is no earlier than the first value group of the tile whose scales were there (a value group is multiplied
    // after the rows have used all scales of its tile).  In order, a tile is n_kst key groups and, behind those of the next, n_vst value groups.
    const int per_tile = g.n_kst + g.n_vst;
    auto depth_of = [&](int slots) { return 1 + (slots + g.n_kst + per_tile - 1) / per_tile; };
    auto control_of = [&](int slots) {
        return (2 * kMaxSlots + 5 + 4 + kMaxDepth + 1) / 2 * 16 + (depth_of(slots) * kKeys * (g.k_sets + (g.shared_kv ? 0 : 1)) + 2 * rt * kRows + 8) * 4 + 2 * (kRows >> g.pk_shift) * 4;
    };
    for (g.n_slots = kMaxSlots; g.n_slots >= 2; --g.n_slots)
        if (g.n_slots * g.slot_bytes + g.q_bytes + control_of(g.n_slots) <= kSmemMost) break;
    if (g.n_slots < 2) return false;
    g.depth = depth_of(g.n_slots);
    const int control = control_of(g.n_slots);
    // the output is staged in the ring and the queries: 4 rt warps of 32 rows, 4 floats between the rows
    const int staged = kRows * rt * ((g.n_vst == 1 ? (g.wv0 + 8 * rt - 1) / (8 * rt) * 8 : 256 / rt) + 4) * 4;
    g.q_bytes = std::max(g.q_bytes, staged - g.n_slots * g.slot_bytes);
    smem = (size_t)g.n_slots * g.slot_bytes + g.q_bytes + control;
    return smem <= (size_t)kSmemMost;
}

template <int NVS, int RT>
cudaError_t launch_inst(const SplitAttention& a, const Geometry& g, size_t smem, cudaStream_t st) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = ask_smem<split_attention_kernel<NVS, RT>>(device, kSmemMost);
    if (e != cudaSuccess) return e;
    const int tt = kRows >> g.pk_shift, tiles = a.n_seq > 1 ? a.M / tt + a.n_seq : (a.M + tt - 1) / tt;
    if (a.work) {
        split_keys_kernel<<<dim3(std::min(g.cap_tiles, std::max(1, kSplitGrid / g.parts)), g.parts), 256, 0, st>>>(a, g);
        ++extra_launches();
    }
    split_attention_kernel<NVS, RT><<<(a.heads >> g.pk_shift) * tiles, kSplitThreads<RT>, smem, st>>>(a, g);
    return cudaGetLastError();
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
    return geometry_of(a, g, smem, 2);
}

size_t split_attention_work_bytes(const SplitAttention& a, int keys) {
    Geometry g;
    size_t smem;
    if (!geometry_of(a, g, smem, 2)) return 0;
    return (size_t)a.n_slots * sizeof(SlotTiles) + 256 + (size_t)((keys + kKeys - 1) / kKeys) * (g.tile_bytes + 4u * kKeys * g.sets);
}

cudaError_t launch_split_attention(const SplitAttention& a, cudaStream_t st) {
    Geometry g;
    size_t smem;
    if (a.M <= 0 || !geometry_of(a, g, smem, 2)) return cudaErrorNotSupported;
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    g.ran_out = split_attention_ran_out(device, st);          // (mapped and unified: one address on both sides)
    if (take_ran_out(device, st)) return cudaErrorLaunchTimeout;
    SplitAttention with = a;
    // Wide values are split in advance in every step: the fetching warps have few registers for them (9 and 24 decoding sequences over 1000
    // cached keys, latent rows of 256 + 32, 4 layers: 1714 and 1833 us split by the row tiles, 1139 and 1250 in advance; over 100 keys 867
    // and 863)
    if (g.cap_tiles <= 0 || (g.n_vst == 1 && (long long)a.M * (a.heads / a.kv_heads) < kSplitOnceRows)) with.work = nullptr;
    if (g.n_vst == 2) return launch_inst<2, 2>(with, g, smem, st);
    // Four threads per row where the keys are split in advance (us, two / four: windowed 4096 rows, 16 heads of 128 over 4 266 / 245, mixed
    // scores, three prompts of 2048 rows 147 / 117, 4096 rows in chunks of 2048 303 / 263, float32 model 80 / 63).  Their fetching warps have half
    // the registers (861 rows of Dia, whose keys every row tile splits for itself, 81 / 107); wide values do not fit theirs (451 / 459).
    Geometry g4;
    size_t smem4;
    if (with.work && geometry_of(a, g4, smem4, 4)) {
        g4.ran_out = g.ran_out;
        return launch_inst<1, 4>(with, g4, smem4, st);
    }
    return launch_inst<1, 2>(with, g, smem, st);
}

}  // namespace dia
