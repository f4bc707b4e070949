// gemm_tcgen05.cu - the dense contractions OFF the decode step (encoder, cross-attention K/V precompute, prompt
// prefill) on the 5th-generation tensor cores.
//
//   Y[M][N] (fp32) = X[M][K] (fp32) . W[K][N] (bf16)           DenseGeneral.forward, dia/layers.py:55-66, M = B*T rows
//
// The reference runs these in fp32 and the K/V a prefill writes are re-read by every later greedy step, so the
// activations may not be rounded to bf16.  X is therefore split into three bf16 terms
// (x = hi + lo + lo2, exact to 24 bits) and each k-step issues three tcgen05.mma into the SAME fp32 accumulator in
// tensor memory: the product has fp32-operand accuracy at bf16 tensor-core speed.
//
// Structure (persistent: one CTA per SM walks the 128 x 256 output tiles, warp-specialised):
//   warp 0    one lane: TMA producer - cp.async.bulk.tensor loads of the weight tile [256 x 64] of a k-block into a
//             3-slot ring and of the three A-term tiles [128 x 64] into a 7-slot ring (both K-major, 128-byte swizzle);
//             the rings run on across tile boundaries, so the next tile's operands are in flight during a tile's tail
//   warp 1    allocates all 512 TMEM columns = two 128 x 256 fp32 accumulators; the warp walks the k-blocks and one
//             elected lane issues tcgen05.mma (M = 128, N = 256, K = 16, kind::f16, bf16 inputs, fp32 accumulate),
//             releases ring slots with tcgen05.commit and hands a finished accumulator to the epilogue
//   warps 2-5 epilogue of tile i (tcgen05.ld, 32 lanes x 32 columns per instruction -> registers -> residual add ->
//             fp32 stores) while the MMAs of tile i + 1 fill the other accumulator
// W is kept as a K-major bf16 copy [N][K] made once per weight (transpose_to_bf16_kernel), so that A and B use the
// same canonical UMMA layout.  Every wait of the kernels of one SM is bounded: a stuck pipeline traps instead of hanging the GPU.
// More than 128 rows run on pairs of SMs (dia_gemm_pair_kernel, whose waits end without a trap); this kernel keeps the shorter ones and small expert groups.
//
// The same kernel serves callers whose activations are bf16 already (terms = 1: one MMA per k-step, the operand is read
// as it is), row tiles that belong to different weight matrices (expert groups: the group of a tile's first row picks
// the matrix, a device-side row count skips the unused tiles), a contraction length that is not a multiple of the
// k-block (the TMA fills the tail of both operands with zeros), a DynamicTanh in front of the residual add, and a gelu whose
// result leaves as the bf16 operand of the product that follows.
#include <algorithm>
#include <atomic>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "engine_internal.h"
#include "gemm_tcgen05.h"
#include "attention_split.h"

namespace dia {

namespace {

// BN = 256: the three A-term tiles (48 KB per k-block) are shared by twice as many output columns - the kernel is bound
// by the operand traffic from L2 (BN = 128 moved 4.3 GB for M = 2048, N = 16384, K = 2048: 13 TB/s at 326 us), and a
// 256-wide MMA (128-cycle floor) also hides the ~100 cycles one tcgen05.mma takes to issue.
constexpr int BM = 128, BN = 256, BK = 64;
constexpr int kTerms = 3;                                   // terms of an fp32 activation (the most a call may stack)
constexpr int kASlots = 7, kBSlots = 3;                     // A-term ring / weight ring: > 2 k-blocks of operands in flight
constexpr int kTileBytes = BM * BK * 2;                     // 16 KB: one [128 x 64] bf16 tile
constexpr int kBTileBytes = BN * BK * 2;                    // 32 KB: the weight tile
constexpr int kGemmThreads = 192;                           // 6 warps
constexpr int kGemmBars = 2 * kASlots + 2 * kBSlots + 4;
constexpr int kGemmSmem = kASlots * kTileBytes + kBSlots * kBTileBytes + 1024 /* alignment slack */ + 256 /* barriers */;
static_assert(kGemmBars * 8 + 8 <= 256, "barrier region");

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    unsigned polls = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (++polls > 20000000u) __trap();                  // seconds: the pipeline is stuck
    }
}
// K-major, 128-byte swizzle: rows of 128 B, 8-row groups 1024 B apart (stride byte offset), version 1 (sm_100)
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    const uint32_t lo = ((smem_addr & 0x3FFFFu) >> 4) | (1u << 16);
    const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace

// gelu in its tanh form, as z sigmoid(2 u) with u = sqrt(2 / pi) (z + 0.044715 z^3): 0.5 (1 + tanh u) = sigmoid(2 u).  Fast
// exponential and division: the result is rounded to bf16.
__device__ __forceinline__ float gelu_to_bf16_range(float z) {
    const float u2 = 1.5957691216057308f * fmaf(0.044715f * z * z, z, z);
    return __fdividef(z, 1.0f + __expf(fminf(-u2, 80.f)));
}

// v = t0 + t1 + t2 in bf16.  An infinity stays one, alone; the largest numbers, which would round up to an infinity, are rounded towards
// zero in their first term.  (Both show in the remainder: one test on the way of all others.  The terms may go to memory and are not
// read back.)
__device__ __forceinline__ void split3(float v, __nv_bfloat16& t0, __nv_bfloat16& t1, __nv_bfloat16& t2) {
    __nv_bfloat16 a = __float2bfloat16_rn(v);
    float r1 = v - __bfloat162float(a);
    if (!(fabsf(r1) <= 3.402823466e38f)) {
        const bool finite = fabsf(v) <= 3.402823466e38f;
        if (finite) a = __float2bfloat16_rz(v);
        r1 = finite ? v - __bfloat162float(a) : 0.f;
    }
    const __nv_bfloat16 b = __float2bfloat16_rn(r1);
    t0 = a;
    t1 = b;
    t2 = __float2bfloat16_rn(r1 - __bfloat162float(b));
}
// The same with every first term rounded towards zero (8 bits, the nearest 8 of the other 16, the at most 8 that are left): no test, for the
// kernels whose accumulators live for 64 products (the test cost a product of 16 rows, whose every CTA splits the rows, 21.0 -> 22.5
// us; sums of all K products in tensor memory, which cuts off, are closer with terms of either sign: 861 rows through Dia's decoder
// 2.8e-5 against 3.0e-5)
__device__ __forceinline__ void split3_down(float v, __nv_bfloat16& t0, __nv_bfloat16& t1, __nv_bfloat16& t2) {
    t0 = __float2bfloat16_rz(v);
    const float f0 = __bfloat162float(t0), r1 = fabsf(f0) <= 3.402823466e38f ? v - f0 : 0.f;
    t1 = __float2bfloat16_rn(r1);
    t2 = __float2bfloat16_rn(r1 - __bfloat162float(t1));
}

// W [K][N] (fp32 or bf16, N contiguous) -> Wt [N][K] bf16 (K contiguous)
__global__ void transpose_to_bf16_kernel(const void* __restrict__ w, int src_bf16, __nv_bfloat16* __restrict__ wt, int K, int N) {
    __shared__ float tile[32][33];
    const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int k = k0 + r, n = n0 + threadIdx.x;
        float v = 0.f;
        if (k < K && n < N)
            v = src_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[(size_t)k * N + n])
                         : reinterpret_cast<const float*>(w)[(size_t)k * N + n];
        tile[r][threadIdx.x] = v;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int n = n0 + r, k = k0 + threadIdx.x;
        if (k < K && n < N) wt[(size_t)n * K + k] = __float2bfloat16_rn(tile[threadIdx.x][r]);
    }
}

// Largest magnitude of every column of W [K][N] into mag (zeros before), as the bits of a float
__global__ void __launch_bounds__(256) column_magnitudes_kernel(const void* __restrict__ w, int src_bf16, uint32_t* __restrict__ mag, int K, int N) {
    const int n = blockIdx.x * 256 + threadIdx.x, k1 = min(K, ((int)blockIdx.y + 1) * 64);
    if (n >= N) return;
    uint32_t m = 0;
#pragma unroll 8
    for (int k = blockIdx.y * 64; k < k1; ++k) {
        const size_t at = (size_t)k * N + n;
        const uint32_t b = src_bf16 ? (uint32_t)reinterpret_cast<const uint16_t*>(w)[at] << 16
                                    : __float_as_uint(__bfloat162float(__float2bfloat16_rn(reinterpret_cast<const float*>(w)[at])));
        m = max(m, b & 0x7fffffffu);
    }
    atomicMax(mag + n, m);
}

// W [K][N] (values of bf16) -> Wt [N][K] fp16, every column times a power of two that brings its largest magnitude to [2^14, 2^15).  fp16
// then holds the 8 bits of every value down to 2^-31 of that; *inexact is set where it does not, and for columns of infinities, NaNs or
// magnitudes whose power of two is out of range.
__global__ void transpose_to_half_kernel(const void* __restrict__ w, int src_bf16, const float* __restrict__ mag, __half* __restrict__ wt, int* __restrict__ inexact,
                                         int K, int N) {
    __shared__ float tile[32][33];
    const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int k = k0 + r, n = n0 + threadIdx.x;
        float v = 0.f;
        if (k < K && n < N)
            v = src_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[(size_t)k * N + n])
                         : __bfloat162float(__float2bfloat16_rn(reinterpret_cast<const float*>(w)[(size_t)k * N + n]));
        tile[r][threadIdx.x] = v;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int n = n0 + r, k = k0 + threadIdx.x;
        if (k >= K || n >= N) continue;
        const int e = (int)(__float_as_uint(mag[n]) >> 23) - 127;
        const bool fits = e >= -112 && e < 128;               // (a column of zeros: e = -127, and zeros)
        const float v = tile[threadIdx.x][r], scaled = fits ? v * __uint_as_float((uint32_t)(141 - e) << 23) : 0.f;
        const __half h = __float2half_rn(scaled);
        if (fits ? __half2float(h) != scaled : mag[n] != 0.f) *inexact = 1;
        wt[(size_t)n * K + k] = h;
    }
}

// Rows of a product's operand.  TERMS 3: three bf16 terms, stacked as [3][M][K]; 0: the rows themselves, in fp32; 2: two fp16 terms, hi =
// fp16(v), lo = fp16(v - hi), each row times a power of two that brings its largest magnitude to [2^14, 2^15): a value keeps 22 bits and more (a
// quarter of all fp32 numbers change by their last bit, the others not) down to 2^-17 of its row's largest, and is off by at most 2^-39 of
// that below.  [2][M][K], and the rows' inverse scales [M] in row_inv.  A row with an infinity or a NaN gives nothing but infinities and
// NaNs in its products: the other values are left out.  norm_w: RMSNorm of the row in front (dia/layers.py:541,560,579,714).
// GATED: the row is silu(x[0 .. K)) x[K .. 2K) (dia/layers.py:95-101).  One CTA per row, which stays in registers up to 8192 channels
// (1722 rows of 8192 gated channels: 51 us for the gate and 22 for the split, 42 together).
template <int TERMS, bool GATED>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, const float* __restrict__ norm_w, float eps, void* __restrict__ out,
                                                         float* __restrict__ row_inv, int M, int K, int aligned) {
    constexpr int kHeld = 8;
    __shared__ float part[8], most[8];
    const int tid = threadIdx.x, row = blockIdx.x, n4 = K >> 2;
    const float* xr = x + (size_t)row * K * (GATED ? 2 : 1);
    auto four = [&](const float* p, int i) {
        return aligned ? reinterpret_cast<const float4*>(p)[i] : make_float4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
    };
    auto raw = [&](int i) {
        float4 v = four(xr, i);
        if (GATED) {
            const float4 u = four(xr, n4 + i);
            v.x = v.x / (1.0f + expf(-v.x)) * u.x; v.y = v.y / (1.0f + expf(-v.y)) * u.y;
            v.z = v.z / (1.0f + expf(-v.z)) * u.z; v.w = v.w / (1.0f + expf(-v.w)) * u.w;
        }
        return v;
    };
    float4 held[kHeld];
#pragma unroll
    for (int j = 0; j < kHeld; ++j)
        if (j * 256 + tid < n4) held[j] = raw(j * 256 + tid);
    float inv = 1.f;
    if (norm_w) {
        float ss = 0.f;
        auto add = [&](const float4& v) { ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss); };
#pragma unroll
        for (int j = 0; j < kHeld; ++j)
            if (j * 256 + tid < n4) add(held[j]);
        for (int i = kHeld * 256 + tid; i < n4; i += 256) add(raw(i));
        ss = warp_sum(ss);
        if ((tid & 31) == 0) part[tid >> 5] = ss;
        __syncthreads();
        float tot = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) tot += part[i];
        inv = 1.0f / sqrtf(tot / (float)K + eps);
    }
    auto value = [&](const float4& v, int i) {
        if (!norm_w) return v;
        const float4 w = four(norm_w, i);
        return make_float4((v.x * inv) * w.x, (v.y * inv) * w.y, (v.z * inv) * w.z, (v.w * inv) * w.w);
    };
    const size_t plane = (size_t)M * K, at = (size_t)row * K;
    if (TERMS != 2) {
        auto put = [&](const float4& v, int i) {
            if (TERMS == 0) {
                reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + at)[i] = v;
                return;
            }
            __nv_bfloat16 t[3][4];
            split3(v.x, t[0][0], t[1][0], t[2][0]); split3(v.y, t[0][1], t[1][1], t[2][1]);
            split3(v.z, t[0][2], t[1][2], t[2][2]); split3(v.w, t[0][3], t[1][3], t[2][3]);
#pragma unroll
            for (int q = 0; q < 3; ++q)
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + q * plane + at + 4 * i) = *reinterpret_cast<const uint2*>(t[q]);
        };
#pragma unroll
        for (int j = 0; j < kHeld; ++j)
            if (j * 256 + tid < n4) put(value(held[j], j * 256 + tid), j * 256 + tid);
        for (int i = kHeld * 256 + tid; i < n4; i += 256) put(value(raw(i), i), i);
        return;
    }
    uint32_t m = 0;                                           // magnitudes as bits: an infinity or a NaN is the largest
    auto see = [&](const float4& v) {
        m = max(max(max(m, __float_as_uint(v.x) & 0x7fffffffu), __float_as_uint(v.y) & 0x7fffffffu),
                max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
    };
#pragma unroll
    for (int j = 0; j < kHeld; ++j)
        if (j * 256 + tid < n4) {
            held[j] = value(held[j], j * 256 + tid);
            see(held[j]);
        }
    for (int i = kHeld * 256 + tid; i < n4; i += 256) see(value(raw(i), i));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((tid & 31) == 0) most[tid >> 5] = __uint_as_float(m);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(most[i]));
    const bool bad = m >= 0x7f800000u;
    const int e = max((int)(m >> 23), 1) - 127, s = 14 - e, s1 = min(s, 100);       // the scale 2^s as 2^s1 2^(s - s1): s may be 140
    const float f1 = bad ? 1.f : __uint_as_float((uint32_t)(s1 + 127) << 23), f2 = bad ? 1.f : __uint_as_float((uint32_t)(s - s1 + 127) << 23);
    if (tid == 0) row_inv[row] = bad ? 1.f : ldexpf(1.f, -s);
    __half* const hi_row = reinterpret_cast<__half*>(out) + at;
    auto put = [&](const float4& v, int i) {
        const float a[4] = {v.x, v.y, v.z, v.w};
        __half hi[4], lo[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float t = bad ? ((__float_as_uint(a[k]) & 0x7f800000u) == 0x7f800000u ? a[k] : 0.f) : a[k] * f1 * f2;
            hi[k] = __float2half_rn(t);
            lo[k] = __float2half_rn(bad ? 0.f : t - __half2float(hi[k]));
        }
        *reinterpret_cast<uint2*>(hi_row + 4 * i) = *reinterpret_cast<const uint2*>(hi);
        *reinterpret_cast<uint2*>(hi_row + plane + 4 * i) = *reinterpret_cast<const uint2*>(lo);
    };
#pragma unroll
    for (int j = 0; j < kHeld; ++j)
        if (j * 256 + tid < n4) put(held[j], j * 256 + tid);
    for (int i = kHeld * 256 + tid; i < n4; i += 256) put(value(raw(i), i), i);
}

__global__ void __launch_bounds__(kGemmThreads, 1)
dia_gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                        float* y, const float* residual, int M, int N, int K, int terms, const float* dyt_w,
                        const float* dyt_b, float dyt_alpha, __nv_bfloat16* y_bf16, const int* row_group, int group_rows,
                        const int* n_rows) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* a_ring = smem;
    unsigned char* b_ring = smem + kASlots * kTileBytes;
    uint64_t* a_full = reinterpret_cast<uint64_t*>(b_ring + kBSlots * kBTileBytes);
    uint64_t* a_empty = a_full + kASlots;
    uint64_t* b_full = a_empty + kASlots;
    uint64_t* b_empty = b_full + kBSlots;
    uint64_t* t_full = b_empty + kBSlots;                   // accumulator complete (MMA warp -> epilogue), one per accumulator
    uint64_t* t_empty = t_full + 2;                         // accumulator drained (epilogue warps -> MMA warp)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_empty + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_kb = (K + BK - 1) / BK;                    // a partial last k-block reads zeros beyond K in both operands
    const int m_lim = n_rows ? min(M, *n_rows) : M;        // row tiles at or beyond it hold no rows: every role skips them
    // tile t = (column block t / tiles_m, row block t % tiles_m): the CTAs of a wave share a few weight blocks and all of A
    const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN, n_tiles = tiles_m * tiles_n;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kASlots; ++i) { mbar_init(&a_full[i], 1); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < kBSlots; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], 4); }
        fence_mbar_init();
    }
    if (warp == 1) {                                        // one warp allocates (and later frees) the accumulator columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ===== TMA producer =====
            unsigned ia = 0, ib = 0;                        // ring positions, running across the tiles
            for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
                const int n0 = (t / tiles_m) * BN, m0 = (t % tiles_m) * BM;
                if (m0 >= m_lim) continue;
                const int b_row0 = n0 + (row_group ? row_group[m0] * group_rows : 0);   // the tile's weight matrix
                for (int kb = 0; kb < n_kb; ++kb) {
                    {
                        const unsigned s = ib % kBSlots;
                        mbar_wait_bounded(&b_empty[s], ((ib / kBSlots) & 1u) ^ 1u);
                        mbar_arrive_expect_tx(&b_full[s], kBTileBytes);
                        tma_load_2d(smem_u32(b_ring + s * kBTileBytes), &map_b, smem_u32(&b_full[s]), kb * BK, b_row0);
                        ++ib;
                    }
                    for (int tm = 0; tm < terms; ++tm) {   // rows of term tm start at tm * M in the stacked matrix
                        const unsigned s = ia % kASlots;
                        mbar_wait_bounded(&a_empty[s], ((ia / kASlots) & 1u) ^ 1u);
                        mbar_arrive_expect_tx(&a_full[s], kTileBytes);
                        tma_load_2d(smem_u32(a_ring + s * kTileBytes), &map_a, smem_u32(&a_full[s]), kb * BK, tm * M + m0);
                        ++ia;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer: the whole warp walks the k-blocks (uniform operands), one elected lane issues =====
        // instruction descriptor: fp32 accumulate, bf16 x bf16, both operands K-major, N = 256, M = 128
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        unsigned ia = 0, ib = 0, it = 0;
        for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
            if ((t % tiles_m) * BM >= m_lim) continue;
            const unsigned acc = it & 1u;
            mbar_wait_bounded(&t_empty[acc], ((it >> 1) & 1u) ^ 1u);      // the epilogue has drained this accumulator
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d = tmem_base + acc * BN;
            for (int kb = 0; kb < n_kb; ++kb) {
                const unsigned sb = ib % kBSlots;
                mbar_wait_bounded(&b_full[sb], (ib / kBSlots) & 1u);
                const uint64_t bdesc = umma_desc(smem_u32(b_ring + sb * kBTileBytes));
                for (int tm = 0; tm < terms; ++tm) {
                    const unsigned sa = ia % kASlots;
                    mbar_wait_bounded(&a_full[sa], (ia / kASlots) & 1u);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t adesc = umma_desc(smem_u32(a_ring + sa * kTileBytes));
                    if (elect_one_sync()) {
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j)       // advance 16 elements = 32 bytes = 2 descriptor units along K
                            umma_bf16(d, adesc + 2 * j, bdesc + 2 * j, idesc, (kb | tm | j) != 0 ? 1u : 0u);
                        umma_commit(&a_empty[sa]);              // the slot is free once these MMAs have read it
                        if (tm == terms - 1) umma_commit(&b_empty[sb]);
                    }
                    __syncwarp();
                    ++ia;
                }
                ++ib;
            }
            if (elect_one_sync()) umma_commit(&t_full[acc]);    // the accumulator is complete
            __syncwarp();
            ++it;
        }
    } else {
        // ===== epilogue: a warp may touch the 32 TMEM lanes of its quarter (warp id mod 4) =====
        const int q = warp & 3;
        unsigned it = 0;
        for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
            const int n0 = (t / tiles_m) * BN, m0 = (t % tiles_m) * BM;
            if (m0 >= m_lim) continue;
            const unsigned acc = it & 1u;
            mbar_wait_bounded(&t_full[acc], (it >> 1) & 1u);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = m0 + q * 32 + lane;
#pragma unroll 1
            for (int cb = 0; cb < BN / 32; ++cb) {
                uint32_t v[32];
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN + cb * 32;
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                      "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                      "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(taddr)
                    : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row < M) {
                    // residual add of the layer (dia/layers.py:555,574,582) fused: y may alias residual (each element is
                    // read and written by the same thread).  Column tail: N need not be a multiple of the tile (logits head).
                    const int c0 = n0 + cb * 32;
                    float* dst = y + (size_t)row * N + c0;
                    const float* res = residual ? residual + (size_t)row * N + c0 : nullptr;
                    if (y_bf16) {                               // the activation of an up product, as the next product's operand
                        __nv_bfloat16* dstb = y_bf16 + (size_t)row * N + c0;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            if (c0 + 4 * i + 4 <= N) {          // (N a multiple of 4: 8-byte stores)
                                uint2 p;
                                __nv_bfloat162 lo = __floats2bfloat162_rn(gelu_to_bf16_range(__uint_as_float(v[4 * i])),
                                                                          gelu_to_bf16_range(__uint_as_float(v[4 * i + 1])));
                                __nv_bfloat162 hi = __floats2bfloat162_rn(gelu_to_bf16_range(__uint_as_float(v[4 * i + 2])),
                                                                          gelu_to_bf16_range(__uint_as_float(v[4 * i + 3])));
                                p.x = *reinterpret_cast<uint32_t*>(&lo);
                                p.y = *reinterpret_cast<uint32_t*>(&hi);
                                *reinterpret_cast<uint2*>(dstb + 4 * i) = p;
                            }
                        }
                        continue;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (c0 + 4 * i + 4 <= N) {
                            float4 a = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                                   __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
                            if (dyt_w) {                        // DynamicTanh of the product: tanh(alpha a) w + b per column
                                const float4 w4 = *reinterpret_cast<const float4*>(dyt_w + c0 + 4 * i);
                                const float4 b4 = *reinterpret_cast<const float4*>(dyt_b + c0 + 4 * i);
                                a.x = fmaf(tanhf(dyt_alpha * a.x), w4.x, b4.x); a.y = fmaf(tanhf(dyt_alpha * a.y), w4.y, b4.y);
                                a.z = fmaf(tanhf(dyt_alpha * a.z), w4.z, b4.z); a.w = fmaf(tanhf(dyt_alpha * a.w), w4.w, b4.w);
                            }
                            if (res) {
                                const float4 r4 = *reinterpret_cast<const float4*>(res + 4 * i);
                                a.x += r4.x; a.y += r4.y; a.z += r4.z; a.w += r4.w;
                            }
                            *reinterpret_cast<float4*>(dst + 4 * i) = a;
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&t_empty[acc]);
            ++it;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * BN));
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// The same product on pairs of SMs: a cluster of two CTAs owns a 256 x BN tile, and one tcgen05.mma of the pair (cta_group::2) multiplies the
// 256 rows of both by the BN columns of both.  Each CTA holds its own 128 rows and half of the columns, so the operands of a k-block that an
// SM takes from L2 shrink from (terms x 16 + 32) to (terms x 16 + 16) KB - which is what bounds the kernel above.
//   warp 0    one lane per CTA: TMA loads of the CTA's halves into a ring of stages; every byte of both CTAs counts on the leader's barrier
//   warp 1    leader only: one elected lane issues the pair's MMAs, commits to the barriers of both CTAs
//   warps 2-5 epilogue of the CTA's 128 rows while the next tile is multiplied into the other accumulator; 32 x 32 blocks turn through
//             shared memory so that whole lines are stored (row by row, 4096 x 2048 x 2048 was bound by those stores)
// us, one SM per tile / pairs: one term 4096 x 8192 x 2048 135 / 94 (1.46 PFLOP/s), 4096 x 2048 x 6144 106 / 80, 1722 x 16384 x 2048 126 / 90;
// three terms 256 / 209 (1.66 PFLOP/s), 4096 x 6144 x 2048 227 / 187.  Bound: the MMAs (four of one term take 512 cycles to run and 540 to
// issue; the products of a long pass are at the power limit).  A wait that runs out ends every role: the tiles that have no result become NaN, and
// the kernel sets the device's word, which the next launch and the calls that wait for the device report.
//
// SUMS: fp32 rows as two fp16 terms (split_rows_kernel) and weights as fp16 (transpose_to_half_kernel), every row and every column with a power
// of two of its own; an accumulator lives for kPairChunk k-blocks and eight epilogue warps add it to the tile's sums in their registers (two
// threads per row, up to 128 columns each) while the next ones are multiplied into the other.  Against three terms and sums of all products
// in tensor memory: 1722 rows, K = 2048, 16384 columns 209 -> 162 us, 2048 columns 37 -> 28, K = 8192 118 -> 85; relative error 7.0e-6 -> 5.8e-7
// (861 frames through two of Dia's decoder layers 1.25e-5 -> 3.9e-6).  A row's numbers keep 22 bits where three terms kept 24, which the sums make up
// for: over Dia's widths and 130 to 3000 rows (normal, gated, positive numbers) 5.8e-7 to 9.0e-7 against 3.5e-6 to 4.0e-5, and 1.2e-6 against 3.5e-6
// in columns that see only the other numbers of rows with one 2^20 times as large.  Chunks of 1, 2 and 4 k-blocks: 282, 215 and 162 us, 1.5e-7, 2.9e-7 and 5.8e-7 (the
// accumulators of a chunk are read while the MMAs update the others, and the two slow each other down).
template <bool SUMS, bool GLU = false>
struct Pair {
    static constexpr int kFirst = SUMS ? 4 : 2, kWarps = SUMS || GLU ? 8 : 4, kThreads = 32 * (kFirst + kWarps);  // (registers go by groups of 4 warps)
    static constexpr int kSumRegs = 208, kFewRegs = 88, kRegs = (kSumRegs * 8 + kFewRegs * 4) / 12;        // 168 a thread at launch
    static constexpr int kSlots = SUMS || GLU ? 12 : 13;                                                          // ring, and 32 x 32 blocks to turn
    static constexpr int kSmem = kSlots * kTileBytes + kWarps * 4096 + 1024 + 256;
};
constexpr int kPairStagesMost = 8, kPairChunk = 4;
constexpr unsigned kPairPolls = 4000000u;                     // a few seconds
static_assert((2 * kPairStagesMost + 4) * 8 + 8 <= 256, "barrier region");

struct PairProduct {
    float* y; const float* residual;
    int M, N, K, BN, stages;
    const float* dyt_w; const float* dyt_b; float dyt_alpha;
    __nv_bfloat16* y_bf16;
    const int* row_group; int group_rows; const int* n_rows;
    int* ran_out;
    const float* row_inv; const float* col_mag;              // SUMS: inverse scales of the rows, largest magnitudes of the columns
    int glu; float glu_limit;                                 // GLU: the gate's form (see glu_value)
    unsigned polls;                                           // looks at a barrier until a wait has run out
};

// the activation of a gated unit on its gate g and up u products, as the kernel that runs by itself has it: 0 silu(g) u, 1 clamped, 2 gelu(g) u
__device__ __forceinline__ float glu_value(int kind, float g, float u, float limit) {
    if (kind == 1) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return g * (1.0f / (1.0f + expf(-(1.702f * g)))) * (u + 1.0f);
    }
    if (kind == 2) return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * fmaf(0.044715f * g * g, g, g))) * u;
    // Zero divided by two is zero; the division's short way does not take it, and rows that are not there made the gate of their tile take 7 us more.  (The
    // numerator is hidden, or the two selections become one again.)
    float n = g == 0.f ? 1.f : g;
    asm("" : "+f"(n));
    const float q = n / (1.0f + expf(-g));
    return (g == 0.f ? g : q) * u;
}

// How often a wait of the pair kernel looks at its barrier, in products that this thread launches.  With 0 each wait runs out before anything has
// been issued, which is how a test sees what then becomes of the outputs.
unsigned& gemm_pair_polls() {
    static thread_local unsigned polls = kPairPolls;
    return polls;
}

__device__ __forceinline__ uint32_t at_rank(const void* local, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
    return a;
}
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity, unsigned polls) {       // one answer for a converged warp
    for (unsigned i = 0; i < polls; ++i)
        if (__any_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return false;
}
__device__ __forceinline__ bool lane_wait(uint64_t* bar, uint32_t parity, unsigned polls) {
    for (unsigned i = 0; i < polls; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// a load of this CTA that counts on a barrier of the pair's leader
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {                // the barrier at this place in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// NaN for rows [row0, row0 + rows) and columns [c0, c1) of a product that has no result (a multiple of 4 columns)
template <bool GLU>
__device__ __noinline__ void pair_no_result(const PairProduct& p, int row0, int rows, int c0, int c1, int lane) {
    const int N = GLU ? p.N >> 1 : p.N;
    const uint32_t nan = 0x7fffffffu, two = 0x7fff7fffu;      // (as fp32 and as two bf16)
    for (int r = 0; r < rows; ++r)
        for (int n = c0 + 4 * lane; n < c1; n += 128) {
            const size_t at = (size_t)(row0 + r) * N + n;
            if (p.y_bf16) *reinterpret_cast<uint2*>(p.y_bf16 + at) = make_uint2(two, two);
            else *reinterpret_cast<uint4*>(p.y + at) = make_uint4(nan, nan, nan, nan);
        }
}

// the inverse of a column's scale 2^(14 - e), where its largest magnitude lies in [2^e, 2^(e + 1)) (0 for a column of zeros)
__device__ __forceinline__ float column_inverse(float magnitude) {
    return __uint_as_float((uint32_t)max((int)(__float_as_uint(magnitude) >> 23) - 14, 0) << 23);
}

__device__ __forceinline__ void tmem_columns16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr)
        : "memory");
}

// GLU: the weights' rows are [gate (N / 2) | up (N / 2)], and a tile is 128 columns of either: the leader's half of the weight tile holds gate rows, the other's
// the up rows of the same columns, so that each CTA's accumulator has both for its rows.  Eight warps take them, apply the gate and write the bf16 operand of the
// product that follows: 268 MB of fp32 products that another kernel read again stay on the chip (4096 rows, two of eight experts of 2048 and a shared one of
// 4096, width 2048: products and gates 397 us apart, 349 together; with four warps the exponentials and divisions took longer than a tile's MMAs).
template <int TERMS, bool SUMS, bool GLU = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Pair<SUMS, GLU>::kThreads, 1)
dia_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ PairProduct p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* turn = smem + Pair<SUMS, GLU>::kSlots * kTileBytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(turn + Pair<SUMS, GLU>::kWarps * 4096);      // (the leader's alone)
    uint64_t* empty = full + kPairStagesMost;
    uint64_t* t_full = empty + kPairStagesMost;
    uint64_t* t_empty = t_full + 2;                                              // (the leader's alone)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_empty + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = blockIdx.x & 1;
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int BN = p.BN, half = BN >> 1, M = p.M, N = GLU ? p.N >> 1 : p.N, ON = GLU ? half : BN;       // columns of the result, of a tile of it
    const int n_kb = (p.K + BK - 1) / BK, n_stages = p.stages;
    const int m_lim = p.n_rows ? min(M, *p.n_rows) : M;
    const int tiles_m = (M + 2 * BM - 1) / (2 * BM), n_tiles = tiles_m * ((N + ON - 1) / ON);
    const int stage_bytes = TERMS * kTileBytes + half * 128;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kPairStagesMost; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], 2 * Pair<SUMS, GLU>::kWarps); }
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;
    if (warp < Pair<SUMS, GLU>::kFirst) {
        if constexpr (SUMS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Pair<SUMS, GLU>::kFewRegs));
        if (warp == 0) {
            if (lane == 0) {
                unsigned i = 0;
                for (int t = pair; t < n_tiles && ok; t += pairs) {
                    const int n0 = (t / tiles_m) * ON, m0 = (t % tiles_m) * 2 * BM;
                    if (m0 >= m_lim) continue;
                    const int a_row = m0 + (int)rank * BM, b_row = n0 + (int)rank * (GLU ? N : half) + (p.row_group ? p.row_group[m0] * p.group_rows : 0);
                    for (int kb = 0; kb < n_kb; ++kb, ++i) {
                        const unsigned s = i % n_stages;
                        if (!lane_wait(&empty[s], ((i / n_stages) & 1u) ^ 1u, p.polls)) { ok = false; break; }
                        if (rank == 0) mbar_arrive_expect_tx(&full[s], 2u * stage_bytes);
                        const uint32_t bar = at_rank(&full[s], 0), dst = smem_u32(smem + s * stage_bytes);
                        tma_load_2d_pair(dst + TERMS * kTileBytes, &map_b, bar, kb * BK, b_row);
#pragma unroll
                        for (int tm = 0; tm < TERMS; ++tm) tma_load_2d_pair(dst + tm * kTileBytes, &map_a, bar, kb * BK, tm * M + a_row);
                    }
                }
                // (the leader's last commits arrive here: not after this CTA has gone)
                for (unsigned j = i > (unsigned)n_stages ? i - n_stages : 0; j < i && ok; ++j) ok = lane_wait(&empty[j % n_stages], (j / n_stages) & 1u, p.polls);
                // (nor do copies arrive that were issued before a wait ran out)
                for (unsigned j = i > (unsigned)n_stages ? i - n_stages : 0; j < i && !ok && rank == 0; ++j) (void)lane_wait(&full[j % n_stages], (j / n_stages) & 1u, p.polls);
            }
        } else if (warp == 1) {
            if (rank == 0) {
                const uint32_t types = SUMS ? 0u : (1u << 7) | (1u << 10);           // fp16 or bf16
                const uint32_t idesc = (1u << 4) | types | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(2 * BM >> 4) << 24);
                unsigned i = 0, it = 0;                           // k-blocks and uses of an accumulator so far
                for (int t = pair; t < n_tiles && ok; t += pairs) {
                    if ((t % tiles_m) * 2 * BM >= m_lim) continue;
                    for (int kb = 0; kb < n_kb; ++kb, ++i) {
                        const bool first = SUMS ? kb % kPairChunk == 0 : kb == 0, last = kb == n_kb - 1 || (SUMS && kb % kPairChunk == kPairChunk - 1);
                        if (first) {
                            if (!pair_wait(&t_empty[it & 1u], ((it >> 1) & 1u) ^ 1u, p.polls)) { ok = false; break; }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        const uint32_t d = tmem_base + (it & 1u) * 256;
                        const unsigned s = i % n_stages;
                        if (!pair_wait(&full[s], (i / n_stages) & 1u, p.polls)) { ok = false; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t at = smem_u32(smem + s * stage_bytes);
                        const uint64_t adesc = umma_desc(at), bdesc = umma_desc(at + TERMS * kTileBytes);
                        if (elect_one_sync()) {
#pragma unroll
                            for (int u = 0; u < TERMS; ++u) {
                                const int tm = SUMS ? TERMS - 1 - u : u;             // the smallest term first
#pragma unroll
                                for (int j = 0; j < BK / 16; ++j)
                                    umma_bf16_pair(d, adesc + (tm * kTileBytes >> 4) + 2 * j, bdesc + 2 * j, idesc, (u | j) != 0 ? 1u : (first ? 0u : 1u));
                            }
                            umma_commit_pair(&empty[s]);
                            if (last) umma_commit_pair(&t_full[it & 1u]);
                        }
                        __syncwarp();
                        if (last) ++it;
                    }
                }
            }
        }
    } else if constexpr (SUMS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Pair<SUMS, GLU>::kSumRegs));      // (there are as many: see pairs_of)
        const int q = warp & 3, h0 = ((warp - Pair<SUMS, GLU>::kFirst) >> 2) * half;
        float* const blk = reinterpret_cast<float*>(turn + (warp - Pair<SUMS, GLU>::kFirst) * 4096);
        const int rr = lane >> 3, ch = lane & 7;
        unsigned i = 0;
        for (int t = pair; t < n_tiles; t += pairs) {
            const int n0 = (t / tiles_m) * ON, m0 = (t % tiles_m) * 2 * BM;
            float sum[128];
#pragma unroll
            for (int c = 0; c < 128; ++c) sum[c] = 0.f;
            for (int kb = 0; kb < n_kb && ok; kb += kPairChunk, ++i) {
                const unsigned acc = i & 1u;
                if (!pair_wait(&t_full[acc], (i >> 1) & 1u, p.polls)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int cb = 0; cb < 4; ++cb) {
                    if (cb * 32 >= half) break;               // (columns of the last block beyond the half are read and not stored)
                    uint32_t v[32];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                        : "r"(tmem_base + ((uint32_t)(q * 32) << 16) + acc * 256 + h0 + cb * 32)
                        : "memory");
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 32; ++e) sum[cb * 32 + e] += __uint_as_float(v[e]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(at_rank(&t_empty[acc], 0)) : "memory");
            }
            const int row0 = m0 + (int)rank * BM + q * 32, rows = min(32, M - row0);
            if (!ok) {                                        // the sums of this tile lack products, and no later one has any
                pair_no_result<GLU>(p, row0, rows, n0 + h0, min(n0 + h0 + half, N), lane);
                continue;
            }
            float ri[8];                                      // (loads ahead of their uses: the output of a tile took 3.2 us with one row after the other)
#pragma unroll
            for (int g = 0; g < 8; ++g) ri[g] = 4 * g + rr < rows ? p.row_inv[row0 + 4 * g + rr] : 0.f;
#pragma unroll
            for (int cb = 0; cb < 4; ++cb) {
                const int n = n0 + h0 + cb * 32 + 4 * ch;     // (BN and N are multiples of 4)
                if (cb * 32 >= half || rows <= 0) break;
                const bool in = n < N && cb * 32 + 4 * ch < half;
                float4 mag = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in) mag = *reinterpret_cast<const float4*>(p.col_mag + n);
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<float4*>(blk + lane * 32 + ((c ^ (lane & 7)) << 2)) =
                        make_float4(sum[cb * 32 + 4 * c], sum[cb * 32 + 4 * c + 1], sum[cb * 32 + 4 * c + 2], sum[cb * 32 + 4 * c + 3]);
                __syncwarp();
                const float f[4] = {column_inverse(mag.x), column_inverse(mag.y), column_inverse(mag.z), column_inverse(mag.w)};
                const size_t at0 = (size_t)(row0 + rr) * N + n;
#pragma unroll
                for (int g0 = 0; g0 < 8; g0 += 4) {
                    float4 add[4];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        add[g] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (p.residual && in && 4 * (g0 + g) + rr < rows) add[g] = *reinterpret_cast<const float4*>(p.residual + at0 + (size_t)(4 * (g0 + g)) * N);
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const int r = 4 * (g0 + g) + rr;
                        const float4 a = *reinterpret_cast<const float4*>(blk + r * 32 + ((ch ^ (r & 7)) << 2));
                        const float o[4] = {a.x, a.y, a.z, a.w}, z[4] = {add[g].x, add[g].y, add[g].z, add[g].w};
                        float y[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)           // (no step out of range that the result is not)
                            y[e] = o[e] * fminf(ri[g0 + g], f[e]) * fmaxf(ri[g0 + g], f[e]) + z[e];
                        if (in && r < rows) *reinterpret_cast<float4*>(p.y + at0 + (size_t)(4 * (g0 + g)) * N) = make_float4(y[0], y[1], y[2], y[3]);
                    }
                }
                __syncwarp();
            }
        }
    } else if constexpr (GLU) {
        const int q = warp & 3, h0 = ((warp - Pair<SUMS, GLU>::kFirst) >> 2) * 64;
        unsigned char* const blk = turn + (warp - Pair<SUMS, GLU>::kFirst) * 4096;
        const int rr = lane >> 3, ch = lane & 7;              // a lane's row of four and its 16-byte piece of 64 columns
        unsigned it = 0;
        for (int t = pair; t < n_tiles; t += pairs) {
            const int n0 = (t / tiles_m) * ON, m0 = (t % tiles_m) * 2 * BM;
            if (m0 >= m_lim) continue;
            const int row0 = m0 + (int)rank * BM + q * 32, rows = min(32, M - row0);
            const unsigned acc = it & 1u;
            ok = ok && pair_wait(&t_full[acc], (it >> 1) & 1u, p.polls);
            if (!ok) {
                pair_no_result<GLU>(p, row0, rows, n0 + h0, n0 + h0 + 64, lane);
                continue;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t from = tmem_base + ((uint32_t)(q * 32) << 16) + acc * 256 + h0;
#pragma unroll 1
            for (int cb = 0; cb < 4; ++cb) {
                uint32_t g[16], u[16];
                tmem_columns16(from + cb * 16, g);
                tmem_columns16(from + half + cb * 16, u);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                uint32_t y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(glu_value(p.glu, __uint_as_float(g[2 * e]), __uint_as_float(u[2 * e]), p.glu_limit),
                                                                   glu_value(p.glu, __uint_as_float(g[2 * e + 1]), __uint_as_float(u[2 * e + 1]), p.glu_limit));
                    y[e] = *reinterpret_cast<const uint32_t*>(&b);
                }
                // lane = row: its 16-byte piece c goes to place c ^ (row % 8) of its 128 bytes, and is read a row per eight lanes
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    *reinterpret_cast<uint4*>(blk + lane * 128 + (((2 * cb + c) ^ (lane & 7)) << 4)) = make_uint4(y[4 * c], y[4 * c + 1], y[4 * c + 2], y[4 * c + 3]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(at_rank(&t_empty[acc], 0)) : "memory");
            ++it;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int r = 4 * e + rr;
                if (r < rows)
                    *reinterpret_cast<uint4*>(p.y_bf16 + (size_t)(row0 + r) * N + n0 + h0 + 8 * ch) = *reinterpret_cast<const uint4*>(blk + r * 128 + ((ch ^ (r & 7)) << 4));
            }
            __syncwarp();
        }
    } else {
        const int q = warp & 3;
        float* const blk = reinterpret_cast<float*>(turn + (warp - Pair<SUMS, GLU>::kFirst) * 4096);
        const int rr = lane >> 3, ch = lane & 7;              // a lane's row of four and its 16-byte piece of a 32-column block
        unsigned it = 0;
        for (int t = pair; t < n_tiles; t += pairs) {
            const int n0 = (t / tiles_m) * ON, m0 = (t % tiles_m) * 2 * BM;
            if (m0 >= m_lim) continue;
            const int row0 = m0 + (int)rank * BM + q * 32, rows = min(32, M - row0);
            const unsigned acc = it & 1u;
            ok = ok && pair_wait(&t_full[acc], (it >> 1) & 1u, p.polls);
            if (!ok) {
                pair_no_result<GLU>(p, row0, rows, n0, min(n0 + BN, N), lane);
                continue;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int cb = 0; cb < BN / 32; ++cb) {
                const int c0 = n0 + cb * 32;
                if (c0 >= N || rows <= 0) break;              // (uniform)
                uint32_t v[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                      "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                      "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(tmem_base + ((uint32_t)(q * 32) << 16) + acc * 256 + cb * 32)
                    : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                // lane = row: its 16-byte piece c goes to place c ^ (row % 8) of its 128 bytes, and is read a row per eight lanes
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4*>(blk + lane * 32 + ((c ^ (lane & 7)) << 2)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
                __syncwarp();
                const int n = c0 + 4 * ch;
                if (n < N) {                                  // (N is a multiple of 4)
                    float4 w4 = make_float4(0.f, 0.f, 0.f, 0.f), b4 = w4;
                    if (p.dyt_w) {
                        w4 = *reinterpret_cast<const float4*>(p.dyt_w + n);
                        b4 = *reinterpret_cast<const float4*>(p.dyt_b + n);
                    }
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        const int r = 4 * g + rr;
                        if (r >= rows) break;
                        float4 a = *reinterpret_cast<const float4*>(blk + r * 32 + ((ch ^ (r & 7)) << 2));
                        const size_t at = (size_t)(row0 + r) * N + n;
                        if (p.y_bf16) {                       // the activation of an up product, as the next product's operand
                            const __nv_bfloat162 lo = __floats2bfloat162_rn(gelu_to_bf16_range(a.x), gelu_to_bf16_range(a.y));
                            const __nv_bfloat162 hi = __floats2bfloat162_rn(gelu_to_bf16_range(a.z), gelu_to_bf16_range(a.w));
                            *reinterpret_cast<uint2*>(p.y_bf16 + at) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                            continue;
                        }
                        if (p.dyt_w) {                        // DynamicTanh of the product: tanh(alpha a) w + b per column
                            a.x = fmaf(tanhf(p.dyt_alpha * a.x), w4.x, b4.x); a.y = fmaf(tanhf(p.dyt_alpha * a.y), w4.y, b4.y);
                            a.z = fmaf(tanhf(p.dyt_alpha * a.z), w4.z, b4.z); a.w = fmaf(tanhf(p.dyt_alpha * a.w), w4.w, b4.w);
                        }
                        if (p.residual) {
                            const float4 r4 = *reinterpret_cast<const float4*>(p.residual + at);
                            a.x += r4.x; a.y += r4.y; a.z += r4.z; a.w += r4.w;
                        }
                        *reinterpret_cast<float4*>(p.y + at) = a;
                    }
                }
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(at_rank(&t_empty[acc], 0)) : "memory");
            ++it;
        }
    }
    if (!ok && lane == 0 && p.ran_out) {
        *reinterpret_cast<volatile int*>(p.ran_out) = 1;
        __threadfence_system();
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync_all();                                       // neither CTA's memory goes while the other still reads it or arrives there
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
    }
}

__device__ __forceinline__ float load_remote(const float* local, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 load_remote4(const float* local, uint32_t rank) {
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}

// ---------------------------------------------------------------------------------------------------------------------
// Y = A W^T in the accuracy of fp32 FMA arithmetic, for callers that asked for it.  The accumulator of a tensor-core product loses
// up to a unit in the last place at every step, towards zero (K = 2048: 2.1e-6 against 3.9e-7 of an FMA chain), so an accumulator
// lives for one k-block only - the two small terms first, then the large one - and the epilogue warps add it to the tile's sums
// in their registers while the next k-blocks are multiplied into the three other accumulators.  128 x 128 tiles: a thread holds
// 128 sums.  Bound: 12 MMAs of 64 cycles per k-block against ~300 issue slots of draining it.  Where the tiles leave most of the chip
// idle, a cluster of gridDim.y CTAs shares a tile: each takes a range of k-blocks, and the sums meet in shared memory.
constexpr int kFN = 128, kFASlots = 6, kFBSlots = 3;
constexpr int kFWarps = 8, kFThreads = 64 + 32 * kFWarps, kFCols = kFN / 2, kFStride = kFCols + 4;      // epilogue warps, columns of one
constexpr int kFStage = kFWarps * 32 * kFStride * 4;          // 32 rows of sums per epilogue warp
constexpr int kFBars = 2 * kFASlots + 2 * kFBSlots + 8;
constexpr int kFSmem = (kFASlots + kFBSlots) * kTileBytes + kFStage + 1024 + 256;
static_assert(kFBars * 8 + 8 <= 256, "barrier region");

__device__ __noinline__ float f32_act(int act, float z) {
    if (act == 2) return fmaxf(z, 0.f) * fmaxf(z, 0.f);
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * fmaf(0.044715f * z * z, z, z)));
}

// TERMS: terms of A (3: fp32 rows, 1: bf16 rows)
template <int TERMS>
__global__ void __launch_bounds__(kFThreads, 1)
dia_gemm_f32_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ F32Product p) {
    const int M = p.M, N = p.N, K = p.K;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* a_ring = smem;
    unsigned char* b_ring = smem + kFASlots * kTileBytes;
    uint64_t* a_full = reinterpret_cast<uint64_t*>(b_ring + kFBSlots * kTileBytes);
    uint64_t* a_empty = a_full + kFASlots;
    uint64_t* b_full = a_empty + kFASlots;
    uint64_t* b_empty = b_full + kFBSlots;
    uint64_t* t_full = b_empty + kFBSlots;                  // [4] a k-block's products are complete / have been added
    uint64_t* t_empty = t_full + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_empty + 4);
    float* stage = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(a_full) + 256);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = gridDim.y, kb_all = (K + BK - 1) / BK, kb_per = (kb_all + S - 1) / S, kb0 = blockIdx.y * kb_per;
    const int n_kb = max(0, min(kb_per, kb_all - kb0));
    const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + kFN - 1) / kFN, n_tiles = tiles_m * tiles_n * p.heads;
    // an epilogue warp's 32 rows of sums, from rows 2 r0 and 2 r0 + 1 on every S-th pair, four columns per lane
    float* const tile = stage + (warp - 2) * 32 * kFStride;
    auto emit = [&](int t, int r0) {
        const int q = warp & 3, hn = t / tiles_m, h = hn / tiles_n, n0 = (hn - h * tiles_n) * kFN, m0 = (t % tiles_m) * BM;
        const int rows = min(32, M - (m0 + q * 32)), c4 = 4 * (lane & 15), n = n0 + ((warp - 2) >> 2) * kFCols + c4;
        if (n >= N) return;
        const size_t m = (size_t)(m0 + q * 32), col = (size_t)h * p.y_hs + n;
        const float* gate = p.gate ? p.gate + m * p.ldg + (p.head_gate ? (size_t)h : (size_t)h * N + n) : nullptr;
#pragma unroll 1
        for (int r = 2 * r0 + (lane >> 4); r < rows; r += 2 * S) {
            float4 v = *reinterpret_cast<const float4*>(tile + r * kFStride + c4);
            if (S > 1) {
                float4 u[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) if (c < S) u[c] = load_remote4(tile + r * kFStride + c4, c);
                v = u[0];
#pragma unroll
                for (int c = 1; c < 8; ++c) if (c < S) { v.x += u[c].x; v.y += u[c].y; v.z += u[c].z; v.w += u[c].w; }
            }
            v.x *= p.alpha; v.y *= p.alpha; v.z *= p.alpha; v.w *= p.alpha;
            if (p.act) { v.x = f32_act(p.act, v.x); v.y = f32_act(p.act, v.y); v.z = f32_act(p.act, v.z); v.w = f32_act(p.act, v.w); }
            if (gate) {
                const float* z = gate + (size_t)r * p.ldg;
                if (p.head_gate) {
                    const float f = 1.0f / (1.0f + expf(-z[0]));
                    v.x *= f; v.y *= f; v.z *= f; v.w *= f;
                } else {
                    v.x *= 1.0f / (1.0f + expf(-z[0])); v.y *= 1.0f / (1.0f + expf(-z[1]));
                    v.z *= 1.0f / (1.0f + expf(-z[2])); v.w *= 1.0f / (1.0f + expf(-z[3]));
                }
            }
            const size_t at = (m + r) * p.ldy + col;
            if (p.dyt_w) {
                const float4 w4 = *reinterpret_cast<const float4*>(p.dyt_w + col), b4 = *reinterpret_cast<const float4*>(p.dyt_b + col);
                v.x = fmaf(tanhf(p.dyt_alpha * v.x), w4.x, b4.x); v.y = fmaf(tanhf(p.dyt_alpha * v.y), w4.y, b4.y);
                v.z = fmaf(tanhf(p.dyt_alpha * v.z), w4.z, b4.z); v.w = fmaf(tanhf(p.dyt_alpha * v.w), w4.w, b4.w);
            }
            if (p.add) {
                const float4 o = *reinterpret_cast<const float4*>(p.add + at);
                v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
            }
            if (p.y) *reinterpret_cast<float4*>(p.y + at) = v;
            if (p.y_bf16) {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.y_bf16) + at) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            }
        }
    };
    // tile t: row block t % tiles_m of column block (t / tiles_m) % tiles_n of head t / (tiles_m tiles_n)
    if (threadIdx.x == 0) {
        for (int i = 0; i < kFASlots; ++i) { mbar_init(&a_full[i], 1); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < kFBSlots; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < 4; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], kFWarps); }
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(4 * kFN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            unsigned ia = 0, ib = 0;
            for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
                const int hn = t / tiles_m, h = hn / tiles_n, n0 = (hn - h * tiles_n) * kFN, m0 = (t % tiles_m) * BM;
                for (int kb = 0; kb < n_kb; ++kb) {
                    const unsigned s = ib % kFBSlots;
                    mbar_wait_bounded(&b_empty[s], ((ib / kFBSlots) & 1u) ^ 1u);
                    mbar_arrive_expect_tx(&b_full[s], kTileBytes);
                    tma_load_2d(smem_u32(b_ring + s * kTileBytes), &map_b, smem_u32(&b_full[s]), (kb0 + kb) * BK, h * N + n0);
                    ++ib;
                    for (int tm = TERMS - 1; tm >= 0; --tm) {          // the smallest term first
                        const unsigned sa = ia % kFASlots;
                        mbar_wait_bounded(&a_empty[sa], ((ia / kFASlots) & 1u) ^ 1u);
                        mbar_arrive_expect_tx(&a_full[sa], kTileBytes);
                        tma_load_2d(smem_u32(a_ring + sa * kTileBytes), &map_a, smem_u32(&a_full[sa]), (kb0 + kb) * BK, (tm * p.heads + h) * M + m0);
                        ++ia;
                    }
                }
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kFN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        unsigned ia = 0, ib = 0;
        for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
            for (int kb = 0; kb < n_kb; ++kb) {
                const unsigned acc = ib & 3u, sb = ib % kFBSlots;
                mbar_wait_bounded(&t_empty[acc], ((ib >> 2) & 1u) ^ 1u);
                mbar_wait_bounded(&b_full[sb], (ib / kFBSlots) & 1u);
                const uint64_t bdesc = umma_desc(smem_u32(b_ring + sb * kTileBytes));
                const uint32_t d = tmem_base + acc * kFN;
                for (int tm = 0; tm < TERMS; ++tm) {
                    const unsigned sa = ia % kFASlots;
                    mbar_wait_bounded(&a_full[sa], (ia / kFASlots) & 1u);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t adesc = umma_desc(smem_u32(a_ring + sa * kTileBytes));
                    if (elect_one_sync()) {
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j) umma_bf16(d, adesc + 2 * j, bdesc + 2 * j, idesc, (tm | j) != 0 ? 1u : 0u);
                        umma_commit(&a_empty[sa]);
                        if (tm == TERMS - 1) {
                            umma_commit(&b_empty[sb]);
                            umma_commit(&t_full[acc]);
                        }
                    }
                    __syncwarp();
                    ++ia;
                }
                ++ib;
            }
        }
    } else {
        const int q = warp & 3;
        unsigned it = 0;
        for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
            float sum[kFCols];
#pragma unroll
            for (int c = 0; c < kFCols; ++c) sum[c] = 0.f;
            for (int kb = 0; kb < n_kb; ++kb, ++it) {
                const unsigned acc = it & 3u;
                mbar_wait_bounded(&t_full[acc], (it >> 2) & 1u);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int cb = 0; cb < kFCols / 32; ++cb) {
                    uint32_t v[32];
                    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * kFN + ((warp - 2) >> 2) * kFCols + cb * 32;
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                        : "r"(taddr)
                        : "memory");
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) sum[cb * 32 + i] += __uint_as_float(v[i]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&t_empty[acc]);
            }
            // The sums go out through shared memory, a row per step and four columns per lane: coalesced, and a short loop where the
            // unrolled one (128 copies of the epilogue) was bound by instruction fetches.
            __syncwarp();
#pragma unroll
            for (int c = 0; c < kFCols; c += 4)
                *reinterpret_cast<float4*>(tile + lane * kFStride + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
            __syncwarp();
            if (S == 1) emit(t, 0);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(4 * kFN));
    }
    if (S > 1) {
        cluster_sync_all();
        if (warp >= 2) emit(blockIdx.x, blockIdx.y);
        cluster_sync_all();                                   // (the sums stay until every CTA has read them)
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Few rows: a cluster of S CTAs owns 128 weight rows, each CTA a range of k-blocks.
//   warp 0    requests the CTA's weight tiles [128 x 64] (TMA, 128-byte swizzle) ahead of the rows - before the kernel's predecessor
//             has ended, when launched early
//   all warps split the rows' k range into three bf16 terms: column term * Mp + m of the [NB x 64] operand of a k-block
//   warp 1    per k-block 4 MMAs (M = 128, N = NB) into an accumulator of its own
//   warps 2-5 add the k-blocks' accumulators in fp32 registers (weight row = lane), then the three terms; the CTAs' partial sums
//             meet in shared memory and every CTA of the cluster adds its share of the outputs, in the order of the k ranges
// Bound: the weights' bytes.  The row kernel reads them once per row from L2 instead: 8 rows x 2048 x 6144 took 35 us.
// An SM holds two of its CTAs at most, whatever the shape: a launch may start before its predecessors have ended, and its CTAs keep
// their half of tensor memory while they wait for them.  With three on an SM a predecessor's CTA could find all of it taken by CTAs
// that wait for that CTA.
constexpr int kRThreads = 192, kRSlotsMost = 8, kRSmemMost = 226 * 1024, kRSmemLeast = 78 * 1024;
static_assert(3 * kRSmemLeast > 228 * 1024, "two CTAs on an SM");

// NB: columns of the rows' operand (32 for up to 8 rows, 96 for up to 32)
template <int NB>
__global__ void __launch_bounds__(kRThreads, 1)
dia_gemm_few_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ FewRowsProduct p, int kb_per, int n_slots) {
    constexpr int Mp = NB / 3 / 8 * 8, kBufs = NB == 32 ? 8 : 2, kCols = 256;      // (two CTAs per SM)
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t w_full[kRSlotsMost], w_empty[kRSlotsMost], t_full[8], t_empty[8];
    __shared__ uint32_t tmem_slot;
    unsigned char* ring = smem;
    unsigned char* rows = ring + n_slots * kTileBytes;                         // [kb_per][NB x 64] bf16
    float* part = reinterpret_cast<float*>(rows + (size_t)kb_per * NB * 128);  // [Mp][128]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = gridDim.y, n_kb = (p.K + BK - 1) / BK, rank = blockIdx.y, n0 = blockIdx.x * BM, M = p.M;
    const int kb0 = rank * kb_per, kbs = max(0, min(kb_per, n_kb - kb0));
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) {
        for (int i = 0; i < kRSlotsMost; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 1); }
        for (int i = 0; i < 8; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], 4); }
        fence_mbar_init();
        for (int kb = 0; kb < min(kbs, n_slots); ++kb) {
            mbar_arrive_expect_tx(&w_full[kb], kTileBytes);
            tma_load_2d(smem_u32(ring + kb * kTileBytes), &map_w, smem_u32(&w_full[kb]), (kb0 + kb) * BK, n0);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // ---- the rows' terms: 8 channels per item ----
    for (int i = tid; i < Mp * kbs * 8; i += kRThreads) {
        const int m = i / (kbs * 8), c = i - m * (kbs * 8), kb = c >> 3, ch = c & 7, k = (kb0 + kb) * BK + ch * 8;
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = 0.f;
        if (m < M && k < p.K) {                               // (K a multiple of 8)
            const float4* src = reinterpret_cast<const float4*>(p.a + (size_t)m * p.lda + k);
            const float4 x = src[0], y = src[1];
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
        }
        __nv_bfloat16 t[3][8];
#pragma unroll
        for (int e = 0; e < 8; ++e) split3_down(v[e], t[0][e], t[1][e], t[2][e]);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int r = q * Mp + m;
            *reinterpret_cast<uint4*>(rows + (size_t)kb * NB * 128 + (r >> 3) * 1024 + (r & 7) * 128 + ((ch ^ (r & 7)) << 4)) =
                *reinterpret_cast<const uint4*>(t[q]);
        }
    }
    for (int i = tid; i < (NB - 3 * Mp) * kbs * 8; i += kRThreads) {           // columns that no row uses
        const int r = 3 * Mp + i / (kbs * 8), c = i % (kbs * 8);
        *reinterpret_cast<uint4*>(rows + (size_t)(c >> 3) * NB * 128 + (r >> 3) * 1024 + (r & 7) * 128 + ((c & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_proxy_async();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (warp == 0) {
        if (lane == 0)
            for (int kb = n_slots; kb < kbs; ++kb) {
                const int s = kb % n_slots;
                mbar_wait_bounded(&w_empty[s], ((kb / n_slots) & 1u) ^ 1u);
                mbar_arrive_expect_tx(&w_full[s], kTileBytes);
                tma_load_2d(smem_u32(ring + s * kTileBytes), &map_w, smem_u32(&w_full[s]), (kb0 + kb) * BK, n0);
            }
    } else if (warp == 1) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        for (int kb = 0; kb < kbs; ++kb) {
            const int s = kb % n_slots, acc = kb % kBufs;
            mbar_wait_bounded(&t_empty[acc], ((kb / kBufs) & 1u) ^ 1u);
            mbar_wait_bounded(&w_full[s], (kb / n_slots) & 1u);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t adesc = umma_desc(smem_u32(ring + s * kTileBytes)), bdesc = umma_desc(smem_u32(rows + (size_t)kb * NB * 128));
            if (elect_one_sync()) {
#pragma unroll
                for (int j = 0; j < BK / 16; ++j) umma_bf16(tmem + acc * NB, adesc + 2 * j, bdesc + 2 * j, idesc, j != 0 ? 1u : 0u);
                umma_commit(&w_empty[s]);
                umma_commit(&t_full[acc]);
            }
            __syncwarp();
        }
    } else {
        const int q = warp & 3;
        float sum[NB];
#pragma unroll
        for (int c = 0; c < NB; ++c) sum[c] = 0.f;
        for (int kb = 0; kb < kbs; ++kb) {
            const int acc = kb % kBufs;
            mbar_wait_bounded(&t_full[acc], (kb / kBufs) & 1u);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t v[NB];
#pragma unroll
            for (int c = 0; c < NB; c += 16)
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                    : "=r"(v[c]), "=r"(v[c + 1]), "=r"(v[c + 2]), "=r"(v[c + 3]), "=r"(v[c + 4]), "=r"(v[c + 5]), "=r"(v[c + 6]), "=r"(v[c + 7]),
                      "=r"(v[c + 8]), "=r"(v[c + 9]), "=r"(v[c + 10]), "=r"(v[c + 11]), "=r"(v[c + 12]), "=r"(v[c + 13]), "=r"(v[c + 14]), "=r"(v[c + 15])
                    : "r"(tmem + ((uint32_t)(q * 32) << 16) + acc * NB + c)
                    : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < NB; ++c) sum[c] += __uint_as_float(v[c]);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&t_empty[acc]);
        }
#pragma unroll
        for (int m = 0; m < Mp; ++m) part[m * BM + q * 32 + lane] = (sum[2 * Mp + m] + sum[Mp + m]) + sum[m];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
    }
    if (S > 1) cluster_sync_all();
    // ---- the outputs of the tile, dealt to the cluster's CTAs ----
    for (int i = rank * kRThreads + tid; i < M * BM; i += S * kRThreads) {
        const int m = i / BM, c = i - m * BM, n = n0 + c;
        if (n >= p.N) continue;
        float v;
        if (S > 1) {
            float u[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) u[r] = r < S ? load_remote(part + i, r) : 0.f;
            v = u[0];
#pragma unroll
            for (int r = 1; r < 8; ++r)
                if (r < S) v += u[r];
        } else {
            v = part[i];
        }
        if (p.act) v = f32_act(p.act, v);
        const size_t at = (size_t)m * p.ldy + n;
        p.y[at] = p.add ? p.add[at] + v : v;
    }
    if (S > 1) cluster_sync_all();                            // (the partial sums stay until every CTA has read them)
}

// three bf16 terms of every head's columns, [3][heads][M][K]
__global__ void __launch_bounds__(256) split3_heads_kernel(const float* __restrict__ x, int ldx, int hs, __nv_bfloat16* __restrict__ xs, int H, int M, int K) {
    const size_t n = (size_t)H * M * K;
    const float* row = x + (size_t)blockIdx.x * ldx;
    for (int i = threadIdx.x; i < H * (K >> 2); i += 256) {   // (K a multiple of 8)
        const int h = i / (K >> 2), k = 4 * (i - h * (K >> 2));
        const size_t o = ((size_t)h * M + blockIdx.x) * K + k;
        __nv_bfloat16 t[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split3_down(row[(size_t)h * hs + k + e], t[0][e], t[1][e], t[2][e]);
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(xs + q * n + o) = *reinterpret_cast<const uint2*>(t[q]);
    }
}

// ---- host side ---------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// a [rows][K] bf16 matrix, K contiguous, read in [box_rows x 64 k] boxes with the 128-byte swizzle
static bool make_map(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t gemm_workspace_bytes(int M, int K) { return (size_t)kTerms * M * K * 2; }

// (the word of waits that ran out: there before a product of these weights can be captured)
static cudaError_t make_ran_out(cudaStream_t st) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) (void)split_attention_ran_out(dev, st);
    return e;
}

cudaError_t launch_transpose_to_bf16(const void* w, int src_bf16, void* wt, int K, int N, cudaStream_t st) {
    const cudaError_t e = make_ran_out(st);
    if (e != cudaSuccess) return e;
    dim3 grid((N + 31) / 32, (K + 31) / 32), block(32, 8);
    transpose_to_bf16_kernel<<<grid, block, 0, st>>>(w, src_bf16, reinterpret_cast<__nv_bfloat16*>(wt), K, N);
    return cudaGetLastError();
}

static bool dense_rows_f32(int terms, int M, int N, int K, int sms);
static cudaError_t run_gemm_f32(const F32Product& p, const void* a_terms, int terms, int splits, cudaStream_t st);

// clusters of two CTAs of the pair kernel that run at the same time
template <int TERMS, bool SUMS, bool GLU = false>
static cudaError_t pairs_of(int dev, int* out) {
    static std::atomic<int> known[64];
    if (dev >= 0 && dev < 64 && (*out = known[dev].load(std::memory_order_relaxed)) > 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(Pair<SUMS, GLU>::kThreads);
    cfg.dynamicSmemBytes = Pair<SUMS, GLU>::kSmem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const auto kernel = dia_gemm_pair_kernel<TERMS, SUMS, GLU>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Pair<SUMS, GLU>::kSmem);
    cudaFuncAttributes built;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&built, kernel);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(out, kernel, &cfg);
    if (e != cudaSuccess) return e;
    if (SUMS && built.numRegs < Pair<SUMS, GLU>::kRegs) return cudaErrorNotSupported;      // (its roles would wait for registers that are not there)
    if (*out < 1) return cudaErrorNotSupported;
    if (dev >= 0 && dev < 64) known[dev].store(*out, std::memory_order_relaxed);
    return cudaSuccess;
}

// Columns of a pair's tile: the width whose rounds of tiles end first.  A round's time grows with its columns where the MMAs bound it (three
// terms, us per k-block alone on the chip: 0.44 at 128, 0.63 at 192, 0.83 at 256) and hardly where issuing four of them does (one term:
// 0.30 and 0.28; two terms with fp32 sums, seven rounds of 32 k-blocks, 16.2 at 128 and 24.5 at 256 a round).  1722 rows x 16384 columns, K = 2048, three terms: 7 rounds of 256 223 us, 7 of 224 209; 3072 columns: 2 of 256 69, 2 of 160 49
static int pair_columns(int terms, int M, int N, int pairs) {
    const int tiles_m = (M + 2 * BM - 1) / (2 * BM), fixed = terms == 1 ? 700 : terms == 2 ? 100 : 30;
    int best = 0;
    long long least = 0;
    for (int bn = 256; bn >= 128; bn -= 32) {
        const long long r = ((long long)tiles_m * ((N + bn - 1) / bn) + pairs - 1) / pairs, cost = r * (fixed + bn);
        if (!best || cost < least) best = bn, least = cost;
    }
    return best;
}
template <int TERMS, bool SUMS, bool GLU = false>
static cudaError_t run_pair(const CUtensorMap& ma, const void* wt, long long wt_rows, PairProduct& q, int dev, cudaStream_t st) {
    int pairs = 0;
    cudaError_t e = pairs_of<TERMS, SUMS, GLU>(dev, &pairs);
    const auto kernel = dia_gemm_pair_kernel<TERMS, SUMS, GLU>;
    if (e == cudaSuccess) e = ask_smem<dia_gemm_pair_kernel<TERMS, SUMS, GLU>>(dev, Pair<SUMS, GLU>::kSmem);
    if (e != cudaSuccess) return e;
    q.polls = gemm_pair_polls();
    q.ran_out = split_attention_ran_out(dev, st);
    if (take_ran_out(dev, st)) return cudaErrorLaunchTimeout;
    q.BN = GLU ? 256 : pair_columns(TERMS, q.M, q.N, pairs);
    q.stages = std::min(kPairStagesMost, Pair<SUMS, GLU>::kSlots * kTileBytes / (TERMS * kTileBytes + q.BN / 2 * 128));
    CUtensorMap mb;
    if (!make_map(&mb, wt, wt_rows, q.K, q.BN / 2)) return cudaErrorNotSupported;
    const int n_tiles = ((q.N + q.BN - 1) / q.BN) * ((q.M + 2 * BM - 1) / (2 * BM));
    kernel<<<2 * std::min(n_tiles, pairs), Pair<SUMS, GLU>::kThreads, Pair<SUMS, GLU>::kSmem, st>>>(ma, mb, q);
    return cudaGetLastError();
}

// A: bf16 [terms * M][K], the terms of the activation stacked (terms = 1: the activation itself); Wt: bf16 [wt_rows][K].
// Returns cudaErrorNotSupported for shapes the tiling does not cover (the caller decides what to do).
cudaError_t launch_gemm_tcgen05_bf16(const void* a_bf16, int terms, const void* wt, long long wt_rows, float* y, int M, int N,
                                     int K, const GemmEpilogue& ep, const GemmGroups* groups, cudaStream_t st) {
    if (!gemm_tcgen05_shape_ok(M, N, K) || terms < 1 || terms > kTerms || wt_rows < N) return cudaErrorNotSupported;
    int dev = 0, sms = 0;
    cudaError_t e0 = current_sms(&dev, &sms);
    if (e0 == cudaSuccess) e0 = ask_smem<dia_gemm_tcgen05_kernel>(dev, kGemmSmem);
    if (e0 != cudaSuccess) return e0;
    CUtensorMap ma, mb;
    if (terms == 1 && !groups && wt_rows == N && dense_rows_f32(1, M, N, K, sms)) {
        const F32Product narrow{nullptr, 0, 0, wt, ep.y_bf16 ? nullptr : y, N, N, ep.y_bf16, 1, M, N, K, 1.f, ep.y_bf16 ? 3 : 0, nullptr, 0, 0,
                                ep.residual, ep.dyt_w, ep.dyt_b, ep.dyt_alpha};
        if (gemm_f32_ok(narrow)) return run_gemm_f32(narrow, a_bf16, 1, 8, st);
    }
    if (!make_map(&ma, a_bf16, (long long)terms * M, K, BM)) return cudaErrorNotSupported;
    if (M > BM && (terms == 1 || terms == kTerms) && (!groups || groups->tile_rows % (2 * BM) == 0)) {
        PairProduct q{};
        q.y = y; q.residual = ep.residual; q.M = M; q.N = N; q.K = K;
        q.dyt_w = ep.dyt_w; q.dyt_b = ep.dyt_b; q.dyt_alpha = ep.dyt_alpha; q.y_bf16 = reinterpret_cast<__nv_bfloat16*>(ep.y_bf16);
        if (groups) { q.row_group = groups->row_group; q.group_rows = groups->group_rows; q.n_rows = groups->n_rows; }
        return terms == 1 ? run_pair<1, false>(ma, wt, wt_rows, q, dev, st) : run_pair<kTerms, false>(ma, wt, wt_rows, q, dev, st);
    }
    if (!make_map(&mb, wt, wt_rows, K, BN)) return cudaErrorNotSupported;
    const int n_tiles = ((N + BN - 1) / BN) * ((M + BM - 1) / BM);
    dia_gemm_tcgen05_kernel<<<std::min(n_tiles, sms), kGemmThreads, kGemmSmem, st>>>(
        ma, mb, y, ep.residual, M, N, K, terms, ep.dyt_w, ep.dyt_b, ep.dyt_alpha,
        reinterpret_cast<__nv_bfloat16*>(ep.y_bf16), groups ? groups->row_group : nullptr,
        groups ? groups->group_rows : 0, groups ? groups->n_rows : nullptr);
    return cudaGetLastError();
}

// Whether product and gate are shorter one after the other: the gate of a tile takes eight warps 8 us, which a short k loop or a single round does not hide, and
// its tiles are 256 columns wide, which leaves more pairs idle.  Estimates in us, fitted to 150 to 4096 rows of widths 512 to 2048 and hidden widths of 256 to 4096,
// dense and grouped (within 2 us).  Measured, together / apart: 1030 rows, 512 -> 2048 26.9 / 24.8, 1024 -> 4096 39.2 / 37.2, 2048 -> 2048 37.2 / 39.2; 600 rows,
// 2048 -> 1024 26.9 / 25.5; 3000 rows, 512 -> 1024 28.0 / 26.9, 2048 -> 2048 51.1 / 62.6; four experts of 256, width 2048, 260 rows 26.9 / 24.9, 2800 29.0 / 29.7
static bool gate_apart(int M, int F, int K, int pairs) {
    const int tiles_m = (M + 2 * BM - 1) / (2 * BM), bn = pair_columns(1, M, 2 * F, pairs);
    const auto rounds = [&](int per_row) { return (int)(((long long)tiles_m * per_row + pairs - 1) / pairs); };
    const double k_blocks = (K + BK - 1) / BK, wide = bn / 256.0, outputs = (double)M * F;
    const double together = 12.0 + 0.3 * k_blocks + (rounds(F / 128) - 1) * std::max(0.34 * k_blocks, 8.3);
    const double of_round = 0.3 * k_blocks * (700 + bn) / 956.0;
    const double apart = 4.5 + 3.0 * wide + of_round + (rounds((2 * F + bn - 1) / bn) - 1) * std::max(of_round, 5.0 * wide) + 4.0 +
                         outputs * (outputs > 7.5e6 ? 2.4e-6 : 1.5e-6);      // (the gate's pass; above, the products leave L2)
    return apart + 0.6 < together;
}

cudaError_t launch_gemm_glu_bf16(const void* a_bf16, const void* wt, long long wt_rows, void* y_bf16, int M, int F, int K, int kind, float limit,
                                 const GemmGroups* groups, cudaStream_t st, bool in_any_case) {
    if (M <= BM || F % 128 || F <= 0 || !gemm_tcgen05_shape_ok(M, 2 * F, K) || wt_rows < 2LL * F || kind < 0 || kind > 2 ||
        (reinterpret_cast<uintptr_t>(y_bf16) & 15) || (groups && groups->tile_rows % (2 * BM)))
        return cudaErrorNotSupported;
    int dev = 0, sms = 0;
    const cudaError_t e = current_sms(&dev, &sms);
    if (e != cudaSuccess) return e;
    if (!groups && wt_rows == 2LL * F && dense_rows_f32(1, M, 2 * F, K, sms)) return cudaErrorNotSupported;      // (fp32 sums stay: see there)
    int pairs = 0;
    const cudaError_t known = pairs_of<1, false, true>(dev, &pairs);
    if (known != cudaSuccess) return known;
    if (!in_any_case && gate_apart(M, F, K, pairs)) return cudaErrorNotSupported;
    CUtensorMap ma;
    if (!make_map(&ma, a_bf16, M, K, BM)) return cudaErrorNotSupported;
    PairProduct q{};
    q.M = M; q.N = 2 * F; q.K = K; q.y_bf16 = reinterpret_cast<__nv_bfloat16*>(y_bf16); q.glu = kind; q.glu_limit = limit;
    if (groups) { q.row_group = groups->row_group; q.group_rows = groups->group_rows; q.n_rows = groups->n_rows; }
    return run_pair<1, false, true>(ma, wt, wt_rows, q, dev, st);
}

bool gemm_f32_ok(const F32Product& p) {
    return p.heads > 0 && gemm_tcgen05_shape_ok(p.M, p.N, p.K) && p.ldy % 4 == 0 && p.y_hs % 4 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(p.y_bf16) & 7) == 0 && (reinterpret_cast<uintptr_t>(p.w) & 15) == 0;
}

// Which kernel takes a product of M fp32 rows.  Up to 32 rows the few-rows kernel (N = 2048, K = 1024, 32 rows: 25 us on the 128 x 256
// tiles, 11 here; N = K = 2048: 42 and 22).
static bool dense_rows_few(int M) { return M <= kGemmFewRowsMost; }
// CTAs that share a 128 x 128 tile of the fp32-sum kernel: as many as the chip has room for, two k-blocks each at least.  Clusters of eight
// up to twelve tiles: more of them do not all find eight free SMs close to one another (three terms, us, with four / eight: 12 tiles K = 2048
// 13.3 / 10.5, 16 tiles K = 1024 9.9 / 14.8, K = 4096 20.4 / 25.2)
static int f32_splits(int tiles, int n_kb, int most, int sms) {
    int s = 1;
    while (2 * s <= most && tiles * 2 * s <= (s == 4 ? 96 : sms) && n_kb >= 4 * s) s *= 2;
    return s;
}
// Beyond 32 rows (and for bf16 rows) the fp32-sum kernel where its rounds of tiles are shorter than those of 128 x 256 tiles on one SM: its
// 128 x 128 tiles are twice as many, and where they leave the chip idle its clusters split K.  Three terms: a k-block of a round takes three quarters
// of one of 128 x 256 tiles (1.1 and 1.4 us).  One term: 21 to 20 units a k-block (100 rows N = 32768, K = 2048 21 us, pairs 33).  Pairs of SMs do not
// count here: they take 0.4 to 0.8 us a k-block (three terms) and 0.34 to 0.46 here (one), but their sums of all K products cut off and are two to ten
// times further off, so what has sums of 64 products keeps them (bf16 rows, all
// positive, 1024 x 2048 x 1024: 12.9 us and 1.7e-6 on pairs, 15.4 us and 8.9e-8 here; 2048 x 1024 x 1536 16.5 and 3.4e-6, 20.5 and 1.0e-7).
static bool dense_rows_f32(int terms, int M, int N, int K, int sms) {
    const int tm = (M + BM - 1) / BM, n_kb = (K + BK - 1) / BK;
    const long long narrow = (long long)tm * ((N + kFN - 1) / kFN), wide = (long long)tm * ((N + BN - 1) / BN);
    const int s = narrow < sms ? f32_splits((int)narrow, n_kb, 8, sms) : 1;
    const long long here = (narrow * s + sms - 1) / sms, there = (wide + sms - 1) / sms;
    const int kb = (n_kb + s - 1) / s;
    return terms == 1 ? here * (21 * kb + 100) < there * (20 * n_kb + 130) : here * kb * 3 < there * n_kb * 4;
}

// splits: the most CTAs that may share a tile (1: a sum's order does not depend on the rows beside it)
static cudaError_t run_gemm_f32(const F32Product& p, const void* a_terms, int terms, int splits, cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaError_t e = current_sms(&dev, &sms);
    const auto kernel = terms == 1 ? dia_gemm_f32_kernel<1> : dia_gemm_f32_kernel<kTerms>;
    if (e == cudaSuccess) e = terms == 1 ? ask_smem<dia_gemm_f32_kernel<1>>(dev, kFSmem) : ask_smem<dia_gemm_f32_kernel<kTerms>>(dev, kFSmem);
    if (e != cudaSuccess) return e;
    CUtensorMap ma, mb;
    if (!make_map(&ma, a_terms, (long long)terms * p.heads * p.M, p.K, BM) || !make_map(&mb, p.w, (long long)p.heads * p.N, p.K, kFN))
        return cudaErrorNotSupported;
    const int n_tiles = p.heads * ((p.N + kFN - 1) / kFN) * ((p.M + BM - 1) / BM), n_kb = (p.K + BK - 1) / BK;
    const int s = f32_splits(n_tiles, n_kb, splits, sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s > 1 ? n_tiles : std::min(n_tiles, sms), s);
    cfg.blockDim = dim3(kFThreads);
    cfg.dynamicSmemBytes = kFSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1;
    attr.val.clusterDim.y = s;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, ma, mb, p);
}

cudaError_t launch_gemm_f32(const F32Product& p, void* work, cudaStream_t st) {
    if (!gemm_f32_ok(p)) return cudaErrorNotSupported;
    split3_heads_kernel<<<p.M, 256, 0, st>>>(p.a, p.lda, p.a_hs, reinterpret_cast<__nv_bfloat16*>(work), p.heads, p.M, p.K);
    ++extra_launches();
    return run_gemm_f32(p, work, kTerms, 1, st);
}

static size_t few_rows_smem(int NB, int kb_per, int n_slots) {
    return 1024 + (size_t)n_slots * kTileBytes + (size_t)kb_per * NB * 128 + (size_t)(NB / 3 / 8 * 8) * BM * 4;
}
// CTAs of a cluster: enough of them to fill the chip, at least two k-blocks each (a rule on N and K alone, so that a row's sums do not
// depend on what shares its step)
static int few_rows_split(int N, int K) {
    const int tiles = (N + BM - 1) / BM, n_kb = (K + BK - 1) / BK;
    int s = 1;
    while (s < 8 && n_kb >= 4 * s && tiles * s < 120) s *= 2;
    return s;
}

bool gemm_few_rows_ok(const FewRowsProduct& p) {
    if (p.M <= 0 || p.M > kGemmFewRowsMost || p.N <= 0 || p.K < BK || p.K % 8 || p.lda % 4 || (reinterpret_cast<uintptr_t>(p.a) & 15) ||
        (reinterpret_cast<uintptr_t>(p.w) & 15))
        return false;
    const int n_kb = (p.K + BK - 1) / BK, s = few_rows_split(p.N, p.K), kb_per = (n_kb + s - 1) / s;
    return few_rows_smem(p.M <= 8 ? 32 : 96, kb_per, std::min(kb_per, 2)) <= kRSmemMost;
}

template <int NB>
static cudaError_t launch_few_rows(const FewRowsProduct& p, bool early, cudaStream_t st) {
    const int n_kb = (p.K + BK - 1) / BK, s = few_rows_split(p.N, p.K), kb_per = (n_kb + s - 1) / s;
    // two CTAs per SM where at least three slots fit: the next launch's weights are then requested while this one still runs
    int n_slots = std::min(kRSlotsMost, kb_per);
    while (n_slots > 3 && few_rows_smem(NB, kb_per, n_slots) > kRSmemMost / 2) --n_slots;
    while (few_rows_smem(NB, kb_per, n_slots) > kRSmemMost) --n_slots;
    const size_t smem = std::max<size_t>(few_rows_smem(NB, kb_per, n_slots), kRSmemLeast);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = ask_smem<dia_gemm_few_rows_kernel<NB>>(dev, kRSmemMost);
    if (e != cudaSuccess) return e;
    CUtensorMap mw;
    if (!make_map(&mw, p.w, p.N, p.K, BM)) return cudaErrorNotSupported;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + BM - 1) / BM, s);
    cfg.blockDim = dim3(kRThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = s;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, dia_gemm_few_rows_kernel<NB>, mw, p, kb_per, n_slots);
}

cudaError_t launch_gemm_few_rows(const FewRowsProduct& p, bool early, cudaStream_t st) {
    if (!gemm_few_rows_ok(p)) return cudaErrorNotSupported;
    return p.M <= 8 ? launch_few_rows<32>(p, early, st) : launch_few_rows<96>(p, early, st);
}

// Whether M fp32 rows go as two fp16 terms to the pair kernel with fp32 sums: beyond 128 rows, what the 128 x 128 tiles of three terms do not take.
bool gemm_half_ok(int M, int N, int K) {
    int dev = 0, sms = 0;
    if (M <= BM || N <= 0 || N % 4 || K < BK || K % BK) return false;
    if (current_sms(&dev, &sms) != cudaSuccess) return false;
    return !dense_rows_f32(kTerms, M, N, K, sms);
}

// k-blocks that the fp32-sum kernel takes for M fp32 rows, one after the other, or 0 where launch_gemm_tcgen05 does not sum them in fp32 by itself
int gemm_sums_blocks(int M, int N, int K, bool always) {
    int dev = 0, sms = 0;
    if (dense_rows_few(M)) return 1;
    if (current_sms(&dev, &sms) != cudaSuccess || (!always && !dense_rows_f32(kTerms, M, N, K, sms))) return 0;
    const int tiles = (M + BM - 1) / BM * ((N + kFN - 1) / kFN), n_kb = (K + BK - 1) / BK, s = tiles < sms ? f32_splits(tiles, n_kb, 8, sms) : 1;
    return (tiles * s + sms - 1) / sms * ((n_kb + s - 1) / s);
}

cudaError_t launch_prepare_half(const void* w, int src_bf16, void* wt, float* mag, int* inexact, int K, int N, cudaStream_t st) {
    cudaError_t e = make_ran_out(st);
    if (e == cudaSuccess) e = cudaMemsetAsync(mag, 0, (size_t)N * 4, st);
    if (e != cudaSuccess) return e;
    column_magnitudes_kernel<<<dim3((N + 255) / 256, (K + 63) / 64), 256, 0, st>>>(w, src_bf16, reinterpret_cast<uint32_t*>(mag), K, N);
    transpose_to_half_kernel<<<dim3((N + 31) / 32, (K + 31) / 32), dim3(32, 8), 0, st>>>(w, src_bf16, mag, reinterpret_cast<__half*>(wt), inexact, K, N);
    ++extra_launches();
    return cudaGetLastError();
}

template <int TERMS>
static void split_rows(const float* x, const float* norm_w, float eps, bool gated, void* out, float* row_inv, int M, int K, cudaStream_t st) {
    const int aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(norm_w)) & 15) == 0;
    if (gated) split_rows_kernel<TERMS, true><<<M, 256, 0, st>>>(x, nullptr, 0.f, out, row_inv, M, K, aligned);
    else split_rows_kernel<TERMS, false><<<M, 256, 0, st>>>(x, norm_w, eps, out, row_inv, M, K, aligned);
}

// y = [residual +] x W for fp32 rows: two fp16 terms and fp32 sums of pieces of 256 products, on pairs of SMs.
cudaError_t launch_gemm_half(const float* x, const float* norm_w, float eps, bool gated, const void* wt, const float* mag, const float* residual, float* y,
                             void* workspace, int M, int N, int K, cudaStream_t st) {
    if (M <= 0 || N <= 0 || N % 4 || K < BK || K % BK || (gated && norm_w)) return cudaErrorNotSupported;
    __half* const terms = reinterpret_cast<__half*>(workspace);
    float* const row_inv = reinterpret_cast<float*>(terms + 2 * (size_t)M * K);
    split_rows<2>(x, norm_w, eps, gated, terms, row_inv, M, K, st);
    ++extra_launches();
    CUtensorMap ma;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!make_map(&ma, terms, 2LL * M, K, BM)) return cudaErrorNotSupported;
    PairProduct q{};
    q.y = y; q.residual = residual; q.M = M; q.N = N; q.K = K;
    q.row_inv = row_inv; q.col_mag = mag;
    return run_pair<2, true>(ma, wt, N, q, dev, st);
}

// fp32 activations: the three-term split (with the row's RMSNorm in front when norm_w is given, or with the gate of [M][2][K] rows), then
// the kernel; sums: the one of fp32 sums, whatever is the faster one
cudaError_t launch_gemm_tcgen05(const float* x, const float* norm_w, float eps, bool gated, const void* wt, const float* residual,
                                float* y, void* workspace, int M, int N, int K, cudaStream_t st, bool sums) {
    if (M <= 0 || N % 4 || N <= 0 || K % BK || K < BK || (gated && norm_w)) return cudaErrorNotSupported;
    const long long n = (long long)M * K;
    FewRowsProduct few{x, K, wt, y, N, M, N, K, 0, residual};
    if (dense_rows_few(M)) {
        const bool made = norm_w || gated;                    // (the rows lie in the workspace)
        if (made) few.a = reinterpret_cast<const float*>(workspace);
        // (the rows are read while outputs are written)
        const bool apart = made || x + n <= y || y + (long long)M * N <= x;
        if (apart && gemm_few_rows_ok(few)) {
            if (made) {
                split_rows<0>(x, norm_w, eps, gated, workspace, nullptr, M, K, st);
                ++extra_launches();
            }
            return launch_gemm_few_rows(few, false, st);
        }
    }
    split_rows<kTerms>(x, norm_w, eps, gated, workspace, nullptr, M, K, st);
    ++extra_launches();
    const F32Product wide{nullptr, 0, 0, wt, y, N, N, nullptr, 1, M, N, K, 1.f, 0, nullptr, 0, 0, residual};
    int dev = 0, sms = 0;
    const cudaError_t e = current_sms(&dev, &sms);
    if (e != cudaSuccess) return e;
    if ((sums || dense_rows_f32(kTerms, M, N, K, sms)) && gemm_f32_ok(wide)) return run_gemm_f32(wide, workspace, kTerms, 8, st);
    const GemmEpilogue ep{residual, nullptr, nullptr, 0.f, nullptr};
    return launch_gemm_tcgen05_bf16(workspace, kTerms, wt, N, y, M, N, K, ep, nullptr, st);
}

}  // namespace dia
