// lm_attention.cu - softmax attention of a handful of rows (decoding) over the pages, split over the keys (sm_100a).
//
//   few_rows_attention_kernel   grouped-query attention (temperature, tanh cap, linear distance bias, a window that keeps the first tokens,
//                               chunks, sink, elementwise gate) and attention over cached latents (the value is the head of the key row), for
//                               up to kAttnRowsKernelMax rows
//
// A CTA takes one (row, up to HT query heads of one key/value head, share of the keys).  Tiles of 32 keys are gathered into shared memory, the
// next one while the last is computed (asynchronous 16-byte copies).  Scores: lane = key, every warp an eighth of the channels for all heads, so
// that an element of a key is read once; a warp per head adds the eight parts and does the online softmax; then thread = channel, a part of
// the tile's keys each where there are fewer channels than threads.  The CTAs of a cluster (shares next to one another) merge their sums
// through each other's shared memory, a part of the outputs each; at most four clusters are left per row and head group, and the last of them
// to arrive merges those, again with all its CTAs.
//
// Bound: latencies (a launch, page numbers, the first tile, four barriers per tile, the merges), then the keys' and values' bytes.  us from the
// kernel before to the end, a warp per key with a dependent softmax per key and one merging CTA / here, over 1000 cached keys: 16 heads of 128
// over 4, one row 16 / 13, eight 53 / 33; 16 heads over latent rows of 256 + 32, one row 34 / 20, eight 34 / 29.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "gemm_tcgen05.h"
#include "lm_device.cuh"
#include "lm_internal.h"

namespace lm {
namespace {

constexpr int kFewKeys = 32, kFewThreads = 256, kFewWarps = 8, kFewCluster = 8;
// Keys of a CTA at least, unless one cluster has room for all: a second cluster costs a merge through global memory (four layers of width 2048, steps of
// one and of eight rows, us: over 100 keys 275 and 356 with all 32 CTAs, 257 and 319 with one cluster; over 600 keys with 16, 32 and 64 keys a CTA 277, 276
// and 291, 372, 368 and 382)
constexpr int kFewLeast = 32;

__device__ __forceinline__ uint32_t shared_at(const void* local, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return a;
}
__device__ __forceinline__ float remote(const float* local, uint32_t rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(shared_at(local, rank)) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// floats of shared memory: queries, key tiles, value tiles, parts of the scores (later the sums), weights, statistics
__host__ __device__ inline int few_smem_floats(int HT, int kdim, int vdim, bool shared_kv) {
    return HT * kdim + 2 * kFewKeys * (kdim + 4) + (shared_kv ? 0 : 2 * kFewKeys * vdim) + HT * kFewThreads + HT * kFewKeys + HT * (4 + kFewCluster);
}

}  // namespace

template <int HT>
__global__ void __launch_bounds__(kFewThreads)
few_rows_attention_kernel(const __grid_constant__ FewAttention p, int cluster_bits) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_last;
    pdl_release();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cluster = 1 << cluster_bits, sp = blockIdx.x, rank = sp & (cluster - 1), cl = sp >> cluster_bits, r = blockIdx.z;
    const int rep = p.heads / p.kv_heads, chunks = (rep + HT - 1) / HT, g = blockIdx.y / chunks, h0 = g * rep + (blockIdx.y % chunks) * HT;
    const int nh = min(HT, (g + 1) * rep - h0), kdim = p.kdim, vdim = p.vdim, KS = kdim + 4, K4 = kdim >> 2;
    float* Q = sm;                                            // [HT][kdim]
    float* Kt = Q + HT * kdim;                                // [2][32][KS]
    float* Vt = p.shared_kv ? Kt : Kt + 2 * kFewKeys * KS;    // [2][32][vdim]
    const int VS = p.shared_kv ? KS : vdim;
    float* parts = p.shared_kv ? Kt + 2 * kFewKeys * KS : Vt + 2 * kFewKeys * vdim;      // [8][HT][32] of a tile's scores; at the end the sums,
    float* sums = parts;                                      // [HT][256]: key groups x channels
    float* P = parts + HT * kFewThreads;                      // [HT][32]
    float* stat = P + HT * kFewKeys;                          // [HT] corrections, then denominators of the cluster
    float *m_s = stat + HT, *l_s = m_s + HT, *all_m = l_s + HT, *w_s = all_m + HT;      // w_s: [HT][8] weights of the cluster's shares
    pdl_wait();
    const int i = p.row_pos[r], lo = first_key(i, p.window, p.chunk), n_keep = p.window > 0 ? min(p.keep_first, lo) : 0;
    // as many clusters as the keys that are there fill (the grid has room for those that there may be)
    static_assert(kFewLeast == 32, "a shift below");
    const int n_keys = n_keep + (i - lo + 1), shares = min((int)gridDim.x >> cluster_bits, ((n_keys - 1) >> (cluster_bits + 5)) + 1);
    if (cl >= shares) return;                                 // (all its CTAs)
    const int per = ((((n_keys - 1) >> cluster_bits) + shares) / shares + 3) & ~3, k0 = min(n_keys, sp * per), k1 = min(n_keys, k0 + per);
    const int* pages = p.table + (size_t)p.row_slot[r] * p.max_pages;
    auto gather = [&](int t0, int buf) {                      // keys t0 .. of the share: warp w rows 4 w .. + 3
        size_t at[4];
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int kk = t0 + warp * 4 + u, j = kk < n_keep ? kk : lo + (kk - n_keep);
            in[u] = kk < k1;
            at[u] = in[u] ? ((size_t)pages[j / p.page_size] * p.kv_heads + g) * p.page_size + j % p.page_size : 0;
        }
        for (int c = lane; c < K4; c += 32)
#pragma unroll
            for (int u = 0; u < 4; ++u) copy16(Kt + (buf * kFewKeys + warp * 4 + u) * KS + 4 * c, p.kcache + at[u] * kdim + 4 * c, in[u]);
        if (!p.shared_kv)
            for (int c = lane; c < vdim >> 2; c += 32)
#pragma unroll
                for (int u = 0; u < 4; ++u) copy16(Vt + (buf * kFewKeys + warp * 4 + u) * vdim + 4 * c, p.vcache + at[u] * vdim + 4 * c, in[u]);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (k0 < k1) gather(k0, 0);
    for (int c = tid; c < HT * K4; c += kFewThreads) {        // (heads beyond nh repeat the last one; they are not stored)
        const int hh = c / K4, d = 4 * (c - hh * K4);
        *reinterpret_cast<float4*>(Q + hh * kdim + d) = *reinterpret_cast<const float4*>(p.q + (size_t)r * p.ldq + (size_t)(h0 + min(hh, nh - 1)) * kdim + d);
    }
    // thread = channel of a value in one of the key groups
    const int W = vdim <= 64 ? 64 : vdim <= 128 ? 128 : 256, groups = kFewThreads / W, col = tid % W, grp = tid / W, gk = kFewKeys / groups;
    float acc[HT];
#pragma unroll
    for (int hh = 0; hh < HT; ++hh) acc[hh] = 0.f;
    constexpr int HW = (HT + kFewWarps - 1) / kFewWarps;      // heads of a warp in the softmax
    float m_run[HW], l_run[HW], mult[HW], slope[HW];
#pragma unroll
    for (int u = 0; u < HW; ++u) {
        const int h = h0 + min(warp + kFewWarps * u, nh - 1);
        m_run[u] = -CUDART_INF_F;
        l_run[u] = 0.f;
        mult[u] = p.scale * (p.temp ? p.temp[h] : 1.f);
        slope[u] = p.slopes ? p.slopes[h] : 0.f;
    }
    const float inv_cap = p.cap > 0.f ? 1.0f / p.cap : 0.f;
    const int c_per = (K4 + kFewWarps - 1) / kFewWarps, c_a = min(K4, warp * c_per), c_b = min(K4, c_a + c_per);
    int buf = 0;
    for (int t0 = k0; t0 < k1; t0 += kFewKeys, buf ^= 1) {
        const bool more = t0 + kFewKeys < k1;
        if (more) gather(t0 + kFewKeys, buf ^ 1);             // (its buffer was left behind the last barrier of the tile before)
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                      // the tile is there (and the queries, the first time)
        {
            const float* kp = Kt + (buf * kFewKeys + lane) * KS;
            float s[HT];
#pragma unroll
            for (int hh = 0; hh < HT; ++hh) s[hh] = 0.f;
#pragma unroll 2
            for (int c = c_a; c < c_b; ++c) {
                const float4 k = *reinterpret_cast<const float4*>(kp + 4 * c);
#pragma unroll
                for (int hh = 0; hh < HT; ++hh) {
                    const float4 q = *reinterpret_cast<const float4*>(Q + hh * kdim + 4 * c);
                    s[hh] = fmaf(q.x, k.x, s[hh]); s[hh] = fmaf(q.y, k.y, s[hh]); s[hh] = fmaf(q.z, k.z, s[hh]); s[hh] = fmaf(q.w, k.w, s[hh]);
                }
            }
#pragma unroll
            for (int hh = 0; hh < HT; ++hh) parts[(warp * HT + hh) * kFewKeys + lane] = s[hh];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < HW; ++u) {
            const int hh = warp + kFewWarps * u;
            if (hh >= HT) break;
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < kFewWarps; ++w) s += parts[(w * HT + hh) * kFewKeys + lane];
            s *= mult[u];
            if (p.cap > 0.f) s = p.cap * tanhf(s * inv_cap);
            const int kk = t0 + lane, j = kk < n_keep ? kk : lo + (kk - n_keep);
            const bool in = kk < k1;
            if (p.slopes) s -= slope[u] * (float)(i - j);
            const float m_new = fmaxf(m_run[u], warp_max(in ? s : -CUDART_INF_F)), base = m_new == -CUDART_INF_F ? 0.f : m_new;
            const float corr = expf(m_run[u] - base), e = in ? expf(s - base) : 0.f;
            l_run[u] = l_run[u] * corr + warp_sum(e);
            m_run[u] = m_new;
            P[hh * kFewKeys + lane] = e;
            if (lane == 0) stat[hh] = corr;
        }
        __syncthreads();
        if (col < vdim) {
#pragma unroll
            for (int hh = 0; hh < HT; ++hh) acc[hh] *= stat[hh];
            const float* vp = Vt + (buf * kFewKeys + grp * gk) * VS + col;
#pragma unroll 2
            for (int j = 0; j < gk; j += 4) {
                const float v0 = vp[j * VS], v1 = vp[(j + 1) * VS], v2 = vp[(j + 2) * VS], v3 = vp[(j + 3) * VS];
#pragma unroll
                for (int hh = 0; hh < HT; ++hh) {
                    const float4 e = *reinterpret_cast<const float4*>(P + hh * kFewKeys + grp * gk + j);
                    acc[hh] = fmaf(e.x, v0, acc[hh]); acc[hh] = fmaf(e.y, v1, acc[hh]); acc[hh] = fmaf(e.z, v2, acc[hh]); acc[hh] = fmaf(e.w, v3, acc[hh]);
                }
            }
        }
        __syncthreads();                                      // the tile, the weights and the corrections are read
    }
    // ---- the share's sums, then the cluster's ----
#pragma unroll
    for (int hh = 0; hh < HT; ++hh) sums[hh * kFewThreads + tid] = acc[hh];
#pragma unroll
    for (int u = 0; u < HW; ++u) {
        const int hh = warp + kFewWarps * u;
        if (hh < HT && lane == 0) { m_s[hh] = m_run[u]; l_s[hh] = l_run[u]; }
    }
    if (groups > 1) {                                         // (the same for all CTAs) the key groups' sums, in their order
        __syncthreads();
        if (grp == 0)
#pragma unroll
            for (int hh = 0; hh < HT; ++hh) {
                float v = acc[hh];
                for (int q = 1; q < groups; ++q) v += sums[hh * kFewThreads + q * W + col];
                sums[hh * kFewThreads + col] = v;
            }
    }
    cluster_barrier();
    for (int hh = warp; hh < nh; hh += kFewWarps) {           // a warp per head: lane = share of the cluster
        const float ms = lane < cluster ? remote(m_s + hh, lane) : -CUDART_INF_F, ls = lane < cluster ? remote(l_s + hh, lane) : 0.f;
        const float m = warp_max(ms), w = ms == -CUDART_INF_F ? 0.f : expf(ms - m), l = warp_sum(ls * w);
        if (lane < kFewCluster) w_s[hh * kFewCluster + lane] = w;
        if (lane == 0) { all_m[hh] = m; stat[hh] = l; }
    }
    __syncthreads();
    const size_t stride = (size_t)vdim + 2;
    auto finish = [&](int hh, int c, float o) {
        const int h = h0 + hh;
        o *= p.out_scale;
        if (p.gate) o *= sigmoidf_(p.gate[(size_t)r * p.ldg + (size_t)h * vdim + c]);
        if (p.head_gate) o *= p.head_gate[(size_t)r * p.ldg + h];
        const size_t at = (size_t)r * p.ldo + (size_t)h * vdim + c;
        p.out[at] = o;
        if (p.out_bf16) reinterpret_cast<__nv_bfloat16*>(p.out_bf16)[at] = __float2bfloat16_rn(o);
    };
    auto denominator = [&](int h, float m, float l) {         // 1 / (l + sink's term) for sums relative to the maximum m
        const float sk = p.sink ? p.sink[h] : -CUDART_INF_F, top = fmaxf(m, sk), f = m == -CUDART_INF_F ? 0.f : expf(m - top);
        const float all = l * f + (p.sink ? expf(sk - top) : 0.f);
        return all > 0.f ? f / all : all == all ? 0.f : all;
    };
    for (int idx = rank * kFewThreads + tid; idx < nh * vdim; idx += cluster * kFewThreads) {
        const int hh = idx / vdim, c = idx - hh * vdim;
        float v[kFewCluster], o = 0.f;
#pragma unroll
        for (int t = 0; t < kFewCluster; ++t) v[t] = t < cluster ? remote(sums + hh * kFewThreads + c, t) : 0.f;
#pragma unroll
        for (int t = 0; t < kFewCluster; ++t) o = fmaf(v[t], w_s[hh * kFewCluster + t], o);
        if (shares == 1) finish(hh, c, o * denominator(h0 + hh, all_m[hh], stat[hh]));
        else p.part[((size_t)(r * p.heads + h0 + hh) * shares + cl) * stride + 2 + c] = o;
    }
    if (shares == 1) {
        cluster_barrier();                                    // (nobody's sums go while another CTA reads them)
        return;
    }
    if (rank == 0 && tid < nh) {
        float* dst = p.part + ((size_t)(r * p.heads + h0 + tid) * shares + cl) * stride;
        dst[0] = all_m[tid];
        dst[1] = stat[tid];
    }
    __threadfence();
    cluster_barrier();
    if (rank == 0 && tid == 0) {
        unsigned* cnt = p.arrived + (size_t)r * gridDim.y + blockIdx.y;
        s_last = atomicAdd(cnt, 1u) == (unsigned)shares - 1u;
        if (s_last) *cnt = 0u;                                // back to zero for the next step
        __threadfence();
    }
    cluster_barrier();
    int last;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(last) : "r"(shared_at(&s_last, 0)) : "memory");
    if (last) {
        __threadfence();
        for (int idx = rank * kFewThreads + tid; idx < nh * vdim; idx += cluster * kFewThreads) {
            const int hh = idx / vdim, c = idx - hh * vdim;
            const float* src = p.part + (size_t)(r * p.heads + h0 + hh) * shares * stride;
            float ms[4], ls[4], os[4], m = -CUDART_INF_F;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                ms[t] = t < shares ? __ldcg(src + t * stride) : -CUDART_INF_F;
                ls[t] = t < shares ? __ldcg(src + t * stride + 1) : 0.f;
                os[t] = t < shares ? __ldcg(src + t * stride + 2 + c) : 0.f;
                m = fmaxf(m, ms[t]);
            }
            float l = 0.f, o = 0.f;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float w = ms[t] == -CUDART_INF_F ? 0.f : expf(ms[t] - m);
                l = fmaf(ls[t], w, l);
                o = fmaf(os[t], w, o);
            }
            finish(hh, c, o * denominator(h0 + hh, m, l));
        }
    }
    cluster_barrier();                                        // (rank 0's word is read)
}

// CTAs of a row and head group that share its keys: a power of two, for up to four CTAs per SM, and 16 keys each at least where the window
// or the chunk bounds them
static int few_shares(int others, long long max_keys, int sms) {
    static_assert(kAttnSplitsMax <= 4 * kFewCluster, "clusters that the last merge reads");
    int S = 1;
    while (S * 2 <= kAttnSplitsMax && others * S * 2 <= 4 * sms && (long long)S * 16 < max_keys) S *= 2;
    return S;
}
static int few_heads(const FewAttention& p) {
    const int rep = p.heads / p.kv_heads;
    return rep >= 9 ? 16 : rep >= 5 ? 8 : rep >= 3 ? 4 : 2;
}

// A key head that one query head reads stays with the kernels that give a key to a warp: nothing is shared between heads here (a model's step
// with 4 heads over 4 in half of its layers, us, there / here: 6 rows over 134 keys 172 / 182, 4 rows over 865 203 / 207)
bool few_rows_attention_ok(const FewAttention& p) {
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (p.heads <= 0 || p.kv_heads <= 0 || p.heads % p.kv_heads || p.heads == p.kv_heads || p.kdim <= 0 || p.vdim <= 0 || p.vdim > kFewThreads || p.kdim % 4 || p.vdim % 4 ||
        p.ldq % 4 || !al(p.q) || !al(p.kcache) || !al(p.vcache))
        return false;
    return few_smem_floats(few_heads(p), p.kdim, p.vdim, p.shared_kv) * 4 <= 220 * 1024;
}

template <int HT>
static cudaError_t launch_few(const FewAttention& p, int M, cudaStream_t st) {
    const size_t smem = (size_t)few_smem_floats(HT, p.kdim, p.vdim, p.shared_kv) * 4;
    int dev = 0, sms = 0;
    cudaError_t e = dia::current_sms(&dev, &sms);
    if (e == cudaSuccess) e = dia::ask_smem<few_rows_attention_kernel<HT>>(dev, 220 * 1024);
    if (e != cudaSuccess) return e;
    const int rep = p.heads / p.kv_heads, groups = p.kv_heads * ((rep + HT - 1) / HT);
    long long max_keys = p.window > 0 ? (long long)p.window + p.keep_first : (long long)p.max_pages * p.page_size;
    if (p.chunk > 0) max_keys = std::min<long long>(max_keys, (long long)p.chunk + (p.window > 0 ? p.keep_first : 0));
    const int S = few_shares(M * groups, max_keys, sms), cluster_bits = S >= kFewCluster ? 3 : S >= 4 ? 2 : S >= 2 ? 1 : 0;
    static_assert(kFewCluster == 8, "its bits");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S, groups, M);
    cfg.blockDim = dim3(kFewThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1 << cluster_bits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, few_rows_attention_kernel<HT>, p, cluster_bits);
}

cudaError_t launch_few_rows_attention(const FewAttention& p, int M, cudaStream_t st) {
    if (M <= 0 || M > kAttnRowsKernelMax || !few_rows_attention_ok(p)) return cudaErrorNotSupported;
    switch (few_heads(p)) {
        case 16: return launch_few<16>(p, M, st);
        case 8: return launch_few<8>(p, M, st);
        case 4: return launch_few<4>(p, M, st);
        default: return launch_few<2>(p, M, st);
    }
}

}  // namespace lm
