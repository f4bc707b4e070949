// lm_delta.cu - the delta rule with one decay per head, many tokens of a sequence at a time (sm_100a).
//
//   S <- a_t S,  u_t = b_t (v_t - S^T k_t),  S <- S + k_t u_t^T,  o_t = S^T q_t          (S [dim][vdim], fp32; see lm_scan.cu)
//
// 32 tokens are one chunk.  With S0 the state in front of it, A_t = a_1 .. a_t and D_tj = a_j+1 .. a_t (products, not quotients: a decay may be 0),
//   (I + L) U = diag(b) (V - diag(A) K S0),   L_tj = b_t D_tj (k_t . k_j) for j < t
//   O = diag(A) Q S0 + P U,                   P_tj = D_tj (q_t . k_j) for j <= t
//   S = A_32 S0 + (diag(D_32) K)^T U
// so that a token no longer waits for the one in front of it: the triangle is inverted once per (chunk, head), of which a step has hundreds, and the
// state passes a chunk in four small products.
//
//   delta_chunk_kernel     per (chunk, head): T = (I + L)^-1 diag(b), P, A and D_32 to the room.  Column j of the inverse is the work of a lane (forward
//                          substitution in registers).  Keys are unit vectors and b <= 1, so T's entries are no larger than 1.
//   delta_columns_kernel   per (sequence, head, 16 value columns): walks the chunks, the longest sequences first.  256 threads: thread (rg, hv, cg) sums half
//                          hv of the channels of K S0 and Q S0 for tokens rg and rg + 16, then owns token rg + 16 hv and columns 2 cg, 2 cg + 1 of U and O,
//                          and dim / 32 channels of the same columns of S in registers (a copy in shared memory feeds the products).
//                          All arithmetic is fp32x2 multiply-adds, pairs along the summed index.
//
// Bound: the loads from shared memory that feed the multiply-adds (16 bytes for each lane: four cycles an instruction, and 2.7 multiply-adds for each): a
// chunk of 32 tokens takes a block 6800 cycles by itself and 10000 beside another, where the serial scan takes 24000.  Layer of 16 heads of 128, us, serial
// scan / chunks: 1024 tokens 323 / 243, 4096 1102 / 729, 2048 beside 1 684 / 399, prompts of 1024, 700, 513, 37 and 1 tokens 574 / 390 (407 with the short ones behind
// the long ones instead of beside them; the blocks in the sequences' order took 68 more, 32 columns a block, which read a third less, 185); 4 heads of 64, 2000 tokens 488 / 256.
// A column's order of operations depends on its sequence's portion alone.  Sequences of fewer tokens stay with the serial scan.
#include <algorithm>
#include <atomic>

#include <cuda_runtime.h>
#include <stdint.h>

#include "fp32_pairs.cuh"
#include "gemm_tcgen05.h"
#include "lm_device.cuh"
#include "lm_internal.h"

namespace lm {

namespace {

constexpr int kC = kDeltaChunk, kCols = 16, kThreads = 128, kColThreads = 256, kTS = kC + 4;      // kTS: row stride of the triangles in shared memory
static_assert(kC == 32, "a lane per column of the triangle");

using dia::f2; using dia::pack2; using dia::fma2;
__device__ __forceinline__ float sum2(f2 v) {
    float x, y;
    dia::unpack2(v, x, y);
    return x + y;
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void copies_started() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_done_but() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct DeltaArgs {
    const float* in; int ld, q_off, k_off, v_off, b_off, a_off;
    int H, G, dim, vdim, n_seq;
    float* state;
    const int *seq_slot, *seq_row0, *seq_count, *row_pos;
    float* o; int ldo;
    float* room;                                              // [chunk][H][kDeltaChunkFloats]: T [t][j], P [t][j], A [t], D_32 [j]
};
// The chunks of sequence s are room places row0 / 32 + s on: no two sequences meet, and there are rows / 32 + sequences places
__device__ __forceinline__ int first_chunk(int row0, int s) { return row0 / kC + s; }

// rows t0 .. of a sequence's portion into shared memory, kC rows of DP channels with stride LD (zeros beyond dim and the portion)
template <int DP, int LD, int THREADS>
__device__ __forceinline__ void stage_rows(float* dst, const float* src, int ld, int dim, int nt) {
    for (int i = threadIdx.x; i < kC * (DP / 4); i += THREADS) {
        const int t = i / (DP / 4), c = 4 * (i % (DP / 4));
        const bool ok = t < nt && c < dim;
        copy16(dst + t * LD + c, src + (ok ? (size_t)t * ld + c : 0), ok);
    }
}

template <int DP>
__global__ void __launch_bounds__(kThreads)
delta_chunk_kernel(const DeltaArgs p) {
    constexpr int LD = DP + 4;
    __shared__ __align__(16) float sk[kC * LD], sq[kC * LD], sg[kC * kTS], sp[kC * kTS], sd[kC * kTS];
    __shared__ float sa[kC], sb[kC];
    __shared__ int s_seq;
    pdl_release();
    pdl_wait();
    const int h = blockIdx.y, g = h / (p.H / p.G), tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) s_seq = -1;
    __syncthreads();
    for (int s = tid; s < p.n_seq; s += kThreads) {
        const int first = first_chunk(p.seq_row0[s], s), n = p.seq_count[s];
        if (n >= kChunkTokensMin && (int)blockIdx.x >= first && (int)blockIdx.x < first + (n + kC - 1) / kC) s_seq = s;
    }
    __syncthreads();
    if (s_seq < 0) return;
    const int row0 = p.seq_row0[s_seq], t0 = ((int)blockIdx.x - first_chunk(row0, s_seq)) * kC, nt = min(kC, p.seq_count[s_seq] - t0);
    const float* base = p.in + (size_t)(row0 + t0) * p.ld;
    stage_rows<DP, LD, kThreads>(sk, base + p.k_off + g * p.dim, p.ld, p.dim, nt);
    stage_rows<DP, LD, kThreads>(sq, base + p.q_off + g * p.dim, p.ld, p.dim, nt);
    copies_started();
    if (tid < kC) {                                           // (tokens beyond the portion: no decay, no write)
        sa[tid] = tid < nt ? base[(size_t)tid * p.ld + p.a_off + h] : 1.f;
        sb[tid] = tid < nt ? base[(size_t)tid * p.ld + p.b_off + h] : 0.f;
    }
    copies_done_but<0>();
    __syncthreads();
    if (tid < kC) {                                           // decays: column j of D, a lane each (products of up to 31 factors: rounded once)
        double d = 1.0;
#pragma unroll
        for (int t = 0; t < kC; ++t) {
            if (t > lane) d *= (double)sa[t];
            sd[t * kTS + lane] = t >= lane ? (float)d : 0.f;
        }
    }
    // the products: threads 0 .. 63 keys with keys, 64 .. 127 queries with keys, 4 x 4 each
    {
        const float* rows = tid < 64 ? sk : sq;
        const int tr = (tid & 63) >> 3, tc = tid & 7;         // rows tr + 8 i, columns tc + 8 j
        f2 acc[4][4] = {};
#pragma unroll 4
        for (int c = 0; c < DP; c += 4) {
            ulonglong2 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[i] = *reinterpret_cast<const ulonglong2*>(rows + (tr + 8 * i) * LD + c);
                b[i] = *reinterpret_cast<const ulonglong2*>(sk + (tc + 8 * i) * LD + c);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i].y, b[j].y, fma2(a[i].x, b[j].x, acc[i][j]));
        }
        float* dst = tid < 64 ? sg : sp;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[(tr + 8 * i) * kTS + tc + 8 * j] = sum2(acc[i][j]);
    }
    __syncthreads();
    for (int i = tid; i < kC * kC; i += kThreads) {
        const int t = i / kC, j = i % kC;
        const float d = sd[t * kTS + j];
        sg[t * kTS + j] = j < t ? sb[t] * d * sg[t * kTS + j] : 0.f;
        sp[t * kTS + j] = j <= t ? d * sp[t * kTS + j] : 0.f;
    }
    __syncthreads();
    float* out = p.room + ((size_t)blockIdx.x * p.H + h) * kDeltaChunkFloats;
    if (tid < 32) {
        float x[kC];                                          // column `lane` of (I + L)^-1
#pragma unroll
        for (int t = 0; t < kC; ++t) {
            float v[4] = {t == lane ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < t; ++i) v[i & 3] = fmaf(-sg[t * kTS + i], x[i], v[i & 3]);
            x[t] = (v[0] + v[1]) + (v[2] + v[3]);
        }
        const float b = sb[lane];
#pragma unroll
        for (int t = 0; t < kC; ++t) out[t * kC + lane] = t >= lane ? x[t] * b : 0.f;
        out[2 * kC * kC + lane] = sa[0] * sd[lane * kTS];     // A
        out[2 * kC * kC + kC + lane] = sd[(kC - 1) * kTS + lane];
    } else {
        for (int i = tid - 32; i < kC * kC; i += kThreads - 32) out[kC * kC + i] = sp[i / kC * kTS + i % kC];
    }
}

// Shared memory of delta_columns_kernel, in floats: keys (two chunks), queries, values (two), triangles T and P and the two vectors, the state as pairs
// along the channel, halves of K S and Q S, R and U as pairs along the token, U times D_32 twice over
template <int DP>
struct Columns {
    static constexpr int LD = DP + 4;
    static constexpr int k = 0, q = k + 2 * kC * LD, v = q + kC * LD, tri = v + 2 * kC * kCols, vec = tri + 2 * kC * kTS, s = vec + 2 * kC,
                         x = s + DP * kCols, r = x + kCols / 4 * kColThreads, u = r + kC * kCols, ud = u + kC * kCols, floats = ud + 2 * kC * kCols;
};

template <int DP>
__global__ void __launch_bounds__(kColThreads, 2)
delta_columns_kernel(const DeltaArgs p) {
    using M = Columns<DP>;
    constexpr int LD = M::LD, ND = DP / 64, NC = kCols / 8, RP = kColThreads / (DP / 4);      // channel pairs and columns of S per thread, rows per pass of the staging
    extern __shared__ __align__(16) float sh[];
    pdl_wait();
    pdl_release();                                            // (behind the wait: the scan of the short sequences relies on it)
    // the longest sequences' blocks start first
    __shared__ int s_seq;
    for (int i = threadIdx.x; i < p.n_seq; i += kColThreads) {
        const int mine = p.seq_count[i];
        int longer = 0;
        for (int e = 0; e < p.n_seq; ++e) {
            const int other = p.seq_count[e];
            longer += other > mine || (other == mine && e < i);
        }
        if (longer == (int)blockIdx.z) s_seq = i;
    }
    __syncthreads();
    const int s = s_seq, h = blockIdx.y, col0 = blockIdx.x * kCols, g = h / (p.H / p.G);
    const int n = p.seq_count[s];
    if (n < kChunkTokensMin) return;
    // two halves of 128 threads: half hv sums channels hv DP / 2 .. of K S and Q S for tokens rg and rg + 16, then has token rg + 16 hv
    const int tid = threadIdx.x, hv = tid >> 7, rg = (tid >> 3) & 15, cg = tid & 7, c0 = NC * cg, tok = rg + 16 * hv;
    const int slot = p.seq_slot[s], row0 = p.seq_row0[s];
    const float* const base = p.in + (size_t)row0 * p.ld;
    const float* const room = p.room + ((size_t)first_chunk(row0, s) * p.H + h) * kDeltaChunkFloats;
    const bool from_zero = p.row_pos[row0] == 0;
    const int d0 = (2 * rg + hv) * (2 * ND);                  // channels of this thread's part of S

    // staging: this thread's row and channels of the first pass
    const int st_t = tid / (DP / 4), st_c = 4 * (tid % (DP / 4)), sv_t = tid / kCols, sv_c = tid % kCols;
    const bool st_ok = st_c < p.dim, sv_ok = col0 + sv_c < p.vdim;
    const float* const k_src = base + (size_t)st_t * p.ld + p.k_off + g * p.dim + (st_ok ? st_c : 0);
    const float* const q_src = base + (size_t)st_t * p.ld + p.q_off + g * p.dim + (st_ok ? st_c : 0);
    const float* const v_src = base + (size_t)sv_t * p.ld + p.v_off + h * p.vdim + (sv_ok ? col0 + sv_c : 0);
    auto stage_rows_of = [&](float* dst, const float* src, int t0) {
#pragma unroll
        for (int i = 0; i < kC / RP; ++i) {
            const bool ok = st_ok && t0 + st_t + i * RP < n;
            copy16(dst + (st_t + i * RP) * LD + st_c, ok ? src + (size_t)(t0 + i * RP) * p.ld : base, ok);
        }
    };
    auto stage_inputs = [&](int t0, int buf) {
        stage_rows_of(sh + M::k + buf * kC * LD, k_src, t0);
        stage_rows_of(sh + M::q, q_src, t0);
#pragma unroll
        for (int i = 0; i < kC * kCols / kColThreads; ++i) {
            const int t = sv_t + i * (kColThreads / kCols);
            const bool ok = sv_ok && t0 + t < n;
            copy4(sh + M::v + buf * kC * kCols + t * kCols + sv_c, ok ? v_src + (size_t)(t0 + i * (kColThreads / kCols)) * p.ld : base, ok);
        }
    };
    auto stage_triangles = [&](int t0) {                      // what the kernel in front has made of the chunk
        const float* src = room + (size_t)(t0 / kC) * p.H * kDeltaChunkFloats;
#pragma unroll
        for (int i = 0; i < 2 * kC * kC / 4 / kColThreads; ++i) {
            const int e = 4 * (tid + i * kColThreads);
            copy16(sh + M::tri + e / kC * kTS + e % kC, src + e, true);
        }
        if (tid < 2 * kC / 4) copy16(sh + M::vec + 4 * tid, src + 2 * kC * kC + 4 * tid, true);
    };
    stage_inputs(0, 0);
    copies_started();
    stage_triangles(0);
    copies_started();

    f2 S[ND][NC];                                             // channels d0 + 2 i, + 1 of columns c0 ..
#pragma unroll
    for (int e = 0; e < NC; ++e) {
        const float* st = p.state + (((size_t)slot * p.H + h) * p.vdim + col0 + c0 + e) * p.dim;
#pragma unroll
        for (int i = 0; i < ND; ++i) {
            const int d = d0 + 2 * i;
            S[i][e] = !from_zero && col0 + c0 + e < p.vdim && d < p.dim ? *reinterpret_cast<const f2*>(st + d) : 0ull;
        }
    }
    auto put_state = [&] {
#pragma unroll
        for (int i = 0; i < ND; ++i)
#pragma unroll
            for (int e = 0; e < NC; e += 2) *reinterpret_cast<ulonglong2*>(sh + M::s + (d0 / 2 + i) * 2 * kCols + 2 * (c0 + e)) = make_ulonglong2(S[i][e], S[i][e + 1]);
    };
    put_state();
    // row tok of a lower triangle m times x: only what a row has (zero times an infinity of a later token is no zero).  A warp's rows lie in one
    // block of four
    auto triangle = [&](const float* m, const float* x, float (&y)[NC]) {
        const float* row = m + tok * kTS;
        const int e = rg & 3, last = tok >> 2;                // the block with the diagonal
        f2 a[NC] = {};
#pragma unroll 2
        for (int b = 0; b <= last; ++b) {
            const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(row + 4 * b);
#pragma unroll
            for (int i = 0; i < NC; i += 2) {
                ulonglong2 u = *reinterpret_cast<const ulonglong2*>(x + 2 * b * 2 * kCols + 2 * (c0 + i)), w = *reinterpret_cast<const ulonglong2*>(x + (2 * b + 1) * 2 * kCols + 2 * (c0 + i));
                if (b == last) {
                    if (e < 1) { u.x &= 0xffffffffull; u.y &= 0xffffffffull; }
                    if (e < 2) w.x = w.y = 0;
                    if (e == 2) { w.x &= 0xffffffffull; w.y &= 0xffffffffull; }
                }
                a[i] = fma2(z.y, w.x, fma2(z.x, u.x, a[i]));
                a[i + 1] = fma2(z.y, w.y, fma2(z.x, u.y, a[i + 1]));
            }
        }
#pragma unroll
        for (int i = 0; i < NC; ++i) y[i] = sum2(a[i]);
    };
    for (int t0 = 0, buf = 0; t0 < n; t0 += kC, buf ^= 1) {
        copies_done_but<1>();                                 // (keys, queries, values; the triangles may be on their way)
        __syncthreads();
        const float* sk = sh + M::k + buf * kC * LD;
        // ---- halves of K S and Q S ----
        float ks[NC], qs[NC];                                 // of token tok
        {
            const float* a0 = sk + rg * LD + hv * (DP / 2);
            const float* b0 = sh + M::q + rg * LD + hv * (DP / 2);
            const float* ss = sh + M::s + hv * (DP / 4) * 2 * kCols + 2 * c0;
            f2 acc[4][NC] = {};                               // K S of rg, rg + 16, Q S of rg, rg + 16
#pragma unroll 2
            for (int c = 0; c < DP / 2; c += 4) {
                const ulonglong2 x[4] = {*reinterpret_cast<const ulonglong2*>(a0 + c), *reinterpret_cast<const ulonglong2*>(a0 + 16 * LD + c),
                                         *reinterpret_cast<const ulonglong2*>(b0 + c), *reinterpret_cast<const ulonglong2*>(b0 + 16 * LD + c)};
#pragma unroll
                for (int e = 0; e < NC; e += 2) {
                    const ulonglong2 y0 = *reinterpret_cast<const ulonglong2*>(ss + c / 2 * 2 * kCols + 2 * e), y1 = *reinterpret_cast<const ulonglong2*>(ss + (c / 2 + 1) * 2 * kCols + 2 * e);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        acc[i][e] = fma2(x[i].y, y1.x, fma2(x[i].x, y0.x, acc[i][e]));
                        acc[i][e + 1] = fma2(x[i].y, y1.y, fma2(x[i].x, y0.y, acc[i][e + 1]));
                    }
                }
            }
            // the other half's token goes to it
            float4* x = reinterpret_cast<float4*>(sh + M::x);
#pragma unroll
            for (int e = 0; e < NC; e += 2) {
                float z[4][2];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    z[i][0] = sum2(acc[i][e]);
                    z[i][1] = sum2(acc[i][e + 1]);
                }
                x[e / 2 * kColThreads + (tid ^ 128)] = hv ? make_float4(z[0][0], z[0][1], z[2][0], z[2][1]) : make_float4(z[1][0], z[1][1], z[3][0], z[3][1]);
                ks[e] = hv ? z[1][0] : z[0][0]; ks[e + 1] = hv ? z[1][1] : z[0][1];
                qs[e] = hv ? z[3][0] : z[2][0]; qs[e + 1] = hv ? z[3][1] : z[2][1];
            }
        }
        copies_done_but<0>();                                 // the triangles
        __syncthreads();
        if (t0 + kC < n) stage_inputs(t0 + kC, buf ^ 1);      // (the queries have been read, the other keys in the turn before)
        copies_started();
        const float* tri = sh + M::tri;
        const float* vec = sh + M::vec;
        const float a_tok = vec[tok];
        // ---- R = V - A K S, as pairs along the token ----
        {
            float* r = sh + M::r + (tok >> 1) * 2 * kCols + (tok & 1);
#pragma unroll
            for (int e = 0; e < NC; e += 2) {
                const float4 other = reinterpret_cast<const float4*>(sh + M::x)[e / 2 * kColThreads + tid];
                ks[e] += other.x; ks[e + 1] += other.y; qs[e] += other.z; qs[e + 1] += other.w;
                const float2 v = *reinterpret_cast<const float2*>(sh + M::v + buf * kC * kCols + tok * kCols + c0 + e);
                r[2 * (c0 + e)] = fmaf(-a_tok, ks[e], v.x);
                r[2 * (c0 + e) + 2] = fmaf(-a_tok, ks[e + 1], v.y);
            }
        }
        __syncthreads();
        // ---- U = T R ----
        {
            float u[NC];
            triangle(tri, sh + M::r, u);
            const float d = vec[kC + tok];
            float* w = sh + M::u + (tok >> 1) * 2 * kCols + (tok & 1);
#pragma unroll
            for (int e = 0; e < NC; e += 2) {
                w[2 * (c0 + e)] = u[e];
                w[2 * (c0 + e) + 2] = u[e + 1];
                *reinterpret_cast<float4*>(sh + M::ud + tok * 2 * kCols + 2 * (c0 + e)) = make_float4(d * u[e], d * u[e], d * u[e + 1], d * u[e + 1]);
            }
        }
        __syncthreads();
        // ---- O = A Q S + P U ----
        {
            float y[NC];
            triangle(tri + kC * kTS, sh + M::u, y);
            if (t0 + tok < n) {
                float* o = p.o + (size_t)(row0 + t0 + tok) * p.ldo + h * p.vdim + col0 + c0;
#pragma unroll
                for (int e = 0; e < NC; ++e)
                    if (col0 + c0 + e < p.vdim) o[e] = fmaf(a_tok, qs[e], y[e]);
            }
        }
        // ---- S = A_32 S + (D_32 K)^T U ----
        {
            f2 add[ND][NC] = {};
#pragma unroll 4
            for (int t = 0; t < kC; ++t) {
                f2 k[ND];
                if constexpr (ND == 2) {
                    const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(sk + t * LD + d0);
                    k[0] = kk.x;
                    k[1] = kk.y;
                } else {
                    k[0] = *reinterpret_cast<const f2*>(sk + t * LD + d0);
                }
#pragma unroll
                for (int e = 0; e < NC; e += 2) {
                    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(sh + M::ud + t * 2 * kCols + 2 * (c0 + e));
#pragma unroll
                    for (int i = 0; i < ND; ++i) {
                        add[i][e] = fma2(k[i], u.x, add[i][e]);
                        add[i][e + 1] = fma2(k[i], u.y, add[i][e + 1]);
                    }
                }
            }
            const f2 a = pack2(vec[kC - 1], vec[kC - 1]);
#pragma unroll
            for (int i = 0; i < ND; ++i)
#pragma unroll
                for (int e = 0; e < NC; ++e) S[i][e] = fma2(S[i][e], a, add[i][e]);
            put_state();                                      // (the state in shared memory was read in front of the last barriers)
        }
        __syncthreads();                                      // the triangles are read
        if (t0 + kC < n) stage_triangles(t0 + kC);
        copies_started();
    }
    copies_done_but<0>();
#pragma unroll
    for (int e = 0; e < NC; ++e) {
        if (col0 + c0 + e >= p.vdim) continue;
        float* st = p.state + (((size_t)slot * p.H + h) * p.vdim + col0 + c0 + e) * p.dim;
#pragma unroll
        for (int i = 0; i < ND; ++i)
            if (d0 + 2 * i < p.dim) *reinterpret_cast<f2*>(st + d0 + 2 * i) = S[i][e];
    }
}

template <int DP>
cudaError_t launch_inst(const DeltaArgs& p, int M, int n_long, int longest_tokens, cudaStream_t st) {
    cudaError_t e = launch_pdl_if(false, delta_chunk_kernel<DP>, dim3(M / kC + p.n_seq, p.H), dim3(kThreads), 0, st, p);
    if (e != cudaSuccess) return e;
    ++dia::extra_launches();
    constexpr int smem = Columns<DP>::floats * 4;
    int dev = 0;
    e = cudaGetDevice(&dev);
    static std::atomic<bool> asked[64];
    if (e == cudaSuccess && (dev < 0 || dev >= 64 || !asked[dev].load(std::memory_order_relaxed))) {
        e = cudaFuncSetAttribute(delta_columns_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess && dev >= 0 && dev < 64) asked[dev].store(true, std::memory_order_relaxed);
    }
    if (e != cudaSuccess) return e;
    // (of M tokens no more than M / kChunkTokensMin sequences are long ones)
    const int columns = (p.vdim + kCols - 1) / kCols, longest = std::min(n_long > 0 ? n_long : p.n_seq, M / kChunkTokensMin);
    int sms = 0;
    e = dia::current_sms(&dev, &sms);
    if (e != cudaSuccess) return e;
    // Beside the kernel in front the blocks crowd on the SMs that empty first.  Where there is one of the larger kind for each SM at most and a walk is long, that
    // costs more than the early start gives (us, 2048 tokens and 1, 128 blocks: 548 early, 400 behind it; 900 and five of 40 300 / 253; 96 and three of 10, 32
    // blocks 58 / 63; four of 300, 512 blocks 257 / 262); a step of one sequence has nothing that starts beside
    const bool spread = DP > 64 && (long long)columns * p.H * longest <= sms && longest_tokens >= 8 * kC;
    return launch_pdl_if(p.n_seq > 1 && !spread, delta_columns_kernel<DP>, dim3(columns, p.H, longest), dim3(kColThreads), (size_t)smem, st, p);
}

}  // namespace

bool delta_chunks_ok(const float* in, int ld, const ScanInputs& si, int H, int G, int dim, int vdim, const float* state) {
    auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    return G > 0 && H > 0 && H % G == 0 && H <= 65535 && dim > 0 && dim <= 128 && dim % 4 == 0 && vdim > 0 && ld % 4 == 0 && si.q_off % 4 == 0 &&
           si.k_off % 4 == 0 && aligned(in) && aligned(state);
}

cudaError_t launch_delta_chunks(const float* in, int ld, const ScanInputs& si, int H, int G, int dim, int vdim, float* state, const SeqMeta& sm,
                                const RowMeta& rm, int n_seq, int M, float* o, int ldo, float* room, int n_long, int longest_tokens, cudaStream_t st) {
    const DeltaArgs p{in, ld, si.q_off, si.k_off, si.v_off, si.beta_off, si.a_off, H, G, dim, vdim, n_seq, state, sm.slot, sm.row0, sm.count, rm.pos, o, ldo, room};
    return dim <= 64 ? launch_inst<64>(p, M, n_long, longest_tokens, st) : launch_inst<128>(p, M, n_long, longest_tokens, st);
}

}  // namespace lm
