// gemm_tcgen05.h - the tensor-core contraction of gemm_tcgen05.cu for callers that hold bf16 activations.
//
//   Y[M][N] (fp32) = residual + f(A[M][K] (bf16) . Wt[N][K]^T (bf16)),  fp32 accumulation in tensor memory
//
// f is the identity, a DynamicTanh per output column, or an activation whose result is kept as the bf16 operand of the next
// product (Yb[M][N] instead of Y).  With row groups, the rows of A are sorted by group, every
// group starts on a multiple of GemmGroups::tile_rows rows, and group g multiplies rows [g * group_rows, g * group_rows + N)
// of Wt.
#pragma once

#include <atomic>

#include <cuda_runtime.h>

namespace dia {

// What is asked for once per device (static: two libraries in one process hold kernels of the same names, and an inline function's statics would be
// theirs together).  SMs of the current device:
static inline cudaError_t current_sms(int* dev, int* sms) {
    static std::atomic<int> known[64];
    const cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess) return e;
    if (*dev < 64 && (*sms = known[*dev].load(std::memory_order_relaxed)) > 0) return cudaSuccess;
    const cudaError_t a = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, *dev);
    if (a == cudaSuccess && *dev < 64) known[*dev].store(*sms, std::memory_order_relaxed);
    return a;
}
// Dynamic shared memory of a kernel, the same size for every launch:
template <auto KERNEL>
static cudaError_t ask_smem(int dev, int bytes) {
    static std::atomic<bool> asked[64];
    if (dev < 64 && asked[dev].load(std::memory_order_relaxed)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < 64) asked[dev].store(true, std::memory_order_relaxed);
    return e;
}

constexpr int kGemmRowTile = 128;            // rows of A per output tile: the padding unit of a row group
constexpr int kGemmPairRows = 256;           // the same of a pair of SMs

struct GemmEpilogue {
    const float* residual;                   // [M][N] added to the result (may alias Y), or null
    const float* dyt_w;                      // [N]: f(a) = tanh(dyt_alpha a) dyt_w + dyt_b; null: f(a) = a
    const float* dyt_b;
    float dyt_alpha;
    void* y_bf16;                            // [M][N] bf16: gelu(result), the tanh form, goes here and nothing to y; null: y
};

struct GemmGroups {
    const int* row_group;                    // device [M]: group of every row of A (read at the first row of a tile)
    int group_rows;                          // rows of Wt per group
    const int* n_rows;                       // device: rows of A in use (row tiles at or beyond it are skipped); null: M
    int tile_rows;                           // every group starts on a multiple of it: kGemmRowTile or kGemmPairRows
};

// K a multiple of 8 (16-byte rows for the TMA), N a multiple of 4 (float4 stores)
// Kernels that launchers on this thread launched beyond one per call, for the caller that counts launches (it takes them)
inline long long& extra_launches() {
    static thread_local long long n = 0;
    return n;
}

inline bool gemm_tcgen05_shape_ok(int M, int N, int K) { return M > 0 && N > 0 && K >= 8 && K % 8 == 0 && N % 4 == 0; }

cudaError_t launch_gemm_tcgen05_bf16(const void* a_bf16, int terms, const void* wt, long long wt_rows, float* y, int M, int N,
                                     int K, const GemmEpilogue& ep, const GemmGroups* groups, cudaStream_t st);
// Yb[M][F] = bf16(glu(gate, up)) of [gate | up] = A[M][K] (bf16) . Wt[2 F][K]^T: the products of launch_gemm_tcgen05_bf16 with the gate in front of the bf16
// rounding (kind: kGlu* of the language models).  cudaErrorNotSupported where that product would not run on pairs of SMs, F is no multiple of 128 or (but for
// in_any_case) the two are the shorter way: the caller then runs the product and the gate one after the other, to the same bits.
cudaError_t launch_gemm_glu_bf16(const void* a_bf16, const void* wt, long long wt_rows, void* y_bf16, int M, int F, int K, int kind, float limit,
                                 const GemmGroups* groups, cudaStream_t st, bool in_any_case = false);

// Per head h < heads: Y[m][h y_hs + n] = act(alpha sum_k A[m][h a_hs + k] W[h][n][k]) [* sigmoid of a gate column], as fp32 FMA
// arithmetic gives it: A (fp32, row stride lda) is split into three bf16 terms (24 bits) in `work` (gemm_f32_work_bytes), every 64
// products of a sum are accumulated in tensor memory and added to the sum in fp32 registers.  W: bf16 [heads * N][K].
struct F32Product {
    const float* a; int lda, a_hs;
    const void* w;
    float* y; int ldy, y_hs;
    void* y_bf16;                            // a bf16 copy of y; null: none
    int heads, M, N, K;
    float alpha;
    int act;                                 // 0: none, 2: max(z, 0)^2, 3: gelu, the tanh form
    const float* gate; int ldg, head_gate;   // gate[m * ldg + h N + n], with head_gate gate[m * ldg + h]; null: none
    const float* add;                        // laid out as y, added last (may be y); null: none
    const float* dyt_w; const float* dyt_b; float dyt_alpha;      // as in GemmEpilogue, in front of add
};
bool gemm_f32_ok(const F32Product& p);
inline size_t gemm_f32_work_bytes(size_t rows, size_t columns) { return 6 * rows * columns; }      // columns: heads * K
cudaError_t launch_gemm_f32(const F32Product& p, void* work, cudaStream_t st);

// The same for at most 32 rows (decoding, a short text): Y[m][n] = [add +] act(sum_k A[m][k] W[n][k]).  The weights are the 128-row
// operand and stream once for all rows; the rows' three terms are the columns of the other operand.  A sum's order depends on N and K
// (and on whether there are more than 8 rows) only.
// early: launched with programmatic stream serialization (the weights are requested before the predecessor has ended).
constexpr int kGemmFewRowsMost = 32;
struct FewRowsProduct {
    const float* a; int lda;
    const void* w;
    float* y; int ldy;
    int M, N, K;
    int act;                                 // as in F32Product
    const float* add;                        // [M][ldy] added to the product (y itself: it is accumulated), or null
};
bool gemm_few_rows_ok(const FewRowsProduct& p);
cudaError_t launch_gemm_few_rows(const FewRowsProduct& p, bool early, cudaStream_t st);

}  // namespace dia
