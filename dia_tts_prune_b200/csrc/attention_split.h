// attention_split.h - softmax attention for many query rows on the tensor cores (attention_split.cu).
//
// Queries, keys, values and softmax weights are fp32; every product takes them as two fp16 terms of a scaled value (22
// significand bits) and is accumulated in fp32.  A row's result depends on the row and the keys that it sees alone.  Serves
// grouped-query attention over paged keys and values, attention over one cached latent per position (the value is the head of the
// key row), and attention whose scores are mixed across heads.
#pragma once

#include <cuda_runtime.h>

namespace dia {

struct SplitAttention {
    // query head h of row r: q + r * ldq + h * qdim, qdim channels
    const float* q; int ldq; int qdim;
    // key of (page, kv head, offset): kcache + ((page * kv_heads + g) * page_size + offset) * kdim; the value likewise in vcache
    // with rows of vrow floats, of which vdim are the value.  table [slot][max_pages] -> page; null: the page is the slot
    const float* kcache; const float* vcache;
    const int* table; int max_pages, page_size;
    int heads, kv_heads, kdim, vdim, vrow;
    // score = q . k * scale * temp_h, capped (cap > 0: cap tanh(score / cap)), minus slopes_h (i - j); temp, slopes: null: none
    float scale, cap;
    const float* temp; const float* slopes;
    const float* sink;                       // [heads] logits that join the denominator only; null: none
    const float* talk;                       // [heads][heads]: score_h <- sum_g talk[h][g] score_g before the softmax; null: none
    // row r: position row_pos[r] of sequence row_slot[r]; rows of a sequence adjacent and in order.  It sees key j <= its
    // position inside its window (window > 0) and its chunk (chunk > 0), and with a window the first keep_first keys
    const int* row_slot; const int* row_pos; int M;
    int window, keep_first, chunk;
    // rows_per_slot > 0: row r is position r % rows_per_slot of slot r / rows_per_slot (at most 16 slots), and with n = n_valid[slot]
    // sees, by mode, 0: the keys up to its own position; 1: [0, n) if its position is below n, else [n, n_keys); 2: [0, n)
    int rows_per_slot, mode, n_keys;
    int n_valid[16];
    // out[r * ldo + h * vdim + c] = softmax-weighted value * out_scale [* sigmoid(gate[r * ldg + h * vdim + c])]
    // [* head_gate[r * ldg + h]], and its bf16 copy (either may be null)
    float* out; int ldo; void* out_bf16;
    float out_scale;
    const float* gate; const float* head_gate; int ldg;
    // Optional (n_seq 0: not given): the step's sequences - slot, first row and row count of each
    const int* seq_slot; const int* seq_row0; const int* seq_count; int n_seq;
    // Optional, with the sequences or with rows_per_slot: room in which a launch in front splits the keys and values that the rows see once for
    // all row tiles (null: every row tile splits them for itself, which takes about twice as long).  n_slots: slots there are.  Keys beyond the
    // room's size are split by the row tiles.
    void* work; size_t work_bytes; int n_slots;
    long long n_tiles;                                        // with the sequences: no more tiles of 64 keys than this are seen (0: not known)
};

// Whether the kernel takes the shape; M does not matter.  Channel counts and strides that are multiples of 4 on 16-byte aligned pointers, values
// of at most 256 channels, keys of at most 4 groups of 128 (mixed scores: as many key heads of at most 128) for which tensor memory has the
// columns, and shared memory for the queries of 128 (token, head) rows beside two slots of 64 keys: latent rows of 256 + 64 channels fit
// from 4 heads on, mixed scores with 4 key heads of 128 channels do not.
bool split_attention_ok(const SplitAttention& a);
// bytes of `work` for `keys` keys of this shape (0: the shape is not taken)
size_t split_attention_work_bytes(const SplitAttention& a, int keys);
int split_attention_keys(const SplitAttention& a, int slot);      // rows_per_slot > 0: how many keys of a slot some row sees
// The word of `device` that a kernel sets when one of its waits has run out (its outputs are NaN then).  Made by the first call outside of a capture: engines
// and weight copies are made with one, so that products that are captured have it.
int* split_attention_ran_out(int device, cudaStream_t st);
bool take_ran_out(int device, cudaStream_t st);                 // whether a wait has run out since the last look; the word is zero afterwards
cudaError_t launch_split_attention(const SplitAttention& a, cudaStream_t st);

}  // namespace dia
