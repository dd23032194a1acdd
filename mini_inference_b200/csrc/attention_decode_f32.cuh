// Decoded tokens in true float32 (csrc/attention_decode_f32.cu): what attention_generic.cu and attention_masked.cu hand over where it takes the sizes
#pragma once
#include "common.cuh"

namespace mi {

struct DecodeF32 {
    const float *q, *k_cache, *v_cache;
    float *out, *o_part, *lse_part;
    const int *decode_segs, *seg_q_start, *seg_kv_len, *block_table, *table_rows;
    int q_stride, num_decode, table_stride, H, KV, D, ps, splits;
    float scale;
    // attention_masked.cu's terms; all off: plain attention
    int block, window, sink, bias_last, keep, gate_stride;
    const float *sink_values, *bias, *slopes, *gate;
    float cap;
};
// Heads of 64 or 128, 1, 2, 4 or 8 query heads to a key head, rows on 16 bytes
bool takes_decode_f32(const DecodeF32& a);
// With splits > 1 the pieces stay in o_part and lse_part, as the other kernels leave them
int decode_f32(const DecodeF32& a, cudaStream_t stream);

}  // namespace mi
