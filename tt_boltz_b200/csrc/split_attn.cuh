// Attention at fp32 accuracy on part planes (split_attn.cu).
#pragma once
#include "split.cuh"

namespace b200pf {
namespace split {

struct AttnArgs {
    // q | k | v, `heads * hd` columns each, as two fp16 parts [2][rows][ld] of q * q_scale, k * k_scale, v * out_scale;
    // q carries log2(e) / sqrt(hd)
    const __half* qkv;
    float qk_scale;                     // q_scale * k_scale
    long long part_stride;
    int ld;
    long long line_rows, pos_rows;      // row of (line, position) = line * line_rows + position * pos_rows
    const float* gate;                  // [rows][heads * hd], applied to the output (already a sigmoid)
    const float* bias;                  // element (head, query - q0, key) at head * bias_hs + (query - q0) * bias_qs + key, times log2(e)
    long long bias_hs, bias_qs;
    bool bias_vec;                      // set by launch_attention
    const uint8_t* mask;                // key (line, position) at mask + line * mask_ls + position * mask_ks; null: none masked
    long long mask_ls, mask_ks;
    float mask_add;                     // added to a masked key's score (base-2 logarithms)
    __half* out;                        // [2][out rows][heads * hd], scaled as v; row of query i: its own row, minus out_row0
    long long out_part_stride, out_row0;
    int lines, heads, q0, n_q, n_k;     // queries q0 .. q0 + n_q - 1 of every line
};
int launch_attention(const AttnArgs& a, int hd, cudaStream_t st);
bool attention_tc_fits(const AttnArgs& a, int hd);                  // split_attn_tc.cu
int launch_attention_tc(const AttnArgs& a, cudaStream_t st);

}  // namespace split
}  // namespace b200pf
