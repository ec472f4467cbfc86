// Operands of the fp32-accurate tensor-core path: an fp32 value kept as a sum of 16-bit parts.
//
//   F16X2   v * scale = hi + lo, two fp16 parts.  hi is off by at most 2^-11 of the value, and lo by at most 2^-12 of what is left:
//           2^-23 of the value together, one ulp of fp32.  `scale` is a power of two chosen when the weights are packed from a
//           bound of |v| (a LayerNorm output is at most sqrt(C) * gain + offset, a projection of it at most that times the row
//           norm), so neither part can overflow and this holds for values down to 2^-15 of the bound; below, the error is at most
//           2^-38 of the bound.  Products: hi*hi + hi*lo + lo*hi, three MMAs; what is left out is at most 2^-22 of the product.
//   BF16X3  v = h + m + l, three bf16 parts (24 bits, the whole fp32 mantissa, and fp32's own range: no scale).
//           Products of total order <= 2: six MMAs.
// Both accumulate in fp32.  A plane stack is [parts][rows][cols] of 16-bit values.
#pragma once

#include <cuda_fp16.h>

#include "pdl.cuh"
#include "sm100.cuh"

namespace b200pf {
namespace split {

__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
    __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
}
// Two values into fp16 part words {hi, lo}.
__device__ __forceinline__ void split_f16x2(float a, float b, uint32_t& hi, uint32_t& lo) {
    hi = pack_f16x2(a, b);
    const float2 left = fma2(__half22float2(*reinterpret_cast<__half2*>(&hi)), make_float2(-1.f, -1.f), make_float2(a, b));
    lo = pack_f16x2(left.x, left.y);
}
// Two values into bf16 part words {h, m, l}.
__device__ __forceinline__ void split_bf16x3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack_bf16x2(a, b);
    const float ra = a - bf16_lo(h), rb = b - bf16_hi(h);
    m = pack_bf16x2(ra, rb);
    l = pack_bf16x2(ra - bf16_lo(m), rb - bf16_hi(m));
}

// ---- host side -----------------------------------------------------------------------------------
// Two-part (fp16) or three-part (bf16) operand of a GEMM: element (part, batch, row, col) at
// ptr + part * part_stride + batch * batch_stride + row * row_stride + col (16-bit elements; strides multiples of 8).
struct Operand {
    const void* ptr;
    int rows, cols, batches;
    long long row_stride, batch_stride, part_stride;
};
// Output of a GEMM: element (part, batch, row, col), strides in elements of its type; `rows_outer` swaps the roles of row and
// batch in memory order only (the operand planes of a triangle multiplication, [channel][line][position], with
// row = channel and batch = line).
struct Output {
    void* ptr;
    int rows, cols, batches, parts;
    long long row_stride, batch_stride, part_stride;
    bool rows_outer;
};

enum Epilogue { EPI_STORE, EPI_ADD, EPI_SWIGLU, EPI_QKVG, EPI_GATE_PLANES, EPI_GATE_ADD, EPI_CONTRACT };

struct Gemm {
    int parts = 2;                  // 2: F16X2, 3: BF16X3
    Epilogue epi = EPI_STORE;
    Operand a[2], b[2];             // second pair: EPI_GATE_ADD (its own K loop and accumulator)
    bool a_batched = false, b_batched = false;
    int a_second_row = 0;           // EPI_GATE_PLANES: row offset of the gate rows in A
    int m_rows = 0, n_rows = 0, batches = 1;
    int k[2] = {0, 0};
    int k_splits = 1;               // > 1: batch index = K split, partial sums stored per batch (EPI_STORE only)
    float alpha[2] = {1.f, 1.f};
    float out_scale = 1.f;          // EPI_SWIGLU, EPI_GATE_PLANES: scale of the stored parts
    const float* bias = nullptr;    // [n_rows]
    const uint8_t* mask = nullptr;  // EPI_GATE_PLANES: position (batch, col) at mask + batch * mask_bs + col * mask_cs
    long long mask_bs = 0, mask_cs = 0;
    int n_split = 0;                // EPI_QKVG: columns below it (q | k | v, a third each) go out as two fp16 parts times
    float qkv_scale[3] = {1.f, 1.f, 1.f};       // these, the others as sigmoid, fp32
    Output out[2];
};
int launch_gemm(const Gemm& g, cudaStream_t st);

}  // namespace split
}  // namespace b200pf
