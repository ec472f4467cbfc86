// Row kernels that produce the part planes the split GEMM reads (split.cuh).
#pragma once
#include "split.cuh"

namespace b200pf {
namespace split {

struct LnArgs {
    const float* x;             // [rows][C] fp32
    const float* gamma;         // gain and offset, times the planes' scale
    const float* beta;
    __half* planes;             // [2][rows][C], or null: heads only
    long long part_stride;
    long long rows;
    // a few dot products per row with the normalised row: row (i, j) of a pair tensor of width n at out[h][i][j], or transposed at
    // out[h][j][i], lines of `head_pitch`
    const float* head_w;        // [heads][C], divided by the planes' scale
    float* head_out;
    long long head_stride;
    int n, transposed, head_pitch;
};
bool ln_supported(int c);
int launch_ln(const LnArgs& a, int c, int heads, cudaStream_t st);

// LayerNorm over the channels of a channel-major tensor t[d][i][pitch]: planes [2][n * n][d]
int launch_ln_channels(const float* t, long long plane_stride, int pitch, const float* gamma, const float* beta, __half* planes,
                       int n, int d, cudaStream_t st);
// bf16 parts [3][rows][c] of an fp32 matrix, c a multiple of 4
int launch_parts(const float* x, __nv_bfloat16* planes, long long count, cudaStream_t st);
// x += sum_p partial[p]
int launch_add_partials(float* x, const float* partial, int n_partial, long long count, cudaStream_t st);

}  // namespace split
}  // namespace b200pf
