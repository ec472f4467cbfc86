// Weights of the fp32-accurate path into 16-bit parts (split.cuh): a layer's bounds in one launch, its parts and scaled vectors in
// another.  Packing runs once per checkpoint and is bound by launches: as some 45 small torch operations and a synchronisation per
// sub-operation, the first call of two template blocks at 16 tokens took 4.2 ms and of two 256-wide blocks 6.2 ms, against 1.4 and
// 2.0 ms on the un-fused kernels, which pack nothing; this way 1.3 and 1.9 ms.
#include "split.cuh"

namespace b200pf {
namespace split {

constexpr int TABLE = 64, STAT_ROWS = 8, PART_VALUES = 2048;      // items of a launch (by value, below 4 KB); a block's share of an item

struct StatTable {
    int n;
    b200pf_stat_item item[TABLE];
};
struct PackTable {
    int n;
    b200pf_pack_item item[TABLE];
};

// The largest of non-negative floats (and NaN, whose bits are above infinity's) by their bits.
__device__ __forceinline__ void raise_to(float* at, float v) { atomicMax(reinterpret_cast<unsigned int*>(at), __float_as_uint(v)); }
__device__ __forceinline__ unsigned int bits_max(unsigned int a, float v) { return max(a, __float_as_uint(v)); }
__device__ __forceinline__ float warp_bits_max(unsigned int a) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, a));
}

// out[item] = {max |w|, max 2-norm of a row, max (sqrt(cols) |w| + |b|)}; a warp per row
__global__ void __launch_bounds__(STAT_ROWS * 32) weight_stats_kernel(const __grid_constant__ StatTable t, float* out) {
    int i = 0, block = blockIdx.x;
    for (; i < t.n; ++i) {
        const int blocks = (t.item[i].rows + STAT_ROWS - 1) / STAT_ROWS;
        if (block < blocks) break;
        block -= blocks;
    }
    if (i == t.n) return;
    const int rows = t.item[i].rows, cols = t.item[i].cols, row = block * STAT_ROWS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* w = t.item[i].w + (long long)row * cols;
    const float* b = t.item[i].b;
    const float root = sqrtf((float)cols);
    unsigned int top = 0, bound = 0;
    float sum = 0.f;
    for (int c = lane; c < cols; c += 32) {
        const float v = fabsf(w[c]);
        top = bits_max(top, v);
        if (b) bound = bits_max(bound, fmaf(root, v, fabsf(b[c])));
        sum = fmaf(v, v, sum);
    }
    const float norm = sqrtf(warp_sum(sum)), m = warp_bits_max(top), x = warp_bits_max(bound);
    if (lane == 0) {
        raise_to(out + 3 * i, m);
        raise_to(out + 3 * i + 1, fabsf(norm));
        raise_to(out + 3 * i + 2, x);
    }
}

__global__ void __launch_bounds__(256) pack_parts_kernel(const __grid_constant__ PackTable t) {
    int i = 0;
    long long block = blockIdx.x;
    for (; i < t.n; ++i) {
        const long long blocks = ((long long)t.item[i].rows * t.item[i].cols + PART_VALUES - 1) / PART_VALUES;
        if (block < blocks) break;
        block -= blocks;
    }
    if (i == t.n) return;
    const b200pf_pack_item& p = t.item[i];
    const long long count = (long long)p.rows * p.cols, end = min(count, (block + 1) * PART_VALUES);
    for (long long at = block * PART_VALUES + threadIdx.x; at < end; at += 256) {
        const float v = p.src ? __fmul_rn(__fmul_rn(p.src[at], p.factor), p.scale) : 0.f;      // scale: a power of two
        if (p.parts == 0) {
            static_cast<float*>(p.dst)[at] = v;
            continue;
        }
        const int row = (int)(at / p.cols), col = (int)(at % p.cols);
        const long long to = (long long)(p.row0 + (p.interleave ? (row >> 5) * 64 + (row & 31) : row)) * p.cols + col;
        const __half hi = __float2half_rn(v);
        static_cast<__half*>(p.dst)[to] = hi;
        static_cast<__half*>(p.dst)[p.part_stride + to] = __float2half_rn(v - __half2float(hi));
    }
}

}  // namespace split
}  // namespace b200pf

using namespace b200pf;
using namespace b200pf::split;

extern "C" int b200pf_weight_stats(const b200pf_stat_item* items, int n, float* out, void* stream) {
    B200PF_REQUIRE(items && out && n > 0, B200PF_ERR_INVALID, "weight_stats: bad arguments");
    for (int i = 0; i < n; ++i)
        B200PF_REQUIRE(items[i].w && items[i].rows > 0 && items[i].cols > 0 && (!items[i].b || items[i].rows == 1), B200PF_ERR_INVALID,
                       "weight_stats: item %d is null, empty or a matrix with an offset", i);
    cudaStream_t st = (cudaStream_t)stream;
    B200PF_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * 3 * n, st));
    for (int first = 0; first < n; first += TABLE) {
        StatTable t = {};
        unsigned blocks = 0;
        for (t.n = 0; t.n < TABLE && first + t.n < n; ++t.n) {
            t.item[t.n] = items[first + t.n];
            blocks += (unsigned)((t.item[t.n].rows + STAT_ROWS - 1) / STAT_ROWS);
        }
        weight_stats_kernel<<<blocks, STAT_ROWS * 32, 0, st>>>(t, out + 3 * first);
        B200PF_LAUNCH_CHECK();
    }
    return B200PF_OK;
}

extern "C" int b200pf_pack_parts(const b200pf_pack_item* items, int n, void* stream) {
    B200PF_REQUIRE(items && n > 0, B200PF_ERR_INVALID, "pack_parts: bad arguments");
    for (int i = 0; i < n; ++i)
        B200PF_REQUIRE(items[i].dst && items[i].rows > 0 && items[i].cols > 0 && items[i].row0 >= 0 && (!items[i].interleave || items[i].rows % 32 == 0),
                       B200PF_ERR_INVALID, "pack_parts: item %d is null, empty or has rows that can't be interleaved", i);
    for (int first = 0; first < n; first += TABLE) {
        PackTable t = {};
        long long blocks = 0;
        for (t.n = 0; t.n < TABLE && first + t.n < n; ++t.n) {
            t.item[t.n] = items[first + t.n];
            blocks += ((long long)t.item[t.n].rows * t.item[t.n].cols + PART_VALUES - 1) / PART_VALUES;
        }
        pack_parts_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(t);
        B200PF_LAUNCH_CHECK();
    }
    return B200PF_OK;
}
