// Outer-product mean (MSA stack -> pair tensor): the stages around its two GEMMs.
//
//   z[i][j][:] += W_o * vec( sum_s a[s][i][:] (x) b[s][j][:] ) / max(1, sum_s mask[s][i] mask[s][j]) + bias
//   a = mask * (LN(m) W_a^T),  b = mask * (LN(m) W_b^T)            (m: [S][N][64], 32 channels each)
//
// The sum over the S sequences is one K-major GEMM with rows (i, c) and columns (j, d)
// (b200pf_opm_outer: the triangle-multiplication contraction kernel writing each pair's 32 x 32 block
// contiguously), the projection a second one over the 1024 (c, d) products (b200pf_trimul_contract with one
// channel).  This file holds what feeds and drains them:
//   opm_producer_kernel : LayerNorm + both projections + mask, written TRANSPOSED (sequence index contiguous) as
//                         the GEMM's K-major operands; fp32 throughout, bf16 on store.
//   opm_mask_bits_kernel: the MSA mask as one bit per sequence, 32 sequences per word and token.
//   opm_finalize_kernel : pair counts by popcount of the two tokens' words, then y / count + bias added into (or
//                         written over) the fp32 pair rows.
#include "cp_async.cuh"
#include "pdl.cuh"

namespace b200pf {
namespace opm {

constexpr int CM = 64;            // MSA channels
constexpr int CH = 32;            // projected channels per side
constexpr int PROD_THREADS = 128, PROD_ROWS = 64;                // sequences per CTA and token
constexpr int XP = CM + 4;        // pitch of a staged row in floats: 16-byte reads of eight rows meet no bank twice
constexpr int PROD_SMEM = (CM * 2 * CH + PROD_ROWS * (XP + CM + 1) + 2 * CM) * 4;               // 50,944: four CTAs per SM
constexpr int FIN_THREADS = 256, FIN_J = 64;
constexpr int MAX_WORDS = 512;    // sequences / 32 the finalize kernel keeps in shared memory (S <= 16384)

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ uint64_t twice(float w) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(w));
    return r;
}
__device__ __forceinline__ void both(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }

// A CTA takes 64 sequences of one token at a time: rows into shared memory, a thread per row for the LayerNorm, then a thread per
// 8 sequences x 8 outputs, all in fp32 and every sum in one order: the mean and the variance over the channels in turn, an output as
// two chains of FMAs (channels 0-3, 8-11, .. on warps 0 and 1, channels 4-7, 12-15, .. on warps 2 and 3) that are added at the end.  The
// operands are rounded to bf16 right behind, and a last bit that flips there moves the whole MSA module's result by 2e-3 of its norm:
// products of two tf32 parts (2^-22 of a product left out) on the tensor cores did that, in 119 us at 1024 sequences x 600 tokens.  The
// same sums by a thread per row, the weights broadcast from shared memory (a 16-byte load per four FMAs), took 226 us there and 19 at
// 122 x 171; here a load serves sixteen FMAs, packed two sequences each: 138 and 12.  What bounds it are those loads, 512 bytes a warp
// into registers at 128 a clock, beside the FMAs.
__global__ void __launch_bounds__(PROD_THREADS, 4)
opm_producer_kernel(const float* m, const uint8_t* mask, const float* gamma, const float* beta, const float* w_ab, __nv_bfloat16* a_t,
                    __nv_bfloat16* b_t, int s_len, int n, int pitch, int vec) {
    extern __shared__ __align__(16) uint8_t smem[];
    float* w_s = reinterpret_cast<float*>(smem);                          // [channel][output]
    float* in_s = w_s + CM * 2 * CH;                                      // [row][XP] as loaded
    float* x_s = in_s + PROD_ROWS * XP;                                   // [channel][row] normalised
    float* keep_s = x_s + CM * PROD_ROWS;
    float* gb_s = keep_s + PROD_ROWS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, s0 = blockIdx.x * PROD_ROWS;
    const int chain = tid >> 6, u = tid & 63, rg = (u & 7) * 4, o0 = (u >> 3) * 8;       // rows rg .. + 3 and 32 + rg .. + 3, outputs o0 .. + 7
    grid_dependency_wait();
    grid_launch_dependents();
    auto load_rows = [&](int tok) {                                       // 16 lanes per row; rows past the end repeat the last one
        for (int i = tid; i < PROD_ROWS * (CM / 4); i += PROD_THREADS) {
            const int r = i >> 4, c = (i & 15) * 4, s = s0 + r;
            cp_async16(in_s + r * XP + c, m + ((long long)(s < s_len ? s : s_len - 1) * n + tok) * CM + c);
        }
        cp_async_commit();
    };
    load_rows(blockIdx.y);
    gb_s[tid] = tid < CM ? gamma[tid] : beta[tid - CM];
    for (int i = tid; i < 2 * CH * (CM / 4); i += PROD_THREADS) {
        const int o = i & (2 * CH - 1), k = (i >> 6) * 4;
        const float4 w = *reinterpret_cast<const float4*>(w_ab + o * CM + k);
        w_s[k * 2 * CH + o] = w.x;
        w_s[(k + 1) * 2 * CH + o] = w.y;
        w_s[(k + 2) * 2 * CH + o] = w.z;
        w_s[(k + 3) * 2 * CH + o] = w.w;
    }
    int turn = 0;
#pragma unroll 1
    for (int tok = blockIdx.y; tok < n; tok += gridDim.y, turn ^= 2) {
        cp_async_wait<0>();
        __syncthreads();
        const int row = ((warp + turn) & 3) * 32 + lane;                  // two warps normalise, the other two the next time: a warp
        const bool ln = row < PROD_ROWS;                                  // stays on its scheduler
        if (ln) {
            const int s = s0 + row;
            const bool keep = mask[(long long)(s < s_len ? s : s_len - 1) * n + tok] != 0;
            float x[CM], sum = 0.f, ss = 0.f;
#pragma unroll
            for (int j = 0; j < CM / 4; ++j) {
                const float4 v = *reinterpret_cast<const float4*>(in_s + row * XP + 4 * j);
                x[4 * j] = v.x; x[4 * j + 1] = v.y; x[4 * j + 2] = v.z; x[4 * j + 3] = v.w;
            }
#pragma unroll
            for (int k = 0; k < CM; ++k) sum += x[k];
            const float mean = sum * (1.f / CM);
#pragma unroll
            for (int k = 0; k < CM; ++k) { x[k] -= mean; ss = fmaf(x[k], x[k], ss); }
            const float rstd = rsqrtf(ss * (1.f / CM) + LN_EPS);
#pragma unroll
            for (int k = 0; k < CM; ++k) x_s[k * PROD_ROWS + row] = fmaf(x[k] * rstd, gb_s[k], gb_s[CM + k]);
            keep_s[row] = keep ? 1.f : 0.f;
        }
        __syncthreads();
        if (tok + (int)gridDim.y < n) load_rows(tok + gridDim.y);         // the next rows arrive under the products
        uint64_t acc[8][4] = {};                                          // output, pair of rows
#pragma unroll 1
        for (int k4 = chain * 4; k4 < CM; k4 += 8)
#pragma unroll
            for (int e = 3; e >= 0; --e) {
                const float* xk = x_s + (k4 + e) * PROD_ROWS + rg;
                const float* wk = w_s + (k4 + e) * 2 * CH + o0;
                const ulonglong2 xa = *reinterpret_cast<const ulonglong2*>(xk), xb = *reinterpret_cast<const ulonglong2*>(xk + PROD_ROWS / 2);
                const float4 wa = *reinterpret_cast<const float4*>(wk), wb = *reinterpret_cast<const float4*>(wk + 4);
                const uint64_t w[8] = {twice(wa.x), twice(wa.y), twice(wa.z), twice(wa.w), twice(wb.x), twice(wb.y), twice(wb.z), twice(wb.w)};
#pragma unroll
                for (int o = 0; o < 8; ++o) {
                    fma2(acc[o][0], w[o], xa.x);
                    fma2(acc[o][1], w[o], xa.y);
                    fma2(acc[o][2], w[o], xb.x);
                    fma2(acc[o][3], w[o], xb.y);
                }
            }
        // the chains meet: each thread gives four of its outputs to the one with the other chain and finishes the other four
        __syncthreads();
        ulonglong2* ex = reinterpret_cast<ulonglong2*>(x_s);              // [chain][output, half of the rows][thread]
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int o = j >> 1, h = 2 * (j & 1);
            ex[(chain * 8 + j) * 64 + u] = chain ? make_ulonglong2(acc[o][h], acc[o][h + 1]) : make_ulonglong2(acc[4 + o][h], acc[4 + o][h + 1]);
        }
        __syncthreads();
        const int oo = o0 + 4 * chain;
        __nv_bfloat16* dst = (oo < CH ? a_t : b_t) + ((long long)tok * CH + (oo & (CH - 1))) * pitch + s0 + rg;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int o = j >> 1, h = 2 * (j & 1);
            const float4 other = *reinterpret_cast<const float4*>(ex + ((chain ^ 1) * 8 + j) * 64 + u);
            const float4 keep = *reinterpret_cast<const float4*>(keep_s + (j & 1) * (PROD_ROWS / 2) + rg);
            float v[4];
            both(chain ? acc[4 + o][h] : acc[o][h], v[0], v[1]);
            both(chain ? acc[4 + o][h + 1] : acc[o][h + 1], v[2], v[3]);
            v[0] = (v[0] + other.x) * keep.x; v[1] = (v[1] + other.y) * keep.y; v[2] = (v[2] + other.z) * keep.z; v[3] = (v[3] + other.w) * keep.w;
            const int s = s0 + (j & 1) * (PROD_ROWS / 2) + rg;
            __nv_bfloat16* at = dst + o * (long long)pitch + (j & 1) * (PROD_ROWS / 2);
            if (vec && s + 4 <= s_len) {
                *reinterpret_cast<uint2*>(at) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (s + e < s_len) at[e] = __float2bfloat16(v[e]);
            }
        }
    }
}

__global__ void opm_mask_bits_kernel(const uint8_t* mask, uint32_t* bits, int s_len, int n, int words) {
    grid_dependency_wait();
    grid_launch_dependents();
    const int tok = blockIdx.x * blockDim.x + threadIdx.x, w = blockIdx.y;
    if (tok >= n) return;
    uint32_t v = 0;
    for (int b = 0; b < 32; ++b) {
        const int s = w * 32 + b;
        if (s < s_len && mask[(long long)s * n + tok]) v |= 1u << b;
    }
    bits[(long long)tok * words + w] = v;
}

__global__ void __launch_bounds__(FIN_THREADS)
opm_finalize_kernel(const __nv_bfloat16* y, const uint32_t* bits, const float* bias, float* z, int i0, int n, int words, int accumulate) {
    grid_dependency_wait();
    grid_launch_dependents();
    __shared__ uint32_t bi_s[MAX_WORDS];
    __shared__ float inv_s[FIN_J];
    const int il = blockIdx.y, i = i0 + il, j0 = blockIdx.x * FIN_J;
    for (int w = threadIdx.x; w < words; w += FIN_THREADS) bi_s[w] = bits[(long long)i * words + w];
    __syncthreads();
    if (threadIdx.x < FIN_J) {
        const int j = j0 + threadIdx.x;
        int cnt = 0;
        if (j < n) {
            const uint32_t* bj = bits + (long long)j * words;
            for (int w = 0; w < words; ++w) cnt += __popc(bi_s[w] & bj[w]);
        }
        inv_s[threadIdx.x] = 1.f / (float)(cnt > 0 ? cnt : 1);
    }
    __syncthreads();
    const int c4 = threadIdx.x & 31;                                  // four channels
    const float4 b4 = reinterpret_cast<const float4*>(bias)[c4];
    for (int jl = threadIdx.x >> 5; jl < FIN_J; jl += FIN_THREADS / 32) {
        const int j = j0 + jl;
        if (j >= n) break;
        const long long row = (long long)il * n + j;
        const uint2 yv = reinterpret_cast<const uint2*>(y + row * 128)[c4];
        const float inv = inv_s[jl];
        float4 o;
        o.x = fmaf(bf16_lo(yv.x), inv, b4.x);
        o.y = fmaf(bf16_hi(yv.x), inv, b4.y);
        o.z = fmaf(bf16_lo(yv.y), inv, b4.z);
        o.w = fmaf(bf16_hi(yv.y), inv, b4.w);
        float4* zp = reinterpret_cast<float4*>(z + row * 128) + c4;
        if (accumulate) {
            const float4 old = *zp;
            o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
        }
        *zp = o;
    }
}

}  // namespace opm
}  // namespace b200pf

using namespace b200pf;

extern "C" int b200pf_opm_producer(const float* m, const uint8_t* mask, const float* ln_gamma, const float* ln_beta,
                                   const float* w_ab, b200pf_bf16* a_t, b200pf_bf16* b_t, int s_len, int n, int pitch,
                                   void* stream) {
    using namespace opm;
    B200PF_REQUIRE(m && mask && ln_gamma && ln_beta && w_ab && a_t && b_t, B200PF_ERR_INVALID, "opm_producer: null pointer");
    B200PF_REQUIRE(aligned16(m) && aligned16(w_ab), B200PF_ERR_INVALID, "opm_producer: m and w_ab must be 16-byte aligned");
    B200PF_REQUIRE(s_len > 0 && n > 0 && n <= 65535 && pitch >= s_len, B200PF_ERR_INVALID, "opm_producer: bad sizes");
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK) return rc;
    B200PF_SMEM_ATTR_ONCE(opm_producer_kernel, PROD_SMEM);
    // four CTAs fit an SM; each takes every gridDim.y-th token of its sequences, so that its copy of the weights serves several
    const int tiles = (s_len + PROD_ROWS - 1) / PROD_ROWS, want = (4 * sms + tiles - 1) / tiles, per = (n + want - 1) / want;
    const int vec = aligned16(a_t) && aligned16(b_t) && pitch % 4 == 0;
    return launch_pdl(opm_producer_kernel, dim3((unsigned)tiles, (unsigned)((n + per - 1) / per)), dim3(PROD_THREADS), PROD_SMEM, (cudaStream_t)stream,
                      m, mask, ln_gamma, ln_beta, w_ab, (__nv_bfloat16*)a_t, (__nv_bfloat16*)b_t, s_len, n, pitch, vec);
}

extern "C" int b200pf_opm_mask_bits(const uint8_t* mask, uint32_t* bits, int s_len, int n, void* stream) {
    using namespace opm;
    B200PF_REQUIRE(mask && bits && s_len > 0 && n > 0, B200PF_ERR_INVALID, "opm_mask_bits: bad arguments");
    const int words = (s_len + 31) / 32;
    B200PF_REQUIRE(words <= 65535, B200PF_ERR_UNSUPPORTED, "opm_mask_bits: too many sequences");
    dim3 grid((unsigned)((n + 127) / 128), (unsigned)words);
    return launch_pdl(opm_mask_bits_kernel, grid, dim3(128), 0, (cudaStream_t)stream, mask, bits, s_len, n, words);
}

extern "C" int b200pf_opm_finalize(const b200pf_bf16* y, const uint32_t* bits, const float* bias, float* z, int s_len,
                                   int i0, int n_i, int n, int accumulate, void* stream) {
    using namespace opm;
    B200PF_REQUIRE(y && bits && bias && z && aligned16(y) && aligned16(z) && aligned16(bias), B200PF_ERR_INVALID,
                   "opm_finalize: null or misaligned pointer");
    const int words = (s_len + 31) / 32;
    B200PF_REQUIRE(s_len > 0 && words <= MAX_WORDS, B200PF_ERR_UNSUPPORTED, "opm_finalize: at most %d sequences", MAX_WORDS * 32);
    B200PF_REQUIRE(n > 0 && i0 >= 0 && n_i > 0 && i0 + n_i <= n && n_i <= 65535, B200PF_ERR_INVALID, "opm_finalize: bad sizes");
    dim3 grid((unsigned)((n + FIN_J - 1) / FIN_J), (unsigned)n_i);
    return launch_pdl(opm_finalize_kernel, grid, dim3(FIN_THREADS), 0, (cudaStream_t)stream, (const __nv_bfloat16*)y, bits, bias, z, i0, n, words, accumulate);
}
