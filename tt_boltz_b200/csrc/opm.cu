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
//                         the GEMM's K-major operands; fp32 factors as two tf32 parts on mma.sync, bf16 on store.
//   opm_mask_bits_kernel: the MSA mask as one bit per sequence, 32 sequences per word and token.
//   opm_finalize_kernel : pair counts by popcount of the two tokens' words, then y / count + bias added into (or
//                         written over) the fp32 pair rows.
#include "pdl.cuh"

namespace b200pf {
namespace opm {

constexpr int CM = 64;            // MSA channels
constexpr int CH = 32;            // projected channels per side
constexpr int PROD_WARPS = 4, PROD_THREADS = PROD_WARPS * 32, PROD_ROWS = PROD_WARPS * 32;      // sequences per CTA and token
constexpr int WF_ENTRIES = 4 * 8 * 32;                           // weight fragments: 4 row blocks of 16, 8 K steps, 32 lanes
constexpr int STG_PITCH = 80;                                    // bytes per staged output row: 32 bf16 and 16 to spread the banks
constexpr int PROD_SMEM = 2 * WF_ENTRIES * 16 + PROD_WARPS * 2 * CH * STG_PITCH;                // 53,248
constexpr int FIN_THREADS = 256, FIN_J = 64;
constexpr int MAX_WORDS = 512;    // sequences / 32 the finalize kernel keeps in shared memory (S <= 16384)

// v = hi + lo, both rounded to tf32's 11 significant bits: 2^-23 of v is left.  cvt and not integer arithmetic: a NaN stays one.
__device__ __forceinline__ void split_tf32(float v, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(v));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(v - __uint_as_float(hi)));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// A warp takes 32 sequences of one token: D[output][sequence] = W x^T, three tf32 MMAs per product (hi*hi, hi*lo, lo*hi: 2^-22 of
// a product is left out), so every output lies as the operands want it.  The sum over the 64 channels may run in any order, so
// lane (g, t) owns channels 16 q + 4 t .. + 3 of row g: the rows arrive as whole 64-byte pieces straight into B fragments, and the
// weights are laid out once per CTA as A fragments in the same order.  A CTA walks several tokens.  One thread per row with the
// weights broadcast from shared memory (4096 FMAs and 1024 shared loads a row, every lane on lines of its own) took 230 us at
// 1024 sequences x 600 tokens.
__global__ void __launch_bounds__(PROD_THREADS, 4)
opm_producer_kernel(const float* m, const uint8_t* mask, const float* gamma, const float* beta, const float* w_ab, __nv_bfloat16* a_t,
                    __nv_bfloat16* b_t, int s_len, int n, int pitch, int vec) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint4* wf = reinterpret_cast<uint4*>(smem);                  // [part][row block][K step][lane]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    uint8_t* stg = smem + 2 * WF_ENTRIES * 16 + warp * (2 * CH * STG_PITCH);
    grid_dependency_wait();
    grid_launch_dependents();
    for (int i = threadIdx.x; i < WF_ENTRIES; i += PROD_THREADS) {
        const int ln = i & 31, ks = (i >> 5) & 7, mb = i >> 8;
        const float* w0 = w_ab + (mb * 16 + (ln >> 2)) * CM + (ks >> 1) * 16 + (ln & 3) * 4 + (ks & 1) * 2;
        const float2 lo8 = *reinterpret_cast<const float2*>(w0), hi8 = *reinterpret_cast<const float2*>(w0 + 8 * CM);
        uint4 h, l;
        split_tf32(lo8.x, h.x, l.x); split_tf32(hi8.x, h.y, l.y); split_tf32(lo8.y, h.z, l.z); split_tf32(hi8.y, h.w, l.w);
        wf[i] = h;
        wf[WF_ENTRIES + i] = l;
    }
    float4 gam[4], bet[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        gam[q] = make_float4(gamma[q * 16 + 4 * t], gamma[q * 16 + 4 * t + 1], gamma[q * 16 + 4 * t + 2], gamma[q * 16 + 4 * t + 3]);
        bet[q] = make_float4(beta[q * 16 + 4 * t], beta[q * 16 + 4 * t + 1], beta[q * 16 + 4 * t + 2], beta[q * 16 + 4 * t + 3]);
    }
    __syncthreads();
    const int s_base = blockIdx.x * PROD_ROWS + warp * 32;
    if (s_base >= s_len) return;
    for (int tok = blockIdx.y; tok < n; tok += gridDim.y) {
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {                   // 16 sequences: two column blocks of 8
            uint32_t xh[2][16], xl[2][16];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int s = s_base + half * 16 + nt * 8 + g;
                const long long row = (long long)(s < s_len ? s : s_len - 1) * n + tok;     // rows past the end repeat the last one
                const float4* src = reinterpret_cast<const float4*>(m + row * CM) + t;
                float4 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = src[q * 4];
                const float keep = mask[row] ? 1.f : 0.f;
                float sum = 0.f;
#pragma unroll
                for (int q = 0; q < 4; ++q) sum += (v[q].x + v[q].y) + (v[q].z + v[q].w);
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                const float mean = sum * (1.f / CM);
                float ss = 0.f;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    v[q].x -= mean; v[q].y -= mean; v[q].z -= mean; v[q].w -= mean;
                    ss += (v[q].x * v[q].x + v[q].y * v[q].y) + (v[q].z * v[q].z + v[q].w * v[q].w);
                }
                ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                ss += __shfl_xor_sync(0xffffffffu, ss, 2);
                const float rstd = rsqrtf(ss * (1.f / CM) + LN_EPS);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    split_tf32(fmaf(v[q].x * rstd, gam[q].x, bet[q].x) * keep, xh[nt][4 * q], xl[nt][4 * q]);
                    split_tf32(fmaf(v[q].y * rstd, gam[q].y, bet[q].y) * keep, xh[nt][4 * q + 1], xl[nt][4 * q + 1]);
                    split_tf32(fmaf(v[q].z * rstd, gam[q].z, bet[q].z) * keep, xh[nt][4 * q + 2], xl[nt][4 * q + 2]);
                    split_tf32(fmaf(v[q].w * rstd, gam[q].w, bet[q].w) * keep, xh[nt][4 * q + 3], xl[nt][4 * q + 3]);
                }
            }
#pragma unroll 1
            for (int mb = 0; mb < 4; ++mb) {
                float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, small[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const uint4 wh = wf[(mb * 8 + ks) * 32 + lane], wl = wf[WF_ENTRIES + (mb * 8 + ks) * 32 + lane];
                    const int e = (ks >> 1) * 4 + (ks & 1) * 2;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        mma_tf32(acc[nt], wh, xh[nt][e], xh[nt][e + 1]);
                        mma_tf32(small[nt], wh, xl[nt][e], xl[nt][e + 1]);
                        mma_tf32(small[nt], wl, xh[nt][e], xh[nt][e + 1]);
                    }
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    uint8_t* at = stg + (mb * 16 + g) * STG_PITCH + (half * 16 + nt * 8 + 2 * t) * 2;
                    *reinterpret_cast<uint32_t*>(at) = pack_bf16x2(acc[nt][0] + small[nt][0], acc[nt][1] + small[nt][1]);
                    *reinterpret_cast<uint32_t*>(at + 8 * STG_PITCH) = pack_bf16x2(acc[nt][2] + small[nt][2], acc[nt][3] + small[nt][3]);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int it = 0; it < 8; ++it) {                         // 64 output rows of 64 bytes, four lanes each
            const int o = it * 8 + g, s = s_base + t * 8;
            const uint4 v = *reinterpret_cast<const uint4*>(stg + o * STG_PITCH + t * 16);
            __nv_bfloat16* dst = (o < CH ? a_t : b_t) + ((long long)tok * CH + (o & (CH - 1))) * pitch + s;
            if (vec && s + 8 <= s_len) {
                *reinterpret_cast<uint4*>(dst) = v;
            } else {
                const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (s + e < s_len) reinterpret_cast<uint16_t*>(dst)[e] = (uint16_t)(w4[e >> 1] >> (16 * (e & 1)));
            }
        }
        __syncwarp();
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
    // four CTAs fit an SM; each takes every gridDim.y-th token of its sequences, so that its weight fragments serve several
    const int tiles = (s_len + PROD_ROWS - 1) / PROD_ROWS, want = (4 * sms + tiles - 1) / tiles, per = (n + want - 1) / want;
    const int vec = aligned16(a_t) && aligned16(b_t) && pitch % 8 == 0;
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
