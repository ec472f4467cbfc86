// softmax(q k^T + bias + mask) v with a gate, at fp32 accuracy: one-pass softmax over 64-key tiles, both products as six
// m16n8k16 bf16 MMAs on three-part operands (split.cuh: 24 bits of every factor, fp32 accumulation).
//
// mma.sync and not tcgen05: q, k, v rows are 24 or 32 wide and the probabilities need three parts of their own, so a tcgen05
// form would have to push three times the probabilities through tensor memory; here they go from the accumulators of the
// first product straight into the A fragments of the second.  A warp owns 16 queries; per 64-key tile it issues 192 MMAs
// (8 clocks each and scheduler: the bound) against some 650 other instructions.  K and V tiles are shared by the CTA's
// warps, double buffered with cp.async; rows are 64 bytes with the 16-byte chunks swizzled by row so that ldmatrix is
// conflict free.  Bias values are the accumulators' initial values.
#include "split_attn.cuh"

namespace b200pf {
namespace split {

constexpr int KT = 64, KV_PART = KT * 64, KV_STAGE = 6 * KV_PART;          // K parts | V parts

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

template <int HD, int NW>
__global__ void __launch_bounds__(NW * 32, 16 / NW) split_attention_kernel(AttnArgs p) {
    constexpr int CH = HD / 8, NE = HD / 8, NT = NW * 32;
    static_assert(HD == 24 || HD == 32, "head width");
    extern __shared__ __align__(128) uint8_t at_smem[];
    float* mterm = reinterpret_cast<float*>(at_smem + 2 * KV_STAGE);            // [2][KT]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int h = blockIdx.y, line = blockIdx.z;
    const int qw = blockIdx.x * (NW * 16) + warp * 16;                           // this warp's first query, relative to q0
    const bool active = qw < p.n_q;
    const int ht = p.heads * HD;
    if (HD == 24) {                                                              // the fourth chunk of every row stays zero
        for (int i = tid; i < 2 * 6 * KT; i += NT) {
            const int key = i % KT, part = i / KT;
            *reinterpret_cast<uint4*>(at_smem + part * KV_PART + key * 64 + ((3 ^ ((key >> 1) & 3)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    grid_dependency_wait();
    grid_launch_dependents();

    const __nv_bfloat16* base = p.qkv + (long long)line * p.line_rows * p.ld + h * HD;
    const long long pos_ld = p.pos_rows * p.ld;
    auto load_tile = [&](int tile) {
        const int k0 = tile * KT;
        const uint32_t st = smem_u32(at_smem + (tile & 1) * KV_STAGE);
        for (int i = tid; i < 6 * KT * CH; i += NT) {
            const int c = i % CH, key = (i / CH) % KT, part = i / (CH * KT);     // parts 0-2: K, 3-5: V
            const int kk = k0 + key;
            const bool in = kk < p.n_k;
            const __nv_bfloat16* src = base + (part >= 3 ? 2 * ht : ht) + (long long)(part >= 3 ? part - 3 : part) * p.part_stride +
                                       (in ? kk : 0) * pos_ld + c * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(st + part * KV_PART + key * 64 + ((c ^ ((key >> 1) & 3)) << 4)),
                         "l"(src), "r"(in ? 16 : 0) : "memory");
        }
        if (tid < KT) {
            const int kk = k0 + tid;
            float m = 0.f;
            if (kk >= p.n_k) m = -INFINITY;
            else if (p.mask && p.mask[line * p.mask_ls + kk * p.mask_ks] == 0) m = p.mask_add;
            mterm[(tile & 1) * KT + tid] = m;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_tile(0);

    const int r0 = min(qw + g, p.n_q - 1), r1 = min(qw + g + 8, p.n_q - 1);      // rows past the end repeat the last one
    uint32_t q[3][2][4];
#pragma unroll
    for (int part = 0; part < 3; ++part)
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const __nv_bfloat16* a = base + part * p.part_stride + (p.q0 + r0) * pos_ld + ks * 16 + 2 * t;
            const __nv_bfloat16* b = base + part * p.part_stride + (p.q0 + r1) * pos_ld + ks * 16 + 2 * t;
            q[part][ks][0] = *reinterpret_cast<const uint32_t*>(a);
            q[part][ks][1] = *reinterpret_cast<const uint32_t*>(b);
            q[part][ks][2] = HD == 24 && ks == 1 ? 0u : *reinterpret_cast<const uint32_t*>(a + 8);
            q[part][ks][3] = HD == 24 && ks == 1 ? 0u : *reinterpret_cast<const uint32_t*>(b + 8);
        }
    const float* bias0 = p.bias + h * p.bias_hs + r0 * p.bias_qs;
    const float* bias1 = p.bias + h * p.bias_hs + r1 * p.bias_qs;
    float o[NE][4];
#pragma unroll
    for (int e = 0; e < NE; ++e) { o[e][0] = o[e][1] = o[e][2] = o[e][3] = 0.f; }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    const int ntiles = (p.n_k + KT - 1) / KT;
    const uint32_t k_lane = (uint32_t)((lane & 7) * 64), k_sw = (uint32_t)(((lane >> 3) ^ ((lane >> 1) & 3)) << 4);     // row lane & 7, chunk lane / 8

#pragma unroll 1
    for (int tile = 0; tile < ntiles; ++tile) {
        float s[8][4];
        {
            const int k0 = tile * KT + 2 * t;
#pragma unroll
            for (int ni = 0; ni < 8; ++ni) {
                const int c0 = min(k0 + 8 * ni, p.n_k - 1), c1 = min(k0 + 8 * ni + 1, p.n_k - 1);
                s[ni][0] = bias0[c0]; s[ni][1] = bias0[c1]; s[ni][2] = bias1[c0]; s[ni][3] = bias1[c1];
            }
        }
        if (tile + 1 < ntiles) {
            load_tile(tile + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (active) {
            const uint32_t kst = smem_u32(at_smem + (tile & 1) * KV_STAGE), vst = kst + 3 * KV_PART;
            const float* mt = mterm + (tile & 1) * KT + 2 * t;
            float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
            for (int ni = 0; ni < 8; ++ni) {
                uint32_t kb[3][4];
#pragma unroll
                for (int part = 0; part < 3; ++part) ldsm4(kb[part], kst + part * KV_PART + ni * 512 + k_lane + k_sw);
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    mma_bf16(s[ni], q[2][ks], kb[0][2 * ks], kb[0][2 * ks + 1]);
                    mma_bf16(s[ni], q[1][ks], kb[1][2 * ks], kb[1][2 * ks + 1]);
                    mma_bf16(s[ni], q[0][ks], kb[2][2 * ks], kb[2][2 * ks + 1]);
                    mma_bf16(s[ni], q[1][ks], kb[0][2 * ks], kb[0][2 * ks + 1]);
                    mma_bf16(s[ni], q[0][ks], kb[1][2 * ks], kb[1][2 * ks + 1]);
                    mma_bf16(s[ni], q[0][ks], kb[0][2 * ks], kb[0][2 * ks + 1]);
                }
                const float2 mv = *reinterpret_cast<const float2*>(mt + 8 * ni);
                s[ni][0] += mv.x; s[ni][1] += mv.y; s[ni][2] += mv.x; s[ni][3] += mv.y;
                mx0 = fmaxf(mx0, fmaxf(s[ni][0], s[ni][1]));
                mx1 = fmaxf(mx1, fmaxf(s[ni][2], s[ni][3]));
            }
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
            // every tile holds a key inside n_k, whose score is finite: the new maxima are finite
            const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
            const float a0 = exp2f(m0 - n0), a1 = exp2f(m1 - n1);                // 0 on the first tile
            m0 = n0; m1 = n1;
            l0 *= a0; l1 *= a1;
            float ot[NE][4];
#pragma unroll
            for (int e = 0; e < NE; ++e) { ot[e][0] = ot[e][1] = ot[e][2] = ot[e][3] = 0.f; }
#pragma unroll
            for (int j = 0; j < 4; ++j) {                                        // 16 keys
                uint32_t pf[3][4];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    float* sv = s[2 * j + u];
                    sv[0] = exp2f(sv[0] - n0); sv[1] = exp2f(sv[1] - n0); sv[2] = exp2f(sv[2] - n1); sv[3] = exp2f(sv[3] - n1);
                    l0 += sv[0] + sv[1]; l1 += sv[2] + sv[3];
                    split_bf16x3(sv[0], sv[1], pf[0][2 * u], pf[1][2 * u], pf[2][2 * u]);
                    split_bf16x3(sv[2], sv[3], pf[0][2 * u + 1], pf[1][2 * u + 1], pf[2][2 * u + 1]);
                }
                // matrices: (keys 0-7, chunk), (keys 8-15, chunk), (keys 0-7, chunk + 1), (keys 8-15, chunk + 1)
                const int key = j * 16 + ((lane >> 3) & 1) * 8 + (lane & 7);
#pragma unroll
                for (int c2 = 0; c2 < 2; ++c2) {
                    uint32_t vb[3][4];
                    const uint32_t off = (uint32_t)(key * 64 + (((c2 * 2 + (lane >> 4)) ^ ((key >> 1) & 3)) << 4));
#pragma unroll
                    for (int part = 0; part < 3; ++part) ldsm4_t(vb[part], vst + part * KV_PART + off);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (c2 * 2 + u >= NE) continue;
                        float (&oe)[4] = ot[(c2 * 2 + u) % NE];
                        mma_bf16(oe, pf[2], vb[0][2 * u], vb[0][2 * u + 1]);
                        mma_bf16(oe, pf[1], vb[1][2 * u], vb[1][2 * u + 1]);
                        mma_bf16(oe, pf[0], vb[2][2 * u], vb[2][2 * u + 1]);
                        mma_bf16(oe, pf[1], vb[0][2 * u], vb[0][2 * u + 1]);
                        mma_bf16(oe, pf[0], vb[1][2 * u], vb[1][2 * u + 1]);
                        mma_bf16(oe, pf[0], vb[0][2 * u], vb[0][2 * u + 1]);
                    }
                }
            }
            // the tensor core truncates every addend to the running sum's ulp, always towards zero: a tile's products start
            // from zero and join the output with a rounded FMA
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                o[e][0] = fmaf(o[e][0], a0, ot[e][0]); o[e][1] = fmaf(o[e][1], a0, ot[e][1]);
                o[e][2] = fmaf(o[e][2], a1, ot[e][2]); o[e][3] = fmaf(o[e][3], a1, ot[e][3]);
            }
        }
        __syncthreads();
    }
    if (!active) return;
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    const float inv[2] = {p.out_scale / l0, p.out_scale / l1};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int qi = qw + g + 8 * half;
        if (qi >= p.n_q) continue;
        const long long row = line * p.line_rows + (p.q0 + qi) * p.pos_rows;
        const float* gp = p.gate + row * ht + h * HD + 2 * t;
        __half* op = p.out + (row - p.out_row0) * ht + h * HD + 2 * t;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const float2 gv = *reinterpret_cast<const float2*>(gp + 8 * e);
            uint32_t hi, lo;
            split_f16x2(o[e][2 * half] * inv[half] * gv.x, o[e][2 * half + 1] * inv[half] * gv.y, hi, lo);
            *reinterpret_cast<uint32_t*>(op + 8 * e) = hi;
            *reinterpret_cast<uint32_t*>(op + p.out_part_stride + 8 * e) = lo;
        }
    }
}

template <int HD, int NW> static int attn_go(const AttnArgs& a, cudaStream_t st) {
    constexpr int smem = 2 * KV_STAGE + 2 * KT * 4;
    auto kern = split_attention_kernel<HD, NW>;
    B200PF_SMEM_ATTR_ONCE(kern, smem);
    return launch_pdl(kern, dim3((unsigned)((a.n_q + NW * 16 - 1) / (NW * 16)), (unsigned)a.heads, (unsigned)a.lines), dim3(NW * 32), smem, st, a);
}

int launch_attention(const AttnArgs& a, int hd, cudaStream_t st) {
    B200PF_REQUIRE(a.qkv && a.gate && a.bias && a.out && aligned16(a.qkv) && a.part_stride % 8 == 0 && a.ld % 8 == 0, B200PF_ERR_INVALID,
                   "split attention: null or misaligned operand");
    B200PF_REQUIRE(a.lines > 0 && a.lines < 65536 && a.heads > 0 && a.n_q > 0 && a.n_k > 0, B200PF_ERR_INVALID, "split attention: bad sizes");
    B200PF_REQUIRE(hd == 24 || hd == 32, B200PF_ERR_UNSUPPORTED, "split attention: head width 24 or 32 (got %d)", hd);
    // eight warps share a K / V tile; with fewer than two such CTAs per SM, four warps per CTA spread the queries further
    const bool wide = (long long)a.lines * a.heads * ((a.n_q + 127) / 128) >= 2 * 148;
    if (hd == 24) return wide ? attn_go<24, 8>(a, st) : attn_go<24, 4>(a, st);
    return wide ? attn_go<32, 8>(a, st) : attn_go<32, 4>(a, st);
}

}  // namespace split
}  // namespace b200pf
