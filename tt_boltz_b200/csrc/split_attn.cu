// softmax(q k^T + bias + mask) v with a gate, at fp32 accuracy: one-pass softmax over 64-key tiles, both products as three
// m16n8k16 fp16 MMAs on two-part operands (split.cuh), fp32 accumulation.
//
// For single lines (the single track) and rows of 24, which fill neither the line groups nor the swizzled rows of the tcgen05 form
// (split_attn_tc.cu: three lines and more, rows of 32); the probabilities go from the accumulators of the first product straight into
// the A fragments of the second.  A warp owns 16 queries; per 64-key tile it issues 96 MMAs.  With three bf16 parts and six MMAs per
// product, and every lane fetching its own bias values, a launch took 462 us at 292 tokens x 4 heads and 528 at 256 x 8; with two
// parts 390 and 430, with staged bias tiles 310 and 311, with one barrier a tile, interleaved accumulators, scores that stay in the
// products' scale, packed fp32 arithmetic (1190 -> 779 instructions per warp and tile) and masks fetched a tile ahead 258 and 245.
// K and V tiles are shared by the CTA's warps, double buffered with
// cp.async; rows are 64 bytes with the 16-byte chunks swizzled by row so that ldmatrix is conflict free.  Bias tiles come with them,
// as whole lines (read by the lanes that want them, 8 bytes of eight rows at a time and behind the tile before, they were the
// longest wait of a tile), and are the accumulators' initial values.
#include "split_attn.cuh"

namespace b200pf {
namespace split {

constexpr int KT = 64, KV_PART = KT * 64, KV_STAGE = 4 * KV_PART;          // K parts | V parts

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

constexpr int BP = KT + 8;               // bias tile pitch in floats: a half-warp's float2 reads of four rows meet no bank twice
constexpr int bias_stage(int nw) { return nw * 16 * BP * 4; }
constexpr float P_SCALE = 16384.f;       // probabilities are at most one: their parts use the upper half of fp16's range

// Two fp32 values in one 64-bit register for the packed instructions (one issue slot, two results).
__device__ __forceinline__ uint64_t f2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_get(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float m;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}

// 2^x of a score below the row's maximum.  PTX documents the instruction as an approximation good to some 2^-22 of its result, with
// results below 2^-126 flushed to zero.  A row's largest probability is 1, so a flushed one is below 2^-126 of the row's sum, and each
// of its products below 2^-126 of the largest value: nothing that 24 bits of either could show.
__device__ __forceinline__ float prob(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The reference of a row that has met no key with a finite score: above that of any other, and so far that two to the difference is 0.
constexpr float NO_KEYS = 3e38f;

// Shared memory of a key group: its K / V, bias and mask tiles
constexpr int group_bytes(int nw) { return 2 * (KV_STAGE + bias_stage(nw) + KT * 4); }

// A CTA is KS groups of NW warps: every group has the CTA's NW * 16 queries and each KS-th key tile, with two stages and a barrier of its own.
template <int HD, int NW, int KS>
__global__ void __launch_bounds__(KS * NW * 32, KS > 1 ? 1 : 16 / NW) split_attention_kernel(AttnArgs p) {
    constexpr int CH = HD / 8, NE = HD / 8, NT = NW * 32;
    static_assert(HD == 24 || HD == 32, "head width");
    extern __shared__ __align__(128) uint8_t at_smem_all[];
    const int kg = KS > 1 ? (int)threadIdx.x / NT : 0;                           // this warp's key group
    uint8_t* at_smem = at_smem_all + kg * group_bytes(NW);
    uint8_t* bias_s = at_smem + 2 * KV_STAGE;                                   // [2][NW * 16 queries][BP]
    float* mterm = reinterpret_cast<float*>(bias_s + 2 * bias_stage(NW));       // [2][KT]
    const int tid = (int)threadIdx.x - kg * NT, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    auto group_sync = [&] {
        if (KS == 1) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(kg + 1), "n"(NT) : "memory");
    };
    const int h = blockIdx.y, line = blockIdx.z;
    const int qw = blockIdx.x * (NW * 16) + warp * 16;                           // this warp's first query, relative to q0
    const bool active = qw < p.n_q;
    const int ht = p.heads * HD;
    if (HD == 24) {                                                              // the fourth chunk of every row stays zero
        for (int i = tid; i < 2 * 4 * KT; i += NT) {
            const int key = i % KT, part = i / KT;
            *reinterpret_cast<uint4*>(at_smem + part * KV_PART + key * 64 + ((3 ^ ((key >> 1) & 3)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    grid_dependency_wait();
    grid_launch_dependents();

    const __half* base = p.qkv + (long long)line * p.line_rows * p.ld + h * HD;
    const long long pos_ld = p.pos_rows * p.ld;
    const int qb = blockIdx.x * (NW * 16);
    const float* brow = p.bias + h * p.bias_hs;
    auto mask_term = [&](int kk) {
        if (kk >= p.n_k) return -INFINITY;
        return p.mask && p.mask[line * p.mask_ls + kk * p.mask_ks] == 0 ? p.mask_add : 0.f;
    };
    float m_next = tid < KT ? mask_term(kg * KT + tid) : 0.f;          // this thread's key of the next tile to be loaded, fetched a tile ahead
    auto load_tile = [&](int tile, int stage) {
        const int k0 = tile * KT;
        {   // K and V parts: four chunk slots per row (HD = 24 leaves the fourth out), NT / 4 rows at a time
            const uint32_t st = smem_u32(at_smem + stage * KV_STAGE);
            const int c = tid & 3;
            if (HD == 32 || c < CH) {
#pragma unroll
                for (int kr = 0; kr < KT; kr += NT / 4) {
                    const int key = kr + (tid >> 2), kk = k0 + key;
                    const bool in = kk < p.n_k;
                    const __half* src = base + ht + (in ? kk : 0) * pos_ld + c * 8;
                    const uint32_t dst = st + key * 64 + ((c ^ ((key >> 1) & 3)) << 4);
#pragma unroll
                    for (int part = 0; part < 4; ++part)                         // parts 0-1: K, 2-3: V
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + part * KV_PART),
                                     "l"(src + (part >= 2 ? ht : 0) + (part & 1) * p.part_stride), "r"(in ? 16 : 0) : "memory");
                }
            }
        }
        const uint32_t bst = smem_u32(bias_s + stage * bias_stage(NW));
        if (p.bias_vec) {
            const int c = (tid % (KT / 4)) * 4, rt = tid / (KT / 4);
            const bool in = k0 + c < p.n_k;
            const float* src = brow + (in ? k0 + c : 0);
#pragma unroll 4
            for (int r = rt; r < NW * 16; r += NT / (KT / 4))
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(bst + (r * BP + c) * 4),
                             "l"(src + min(qb + r, p.n_q - 1) * p.bias_qs), "r"(in ? 16 : 0) : "memory");
        } else {
            const int c = tid % KT, rt = tid / KT;
            const bool in = k0 + c < p.n_k;
            const float* src = brow + (in ? k0 + c : 0);
#pragma unroll 4
            for (int r = rt; r < NW * 16; r += NT / KT)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(bst + (r * BP + c) * 4),
                             "l"(src + min(qb + r, p.n_q - 1) * p.bias_qs), "r"(in ? 4 : 0) : "memory");
        }
        if (tid < KT) mterm[stage * KT + tid] = m_next;
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (tid < KT) m_next = mask_term(k0 + KS * KT + tid);
    };
    load_tile(kg, 0);

    const int r0 = min(qw + g, p.n_q - 1), r1 = min(qw + g + 8, p.n_q - 1);      // rows past the end repeat the last one
    uint32_t q[2][2][4];
#pragma unroll
    for (int part = 0; part < 2; ++part)
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const __half* a = base + part * p.part_stride + (p.q0 + r0) * pos_ld + ks * 16 + 2 * t;
            const __half* b = base + part * p.part_stride + (p.q0 + r1) * pos_ld + ks * 16 + 2 * t;
            q[part][ks][0] = *reinterpret_cast<const uint32_t*>(a);
            q[part][ks][1] = *reinterpret_cast<const uint32_t*>(b);
            q[part][ks][2] = HD == 24 && ks == 1 ? 0u : *reinterpret_cast<const uint32_t*>(a + 8);
            q[part][ks][3] = HD == 24 && ks == 1 ? 0u : *reinterpret_cast<const uint32_t*>(b + 8);
        }
    float o[NE][4];
#pragma unroll
    for (int e = 0; e < NE; ++e) { o[e][0] = o[e][1] = o[e][2] = o[e][3] = 0.f; }
    // Scores stay in the scaled domain of the products (qk is a power of two, so that moves no value); c0 / c1 are the rows'
    // references as they enter the exponent, minus the maximum so far, and l0 / l1 the sums of the probabilities.
    float c0 = INFINITY, c1 = INFINITY, mq0 = -INFINITY, mq1 = -INFINITY;
    uint64_t l0 = f2(0.f, 0.f), l1 = l0;
    const int ntiles = (p.n_k + KT - 1) / KT;
    const float qk = p.qk_scale, qk_inv = 1.f / p.qk_scale;                      // powers of two
    const uint64_t qk2 = f2(qk, qk), qk_inv2 = f2(qk_inv, qk_inv), p_scale2 = f2(P_SCALE, P_SCALE);
    const uint32_t k_lane = (uint32_t)((lane & 7) * 64), k_sw = (uint32_t)(((lane >> 3) ^ ((lane >> 1) & 3)) << 4);     // row lane & 7, chunk lane / 8

#pragma unroll 1
    for (int tile = kg, stage = 0; tile < ntiles; tile += KS, stage ^= 1) {
        // one barrier per tile: behind it this tile has arrived, and every warp of the group is through the tile before, whose
        // stage the next one overwrites
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        group_sync();
        if (tile + KS < ntiles) load_tile(tile + KS, stage ^ 1);
        if (active) {
            float s[8][4];
            const float* bt = reinterpret_cast<const float*>(bias_s + stage * bias_stage(NW)) + (warp * 16 + g) * BP + 2 * t;
#pragma unroll
            for (int ni = 0; ni < 8; ++ni) {
                const float2 b0 = *reinterpret_cast<const float2*>(bt + 8 * ni), b1 = *reinterpret_cast<const float2*>(bt + 8 * BP + 8 * ni);
                f2_get(f2_mul(f2(b0.x, b0.y), qk2), s[ni][0], s[ni][1]);
                f2_get(f2_mul(f2(b1.x, b1.y), qk2), s[ni][2], s[ni][3]);
            }
            const uint32_t kst = smem_u32(at_smem + stage * KV_STAGE), vst = kst + 2 * KV_PART;
            const float* mt = mterm + stage * KT;
            const float2 mine = *reinterpret_cast<const float2*>(mt + 2 * lane);
            const bool masked = __any_sync(0xffffffffu, mine.x != 0.f || mine.y != 0.f);
#pragma unroll
            for (int n2 = 0; n2 < 8; n2 += 2) {          // two column blocks at a time: their accumulators' chains interleave
                uint32_t kb[2][2][4];
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int part = 0; part < 2; ++part) ldsm4(kb[u][part], kst + part * KV_PART + (n2 + u) * 512 + k_lane + k_sw);
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) mma_f16(s[n2 + u], q[1][ks], kb[u][0][2 * ks], kb[u][0][2 * ks + 1]);
#pragma unroll
                    for (int u = 0; u < 2; ++u) mma_f16(s[n2 + u], q[0][ks], kb[u][1][2 * ks], kb[u][1][2 * ks + 1]);
#pragma unroll
                    for (int u = 0; u < 2; ++u) mma_f16(s[n2 + u], q[0][ks], kb[u][0][2 * ks], kb[u][0][2 * ks + 1]);
                }
            }
            if (masked) {
#pragma unroll
                for (int ni = 0; ni < 8; ++ni) {
                    const float2 mv = *reinterpret_cast<const float2*>(mt + 8 * ni + 2 * t);
                    s[ni][0] = fmaf(mv.x, qk, s[ni][0]); s[ni][1] = fmaf(mv.y, qk, s[ni][1]);
                    s[ni][2] = fmaf(mv.x, qk, s[ni][2]); s[ni][3] = fmaf(mv.y, qk, s[ni][3]);
                }
            }
            float mx0 = mq0, mx1 = mq1;
#pragma unroll
            for (int ni = 0; ni < 8; ++ni) {
                mx0 = max3(mx0, s[ni][0], s[ni][1]);
                mx1 = max3(mx1, s[ni][2], s[ni][3]);
            }
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
            // The maximum of keys that the bias excludes (-inf) is -inf; a finite reference gives each of them, and whatever they are
            // joined with later, a zero.  A key group may have no other keys than such ones.
            mq0 = mx0; mq1 = mx1;
            const float d0 = fminf(-mx0 * qk_inv, NO_KEYS), d1 = fminf(-mx1 * qk_inv, NO_KEYS);
            const float a0 = exp2f(d0 - c0), a1 = exp2f(d1 - c1);                // 0 on the first tile
            c0 = d0; c1 = d1;
            const uint64_t c02 = f2(d0, d0), c12 = f2(d1, d1), a02 = f2(a0, a0), a12 = f2(a1, a1);
            l0 = f2_mul(l0, a02); l1 = f2_mul(l1, a12);
            float ot[NE][4];
#pragma unroll
            for (int e = 0; e < NE; ++e) { ot[e][0] = ot[e][1] = ot[e][2] = ot[e][3] = 0.f; }
#pragma unroll
            for (int j = 0; j < 4; ++j) {                                        // 16 keys
                // matrices: (keys 0-7, chunk), (keys 8-15, chunk), (keys 0-7, chunk + 1), (keys 8-15, chunk + 1)
                const int key = j * 16 + ((lane >> 3) & 1) * 8 + (lane & 7);
                uint32_t vb[2][2][4];
#pragma unroll
                for (int c2 = 0; c2 < 2; ++c2)
#pragma unroll
                    for (int part = 0; part < 2; ++part)
                        ldsm4_t(vb[c2][part], vst + part * KV_PART + (uint32_t)(key * 64 + (((c2 * 2 + (lane >> 4)) ^ ((key >> 1) & 3)) << 4)));
                uint32_t pf[2][4];
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const float* sv = s[2 * j + u] + 2 * r;
                        // The score minus the maximum, rounded once: never above zero, and finest for the keys that matter.  The parts'
                        // scale comes behind, exactly: in the reference (14 - maximum) it rounds the exponents of a row's largest
                        // probabilities at 2^-20 and takes the attention's error against 64 bits from 1.74e-7 to 2.61e-7 (292 keys,
                        // normal scores); the multiplication takes no time that shows (260 us a launch at 292 x 4 both ways).
                        float x0, x1;
                        f2_get(f2_fma(f2(sv[0], sv[1]), qk_inv2, r ? c12 : c02), x0, x1);
                        const uint64_t pr = f2(prob(x0), prob(x1));
                        if (r) l1 = f2_add(l1, pr);
                        else l0 = f2_add(l0, pr);
                        f2_get(f2_mul(pr, p_scale2), x0, x1);
                        split_f16x2(x0, x1, pf[0][2 * u + r], pf[1][2 * u + r]);
                    }
#pragma unroll
                for (int e = 0; e < NE; ++e) mma_f16(ot[e], pf[1], vb[e >> 1][0][2 * (e & 1)], vb[e >> 1][0][2 * (e & 1) + 1]);
#pragma unroll
                for (int e = 0; e < NE; ++e) mma_f16(ot[e], pf[0], vb[e >> 1][1][2 * (e & 1)], vb[e >> 1][1][2 * (e & 1) + 1]);
#pragma unroll
                for (int e = 0; e < NE; ++e) mma_f16(ot[e], pf[0], vb[e >> 1][0][2 * (e & 1)], vb[e >> 1][0][2 * (e & 1) + 1]);
            }
            // the tensor core truncates every addend to the running sum's ulp, always towards zero: a tile's products start
            // from zero and join the output with a rounded FMA
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                f2_get(f2_fma(f2(o[e][0], o[e][1]), a02, f2(ot[e][0], ot[e][1])), o[e][0], o[e][1]);
                f2_get(f2_fma(f2(o[e][2], o[e][3]), a12, f2(ot[e][2], ot[e][3])), o[e][2], o[e][3]);
            }
        }
    }
    float sum[2], x, y;
    f2_get(l0, x, y);
    sum[0] = x + y;
    f2_get(l1, x, y);
    sum[1] = x + y;
    if constexpr (KS > 1) {
        // the groups' sums and outputs meet in the first one, each brought from its own maximum to the largest
        constexpr int NV = 4 + 4 * NE;
        group_sync();                                            // every warp of the group is through its last tile
        float* mine = reinterpret_cast<float*>(at_smem) + tid;
        if (kg > 0) {
            mine[0] = c0; mine[NT] = c1; mine[2 * NT] = sum[0]; mine[3 * NT] = sum[1];
#pragma unroll
            for (int e = 0; e < 4 * NE; ++e) mine[(4 + e) * NT] = o[e >> 2][e & 3];
        }
        __syncthreads();
        if (kg > 0) return;
        static_assert(NV * NT * 4 <= KV_STAGE, "a group's results lie over its first tile");
#pragma unroll 1
        for (int k = 1; k < KS; ++k) {
            const float* other = reinterpret_cast<const float*>(at_smem_all + k * group_bytes(NW)) + tid;
            const float d0 = fminf(c0, other[0]), d1 = fminf(c1, other[NT]);         // c0 and c1 are minus the maxima
            const float a0 = exp2f(d0 - c0), a1 = exp2f(d1 - c1), b0 = exp2f(d0 - other[0]), b1 = exp2f(d1 - other[NT]);
            c0 = d0; c1 = d1;
            sum[0] = fmaf(sum[0], a0, other[2 * NT] * b0);
            sum[1] = fmaf(sum[1], a1, other[3 * NT] * b1);
#pragma unroll
            for (int e = 0; e < 4 * NE; ++e) o[e >> 2][e & 3] = fmaf(o[e >> 2][e & 3], e & 2 ? a1 : a0, other[(4 + e) * NT] * (e & 2 ? b1 : b0));
        }
    }
    if (!active) return;
    float inv[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        float x = sum[r];
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        inv[r] = 1.f / (x * P_SCALE);
    }
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

template <int HD, int NW, int KS> static int attn_go(const AttnArgs& a, cudaStream_t st) {
    constexpr int smem = KS * group_bytes(NW);         // NW = 8: 107,008, two CTAs per SM; three groups of four 210,432
    auto kern = split_attention_kernel<HD, NW, KS>;
    B200PF_SMEM_ATTR_ONCE(kern, smem);
    return launch_pdl(kern, dim3((unsigned)((a.n_q + NW * 16 - 1) / (NW * 16)), (unsigned)a.heads, (unsigned)a.lines), dim3(KS * NW * 32), smem, st, a);
}
// A line by itself gives a scheduler one warp, whose chains nothing overlaps, up to some 1000 queries; with three key groups per CTA it has
// three (an SM's shared memory holds their tiles): 33.6 -> 19.8 us at 509 tokens x 16 heads, 26.7 -> 17.1 at 400, 22.2 -> 14.5 at 300, 17.6 ->
// 13.0 at 203, 60.8 -> 52 at 1024; beside the pair track, whose kernels wait for the SMs that it holds, a block takes 1303 -> 1289, 518 -> 509 at 300
// and 261 -> 258.5 at 203.  Two groups: 20.7, 17.4, 14.4 and 12.9; four with a stage each: 19.6, 17.7, 15.8 and 13.6.  Two tiles of
// keys aren't worth it (130 -> 133 a block at 117).  1024 keys stay below where 16 heads need a third round of such CTAs, one per SM: 77 -> 67
// at 1025 and 73 -> 65 at 1100, where two rounds still do, would gain too, but 1300, 1500 and 2048 lose (85 -> 97, 96 -> 110, 149 -> 170).
// The choice looks at the keys only: a range of the queries has the bits of all of them.
template <int HD> static int attn_pick(const AttnArgs& a, int sms, cudaStream_t st) {
    if (a.lines == 1 && a.n_k > 2 * KT && a.n_k <= 1024) return attn_go<HD, 4, 3>(a, st);
    // eight warps share a K / V tile; with fewer than two such CTAs per SM, four warps per CTA spread the queries further
    if ((long long)a.lines * a.heads * ((a.n_q + 127) / 128) >= 2LL * sms) return attn_go<HD, 8, 1>(a, st);
    return attn_go<HD, 4, 1>(a, st);
}

int launch_attention(const AttnArgs& args, int hd, cudaStream_t st) {
    AttnArgs a = args;
    // 16-byte pieces of the bias rows where every one starts on a 16-byte boundary and ends inside its row, single values elsewhere
    a.bias_vec = aligned16(a.bias) && a.bias_hs % 4 == 0 && a.bias_qs % 4 == 0 && a.n_k % 4 == 0;
    B200PF_REQUIRE(a.qkv && a.gate && a.bias && a.out && aligned16(a.qkv) && a.part_stride % 8 == 0 && a.ld % 8 == 0, B200PF_ERR_INVALID,
                   "split attention: null or misaligned operand");
    B200PF_REQUIRE(a.lines > 0 && a.lines < 65536 && a.heads > 0 && a.n_q > 0 && a.n_k > 0, B200PF_ERR_INVALID, "split attention: bad sizes");
    B200PF_REQUIRE(hd == 24 || hd == 32, B200PF_ERR_UNSUPPORTED, "split attention: head width 24 or 32 (got %d)", hd);
    // 322 -> 199 us for the whole sub-operation at 292 tokens x 4 heads, 77 -> 53 at 130, 33 -> 27 at 65, 27 -> 22 at 48
    if (attention_tc_fits(a, hd)) return launch_attention_tc(a, st);
    int sms, rc;
    if ((rc = device_multiprocessors(&sms)) != B200PF_OK) return rc;      // its CTAs share an SM: a CtaLimit does not mean them
    return hd == 24 ? attn_pick<24>(a, sms, st) : attn_pick<32>(a, sms, st);
}

}  // namespace split
}  // namespace b200pf
