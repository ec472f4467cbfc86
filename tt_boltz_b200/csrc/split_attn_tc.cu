// softmax(q k^T + bias + mask) v with a gate, at fp32 accuracy, on tcgen05: the triangle attention of the fp32 tier.
//
// One CTA works on (head, 128 queries, three consecutive lines, which share the bias tiles).  Roles (512 threads):
//   warps 0-11   softmax group g = warp / 4 -> line l + g   (thread = query row = TMEM lane)
//   warp  12     TMA producer   (bias tiles shared by the lines; q, k, v parts of all three in one box each)
//   warps 13-15  MMA issuers, one per group
// Per 64-key tile and group: S = q k^T as three fp16 MMAs per product (split.cuh; small terms first) into 64 columns of tensor memory; the
// softmax thread reads its row, adds the fp32 bias from the shared tile with one FMA per score, takes the row's maximum (a row is a thread:
// no shuffles), and writes the probabilities' two parts over the scores' columns, the A operands of O = p v.  A tile's products start from
// zero and join the output, which stays in registers, with a rounded FMA: the tensor core truncates every addend to the running sum's ulp.
// v lies as it comes, keys by channels: an MN-major B operand.  Scores are double buffered, so that a tile's products run under the softmax
// of the one before.  TMEM columns per group: S / P 2 x 64 | O 32, 480 in all.
//
// The mma.sync kernel that it takes the place of (split_attn.cu, which stays for what does not fit here: fewer than three lines, rows of 24,
// a range of the queries, bias rows off 16-byte boundaries) spent a tile on 96 MMAs and 680 other instructions in dependent chains with 3.6
// warps per scheduler: 261 us a launch at 292 tokens x 4 heads, 246 at 256 x 8; now 137 and some 135.  Errors of the whole sub-operation
// against 64 bits: 1.18e-6 for 1.23e-6 at 292 x 4, 1.99e-6 for 2.12e-6 at 256 x 8.
// What bounds it: a 64-key tile of the three groups takes 4 k clocks, 2 k of them the exponentials and parts (1.5 k are the exp2 unit's),
// 1.1 k scores and maximum, 0.4 k waits; an item's end (gates, transposition, store) another 4.6 k.  On the way: masks fetched by the
// softmax warps +12 us, a row per lane for gates and stores +24, the next item's scores ahead of this one's last P V +5.
// Every wait is bounded; a wait that runs out raises the status word and the CTA unwinds.
#include "split_attn.cuh"
#include "tmap.cuh"

namespace b200pf {
namespace split {
namespace tc {

constexpr int AQ = 128, AK = 64, HD = 32, NG = 3, ST = 2;
constexpr int ROW_BYTES = HD * 2;                                  // 64: rows of q, k and v parts, 64-byte swizzle
constexpr int Q_BYTES = AQ * ROW_BYTES, KV_BYTES = AK * ROW_BYTES;  // one line, one part: 8192, 4096
constexpr int Q_TILE = 2 * NG * Q_BYTES, KV_TILE = 2 * NG * KV_BYTES;       // [part][line][row]
constexpr int BIAS_BOX = AQ * 128, BIAS_TILE = 2 * BIAS_BOX;       // two boxes of [128 queries][32 keys] fp32, 128-byte swizzle
constexpr int OFF_BIAS = 0, OFF_Q = ST * BIAS_TILE, OFF_K = OFF_Q + Q_TILE, OFF_V = OFF_K + ST * KV_TILE;
constexpr int OFF_BAR = OFF_V + ST * KV_TILE;
constexpr int SMEM_BYTES = OFF_BAR + 512;                          // 213,504
constexpr int TMA_WARP = 12, MMA_WARP0 = 13, THREADS = 16 * 32;
constexpr uint32_t GROUP_COLS = 160, COL_O = 128;
constexpr float P_SCALE = 16384.f;       // probabilities are at most one: their parts use the upper half of fp16's range

struct Bars {
    uint64_t k_full[ST], k_empty[ST], v_full[ST], v_empty[ST], b_full[ST], b_empty[ST], q_full, q_empty;
    uint64_t s_full[NG][2], p_full[NG], pv_done[NG];
    uint2 keep[NG][2];                  // with s_full: one bit per key of the tile, 1 = attends
    uint32_t tmem_slot;
    int abort_flag;
};
static_assert(sizeof(Bars) <= 512, "barriers");

// Rows of 64 bytes with the 64-byte swizzle, 8-row groups 512 bytes apart: K-major for q and k, MN-major (rows are the contraction, one
// 32-channel atom wide) for v.
__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}
constexpr uint32_t idesc_f16(int m, int n, bool b_mn) {            // fp16 x fp16 -> fp32
    return (1u << 4) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}
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
// 2^x of a score below the row's maximum, good to some 2^-22 of the result; below 2^-126 flushed to zero, which is below 2^-126 of the
// row's sum.
__device__ __forceinline__ float prob(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}

// Half a row's scores (32 keys): the accumulators plus the bias, and the masked keys' term; keys at or beyond `left` are excluded.
// `keep`: bit e, key e attends.  Both are uniform over the warp.
__device__ __forceinline__ void scores32(float (&t)[32], uint32_t s_addr, const uint8_t* bias_row, int row, uint64_t qk_inv2, uint32_t keep, float mask_add, int left) {
#pragma unroll
    for (int hc = 0; hc < 2; ++hc) {
        uint32_t sr[16];
        tmem_ld_32x16(s_addr + hc * 16, sr);
        float4 b[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(bias_row + (((hc * 4 + c) ^ (row & 7)) << 4));
        sm100::tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int e = hc * 16 + c * 4, q = c * 4;
            f2_get(f2_fma(f2(__uint_as_float(sr[q]), __uint_as_float(sr[q + 1])), qk_inv2, f2(b[c].x, b[c].y)), t[e], t[e + 1]);
            f2_get(f2_fma(f2(__uint_as_float(sr[q + 2]), __uint_as_float(sr[q + 3])), qk_inv2, f2(b[c].z, b[c].w)), t[e + 2], t[e + 3]);
        }
    }
    if (keep != 0xffffffffu || left < 32) {
#pragma unroll
        for (int e = 0; e < 32; ++e) t[e] = e >= left ? -INFINITY : (keep >> e) & 1u ? t[e] : t[e] + mask_add;
    }
}
__device__ __forceinline__ float max32(const float (&t)[32], float m) {
    float m4[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int e = 0; e < 32; e += 8)
#pragma unroll
        for (int i = 0; i < 4; ++i) m4[i] = max3(m4[i], t[e + 2 * i], t[e + 2 * i + 1]);
    return fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
}
// Probabilities of 32 keys relative to the maximum -m, their sum, and their two parts into tensor memory.
__device__ __forceinline__ void probs32(const float (&t)[32], float negm, uint64_t& la, uint64_t& lb, uint32_t p_addr) {
    uint32_t hi[16], lo[16];
    const uint64_t negm2 = f2(negm, negm), scale2 = f2(P_SCALE, P_SCALE);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        float x0, x1;
        f2_get(f2_add(f2(t[2 * e], t[2 * e + 1]), negm2), x0, x1);
        const uint64_t pr = f2(prob(x0), prob(x1));
        if (e & 1) lb = f2_add(lb, pr);
        else la = f2_add(la, pr);
        f2_get(f2_mul(pr, scale2), x0, x1);
        split_f16x2(x0, x1, hi[e], lo[e]);
    }
    sm100::tmem_st_32x16(p_addr, hi);
    sm100::tmem_st_32x16(p_addr + 16, lo);
}

__global__ void __launch_bounds__(THREADS, 1)
split_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_bias,
                          AttnArgs p, unsigned int* status) {
    using namespace sm100;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {       // swizzled tiles need 1024-byte alignment; there is no slack to fix it up
        grid_dependency_wait();
        if (threadIdx.x == 0) atomicOr(status, DEV_STATUS_BAD_INDEX);
        return;
    }
    Bars* B = reinterpret_cast<Bars*>(smem + OFF_BAR);
    volatile int* abort_flag = &B->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int qtiles = (p.n_q + AQ - 1) / AQ, T = (p.n_k + AK - 1) / AK;
    const int trios = (p.lines + NG - 1) / NG;
    const int items = trios * p.heads * qtiles;                        // checked to be an int where it is launched
    const uint32_t my_items = (int)blockIdx.x < items ? (uint32_t)((items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) : 0u;
    const uint32_t total = my_items * (uint32_t)T;                     // tiles of this CTA

    if (tid == 0) {
        for (int i = 0; i < ST; ++i) {
            mbar_init(&B->k_full[i], 1); mbar_init(&B->k_empty[i], NG);
            mbar_init(&B->v_full[i], 1); mbar_init(&B->v_empty[i], NG);
            mbar_init(&B->b_full[i], 1); mbar_init(&B->b_empty[i], NG * 4);
        }
        mbar_init(&B->q_full, 1); mbar_init(&B->q_empty, NG);
        for (int g = 0; g < NG; ++g) {
            mbar_init(&B->s_full[g][0], 2); mbar_init(&B->s_full[g][1], 2);          // the products, and the key bits
            mbar_init(&B->p_full[g], 4); mbar_init(&B->pv_done[g], 1);
        }
        B->abort_flag = 0;
        fence_barrier_init();
    }
    if (tid == TMA_WARP * 32) { tma_prefetch_desc(&map_q); tma_prefetch_desc(&map_kv); tma_prefetch_desc(&map_bias); }
    if (warp == MMA_WARP0) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dependency_wait();                 // behind the CTA's barrier: every warp goes to work by itself from here on
    grid_launch_dependents();
    const uint32_t tmem_base = B->tmem_slot;

    auto decode = [&](int it, int& qt, int& h, int& line0) {
        const int u = it / qtiles;
        qt = it - u * qtiles;
        line0 = u / p.heads;
        h = u - line0 * p.heads;
        line0 *= NG;
    };

    if (warp == TMA_WARP) {
        if (lane == 0) {
            // ------------------------------ TMA producer ------------------------------
            uint32_t G = 0, k = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++k) {
                int qt, h, line0;
                decode(it, qt, h, line0);
                ok = mbar_wait(&B->q_empty, (k & 1) ^ 1, abort_flag);
                if (!ok) break;
                mbar_arrive_expect_tx(&B->q_full, Q_TILE);
                tma_load_5d(smem + OFF_Q, &map_q, &B->q_full, 0, h, qt * AQ, line0, 0);          // lines past the last one arrive as zeros
                for (int j = 0; j < T; ++j, ++G) {
                    const uint32_t st = G % ST, ph = ((G / ST) & 1) ^ 1;
                    ok = mbar_wait(&B->k_empty[st], ph, abort_flag);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&B->k_full[st], KV_TILE);
                    tma_load_5d(smem + OFF_K + st * KV_TILE, &map_kv, &B->k_full[st], 0, p.heads + h, j * AK, line0, 0);
                    ok = mbar_wait(&B->b_empty[st], ph, abort_flag);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&B->b_full[st], BIAS_TILE);
                    tma_load_4d(smem + OFF_BIAS + st * BIAS_TILE, &map_bias, &B->b_full[st], j * AK, qt * AQ, h, 0);
                    tma_load_4d(smem + OFF_BIAS + st * BIAS_TILE + BIAS_BOX, &map_bias, &B->b_full[st], j * AK + 32, qt * AQ, h, 0);
                    ok = mbar_wait(&B->v_empty[st], ph, abort_flag);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&B->v_full[st], KV_TILE);
                    tma_load_5d(smem + OFF_V + st * KV_TILE, &map_kv, &B->v_full[st], 0, 2 * p.heads + h, j * AK, line0, 0);
                }
            }
            if (!ok) {
                atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
                uint64_t t0 = global_timer_ns();
                while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
            }
        }
    } else if (warp >= MMA_WARP0) {
        // ------------------------------ MMA issuer of group g ------------------------------
        // The whole warp runs the loop and waits; one elected lane issues (see sm100::elect_one).
        const uint32_t g = (uint32_t)__shfl_sync(0xffffffffu, warp - MMA_WARP0, 0);
        constexpr uint32_t idesc_s = idesc_f16(AQ, AK, false), idesc_o = idesc_f16(AQ, HD, true);
        constexpr uint32_t Q_PART = (NG * Q_BYTES) >> 4, KV_PART = (NG * KV_BYTES) >> 4, KV_STEP = KV_TILE >> 4;      // 16-byte units
        const uint64_t d_q = desc_sw64(smem_u32(smem + OFF_Q + g * Q_BYTES));
        const uint64_t d_k = desc_sw64(smem_u32(smem + OFF_K + g * KV_BYTES)), d_v = desc_sw64(smem_u32(smem + OFF_V + g * KV_BYTES));
        const uint32_t t_s = tmem_base + g * GROUP_COLS, t_o = t_s + COL_O;
        const bool short_last = p.n_k - (T - 1) * AK <= AK / 2;        // a last tile of at most 32 keys: half of its products
        uint32_t js = 0, ks = 0, jp = 0;                               // the next S: tile of its item, and item; the next P V: tile of its item
        // The key mask of a line is the same for all its queries: the issuer makes bits of it (lane l holds keys l and 32 + l of the next S,
        // fetched a tile ahead), which come with the scores.  In the twelve softmax warps this was a seventh of a tile's time.
        uint32_t m0 = 1, m1 = 1;
        auto mask_fetch = [&] {
            const int it = (int)(blockIdx.x + ks * gridDim.x);
            if (!p.mask || it >= items) return;
            int qt, h, line0;
            decode(it, qt, h, line0);
            const int line = line0 + (int)g < p.lines ? line0 + (int)g : p.lines - 1, key = (int)js * AK + lane;
            const uint8_t* at = p.mask + line * p.mask_ls + key * p.mask_ks;
            m0 = key < p.n_k ? *at : 1u;
            m1 = key + 32 < p.n_k ? at[32 * p.mask_ks] : 1u;
        };
        if (total > 0) mask_fetch();
        auto scores = [&](uint32_t G) {
            const uint32_t st = G % ST;
            if (js == 0 && !mbar_wait_warp(&B->q_full, ks & 1, abort_flag)) return false;
            if (!mbar_wait_warp(&B->k_full[st], (G / ST) & 1, abort_flag)) return false;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t dk = d_k + st * KV_STEP;
                const uint32_t ts = t_s + (G & 1) * AK;
#pragma unroll
                for (int part = 0; part < 3; ++part)                   // lo x hi, hi x lo, hi x hi
#pragma unroll
                    for (int kk = 0; kk < HD / 16; ++kk)
                        umma_bf16(ts, d_q + (part == 0 ? Q_PART : 0) + kk * 2, dk + (part == 1 ? KV_PART : 0) + kk * 2, idesc_s, part || kk ? 1u : 0u);
                umma_commit(&B->s_full[g][G & 1]);
                umma_commit(&B->k_empty[st]);
                if (js + 1 == (uint32_t)T) umma_commit(&B->q_empty);
            }
            const uint32_t k0 = __ballot_sync(0xffffffffu, m0 != 0), k1 = __ballot_sync(0xffffffffu, m1 != 0);
            if (lane == 0) {
                B->keep[g][G & 1] = make_uint2(k0, k1);
                mbar_arrive(&B->s_full[g][G & 1]);
            }
            if (++js == (uint32_t)T) { js = 0; ++ks; }
            mask_fetch();
            return true;
        };
        bool ok = total == 0 || scores(0);
        if (ok && total > 1) ok = scores(1);
        for (uint32_t G = 0; G < total && ok; ++G) {
            const uint32_t st = G % ST;
            ok = mbar_wait_warp(&B->p_full[g], G & 1, abort_flag) && mbar_wait_warp(&B->v_full[st], (G / ST) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t dv = d_v + st * KV_STEP;
                const uint32_t tp = t_s + (G & 1) * AK;
                const bool half = short_last && jp + 1 == (uint32_t)T;
#pragma unroll
                for (int part = 0; part < 3; ++part)                   // lo x hi, hi x lo, hi x hi
#pragma unroll
                    for (int kk = 0; kk < AK / 16; ++kk)               // 16 keys: 8 columns of P (of 32 keys: hi 16, lo 16), two 8-row groups of v
                        if (kk < AK / 32 || !half)
                            umma_bf16_ts(t_o, tp + (part == 0 ? 16 : 0) + (kk >> 1) * 32 + (kk & 1) * 8, dv + (part == 1 ? KV_PART : 0) + kk * (1024 >> 4), idesc_o, part || kk ? 1u : 0u);
                umma_commit(&B->pv_done[g]);
                umma_commit(&B->v_empty[st]);
            }
            __syncwarp();
            if (++jp == (uint32_t)T) jp = 0;
            // Scores of tile G + 2, whose columns hold this tile's P.  Those of the next item's first tile wait for its q, and this item's last
            // P V must not wait with them: they go out behind it.
            if (jp + 1 == (uint32_t)T && T > 1) continue;
            if (jp == 0 && T > 1 && G + 1 < total) ok = mbar_wait_warp(&B->pv_done[g], G & 1, abort_flag) && scores(G + 1);
            if (ok && G + 2 < total) ok = mbar_wait_warp(&B->pv_done[g], G & 1, abort_flag) && scores(G + 2);
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else {
        // ------------------------------ softmax groups ------------------------------
        const int g = warp >> 2, quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t t_s = tmem_base + ((uint32_t)(quarter * 32) << 16) + g * GROUP_COLS, t_o = t_s + COL_O;
        const int ht = p.heads * HD;
        const float qk_inv = 1.f / p.qk_scale;                         // a power of two
        const uint64_t qk_inv2 = f2(qk_inv, qk_inv);
        uint32_t G = 0;
        bool ok = true;
        // a tile's output joins the sum: o = o * a + O
        auto join = [&](float* o, const uint32_t (&ot)[16], float a) {
            const uint64_t a2 = f2(a, a);
#pragma unroll
            for (int e = 0; e < 16; e += 2)
                f2_get(f2_fma(f2(o[e], o[e + 1]), a2, f2(__uint_as_float(ot[e]), __uint_as_float(ot[e + 1]))), o[e], o[e + 1]);
        };
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            int qt, h, line0;
            decode(it, qt, h, line0);
            const int line = line0 + g < p.lines ? line0 + g : p.lines - 1;
            float m = -INFINITY, a_prev = 0.f;
            uint64_t la = f2(0.f, 0.f), lb = la;
            float o[HD];
#pragma unroll
            for (int e = 0; e < HD; ++e) o[e] = 0.f;
#pragma unroll 1
            for (int j = 0; j < T; ++j, ++G) {
                const uint32_t st = G % ST;
                const int left = p.n_k - j * AK;
                ok = mbar_wait(&B->b_full[st], (G / ST) & 1, abort_flag) && mbar_wait(&B->s_full[g][G & 1], (G >> 1) & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint2 keep = B->keep[g][G & 1];
                const uint32_t ts = t_s + (G & 1) * AK;
                const uint8_t* bias_row = smem + OFF_BIAS + st * BIAS_TILE + row * 128;
                const bool whole = left > 32;            // a last tile of at most 32 keys has no second half to work on
                // The second half's scores wait in tensor memory for the maximum, the first half's in registers (both in registers spill).
                // Every tile holds a key inside n_k, whose score is finite: the new maximum is finite.
                float t[32], mx = m;
                if (whole) {
                    scores32(t, ts + 32, bias_row + BIAS_BOX, row, qk_inv2, keep.y, p.mask_add, left - 32);
                    mx = max32(t, mx);
                    uint32_t w[32];
#pragma unroll
                    for (int e = 0; e < 32; ++e) w[e] = __float_as_uint(t[e]);
                    tmem_st_32x32(ts + 32, w);
                }
                scores32(t, ts, bias_row, row, qk_inv2, keep.x, p.mask_add, left);
                mx = max32(t, mx);
                __syncwarp();
                if (lane == 0) mbar_arrive(&B->b_empty[st]);
                const float a = prob(m - mx);            // 0 on the first tile
                m = mx;
                const uint64_t a2 = f2(a, a);
                la = f2_mul(la, a2);
                lb = f2_mul(lb, a2);
                probs32(t, -m, la, lb, ts);
                if (whole) {
                    tmem_st_wait();
                    uint32_t w[32];
                    tmem_ld_32x32(ts + 32, w);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) t[e] = __uint_as_float(w[e]);
                    probs32(t, -m, la, lb, ts + 32);
                }
                if (j > 0) {                             // the tile before: its product was done while this one's softmax ran
                    ok = mbar_wait(&B->pv_done[g], (G & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint32_t ot[16];
                        tmem_ld_32x16(t_o + hf * 16, ot);
                        tmem_ld_wait();
                        join(o + hf * 16, ot, a_prev);
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&B->p_full[g]);
                a_prev = a;
            }
            if (!ok) break;
            // A row of gates is 128 bytes, of a part of the output 64: eight lanes share a row, so that a load or store touches four rows and
            // not 32 (with a row per lane the 24 of them took 6 to 10 k clocks of an item's 45 k).  Lane i of an eight holds channels 4 i of its
            // eight rows, k = 0 .. 7.
            const int i8 = lane & 7, q8 = qt * AQ + quarter * 32 + (lane & 24);
            const bool store = line0 + g < p.lines;
            const long long r0 = line * p.line_rows;
            float4 gate[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                gate[k] = store && q8 + k < p.n_q ? *reinterpret_cast<const float4*>(p.gate + (r0 + (q8 + k) * p.pos_rows) * ht + h * HD + 4 * i8) : make_float4(0.f, 0.f, 0.f, 0.f);
            ok = mbar_wait(&B->pv_done[g], (G & 1) ^ 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                uint32_t ot[16];
                tmem_ld_32x16(t_o + hf * 16, ot);
                tmem_ld_wait();
                join(o + hf * 16, ot, a_prev);
            }
            tc_fence_before();
            float x, y;
            f2_get(f2_add(la, lb), x, y);
            const float inv = 1.f / ((x + y) * P_SCALE);
#pragma unroll
            for (int e = 0; e < HD; ++e) o[e] *= inv;
            // 8 x 8 transposition of four-channel pieces over the lanes of an eight
#pragma unroll
            for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if ((c & bit) == 0)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float& u = o[4 * c + e];
                            float& v = o[4 * (c | bit) + e];
                            const bool up = (lane & bit) != 0;
                            const float got = __shfl_xor_sync(0xffffffffu, up ? u : v, bit);
                            if (up) u = got;
                            else v = got;
                        }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (store && q8 + k < p.n_q) {
                    __half* op = p.out + (r0 + (q8 + k) * p.pos_rows - p.out_row0) * ht + h * HD + 4 * i8;
                    uint2 hi, lo;
                    split_f16x2(o[4 * k] * gate[k].x, o[4 * k + 1] * gate[k].y, hi.x, lo.x);
                    split_f16x2(o[4 * k + 2] * gate[k].z, o[4 * k + 3] * gate[k].w, hi.y, lo.y);
                    *reinterpret_cast<uint2*>(op) = hi;
                    *reinterpret_cast<uint2*>(op + p.out_part_stride) = lo;
                }
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP0) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

}  // namespace tc

bool attention_tc_fits(const AttnArgs& a, int hd) {
    return hd == tc::HD && a.lines >= tc::NG && a.q0 == 0 && a.n_q == a.n_k && aligned16(a.bias) && a.bias_hs % 4 == 0 && a.bias_qs % 4 == 0 &&
           (long long)((a.lines + tc::NG - 1) / tc::NG) * a.heads * ((a.n_q + tc::AQ - 1) / tc::AQ) <= (1 << 30) && aligned16(a.gate) && aligned16(a.out) && a.out_part_stride % 8 == 0 && a.line_rows > 0 && a.pos_rows > 0;
}

int launch_attention_tc(const AttnArgs& a, cudaStream_t st) {
    using namespace tc;
    CUtensorMap mq, mkv, mb;
    int rc, sms;
    if ((rc = multiprocessors(&sms)) != B200PF_OK) return rc;
    {   // coordinates (channel, head of q | k | v, position, line, part)
        cuuint64_t dims[5] = {(cuuint64_t)HD, (cuuint64_t)3 * a.heads, (cuuint64_t)a.n_k, (cuuint64_t)a.lines, 2};
        cuuint64_t str[4] = {(cuuint64_t)HD * 2, (cuuint64_t)a.pos_rows * a.ld * 2, (cuuint64_t)a.line_rows * a.ld * 2, (cuuint64_t)a.part_stride * 2};
        cuuint32_t boxq[5] = {HD, 1, AQ, NG, 2}, boxk[5] = {HD, 1, AK, NG, 2};
        if ((rc = tmap_encode(&mq, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.qkv, 5, dims, str, boxq, CU_TENSOR_MAP_SWIZZLE_64B, "q parts")) != B200PF_OK) return rc;
        if ((rc = tmap_encode(&mkv, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.qkv, 5, dims, str, boxk, CU_TENSOR_MAP_SWIZZLE_64B, "k, v parts")) != B200PF_OK) return rc;
    }
    {
        cuuint64_t dims[4] = {(cuuint64_t)a.n_k, (cuuint64_t)a.n_q, (cuuint64_t)a.heads, 1};
        cuuint64_t str[3] = {(cuuint64_t)a.bias_qs * 4, (cuuint64_t)a.bias_hs * 4, (cuuint64_t)a.bias_hs * 4 * a.heads};
        cuuint32_t box[4] = {32, AQ, 1, 1};
        if ((rc = tmap_encode(&mb, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.bias, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "bias")) != B200PF_OK) return rc;
    }
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "split attention: no device status word");
    B200PF_SMEM_ATTR_ONCE(split_attention_tc_kernel, SMEM_BYTES);
    const long long items = (long long)((a.lines + NG - 1) / NG) * a.heads * ((a.n_q + AQ - 1) / AQ);
    return launch_pdl(split_attention_tc_kernel, dim3((unsigned)(items < sms ? items : sms)), dim3(THREADS), SMEM_BYTES, st, mq, mkv, mb, a, status);
}

}  // namespace split
}  // namespace b200pf
