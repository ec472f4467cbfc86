// GEMM at fp32 accuracy on the 5th-generation tensor cores: D[m][n] = sum_k A[m][k] B[n][k] with A and B given as 16-bit
// part planes (split.cuh) and fp32 accumulation in tensor memory.
//
// One k-block of 64 brings every part of both operands into shared memory once and multiplies them three (fp16 parts) or
// six (bf16 parts) times, so the kernel asks L2 for a half / a third of the bytes per MMA of a plain bf16 GEMM.  Those bytes bound it
// for large K, less so on CTA pairs (launch_one), its epilogue for K = 64, and latency for the single track's few hundred rows.
// Persistent, warp-specialised: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 epilogue (two warps per TMEM lane quarter,
// each half of the columns).  Two accumulator sets let the epilogue of a tile run under the next tile's MMAs.  Every result
// leaves through a swizzled staging slot per warp and a TMA store (or reduce-add), which also clips ragged edges.
#include "split.cuh"
#include "tmap.cuh"

namespace b200pf {
namespace split {

constexpr int THREADS = 320, EPI_WARPS = 8, STG_BYTES = 4096;
constexpr int SMEM_MAX = 232448, SMEM_FIXED = 1024 + 256 + EPI_WARPS * STG_BYTES;

struct Dev {
    int m_rows, n_rows, batches, bn;
    int a_batched, b_batched, a_second_row;
    int k[2], k_splits, kb_per_split;
    float alpha[2], out_scale, qkv_scale[3];
    const float* bias;
    const uint8_t* mask;
    long long mask_bs, mask_cs;
    int n_split;
};

// Products of the parts, smallest first: (lo, hi), (hi, lo), (hi, hi) and (l, h), (m, m), (h, l), (m, h), (h, m), (h, h).
constexpr int n_products(int pl) { return pl == 2 ? 3 : 6; }
__host__ __device__ constexpr int product_a(int pl, int q) { return pl == 2 ? (q == 0 ? 1 : 0) : (q == 0 ? 2 : q == 1 || q == 3 ? 1 : 0); }
__host__ __device__ constexpr int product_b(int pl, int q) { return pl == 2 ? (q == 1 ? 1 : 0) : (q == 2 ? 2 : q == 1 || q == 4 ? 1 : 0); }

template <int PL> __host__ __device__ constexpr uint32_t make_idesc(int m, int n) {
    // fp32 accumulator; fp16 (0) or bf16 (1) operands, both K-major
    return (1u << 4) | (PL == 3 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
constexpr int stage_bytes(int pl, int bn, int na, bool pair) { return pl * (na * 128 + (pair ? bn / 2 : bn)) * 128; }
constexpr int stages_of(int pl, int bn, int na, bool pair) {
    int s = (SMEM_MAX - SMEM_FIXED) / stage_bytes(pl, bn, na, pair);
    return s > 4 ? 4 : s;
}

// 1 / (1 + e^-(a y)), a power of two: 2^t of t = -a y log2(e) with the product's rounding error put back to first order (rounded alone it
// would cost |t| 2^-24), and the reciprocal as the instruction gives it.  Both approximations are good to some 2^-22; with expf and a
// division, twice the instructions, the epilogues below were issue bound: 7088 -> 6527 us for four attention-free blocks at 331 tokens x
// 256, 4000 -> 3691 for two 256-wide blocks at 256, 2126 -> 1826 for two template blocks at 292.  Errors of the sub-operations
// against 64 bits where gains are around one: a little smaller (transition 1.043e-6 for 1.056e-6 at 64 channels, tri-mul 2.75e-7 for 2.79e-7); with
// gains of 8, arguments of 3 to 6, the transition's is 0.4 % larger (a Newton step on the reciprocal takes that back and costs 0.4 to 1.5 % of
// those cases).  Two at a time on packed
// instructions, with the products around them and the parts' remainders (split_f16x2): 14 instructions for 20 and the same bits, template
// 1234 -> 1176 us, wide 3153 -> 3063, fold 6293 -> 6179.  Arguments beyond 87 saturate; a NaN stays one.
struct Sigmoid {
    float most, least, q, q_lo;
    __device__ explicit Sigmoid(float a) : most(87.f / a), least(-87.f / a), q(-1.44269504f * a), q_lo(-1.92596299e-8f * a) {}
    __device__ __forceinline__ float limited(float y) const {
        float c;
        asm("min.NaN.f32 %0, %1, %2;" : "=f"(c) : "f"(y), "f"(most));
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(c) : "f"(c), "f"(least));
        return c;
    }
    __device__ __forceinline__ float2 operator()(float y0, float y1) const {
        const float2 c = make_float2(limited(y0), limited(y1)), q2 = make_float2(q, q), t = mul2(c, q2);
        const float2 left = mul2(fma2(c, make_float2(q_lo, q_lo), fma2(c, q2, make_float2(-t.x, -t.y))), make_float2(0.693147181f, 0.693147181f));
        float2 e, r;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(t.x));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(t.y));
        const float2 d = add2(make_float2(1.f, 1.f), fma2(e, left, e));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d.x));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d.y));
        return r;
    }
};

// PAIR: two CTAs of a cluster share the columns of a tile of 256 rows, 128 each: each loads its rows of A and half of B's, the even one issues
// the MMAs (cta_group::2), each drains its own rows.
template <int PL, int BN, int NA, int NK, int EPI, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1)
split_gemm_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
                  const __grid_constant__ CUtensorMap map_b0, const __grid_constant__ CUtensorMap map_b1,
                  const __grid_constant__ CUtensorMap map_o0, const __grid_constant__ CUtensorMap map_o1, Dev p, unsigned int* status) {
    using namespace sm100;
    // The leading product and the small ones have an accumulator each, for three parts and for the long sums of a contraction.
    // The tensor core truncates when it aligns an addend, so every MMA into a running sum costs up to an ulp of that sum, all in
    // one direction: with 6 K / 16 of them in one accumulator a 300-long contraction was biased by 7e-7; the small products'
    // sums have no ulps to lose.
    constexpr bool SMALL = PL == 3 || EPI == EPI_CONTRACT;
    constexpr int NACC = SMALL ? 2 : NA * NK, ACC_COLS = NACC * BN, TMEM_COLS = 2 * ACC_COLS;
    constexpr int STAGES = stages_of(PL, BN, NA, PAIR), A_PART = 128 * 128;
    static_assert(STAGES >= 2 && TMEM_COLS <= 512, "tile too large");
    constexpr int STAGE = stage_bytes(PL, BN, NA, PAIR);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* stg_base = smem + STAGES * STAGE;
    uint64_t* bars = reinterpret_cast<uint64_t*>(stg_base + EPI_WARPS * STG_BYTES);
    uint64_t* full = bars;                                 // of a pair the even CTA's: both CTAs' loads
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;
    uint64_t* acc_empty = acc_full + 2;                    // of a pair the even CTA's: both CTAs' epilogue warps
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bn = p.bn;                                   // columns of a tile: a multiple of 32, at most BN
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
    const int worker = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, workers = PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x;
    constexpr int TILE_M = PAIR ? 256 : 128;
    const int mt = (p.m_rows + TILE_M - 1) / TILE_M, nt = (p.n_rows + bn - 1) / bn;
    const long long tiles = (long long)p.batches * mt * nt;
    const int b_rows = PAIR ? bn / 2 : bn;                 // of a tile's B rows this CTA's
    const uint32_t b_part = (uint32_t)b_rows * 128;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], PAIR ? 2 : 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], PAIR ? 2 * EPI_WARPS : EPI_WARPS); }
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) {
        if (PAIR) { tmem_alloc_pair(tmem_slot, TMEM_COLS); tmem_relinquish_pair(); }
        else { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&map_a0); tma_prefetch_desc(&map_b0); tma_prefetch_desc(&map_o0);
        if (NK == 2) { tma_prefetch_desc(&map_a1); tma_prefetch_desc(&map_b1); }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();                              // the other CTA's barriers and tensor memory are ready
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dependency_wait();
    grid_launch_dependents();

    // k range of phase `ph` for batch `bt` in 64-wide blocks
    auto kb_range = [&](int ph, int bt, int& kb0, int& kb1) {
        const int total = (p.k[ph] + 63) / 64;
        if (p.k_splits > 1) { kb0 = bt * p.kb_per_split; kb1 = min(total, kb0 + p.kb_per_split); }
        else { kb0 = 0; kb1 = total; }
    };

    if (warp == 0 && lane == 0) {
        const uint32_t full0 = PAIR ? map_to_cta(&full[0], 0) : 0u;
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (long long t = worker; t < tiles && ok; t += workers) {
            const int bt = (int)(t / (mt * nt)), rem = (int)(t % (mt * nt));
            const int m0 = (rem / nt) * TILE_M + (int)rank * 128, n0 = (rem % nt) * bn + (int)rank * b_rows;
            const int ba = p.a_batched ? bt : 0, bb = p.b_batched ? bt : 0;
#pragma unroll
            for (int ph = 0; ph < NK; ++ph) {
                const CUtensorMap* ma = ph == 0 ? &map_a0 : &map_a1;
                const CUtensorMap* mb = ph == 0 ? &map_b0 : &map_b1;
                int kb0, kb1;
                kb_range(ph, bt, kb0, kb1);
                for (int kb = kb0; kb < kb1 && ok; ++kb) {
                    ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag);
                    if (!ok) break;
                    uint8_t* sa = smem + stage * STAGE;
                    uint8_t* sb = sa + NA * PL * A_PART;
                    const uint32_t bytes = (uint32_t)(PL * (NA * A_PART)) + PL * b_part;
                    if (!PAIR || rank == 0) mbar_arrive_expect_tx(&full[stage], bytes);
                    else mbar_arrive_expect_tx_cluster(full0 + stage * 8, bytes);
                    auto load = [&](uint8_t* dst, const CUtensorMap* map, int c1, int c2, int c3) {
                        if (PAIR) tma_load_4d_pair(dst, map, full0 + stage * 8, kb * 64, c1, c2, c3);
                        else tma_load_4d(dst, map, &full[stage], kb * 64, c1, c2, c3);
                    };
#pragma unroll
                    for (int pl = 0; pl < PL; ++pl) {
#pragma unroll
                        for (int na = 0; na < NA; ++na) load(sa + (na * PL + pl) * A_PART, ma, m0 + na * p.a_second_row, ba, pl);
                        load(sb + pl * b_part, mb, n0, bb, pl);
                    }
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
        if (!ok) {   // give copies in flight time to land before the CTA's shared memory goes away
            atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
            uint64_t t0 = global_timer_ns();
            while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
    } else if (warp == 1 && rank == 0) {
        const uint32_t idesc = make_idesc<PL>(TILE_M, bn);
        auto commit = [&](uint64_t* bar) {
            if (PAIR) { umma_commit_pair(smem_u32(bar)); umma_commit_pair(map_to_cta(bar, 1)); }
            else umma_commit(bar);
        };
        const uint64_t d0 = make_desc_k_sw128(smem_u32(smem));
        uint32_t stage = 0, phase = 0, it = 0;
        bool ok = true;
        for (long long t = worker; t < tiles && ok; t += workers, ++it) {
            const int bt = (int)(t / (mt * nt));
            const uint32_t ab = it & 1;
            ok = mbar_wait_warp(&acc_empty[ab], ((it >> 1) & 1) ^ 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int ph = 0; ph < NK; ++ph) {
                int kb0, kb1;
                kb_range(ph, bt, kb0, kb1);
                for (int kb = kb0; kb < kb1 && ok; ++kb) {
                    ok = mbar_wait_warp(&full[stage], phase, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const int ksteps = min(4, (p.k[ph] - kb * 64 + 15) >> 4);         // a short last block is zero-filled
                    if (elect_one()) {
                        const uint64_t da = d0 + stage * (uint64_t)(STAGE >> 4), db = da + ((NA * PL * A_PART) >> 4);
#pragma unroll
                        for (int q = 0; q < n_products(PL); ++q) {
#pragma unroll
                            for (int na = 0; na < NA; ++na) {
                                const bool lead = q == n_products(PL) - 1;
                                const uint32_t d = tmem_base + ab * ACC_COLS + (SMALL ? (lead ? 0 : BN) : (na + ph) * BN);
                                const uint64_t xa = da + (na * PL + product_a(PL, q)) * (A_PART >> 4), xb = db + product_b(PL, q) * (b_part >> 4);
#pragma unroll
                                for (int kk = 0; kk < 4; ++kk)
                                    if (kk < ksteps) {
                                        const uint32_t add = (kb > kb0 || kk > 0 || (q > 0 && !(SMALL && lead))) ? 1u : 0u;
                                        if (PAIR) umma_bf16_pair(d, xa + kk * 2, xb + kk * 2, idesc, add);
                                        else umma_bf16(d, xa + kk * 2, xb + kk * 2, idesc, add);
                                    }
                            }
                        }
                        commit(&empty[stage]);
                        if (ph == NK - 1 && kb + 1 == kb1) commit(&acc_full[ab]);
                    }
                    __syncwarp();
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else if (warp >= 2) {
        const int quarter = warp & 3, chalf = (warp - 2) >> 2;
        uint8_t* stg = stg_base + (warp - 2) * STG_BYTES;
        uint32_t it = 0, slot = 0;
        bool ok = true, whole = false;      // whole: the last store was of all 4096 staging bytes
        // 32 rows x 32 fp32 values, 128-byte swizzle
        auto put_f32 = [&](const float (&v)[32], const CUtensorMap* map, bool add, int c0, int c1, int c2) {
            if (lane == 0) bulk_wait_read0();
            whole = true;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j)
                *reinterpret_cast<float4*>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                if (add) tma_reduce_add_4d(map, stg, c0, c1, c2, 0);
                else tma_store_4d(map, stg, c0, c1, c2, 0);
                bulk_commit();
            }
        };
        // 32 rows x 32 16-bit values of one part, 64-byte swizzle, two slots in turn: the store before may still read the other
        // slot, unless it was put_f32's, which reads both (a gate tile whose CTA's next tile holds q, k or v)
        auto put_part = [&](const uint32_t (&w)[16], const CUtensorMap* map, int c0, int c1, int c2, int part) {
            if (lane == 0) {
                if (whole) bulk_wait_read0();
                else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            }
            whole = false;
            __syncwarp();
            uint8_t* s = stg + slot * 2048;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<uint4*>(s + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) { tma_store_4d(map, s, c0, c1, c2, part); bulk_commit(); }
            slot ^= 1;
        };
        const Sigmoid sig(EPI == EPI_GATE_ADD ? p.alpha[1] : EPI == EPI_QKVG ? 1.f : p.alpha[0]);
        const float ao = p.alpha[0] * p.out_scale;                          // powers of two
        for (long long t = worker; t < tiles && ok; t += workers, ++it) {
            const int bt = (int)(t / (mt * nt)), rem = (int)(t % (mt * nt));
            const int m0 = (rem / nt) * TILE_M + (int)rank * 128 + quarter * 32, n0 = (rem % nt) * bn;
            const uint32_t ab = it & 1;
            uint32_t bits = 0;                                              // mask of the warp's next 32 columns, asked for ahead of the wait
            auto mask_bits = [&](int col) {
                const bool keep = col + lane < p.n_rows && *(p.mask + bt * p.mask_bs + (long long)(col + lane) * p.mask_cs) != 0;
                return __ballot_sync(0xffffffffu, keep);
            };
            if (EPI == EPI_GATE_PLANES) bits = mask_bits(n0 + (chalf ? (bn / 32 + 1) / 2 : 0) * 32);
            ok = mbar_wait(&acc_full[ab], (it >> 1) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t tb = tmem_base + ((uint32_t)(quarter * 32) << 16) + ab * ACC_COLS;
            const int per = EPI == EPI_SWIGLU ? 64 : 32;                    // accumulator columns per round
            const int rounds = bn / per, r0 = chalf ? (rounds + 1) / 2 : 0, r1 = chalf ? rounds : (rounds + 1) / 2;
            if (m0 < p.m_rows) {
#pragma unroll 1
                for (int r = r0; r < r1; ++r) {
                    const int col = n0 + r * per;
                    if (col >= p.n_rows) break;
                    uint32_t x[32], y[32];
                    tmem_ld_32x32(tb + r * per, x);
                    if (EPI == EPI_SWIGLU) tmem_ld_32x32(tb + r * per + 32, y);
                    if (NACC == 2) tmem_ld_32x32(tb + BN + r * per, y);
                    tmem_ld_wait();
                    float v[32];
                    if (EPI == EPI_STORE || EPI == EPI_CONTRACT || EPI == EPI_ADD || EPI == EPI_QKVG) {
#pragma unroll
                        for (int e = 0; e < 32; e += 2) {
                            float2 u = make_float2(__uint_as_float(x[e]), __uint_as_float(x[e + 1]));
                            if (SMALL) u = add2(u, make_float2(__uint_as_float(y[e]), __uint_as_float(y[e + 1])));
                            u = mul2(u, make_float2(p.alpha[0], p.alpha[0]));
                            v[e] = u.x; v[e + 1] = u.y;
                        }
                        if (p.bias) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) v[e] += col + e < p.n_rows ? *(p.bias + col + e) : 0.f;
                        }
                        if (EPI == EPI_STORE || EPI == EPI_CONTRACT) put_f32(v, &map_o0, false, col, m0, bt);
                        else if (EPI == EPI_ADD) put_f32(v, &map_o0, true, col, m0, bt);
                        else if (col < p.n_split) {
                            const int third = p.n_split / 3;            // a multiple of 32: one of q, k, v per round
                            const float sc = p.qkv_scale[col < third ? 0 : col < 2 * third ? 1 : 2];
                            uint32_t w[2][16];
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                const float2 u = mul2(make_float2(v[2 * e], v[2 * e + 1]), make_float2(sc, sc));
                                split_f16x2(u.x, u.y, w[0][e], w[1][e]);
                            }
                            put_part(w[0], &map_o0, col, m0, bt, 0);
                            put_part(w[1], &map_o0, col, m0, bt, 1);
                        } else {
#pragma unroll
                            for (int e = 0; e < 32; e += 2) {
                                const float2 g = sig(v[e], v[e + 1]);
                                v[e] = g.x; v[e + 1] = g.y;
                            }
                            put_f32(v, &map_o1, false, col - p.n_split, m0, bt);
                        }
                    } else if (EPI == EPI_SWIGLU) {
#pragma unroll
                        for (int e = 0; e < 32; e += 2) {
                            const float2 f1 = make_float2(__uint_as_float(x[e]), __uint_as_float(x[e + 1])), f2 = make_float2(__uint_as_float(y[e]), __uint_as_float(y[e + 1]));
                            const float2 h = mul2(mul2(mul2(f1, make_float2(p.alpha[0], p.alpha[0])), sig(f1.x, f1.y)), mul2(f2, make_float2(ao, ao)));
                            v[e] = h.x; v[e + 1] = h.y;
                        }
                        uint32_t w[2][16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) split_f16x2(v[2 * e], v[2 * e + 1], w[0][e], w[1][e]);
                        put_part(w[0], &map_o0, col >> 1, m0, bt, 0);
                        put_part(w[1], &map_o0, col >> 1, m0, bt, 1);
                    } else if (EPI == EPI_GATE_PLANES) {
#pragma unroll
                        for (int e = 0; e < 32; e += 2) {
                            const float2 u = mul2(mul2(make_float2(__uint_as_float(x[e]), __uint_as_float(x[e + 1])), make_float2(ao, ao)),
                                                  sig(__uint_as_float(y[e]), __uint_as_float(y[e + 1])));
                            v[e] = (bits >> e) & 1u ? u.x : 0.f;
                            v[e + 1] = (bits >> (e + 1)) & 1u ? u.y : 0.f;
                        }
                        if (r + 1 < r1) bits = mask_bits(col + 32);
                        uint32_t w[2][16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) split_f16x2(v[2 * e], v[2 * e + 1], w[0][e], w[1][e]);
                        put_part(w[0], &map_o0, col, bt, m0, 0);
                        put_part(w[1], &map_o0, col, bt, m0, 1);
                    } else {
#pragma unroll
                        for (int e = 0; e < 32; e += 2) {
                            const float2 u = mul2(mul2(make_float2(__uint_as_float(x[e]), __uint_as_float(x[e + 1])), make_float2(p.alpha[0], p.alpha[0])),
                                                  sig(__uint_as_float(y[e]), __uint_as_float(y[e + 1])));
                            v[e] = u.x; v[e + 1] = u.y;
                        }
                        put_f32(v, &map_o0, true, col, m0, bt);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_remote(map_to_cta(&acc_empty[ab], 0));
                else mbar_arrive(&acc_empty[ab]);
            }
        }
        if (lane == 0) bulk_wait0();
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();                              // nobody signals or reads the other CTA after this
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
        else tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

static int operand_map(CUtensorMap* m, const Operand& o, int parts, int box_rows, const char* what) {
    B200PF_REQUIRE(o.ptr && aligned16(o.ptr) && o.row_stride % 8 == 0 && o.batch_stride % 8 == 0 && o.part_stride % 8 == 0, B200PF_ERR_INVALID,
                   "split_gemm: operand %s is null, misaligned or has strides that are not multiples of 8", what);
    cuuint64_t dims[4] = {(cuuint64_t)o.cols, (cuuint64_t)o.rows, (cuuint64_t)o.batches, (cuuint64_t)parts};
    cuuint64_t str[3] = {(cuuint64_t)o.row_stride * 2, (cuuint64_t)(o.batches > 1 ? o.batch_stride : o.part_stride) * 2, (cuuint64_t)o.part_stride * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
    return tmap_encode(m, parts == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, o.ptr, 4, dims, str, box,
                       CU_TENSOR_MAP_SWIZZLE_128B, what);
}

static int output_map(CUtensorMap* m, const Output& o) {
    const int es = o.parts == 1 ? 4 : 2;
    B200PF_REQUIRE(o.ptr && aligned16(o.ptr) && o.row_stride * es % 16 == 0 && o.batch_stride * es % 16 == 0 && o.part_stride * es % 16 == 0,
                   B200PF_ERR_INVALID, "split_gemm: output is null, misaligned or has strides that are not multiples of 16 bytes");
    const CUtensorMapDataType dt = o.parts == 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : o.parts == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const long long any = o.row_stride * o.rows;       // stride of a dimension of extent 1: anything valid
    const long long bs = o.batches > 1 ? o.batch_stride : any, ps = o.parts > 1 ? o.part_stride : any;
    cuuint64_t dims[4] = {(cuuint64_t)o.cols, (cuuint64_t)(o.rows_outer ? o.batches : o.rows), (cuuint64_t)(o.rows_outer ? o.rows : o.batches), (cuuint64_t)o.parts};
    cuuint64_t str[3] = {(cuuint64_t)(o.rows_outer ? bs : o.row_stride) * es, (cuuint64_t)(o.rows_outer ? o.row_stride : bs) * es, (cuuint64_t)ps * es};
    cuuint32_t box[4] = {32, o.rows_outer ? 1u : 32u, o.rows_outer ? 32u : 1u, 1};
    return tmap_encode(m, dt, o.ptr, 4, dims, str, box, o.parts == 1 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, "split output");
}

template <int PL, int BN, int NA, int NK, int EPI, bool PAIR>
static int launch_tiles(const Gemm& g, int bn, int sms, cudaStream_t st) {
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "split_gemm: no device status word");
    CUtensorMap a[2], b[2], o[2];
    int rc;
    for (int i = 0; i < NK; ++i) {
        if ((rc = operand_map(&a[i], g.a[i], PL, 128, "A")) != B200PF_OK) return rc;
        if ((rc = operand_map(&b[i], g.b[i], PL, PAIR ? bn / 2 : bn, "B")) != B200PF_OK) return rc;
    }
    if (NK == 1) { a[1] = a[0]; b[1] = b[0]; }
    if ((rc = output_map(&o[0], g.out[0])) != B200PF_OK) return rc;
    if (EPI == EPI_QKVG) { if ((rc = output_map(&o[1], g.out[1])) != B200PF_OK) return rc; }
    else o[1] = o[0];
    constexpr int smem = stages_of(PL, BN, NA, PAIR) * stage_bytes(PL, BN, NA, PAIR) + SMEM_FIXED;
    constexpr auto kern = split_gemm_kernel<PL, BN, NA, NK, EPI, PAIR>;
    B200PF_SMEM_ATTR_ONCE(kern, smem);
    Dev d;
    d.m_rows = g.m_rows; d.n_rows = g.n_rows; d.bn = bn;
    d.batches = g.k_splits > 1 ? g.k_splits : g.batches;
    d.a_batched = g.a_batched; d.b_batched = g.b_batched; d.a_second_row = g.a_second_row;
    d.k[0] = g.k[0]; d.k[1] = g.k[1]; d.k_splits = g.k_splits;
    d.kb_per_split = ((g.k[0] + 63) / 64 + g.k_splits - 1) / g.k_splits;
    d.alpha[0] = g.alpha[0]; d.alpha[1] = g.alpha[1]; d.out_scale = g.out_scale;
    d.bias = g.bias; d.mask = g.mask; d.mask_bs = g.mask_bs; d.mask_cs = g.mask_cs;
    for (int i = 0; i < 3; ++i) d.qkv_scale[i] = g.qkv_scale[i];
    d.n_split = g.n_split;
    constexpr int TILE_M = PAIR ? 256 : 128;
    const long long tiles = (long long)d.batches * ((g.m_rows + TILE_M - 1) / TILE_M) * ((g.n_rows + bn - 1) / bn);
    if (PAIR) {
        int pairs;
        if ((rc = resident_pairs<kern>(THREADS, smem, &pairs)) != B200PF_OK) return rc;
        if (pairs > sms / 2) pairs = sms / 2;
        return launch_pdl_pairs(kern, (unsigned)(tiles < pairs ? tiles : pairs), dim3(THREADS), smem, st, a[0], a[1], b[0], b[1], o[0], o[1], d, status);
    }
    return launch_pdl(kern, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(THREADS), smem, st, a[0], a[1], b[0], b[1], o[0], o[1], d, status);
}

// CTA pairs where there is a tile for every CTA, more than one k-block (which would gain nothing) and pairing leaves few rows empty (an odd
// number of 128-row tiles wastes one; with the contraction's at 3, 331 tokens x 256 channels, the triangle multiplication takes 432 -> 448 us,
// at 9, 1100 x 64 and x 128, 1361 -> 1287 and 2836 -> 2664; between them, 5 and 7, pairs would gain 2 to 3 %): a k-block then brings 64 KB for 96 (256 columns), 48 for 64 (128) or 80 for 96 (two A tiles) into each SM per 256 x `bn` outputs, and some 9 TB/s out of
// L2 are what bounds these GEMMs otherwise.  At 331 tokens x 256 channels: transition 274 -> 220 us (tensor pipe 92 %) and 153 -> 140, output
// gate 94 -> 86, operand planes 176 -> 175 (their epilogue, 35 us, and L2); contraction at 256 tokens 49 -> 43; odd ones (331) stay.  Two 256-wide blocks
// run 1.04 (110 tokens) to 1.10 times (200) as fast, four attention-free ones 1.03 to 1.14, 64 channels 1.00 to 1.01.  K-blocks of 32, with more stages, are
// slower (220 -> 250, 98 -> 109); for the planes, stores of 64 columns change nothing.  Three parts have more products per byte.
template <int PL, int BN, int NA, int NK, int EPI>
static int launch_one(const Gemm& g, int bn, int sms, cudaStream_t st) {
    if constexpr (PL == 2) {
        const long long mt = (g.m_rows + 127) / 128, tiles = (long long)(g.k_splits > 1 ? g.k_splits : g.batches) * mt * ((g.n_rows + bn - 1) / bn);
        if (g.k[0] > 64 && tiles >= sms && (mt % 2 == 0 || mt >= 9)) return launch_tiles<PL, BN, NA, NK, EPI, true>(g, bn, sms, st);
    }
    return launch_tiles<PL, BN, NA, NK, EPI, false>(g, bn, sms, st);
}

// Tile width for `n` columns: the widest tile (at most `most`, a multiple of `step`) whose waves of CTAs, times the bytes a tile
// stages per k-block, come to the least: narrow tiles only where wide ones leave SMs without work.
static int pick_bn(long long row_tiles, int n, int most, int step, int sms) {
    int best = step;
    double best_cost = 1e30;
    for (int bn = most; bn >= step; bn -= step) {
        if (bn > step && bn - step >= n) continue;
        const long long tiles = row_tiles * ((n + bn - 1) / bn);
        const long long waves = (tiles + sms - 1) / sms;
        const double cost = (double)waves * (128 + bn + 64);
        if (cost < best_cost - 1e-9) { best_cost = cost; best = bn; }
    }
    return best;
}

int launch_gemm(const Gemm& g, cudaStream_t st) {
    B200PF_REQUIRE(g.m_rows > 0 && g.n_rows > 0 && g.batches > 0 && g.k[0] > 0, B200PF_ERR_INVALID, "split_gemm: empty problem");
    const int kb_total = (g.k[0] + 63) / 64;
    B200PF_REQUIRE(g.k_splits == 1 || (g.epi == EPI_STORE && g.batches == 1 && g.k_splits > 1 &&
                                       (g.k_splits - 1) * ((kb_total + g.k_splits - 1) / g.k_splits) < kb_total),
                   B200PF_ERR_INVALID, "split_gemm: every K split needs a k-block of its own");
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK) return rc;
    const long long row_tiles = (long long)(g.k_splits > 1 ? g.k_splits : g.batches) * ((g.m_rows + 127) / 128);
#define SG(PL, BN, NA, NK, EPI) return launch_one<PL, BN, NA, NK, EPI>(g, bn, sms, st)
    switch (g.epi) {
        case EPI_STORE: {
            if (g.parts == 3) { const int bn = pick_bn(row_tiles, g.n_rows, 128, 32, sms); SG(3, 128, 1, 1, EPI_STORE); }
            const int bn = pick_bn(row_tiles, g.n_rows, 256, 32, sms);
            if (bn > 128) SG(2, 256, 1, 1, EPI_STORE);
            SG(2, 128, 1, 1, EPI_STORE);
        }
        case EPI_CONTRACT: { const int bn = pick_bn(row_tiles, g.n_rows, 128, 32, sms); SG(2, 128, 1, 1, EPI_CONTRACT); }
        case EPI_ADD: {
            if (g.parts == 3) { const int bn = pick_bn(row_tiles, g.n_rows, 128, 32, sms); SG(3, 128, 1, 1, EPI_ADD); }
            const int bn = pick_bn(row_tiles, g.n_rows, 256, 32, sms);
            if (bn > 128) SG(2, 256, 1, 1, EPI_ADD);
            SG(2, 128, 1, 1, EPI_ADD);
        }
        case EPI_SWIGLU: {
            const int bn = pick_bn(row_tiles, g.n_rows, 256, 64, sms);
            if (bn > 128) SG(2, 256, 1, 1, EPI_SWIGLU);
            SG(2, 128, 1, 1, EPI_SWIGLU);
        }
        case EPI_QKVG: {
            const int bn = pick_bn(row_tiles, g.n_rows, 256, 32, sms);
            if (bn > 128) SG(2, 256, 1, 1, EPI_QKVG);
            SG(2, 128, 1, 1, EPI_QKVG);
        }
        case EPI_GATE_PLANES: { const int bn = pick_bn(row_tiles, g.n_rows, 128, 32, sms); SG(2, 128, 2, 1, EPI_GATE_PLANES); }
        case EPI_GATE_ADD: { const int bn = pick_bn(row_tiles, g.n_rows, 128, 32, sms); SG(2, 128, 1, 2, EPI_GATE_ADD); }
    }
#undef SG
    B200PF_REQUIRE(false, B200PF_ERR_UNSUPPORTED, "split_gemm: unknown epilogue");
}

}  // namespace split
}  // namespace b200pf
