// Pair transition on tcgen05:  z += W3( silu(W1 LN(z)) * (W2 LN(z)) )  per tile of 128 positions.
//
// The 512-wide hidden layer is walked in 8 chunks of 64 channels.  Per chunk c:
//   GEMM1  D1 (128 x 128 fp32, TMEM) = A (LN(z) tile, smem) x [fc1 rows | fc2 rows of the chunk]^T
//   epilogue-1 (thread = position)  h = silu(f1) * f2 -> packed bf16 pairs -> TMEM (tcgen05.st)
//   GEMM2  D2 (128 x 128 fp32, TMEM) += h (A operand read from TMEM) x W3[:, chunk]^T
// The hidden activations never leave the SM (they do not even touch shared memory).  After the last chunk the
// update leaves through TMA reduce-add into z.  silu uses one MUFU: the host halves fc1, so with
// a = f1/2:  silu(f1) = a + a*tanh(a).
// Weights (384 KB bf16) do not fit in shared memory: a warp streams them from L2 with TMA, chunk by chunk, through a ring.
//
// Two kernels, by how many tiles there are (D1 and h are double buffered in both, so that the tensor core works on one chunk while
// the epilogue works on another):
//   transition_one_kernel   at most one tile per CTA: the eight epilogue warps normalise it themselves.
//   transition_pair_kernel  more: CTA pairs, each CTA with a tile of its own and half of every chunk's weight rows (cta_group::2), LayerNorm
//     loaders a tile ahead, the update staged whole and reduced under the next tile.
// A lone CTA's 384 KB of weights per tile were some 7 TB/s out of L2 at 1024 tokens, and with 470 to 520 us there, 71.5 at 400 and 26.8 at
// 203 neither a staging tile for the whole update (508 against 500, 72.7 against 71.4) nor two tiles at a time in one CTA, which shares the
// weights but leaves tensor memory for one D1 per tile (499, 74.0; chunks of 32 hidden channels with two: 548, 84), was faster.  The pairs
// take 457 to 466 at 1024, 66 at 400, 26.4 at 203; blocks of the trunk gain 1 to 2 % from 150 to 600 tokens.  An epilogue warp spends 600
// clocks of a chunk's 1550 on its hidden values (512 of them the tanh unit's), 200 waiting for D1 and 240 for h, 470 on the update.
// One tile per CTA: 12.2 -> 11.5 us at 117 tokens, 10.9 at 45 as before.
#include "rowtc.cuh"
#include "tmap.cuh"

namespace b200pf {
namespace trz {

using namespace rtc;

constexpr int CHUNKS = 8;
constexpr int W12_BYTES = 128 * 128 * 2;                  // [128 rows][128 K]: two k-blocks of 16 KB
constexpr int W3_BYTES = 128 * 64 * 2;                    // [128 out][64 hidden]
constexpr int EPI_WARPS = 8;

struct Args {
    const float* z;
    const float* ln_gamma;
    const float* ln_beta;
    long long rows_flat;
};

__device__ __forceinline__ float tanh_approx(float x) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
    return t;
}
// LayerNorm gain and offset of this lane's channels, and one warp's 16 rows of a tile (8 lanes per row) normalised into the A tile.
struct Affine {
    float4 gam[4], bet[4];
    __device__ __forceinline__ Affine(const Args& p) {
        const int sub = threadIdx.x & 7;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            gam[j] = reinterpret_cast<const float4*>(p.ln_gamma)[j * 8 + sub];
            bet[j] = reinterpret_cast<const float4*>(p.ln_beta)[j * 8 + sub];
        }
    }
};
__device__ __forceinline__ void normalise16(const Args& p, long long base, int row0, uint8_t* a_tile, const Affine& w) {
    const int lane = threadIdx.x & 31, sub = lane & 7, rq = lane >> 3;
    float4 v[4][4];
    // rows beyond the last one repeat row 0: the reduce-add clips them
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long f = base + row0 + i * 4 + rq;
        const float4* src = reinterpret_cast<const float4*>(p.z + (f < p.rows_flat ? f : 0) * KC);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = src[j * 8 + sub];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = row0 + i * 4 + rq;
        float2 t = add2(low2(v[i][0]), high2(v[i][0]));
#pragma unroll
        for (int j = 1; j < 4; ++j) t = add2(t, add2(low2(v[i][j]), high2(v[i][j])));
        float s = t.x + t.y;
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        const float mean = s * (1.f / KC);
        float2 sq = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) centre4(v[i][j], make_float2(-mean, -mean), sq);
        float ss = sq.x + sq.y;
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        ss += __shfl_xor_sync(0xffffffffu, ss, 4);
        const float rstd = rsqrtf(ss * (1.f / KC) + LN_EPS);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint2 o;
            const float4 y = affine4(v[i][j], make_float2(rstd, rstd), w.gam[j], w.bet[j]);
            o.x = pack_bf16x2(y.x, y.y);
            o.y = pack_bf16x2(y.z, y.w);
            const int chunk = (j & 1) * 4 + (sub >> 1);
            *reinterpret_cast<uint2*>(a_tile + (j >> 1) * A_KB_BYTES + sw128(row, chunk) + (sub & 1) * 8) = o;
        }
    }
}

// 32 hidden channels of this thread's position: f1 and f2 from tensor memory, silu(f1) * f2 back as packed bf16.
__device__ __forceinline__ void hidden32(uint32_t t_f1, uint32_t t_f2, uint32_t t_h) {
    using namespace sm100;
    uint32_t f1[32], f2[32], hw[16];
    tmem_ld_32x32(t_f1, f1);
    tmem_ld_32x32(t_f2, f2);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const float2 a = make_float2(__uint_as_float(f1[2 * e]), __uint_as_float(f1[2 * e + 1]));
        const float2 h = mul2(fma2(a, make_float2(tanh_approx(a.x), tanh_approx(a.y)), a), make_float2(__uint_as_float(f2[2 * e]), __uint_as_float(f2[2 * e + 1])));
        hw[e] = pack_bf16x2(h.x, h.y);
    }
    tmem_st_32x16(t_h, hw);
}
// D = A tile x [128 weight rows]^T over K = 128, and D (+)= h x W3 chunk over K = 64.  Operands are descriptors of their first
// k-block; the address field counts 16-byte units.
__device__ __forceinline__ void gemm1(uint32_t d, uint64_t da, uint64_t dw) {
#pragma unroll
    for (int ks = 0; ks < 8; ++ks)
        sm100::umma_bf16(d, da + (ks >> 2) * (A_KB_BYTES >> 4) + (ks & 3) * 2, dw + (ks >> 2) * ((128 * 128) >> 4) + (ks & 3) * 2,
                         sm100::make_idesc_bf16(TM, 128), ks ? 1u : 0u);
}
__device__ __forceinline__ void gemm2(uint32_t d, uint32_t th, uint64_t dw3, bool first) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)               // 64 hidden = 4 k-steps; h: 8 TMEM columns per step
        sm100::umma_bf16_ts(d, th + kk * 8, dw3 + kk * 2, sm100::make_idesc_bf16(TM, 128), (!first || kk) ? 1u : 0u);
}
// A warp that gave up leaves its own copies time to land.
__device__ __forceinline__ void linger() {
    const uint64_t t0 = sm100::global_timer_ns();
    while (sm100::global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
}

// ------------------------------------------------------------------------------------------------
// several tiles per CTA
// ------------------------------------------------------------------------------------------------
namespace pair {
// warps 0-5 LayerNorm loaders (16 rows at a time, round robin), warp 6 MMA issuer, warp 7 weight TMA, warps 8-15 epilogue
constexpr int LOAD_WARPS = 6, MMA_WARP = 6, TMA_WARP = 7, EPI_WARP0 = 8, THREADS = 16 * 32;
constexpr int PASS_ROWS = 16, PASSES = TM / PASS_ROWS;
constexpr int WSTAGES = 4, W12_HALF = W12_BYTES / 2, W3_HALF = W3_BYTES / 2;              // this CTA's half of a chunk's rows
constexpr int OFF_W12 = 0, OFF_W3 = WSTAGES * W12_HALF, OFF_A = OFF_W3 + WSTAGES * W3_HALF;
constexpr int OFF_STG = OFF_A + 2 * A_TILE_BYTES;         // staging: per epilogue warp 2 boxes of [32 pos][32 fp32], 128-byte swizzle
constexpr int STG_BOX = 32 * 128;
constexpr int OFF_BAR = OFF_STG + EPI_WARPS * 2 * STG_BOX;
constexpr int SMEM_BYTES = OFF_BAR + 256;                 // 229,632
// TMEM columns
constexpr uint32_t COL_D1 = 0, COL_D2 = 256, COL_H = 384;

struct Bars {
    uint64_t w12_full[WSTAGES], w3_full[WSTAGES], a_peer[2], h_full[2], d2_empty;          // of the even CTA: arrivals of both, or of the odd one
    uint64_t w12_empty[WSTAGES], w3_empty[WSTAGES], a_full[2], a_empty[2], d1_full[2], h_empty[2], d2_full;        // one per CTA
    uint32_t tmem_slot;
    int abort_flag;
};
static_assert(sizeof(Bars) <= 256, "barriers");
}  // namespace pair

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair::THREADS, 1)
transition_pair_kernel(const __grid_constant__ CUtensorMap map_w12, const __grid_constant__ CUtensorMap map_w3,
                       const __grid_constant__ CUtensorMap map_z, Args p, unsigned int* status) {
    using namespace sm100;
    using namespace pair;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {
        grid_dependency_wait();
        if (threadIdx.x == 0) atomicOr(status, DEV_STATUS_BAD_INDEX);
        return;
    }
    Bars* B = reinterpret_cast<Bars*>(smem + OFF_BAR);
    volatile int* abort_flag = &B->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const uint32_t rank = cluster_ctarank();                                  // 0: issues the MMAs
    // the pair's tiles come two by two, an even one for the even CTA and an odd one (which may lie behind the last) for the odd CTA
    const int couples = (int)((p.rows_flat + 2 * TM - 1) / (2 * TM)), pairs = (int)gridDim.x >> 1, first_couple = (int)blockIdx.x >> 1;
    const uint32_t mine = first_couple < couples ? (uint32_t)((couples - first_couple + pairs - 1) / pairs) : 0u;
    auto row_of = [&](uint32_t it) { return (2LL * (first_couple + (long long)it * pairs) + rank) * TM; };          // first row of this CTA's tile `it`

    if (tid == 0) {
        for (int i = 0; i < WSTAGES; ++i) {
            mbar_init(&B->w12_full[i], 2); mbar_init(&B->w12_empty[i], 1);
            mbar_init(&B->w3_full[i], 2); mbar_init(&B->w3_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->a_full[i], PASSES); mbar_init(&B->a_peer[i], 1); mbar_init(&B->a_empty[i], 1);
            mbar_init(&B->d1_full[i], 1); mbar_init(&B->h_full[i], 2 * EPI_WARPS); mbar_init(&B->h_empty[i], 1);
        }
        mbar_init(&B->d2_full, 1); mbar_init(&B->d2_empty, 2 * EPI_WARPS);
        B->abort_flag = 0;
        fence_barrier_init();
    }
    if (tid == 32) { tma_prefetch_desc(&map_w12); tma_prefetch_desc(&map_w3); tma_prefetch_desc(&map_z); }
    if (warp == MMA_WARP) { tmem_alloc_pair(&B->tmem_slot, 512); tmem_relinquish_pair(); }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                              // the other CTA's barriers and tensor memory are ready
    tc_fence_after();
    grid_dependency_wait();                 // behind the barriers: every warp goes to work by itself from here on
    grid_launch_dependents();
    const uint32_t tmem_base = B->tmem_slot;

    if (warp < LOAD_WARPS) {
        // ---------------------------- LayerNorm loaders ----------------------------
        const Affine w(p);
        // Pass u is rows 16 (u % 8) of tile 1 + u / 8 of this CTA (the epilogue warps normalise its first).
        bool ok = true;
        for (uint32_t u = warp; ok && 1 + u / PASSES < mine; u += LOAD_WARPS) {
            const uint32_t it = 1 + u / PASSES, slot = it & 1, ph = (it >> 1) & 1;
            ok = mbar_wait(&B->a_empty[slot], ph ^ 1, abort_flag);
            if (!ok) break;
            {   // ask L2 for this warp's next 16 rows (two lanes per row, two 128-byte lines each)
                const uint32_t un = u + LOAD_WARPS;
                const long long fn = row_of(1 + un / PASSES) + un % PASSES * PASS_ROWS + (lane & 15);
                if (fn < p.rows_flat) {
                    const char* rowp = reinterpret_cast<const char*>(p.z + fn * KC) + (lane >> 4) * 256;
#pragma unroll
                    for (int j = 0; j < 2; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(rowp + j * 128));
                }
            }
            normalise16(p, row_of(it), (int)(u % PASSES) * PASS_ROWS, smem + OFF_A + slot * A_TILE_BYTES, w);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->a_full[slot]);
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else if (warp == TMA_WARP) {
        if (lane == 0) {
            // ---------------------------- weight TMA: this CTA's half of the rows ----------------------------
            const uint32_t full12 = map_to_cta(&B->w12_full[0], 0), full3 = map_to_cta(&B->w3_full[0], 0);
            bool ok = true;
            for (uint32_t G = 0; G < mine * CHUNKS; ++G) {
                const uint32_t st = G % WSTAGES, ph = (G / WSTAGES) & 1, c = G % CHUNKS;
                ok = mbar_wait(&B->w12_empty[st], ph ^ 1, abort_flag);
                if (!ok) break;
                uint8_t* ws = smem + OFF_W12 + st * W12_HALF;
                if (rank == 0) mbar_arrive_expect_tx(&B->w12_full[st], W12_HALF);
                else mbar_arrive_expect_tx_cluster(full12 + st * 8, W12_HALF);
                tma_load_4d_pair(ws, &map_w12, full12 + st * 8, 0, (int)rank * 64, (int)c, 0);
                tma_load_4d_pair(ws + 64 * 128, &map_w12, full12 + st * 8, 64, (int)rank * 64, (int)c, 0);
                ok = mbar_wait(&B->w3_empty[st], ph ^ 1, abort_flag);
                if (!ok) break;
                if (rank == 0) mbar_arrive_expect_tx(&B->w3_full[st], W3_HALF);
                else mbar_arrive_expect_tx_cluster(full3 + st * 8, W3_HALF);
                tma_load_4d_pair(smem + OFF_W3 + st * W3_HALF, &map_w3, full3 + st * 8, 0, (int)rank * 64, (int)c, 0);
            }
            if (!ok) {
                atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
                linger();
            }
        }
    } else if (warp == MMA_WARP && rank == 1) {
        // ---------------------------- odd CTA: tells the even one that its A tile is there ----------------------------
        // One arrival a tile from a warp with nothing in flight: the loaders, arriving there themselves, each waited 1 900 clocks for
        // their release at cluster scope, as long as half a pass.
        const uint32_t peer = map_to_cta(&B->a_peer[0], 0);
        bool ok = true;
        for (uint32_t it = 0; it < mine && ok; ++it) {
            ok = mbar_wait_warp(&B->a_full[it & 1], (it >> 1) & 1, abort_flag);
            if (ok && elect_one()) mbar_arrive_cluster(peer + (it & 1) * 8);
            __syncwarp();
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else if (warp == MMA_WARP) {
        // ---------------------------- MMA issuer (even CTA only) ----------------------------
        // The whole warp runs the loop and waits; one elected lane issues (see sm100::elect_one).
        constexpr uint32_t idesc = make_idesc_bf16(2 * TM, 128);
        const uint64_t d_a = make_desc_k_sw128(smem_u32(smem + OFF_A));
        const uint64_t d_w12 = make_desc_k_sw128(smem_u32(smem + OFF_W12)), d_w3 = make_desc_k_sw128(smem_u32(smem + OFF_W3));
        const uint32_t total = mine * CHUNKS;
        auto commit_both = [&](uint64_t* bar) {
            umma_commit_pair(smem_u32(bar));
            umma_commit_pair(map_to_cta(bar, 1));
        };
        auto first = [&](uint32_t G) {
            const uint32_t st = G % WSTAGES, it = G / CHUNKS, c = G % CHUNKS;
            if (c == 0 && !(mbar_wait_warp(&B->a_full[it & 1], (it >> 1) & 1, abort_flag) && mbar_wait_warp(&B->a_peer[it & 1], (it >> 1) & 1, abort_flag))) return false;
            if (!mbar_wait_warp(&B->w12_full[st], (G / WSTAGES) & 1, abort_flag)) return false;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t da = d_a + (it & 1) * (uint64_t)(A_TILE_BYTES >> 4), dw = d_w12 + st * (uint64_t)(W12_HALF >> 4);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma_bf16_pair(tmem_base + COL_D1 + (G & 1) * 128, da + (ks >> 2) * (A_KB_BYTES >> 4) + (ks & 3) * 2,
                                   dw + (ks >> 2) * ((64 * 128) >> 4) + (ks & 3) * 2, idesc, ks ? 1u : 0u);
                commit_both(&B->d1_full[G & 1]);
                commit_both(&B->w12_empty[st]);
                if (c + 1 == CHUNKS) commit_both(&B->a_empty[it & 1]);
            }
            __syncwarp();
            return true;
        };
        bool ok = total == 0 || (first(0) && first(1));
        for (uint32_t G = 0; G < total && ok; ++G) {
            const uint32_t st = G % WSTAGES, it = G / CHUNKS, c = G % CHUNKS;
            ok = mbar_wait_warp(&B->h_full[G & 1], (G >> 1) & 1, abort_flag);
            if (ok && G + 2 < total) ok = first(G + 2);          // ahead of this chunk's second product: the epilogue waits for it
            ok = ok && mbar_wait_warp(&B->w3_full[st], (G / WSTAGES) & 1, abort_flag) &&
                 (c != 0 || mbar_wait_warp(&B->d2_empty, (it & 1) ^ 1, abort_flag));        // D2 of the tile before has been read out
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t dw = d_w3 + st * (uint64_t)(W3_HALF >> 4);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)               // 64 hidden = 4 k-steps; h: 8 TMEM columns per step
                    umma_bf16_ts_pair(tmem_base + COL_D2, tmem_base + COL_H + (G & 1) * 32 + kk * 8, dw + kk * 2, idesc, (c | kk) ? 1u : 0u);
                commit_both(&B->w3_empty[st]);
                commit_both(&B->h_empty[G & 1]);
                if (c + 1 == CHUNKS) commit_both(&B->d2_full);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else {
        // ---------------------------- epilogue ----------------------------
        const int quarter = warp & 3, eh = (warp - EPI_WARP0) >> 2;
        uint8_t* stg = smem + OFF_STG + (warp - EPI_WARP0) * 2 * STG_BOX;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        bool ok = true;
        if (mine > 0) {
            const Affine w(p);
            normalise16(p, row_of(0), (warp - EPI_WARP0) * PASS_ROWS, smem + OFF_A, w);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->a_full[0]);
        }
        const uint32_t h_full0 = map_to_cta(&B->h_full[0], 0), d2_empty0 = map_to_cta(&B->d2_empty, 0);
        auto hidden = [&](uint32_t G) {
            const uint32_t buf = G & 1, d1 = tmem_base + lane_off + COL_D1 + buf * 128 + eh * 32;
            if (!mbar_wait(&B->d1_full[buf], (G >> 1) & 1, abort_flag)) return false;
            tc_fence_after();
            // this warp: hidden channels 32*eh .. +31 of the chunk: f1 at columns [32 eh, +32), f2 at [64 + 32 eh, +32)
            if (!mbar_wait(&B->h_empty[buf], ((G >> 1) & 1) ^ 1, abort_flag)) return false;
            hidden32(d1, d1 + 64, tmem_base + lane_off + COL_H + buf * 32 + eh * 16);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(h_full0 + buf * 8);
            return true;
        };
        // D2 of the CTA's tile number `it` -> fp32 staging -> TMA reduce-add into z; this warp: output channels 64 eh .. + 63.
        auto drain = [&](uint32_t it) {
            if (!mbar_wait(&B->d2_full, it & 1, abort_flag)) return false;
            tc_fence_after();
            uint32_t d[2][32];
            tmem_ld_32x32(tmem_base + lane_off + COL_D2 + eh * 64, d[0]);
            tmem_ld_32x32(tmem_base + lane_off + COL_D2 + eh * 64 + 32, d[1]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive_remote(d2_empty0); bulk_wait_read0(); }      // the tile before has left the staging tile
            __syncwarp();
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<uint4*>(stg + b * STG_BOX + sw128(lane, j)) = make_uint4(d[b][4 * j], d[b][4 * j + 1], d[b][4 * j + 2], d[b][4 * j + 3]);
            fence_proxy_async();
            __syncwarp();
            const long long row = row_of(it) + quarter * 32;
            if (lane == 0 && row < p.rows_flat) {
                tma_reduce_add_4d(&map_z, stg, eh * 64, (int)row, 0, 0);
                tma_reduce_add_4d(&map_z, stg + STG_BOX, eh * 64 + 32, (int)row, 0, 0);
                bulk_commit();
            }
            return true;
        };
        for (uint32_t G = 0; G < mine * CHUNKS && ok; ++G) {
            ok = hidden(G);
            if (ok && G % CHUNKS == 0 && G > 0) ok = drain(G / CHUNKS - 1);        // behind the next tile's first chunk, whose products are there already
        }
        if (ok && mine > 0) ok = drain(mine - 1);
        if (lane == 0) bulk_wait0();
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                              // nobody signals or reads the other CTA after this
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc_pair(tmem_base, 512); }
}

// ------------------------------------------------------------------------------------------------
// one tile per CTA
// ------------------------------------------------------------------------------------------------
namespace one {
constexpr int MMA_WARP = 8, TMA_WARP = 9, THREADS = 10 * 32;                  // warps 0-7 LayerNorm, then epilogue
constexpr int WSTAGES = 3, WSTAGE = W12_BYTES + W3_BYTES;                     // 49,152
constexpr int OFF_A = WSTAGES * WSTAGE;
constexpr int OFF_STG = OFF_A + A_TILE_BYTES;             // staging: per epilogue warp [32 pos][32 fp32], 128-byte swizzle
constexpr int STG_BOX = 32 * 128;
constexpr int OFF_BAR = OFF_STG + EPI_WARPS * STG_BOX;
constexpr int SMEM_BYTES = OFF_BAR + 128;                 // 213,120
// TMEM columns
constexpr uint32_t COL_D1 = 0, COL_D2 = 256, COL_H = 384;

struct Bars {
    uint64_t w_full[WSTAGES], w_empty[WSTAGES], a_full, d1_full[2], h_full[2], d2_full;
    uint32_t tmem_slot;
    int abort_flag;
};
static_assert(sizeof(Bars) <= 128, "barriers");
}  // namespace one

__global__ void __launch_bounds__(one::THREADS, 1)
transition_one_kernel(const __grid_constant__ CUtensorMap map_w12, const __grid_constant__ CUtensorMap map_w3,
                      const __grid_constant__ CUtensorMap map_z, Args p, unsigned int* status) {
    using namespace sm100;
    using namespace one;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {
        grid_dependency_wait();
        if (threadIdx.x == 0) atomicOr(status, DEV_STATUS_BAD_INDEX);
        return;
    }
    Bars* B = reinterpret_cast<Bars*>(smem + OFF_BAR);
    volatile int* abort_flag = &B->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;

    if (tid == 0) {
        for (int i = 0; i < WSTAGES; ++i) { mbar_init(&B->w_full[i], 1); mbar_init(&B->w_empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&B->d1_full[i], 1); mbar_init(&B->h_full[i], EPI_WARPS); }
        mbar_init(&B->a_full, EPI_WARPS);
        mbar_init(&B->d2_full, 1);
        B->abort_flag = 0;
        fence_barrier_init();
    }
    if (tid == 32) { tma_prefetch_desc(&map_w12); tma_prefetch_desc(&map_w3); tma_prefetch_desc(&map_z); }
    if (warp == MMA_WARP) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dependency_wait();                 // behind the CTA's barrier: every warp goes to work by itself from here on
    grid_launch_dependents();
    const uint32_t tmem_base = B->tmem_slot;

    if (warp == TMA_WARP) {
        if (lane == 0) {
            // ---------------------------- weight TMA ----------------------------
            bool ok = true;
            for (uint32_t c = 0; c < CHUNKS; ++c) {
                const uint32_t stage = c % WSTAGES, ph = (c / WSTAGES) & 1;
                ok = mbar_wait(&B->w_empty[stage], ph ^ 1, abort_flag);
                if (!ok) break;
                uint8_t* ws = smem + stage * WSTAGE;
                mbar_arrive_expect_tx(&B->w_full[stage], WSTAGE);
                tma_load_4d(ws, &map_w12, &B->w_full[stage], 0, 0, (int)c, 0);
                tma_load_4d(ws + 128 * 128, &map_w12, &B->w_full[stage], 64, 0, (int)c, 0);
                tma_load_4d(ws + W12_BYTES, &map_w3, &B->w_full[stage], 0, 0, (int)c, 0);
            }
            if (!ok) {
                atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
                linger();
            }
        }
    } else if (warp == MMA_WARP) {
        // ---------------------------- MMA issuer ----------------------------
        // The whole warp runs the loop and waits; one elected lane issues (see sm100::elect_one).
        const uint64_t d_a = make_desc_k_sw128(smem_u32(smem + OFF_A));
        const uint64_t d_w = make_desc_k_sw128(smem_u32(smem)), d_w3 = make_desc_k_sw128(smem_u32(smem + W12_BYTES));
        auto first = [&](uint32_t c) {
            if (!mbar_wait_warp(&B->w_full[c % WSTAGES], (c / WSTAGES) & 1, abort_flag)) return false;
            tc_fence_after();
            if (elect_one()) {
                gemm1(tmem_base + COL_D1 + (c & 1) * 128, d_a, d_w + (c % WSTAGES) * (uint64_t)(WSTAGE >> 4));
                umma_commit(&B->d1_full[c & 1]);
            }
            __syncwarp();
            return true;
        };
        bool ok = mbar_wait_warp(&B->a_full, 0, abort_flag) && first(0);
        for (uint32_t c = 0; c < CHUNKS && ok; ++c) {
            if (c + 1 < CHUNKS) ok = first(c + 1);
            ok = ok && mbar_wait_warp(&B->h_full[c & 1], (c >> 1) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                gemm2(tmem_base + COL_D2, tmem_base + COL_H + (c & 1) * 32, d_w3 + (c % WSTAGES) * (uint64_t)(WSTAGE >> 4), c == 0);
                umma_commit(&B->w_empty[c % WSTAGES]);
                if (c + 1 == CHUNKS) umma_commit(&B->d2_full);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else {
        // ---------------------------- LayerNorm and epilogue ----------------------------
        const int quarter = warp & 3, eh = warp >> 2;
        uint8_t* stg = smem + OFF_STG + warp * STG_BOX;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        bool ok = true;
        {
            const Affine w(p);
            normalise16(p, (long long)blockIdx.x * TM, warp * 16, smem + OFF_A, w);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->a_full);
        }
        for (uint32_t c = 0; c < CHUNKS; ++c) {
            const uint32_t buf = c & 1, d1 = tmem_base + lane_off + COL_D1 + buf * 128 + eh * 32;
            ok = mbar_wait(&B->d1_full[buf], (c >> 1) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            // this warp: hidden channels 32*eh .. +31 of the chunk: f1 at columns [32 eh, +32), f2 at [64 + 32 eh, +32)
            hidden32(d1, d1 + 64, tmem_base + lane_off + COL_H + buf * 32 + eh * 16);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->h_full[buf]);
        }
        // update: D2 -> fp32 staging -> TMA reduce-add into z; this warp: output channels 64*eh .. +63
        if (ok && (ok = mbar_wait(&B->d2_full, 0, abort_flag))) {
            tc_fence_after();
            const long long row = (long long)blockIdx.x * TM + quarter * 32;
#pragma unroll
            for (int rd = 0; rd < 2; ++rd) {
                uint32_t d[32];
                tmem_ld_32x32(tmem_base + lane_off + COL_D2 + eh * 64 + rd * 32, d);
                tmem_ld_wait();
                if (rd == 1) {
                    if (lane == 0) bulk_wait_read0();
                    __syncwarp();
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<uint4*>(stg + sw128(lane, j)) = make_uint4(d[4 * j], d[4 * j + 1], d[4 * j + 2], d[4 * j + 3]);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0 && row < p.rows_flat) {
                    tma_reduce_add_4d(&map_z, stg, eh * 64 + rd * 32, (int)row, 0, 0);
                    bulk_commit();
                }
            }
            if (lane == 0) bulk_wait0();
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

}  // namespace trz
}  // namespace b200pf

using namespace b200pf;

extern "C" int b200pf_transition_z_tc(float* z, const float* ln_gamma, const float* ln_beta,
                                      const b200pf_bf16* w12, const b200pf_bf16* w3, long long n_rows_flat, void* stream) {
    using namespace trz;
    B200PF_REQUIRE(z && ln_gamma && ln_beta && w12 && w3 && n_rows_flat > 0, B200PF_ERR_INVALID, "transition_z_tc: bad argument");
    B200PF_REQUIRE(n_rows_flat < (1ll << 31), B200PF_ERR_UNSUPPORTED, "transition_z_tc: too many rows");
    B200PF_REQUIRE(aligned16(z) && aligned16(w12) && aligned16(w3) && aligned16(ln_gamma) && aligned16(ln_beta),
                   B200PF_ERR_INVALID, "transition_z_tc: pointers must be 16-byte aligned");
    CUtensorMap m12, m3, mz;
    int rc;
    const long long tiles = (n_rows_flat + TM - 1) / TM;
    int sms;
    if ((rc = multiprocessors(&sms)) != B200PF_OK) return rc;
    const bool one_each = tiles <= sms;
    {
        cuuint64_t dims[4] = {128, 128, CHUNKS, 1};
        cuuint64_t str[3] = {256, 128 * 256, 128 * 256 * CHUNKS};
        cuuint32_t box[4] = {64, one_each ? 128u : 64u, 1, 1};
        if ((rc = tmap_encode(&m12, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w12, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "w12")) != B200PF_OK) return rc;
    }
    {
        cuuint64_t dims[4] = {64, 128, CHUNKS, 1};
        cuuint64_t str[3] = {128, 128 * 128, 128 * 128 * CHUNKS};
        cuuint32_t box[4] = {64, one_each ? 128u : 64u, 1, 1};
        if ((rc = tmap_encode(&m3, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w3, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "w3")) != B200PF_OK) return rc;
    }
    {
        cuuint64_t dims[4] = {128, (cuuint64_t)n_rows_flat, 1, 1};
        cuuint64_t str[3] = {512, (cuuint64_t)n_rows_flat * 512, (cuuint64_t)n_rows_flat * 512};
        cuuint32_t box[4] = {32, 32, 1, 1};
        if ((rc = tmap_encode(&mz, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, z, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "z")) != B200PF_OK) return rc;
    }
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "transition_z_tc: no device status word");
    B200PF_SMEM_ATTR_ONCE(transition_pair_kernel, pair::SMEM_BYTES);
    B200PF_SMEM_ATTR_ONCE(transition_one_kernel, one::SMEM_BYTES);
    Args a{z, ln_gamma, ln_beta, n_rows_flat};
    if (one_each)
        return launch_pdl(transition_one_kernel, dim3((unsigned)tiles), dim3(one::THREADS), one::SMEM_BYTES, (cudaStream_t)stream, m12, m3, mz, a, status);
    int pairs;
    if ((rc = resident_pairs<transition_pair_kernel>(pair::THREADS, pair::SMEM_BYTES, &pairs)) != B200PF_OK) return rc;
    if (pairs > sms / 2) pairs = sms > 1 ? sms / 2 : 1;
    const long long couples = (tiles + 1) / 2;
    return launch_pdl(transition_pair_kernel, dim3(2u * (unsigned)(couples < pairs ? couples : pairs)), dim3(pair::THREADS), pair::SMEM_BYTES, (cudaStream_t)stream,
                      m12, m3, mz, a, status);
}
