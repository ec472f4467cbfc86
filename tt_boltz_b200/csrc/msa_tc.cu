// The MSA stack's row-wise work on tcgen05, one kernel per stage (64-channel activations m[S][N][64]):
//   msa_transition_kernel   m += W3 (silu(W1 LN(m)) * (W2 LN(m)))
//   pwa_value_kernel        v[head][s][d][token] = W_m LN(m), the K-major operand of the averaging GEMM
//   pwa_output_kernel       m += W_o (sigmoid(W_g LN(m)) * o), o[head][s][d][token] what that GEMM returned
// Persistent CTAs over tiles of 128 rows: loader warps normalise the rows into a bf16 tile in shared memory (K-major, 128-byte
// swizzle), one warp issues the MMAs against weights that stay in shared memory, eight epilogue warps read tensor memory, and
// m is updated by TMA reduce-add, so neither a projection nor a hidden layer goes through memory.
// What bounds them is memory and, for the transition and the output, the special-function results per gate value: at 1024 sequences x 600
// tokens the transition takes 142 us, the value kernel 106 us, the output kernel 138 us.  As LayerNorm, GEMM,
// activation, transposition and add kernels of their own the same work took about 500 and 680 us and moved 4 to 5 times as much.
#include "rowtc.cuh"

namespace b200pf {
namespace msatc {

using rtc::sw128;
using rtc::TM;

constexpr int CM = 64;                                    // MSA channels: one 128-byte k-block
constexpr int X_BYTES = TM * 128;                         // normalised tile: [128 rows][64] bf16
constexpr int BOX = 128 * 128;                            // [128 rows][128 bytes], 128-byte swizzle
constexpr int LOAD_WARPS = 6, MMA_WARP = 6, TMA_WARP = 7, EPI_WARP0 = 8, EPI_WARPS = 8, THREADS = 16 * 32;
constexpr int PASS_ROWS = 32, PASSES = TM / PASS_ROWS;    // a loader warp's unit of work

// 32 rows of 64 channels -> bf16 rows row0 .. row0 + 31 of the tile; called by one warp.  Eight lanes per row, two float4
// each; eight rows per lane at once, so that a warp has all of its loads in flight.  Rows >= valid are written as zeros.
__device__ __forceinline__ void ln64_rows32(const float* src, int row0, int valid, const float4 (&gam)[2], const float4 (&bet)[2], uint8_t* tile, int lane) {
    const int sub = lane & 7, rq = lane >> 3;
    float4 v[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = row0 + i * 4 + rq;
        const float4* p = reinterpret_cast<const float4*>(src + (long long)(row < valid ? row : 0) * CM) + sub;
        v[i][0] = p[0];
        v[i][1] = p[8];
    }
    float s[8], ss[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 t = add2(add2(low2(v[i][0]), high2(v[i][0])), add2(low2(v[i][1]), high2(v[i][1])));
        s[i] = t.x + t.y;
    }
#pragma unroll
    for (int step = 1; step < 8; step <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], step);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float mean = s[i] * (1.f / CM);
        float2 sq = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 2; ++j) centre4(v[i][j], make_float2(-mean, -mean), sq);
        ss[i] = sq.x + sq.y;
    }
#pragma unroll
    for (int step = 1; step < 8; step <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], step);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = row0 + i * 4 + rq;
        const float rstd = rsqrtf(ss[i] * (1.f / CM) + LN_EPS);
        const bool keep = row < valid;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint2 o;
            const float4 y = affine4(v[i][j], make_float2(rstd, rstd), gam[j], bet[j]);
            o.x = keep ? pack_bf16x2(y.x, y.y) : 0u;
            o.y = keep ? pack_bf16x2(y.z, y.w) : 0u;
            *reinterpret_cast<uint2*>(tile + sw128(row, j * 4 + (sub >> 1)) + (sub & 1) * 8) = o;
        }
    }
}

// Asks L2 for rows row0 + lane of the tile after this one (two 128-byte lines each).
__device__ __forceinline__ void prefetch_rows(const float* src, int row, int valid) {
    if (row < valid) {
        const char* p = reinterpret_cast<const char*>(src + (long long)row * CM);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 128));
    }
}

// Tiles: a tensor seen as `lines` lines of `span` rows, 128 rows of one line per tile.
struct Tiling {
    int lines, span, tpl, tiles;
};
struct LnRows {
    const float* m;                  // [lines][span][64]
    const float *gamma, *beta;
    Tiling t;
};

// The loader warps' loop, the same in all three kernels.
__device__ __forceinline__ bool load_loop(const LnRows& p, uint8_t* x0, uint64_t* x_full, uint64_t* x_empty, volatile int* abort_flag, int warp, int lane) {
    using namespace sm100;
    float4 gam[2], bet[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        gam[j] = reinterpret_cast<const float4*>(p.gamma)[j * 8 + (lane & 7)];
        bet[j] = reinterpret_cast<const float4*>(p.beta)[j * 8 + (lane & 7)];
    }
    // Passes go round robin over the loader warps: pass u is rows 32 (u % 4) of this CTA's tile u / 4.
    for (uint32_t u = warp;; u += LOAD_WARPS) {
        const uint32_t it = u / PASSES, stage = it & 1, ph = (it >> 1) & 1;
        const int t = (int)(blockIdx.x + it * gridDim.x), row0 = (int)(u % PASSES) * PASS_ROWS;
        if (t >= p.t.tiles) break;
        if (!mbar_wait(&x_empty[stage], ph ^ 1, abort_flag)) return false;
        const int tn = (int)(blockIdx.x + (u + LOAD_WARPS) / PASSES * gridDim.x);
        if (tn < p.t.tiles) {
            const int ln = tn / p.t.tpl, pn = (tn - ln * p.t.tpl) * TM;
            prefetch_rows(p.m + ((long long)ln * p.t.span + pn) * CM, (int)((u + LOAD_WARPS) % PASSES) * PASS_ROWS + lane, p.t.span - pn);
        }
        const int line = t / p.t.tpl, pos0 = (t - line * p.t.tpl) * TM;
        ln64_rows32(p.m + ((long long)line * p.t.span + pos0) * CM, row0, p.t.span - pos0, gam, bet, x0 + stage * X_BYTES, lane);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&x_full[stage]);
    }
    return true;
}

// 1 / (1 + e^-x) of two values, each by itself (the packed instructions round either half alone; 0 where the exponential overflows).  One
// reciprocal of the denominators' product is three special-function results for four and takes the transition from 142 to 130 us and the
// output from 138 to 125 at 1024 x 600, but two more roundings a gate (rms error 0.99 for 0.79 units of 2^-24 at arguments around one), and in
// the output, where the two are neighbouring tokens, either's bits hang on the other, and a NaN of one is both's.  With a correction of
// the two by their own residuals (0.76) the transition takes 143.
__device__ __forceinline__ float2 sigmoids(float2 x) {
    const float2 t = mul2(x, make_float2(-1.44269504f, -1.44269504f));
    float2 e, s;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(t.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(t.y));
    const float2 d = add2(e, make_float2(1.f, 1.f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s.x) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s.y) : "f"(d.y));
    return s;
}

// A warp's [32 rows][32 fp32] block of an update into m by TMA reduce-add, through a staging tile of its own (STG_WARP bytes): no warp
// waits for another.
constexpr int STG_WARP = 32 * 128;
__device__ __forceinline__ void reduce_update(const CUtensorMap* map_m, uint8_t* stg, const uint32_t (&d)[32], int lane, int col, int pos, int span, int line) {
    using namespace sm100;
    if (lane == 0) bulk_wait_read0();                          // the tile before has left the staging tile
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(stg + sw128(lane, j)) = make_uint4(d[4 * j], d[4 * j + 1], d[4 * j + 2], d[4 * j + 3]);
    fence_proxy_async();
    __syncwarp();
    if (lane == 0 && pos < span) {
        tma_reduce_add_4d(map_m, stg, col, pos, line, 0);
        bulk_commit();
    }
}

// ------------------------------------------------------------------------------------------------
// transition
// ------------------------------------------------------------------------------------------------
namespace tr {
constexpr int CHUNKS = 4;                                 // 64 hidden channels each: 64 rows of fc1, then 64 of fc2
constexpr int W3_KB = 64 * 128;                           // [64 out][64 hidden]
constexpr int OFF_W12 = 0, OFF_W3 = CHUNKS * BOX, OFF_X = OFF_W3 + CHUNKS * W3_KB, OFF_STG = OFF_X + 2 * X_BYTES;
constexpr int OFF_BAR = OFF_STG + 2 * BOX, SMEM = OFF_BAR + 256;          // 164,096
constexpr uint32_t COL_D1 = 0, COL_D2 = 256, COL_H = 384;                 // 2 x 128 | 2 x 64 | 2 x 32
struct Bars {
    uint64_t w_full, x_full[2], x_empty[2], d1_full[2], h_full[2], d2_full[2], d2_empty[2];
    uint32_t tmem_slot;
    int abort_flag;
};
}  // namespace tr

__global__ void __launch_bounds__(THREADS, 1)
msa_transition_kernel(const __grid_constant__ CUtensorMap map_w12, const __grid_constant__ CUtensorMap map_w3, const __grid_constant__ CUtensorMap map_m,
                      LnRows p, unsigned int* status) {
    using namespace sm100;
    using namespace tr;
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
        mbar_init(&B->w_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->x_full[i], PASSES); mbar_init(&B->x_empty[i], 1);
            mbar_init(&B->d1_full[i], 1); mbar_init(&B->h_full[i], EPI_WARPS);
            mbar_init(&B->d2_full[i], 1); mbar_init(&B->d2_empty[i], EPI_WARPS);
        }
        B->abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == MMA_WARP) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    if (tid == 32) { tma_prefetch_desc(&map_w12); tma_prefetch_desc(&map_w3); tma_prefetch_desc(&map_m); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = B->tmem_slot;
    grid_dependency_wait();                 // behind the CTA's barrier: every warp goes to work by itself from here on
    grid_launch_dependents();

    bool ok = true;
    if (warp < LOAD_WARPS) {
        ok = load_loop(p, smem + OFF_X, B->x_full, B->x_empty, abort_flag, warp, lane);
    } else if (warp == MMA_WARP) {
        // D1[c & 1] = x W12[chunk]^T while the epilogue turns the chunk before into h; D2 += h W3[:, chunk]^T
        constexpr uint32_t idesc1 = make_idesc_bf16(TM, 128), idesc2 = make_idesc_bf16(TM, 64);
        const uint64_t d_x = make_desc_k_sw128(smem_u32(smem + OFF_X)), d_w12 = make_desc_k_sw128(smem_u32(smem + OFF_W12)),
                       d_w3 = make_desc_k_sw128(smem_u32(smem + OFF_W3));
        uint32_t it = 0, h_cnt[2] = {0, 0};
        if (elect_one()) {
            mbar_arrive_expect_tx(&B->w_full, CHUNKS * (BOX + W3_KB));
            for (int c = 0; c < CHUNKS; ++c) {
                tma_load_4d(smem + OFF_W12 + c * BOX, &map_w12, &B->w_full, 0, c * 128, 0, 0);
                tma_load_4d(smem + OFF_W3 + c * W3_KB, &map_w3, &B->w_full, c * 64, 0, 0, 0);
            }
        }
        __syncwarp();
        ok = mbar_wait_warp(&B->w_full, 0, abort_flag);
        auto gemm1 = [&](uint32_t stage, int c) {
            if (elect_one()) {
                const uint64_t dx = d_x + stage * (uint64_t)(X_BYTES >> 4), dw = d_w12 + c * (uint64_t)(BOX >> 4);
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16(tmem + COL_D1 + (c & 1) * 128, dx + 2 * k, dw + 2 * k, idesc1, k ? 1u : 0u);
                umma_commit(&B->d1_full[c & 1]);
                if (c + 1 == CHUNKS) umma_commit(&B->x_empty[stage]);
            }
            __syncwarp();
        };
        for (int t = blockIdx.x; t < p.t.tiles && ok; t += gridDim.x, ++it) {
            const uint32_t stage = it & 1, ph = (it >> 1) & 1;
            ok = mbar_wait_warp(&B->x_full[stage], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
            gemm1(stage, 0);
            for (int c = 0; c < CHUNKS && ok; ++c) {
                if (c + 1 < CHUNKS) gemm1(stage, c + 1);       // the h of chunk c - 1, which read that buffer, has been waited for
                ok = mbar_wait_warp(&B->h_full[c & 1], h_cnt[c & 1] & 1, abort_flag);
                if (!ok) break;
                ++h_cnt[c & 1];
                if (c == 0) ok = mbar_wait_warp(&B->d2_empty[stage], ph ^ 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16_ts(tmem + COL_D2 + stage * 64, tmem + COL_H + (c & 1) * 32 + k * 8, d_w3 + c * (uint64_t)(W3_KB >> 4) + 2 * k, idesc2,
                                     (c | k) ? 1u : 0u);
                    if (c + 1 == CHUNKS) umma_commit(&B->d2_full[stage]);
                }
                __syncwarp();
            }
        }
    } else if (warp >= EPI_WARP0) {
        const int quarter = warp & 3, half = (warp - EPI_WARP0) >> 2;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        uint32_t it = 0, d1_cnt[2] = {0, 0};
        for (int t = blockIdx.x; t < p.t.tiles && ok; t += gridDim.x, ++it) {
            const uint32_t stage = it & 1, ph = (it >> 1) & 1;
#pragma unroll 1
            for (int c = 0; c < CHUNKS; ++c) {
                const uint32_t buf = c & 1;
                ok = mbar_wait(&B->d1_full[buf], d1_cnt[buf] & 1, abort_flag);
                if (!ok) break;
                ++d1_cnt[buf];
                tc_fence_after();
                // hidden channels 32 half .. + 31 of the chunk: fc1 in columns [32 half, + 32), fc2 64 further
                uint32_t f1[32], f2[32], hw[16];
                tmem_ld_32x32(tmem + lane_off + COL_D1 + buf * 128 + half * 32, f1);
                tmem_ld_32x32(tmem + lane_off + COL_D1 + buf * 128 + 64 + half * 32, f2);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float a0 = __uint_as_float(f1[2 * e]), a1 = __uint_as_float(f1[2 * e + 1]);
                    const float2 u = mul2(mul2(make_float2(a0, a1), sigmoids(make_float2(a0, a1))), make_float2(__uint_as_float(f2[2 * e]), __uint_as_float(f2[2 * e + 1])));
                    hw[e] = pack_bf16x2(u.x, u.y);
                }
                tmem_st_32x16(tmem + lane_off + COL_H + buf * 32 + half * 16, hw);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&B->h_full[buf]);
            }
            if (!ok) break;
            ok = mbar_wait(&B->d2_full[stage], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
            uint32_t d[32];
            tmem_ld_32x32(tmem + lane_off + COL_D2 + stage * 64 + half * 32, d);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->d2_empty[stage]);
            const int line = t / p.t.tpl, pos0 = (t - line * p.t.tpl) * TM;
            reduce_update(&map_m, smem + OFF_STG + (warp - EPI_WARP0) * STG_WARP, d, lane, half * 32, pos0 + quarter * 32, p.t.span, line);
        }
        if (lane == 0) bulk_wait0();
    }
    if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------------------------------------------------------
// pair-weighted averaging: values
// ------------------------------------------------------------------------------------------------
namespace va {
constexpr int OFF_W = 0, OFF_X = 2 * BOX, OFF_STG = OFF_X + 2 * X_BYTES, OFF_BAR = OFF_STG + 4 * BOX, SMEM = OFF_BAR + 128;      // 131,200
struct Bars {
    uint64_t w_full, x_full[2], x_empty[2], d_full[2], d_empty[2];
    uint32_t tmem_slot;
    int abort_flag;
};
}  // namespace va

__global__ void __launch_bounds__(THREADS, 1)
pwa_value_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_v, LnRows p, unsigned int* status) {
    using namespace sm100;
    using namespace va;
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
        mbar_init(&B->w_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->x_full[i], PASSES); mbar_init(&B->x_empty[i], 1);
            mbar_init(&B->d_full[i], 1); mbar_init(&B->d_empty[i], EPI_WARPS);
        }
        B->abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == MMA_WARP) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    if (tid == 32) { tma_prefetch_desc(&map_w); tma_prefetch_desc(&map_v); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = B->tmem_slot;
    grid_dependency_wait();                 // behind the CTA's barrier: every warp goes to work by itself from here on
    grid_launch_dependents();

    bool ok = true;
    if (warp < LOAD_WARPS) {
        ok = load_loop(p, smem + OFF_X, B->x_full, B->x_empty, abort_flag, warp, lane);
    } else if (warp == MMA_WARP) {
        // D[stage][channel half] (128 channels x 128 tokens) = W_m[half] x^T: the epilogue thread holds a channel's tokens
        constexpr uint32_t idesc = make_idesc_bf16(128, TM);
        const uint64_t d_w = make_desc_k_sw128(smem_u32(smem + OFF_W)), d_x = make_desc_k_sw128(smem_u32(smem + OFF_X));
        uint32_t it = 0;
        if (elect_one()) {
            mbar_arrive_expect_tx(&B->w_full, 2 * BOX);
            for (int h = 0; h < 2; ++h) tma_load_4d(smem + OFF_W + h * BOX, &map_w, &B->w_full, 0, h * 128, 0, 0);
        }
        __syncwarp();
        ok = mbar_wait_warp(&B->w_full, 0, abort_flag);
        for (int t = blockIdx.x; t < p.t.tiles && ok; t += gridDim.x, ++it) {
            const uint32_t stage = it & 1, ph = (it >> 1) & 1;
            ok = mbar_wait_warp(&B->x_full[stage], ph, abort_flag) && mbar_wait_warp(&B->d_empty[stage], ph ^ 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t dx = d_x + stage * (uint64_t)(X_BYTES >> 4);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem + stage * 256 + h * 128, d_w + h * (uint64_t)(BOX >> 4) + 2 * k, dx + 2 * k, idesc, k ? 1u : 0u);
                umma_commit(&B->x_empty[stage]);
                umma_commit(&B->d_full[stage]);
            }
            __syncwarp();
        }
    } else if (warp >= EPI_WARP0) {
        // thread = channel 128 h + 32 quarter + lane, i.e. head 4 h + quarter, 64 tokens of its half; a box is [32 d][64 tokens]
        const int quarter = warp & 3, half = (warp - EPI_WARP0) >> 2;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        uint8_t* stg = smem + OFF_STG + (warp - EPI_WARP0) * 2 * STG_WARP;
        uint32_t it = 0;
        for (int t = blockIdx.x; t < p.t.tiles && ok; t += gridDim.x, ++it) {
            const uint32_t stage = it & 1, ph = (it >> 1) & 1;
            ok = mbar_wait(&B->d_full[stage], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (lane == 0) bulk_wait_read0();
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t r[2][32];
                tmem_ld_32x32(tmem + lane_off + stage * 256 + h * 128 + half * 64, r[0]);
                tmem_ld_32x32(tmem + lane_off + stage * 256 + h * 128 + half * 64 + 32, r[1]);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int e = j * 8 + q * 2;
                        w[q] = pack_bf16x2(__uint_as_float(r[e >> 5][e & 31]), __uint_as_float(r[e >> 5][(e & 31) + 1]));
                    }
                    *reinterpret_cast<uint4*>(stg + h * STG_WARP + sw128(lane, j)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->d_empty[stage]);
            fence_proxy_async();
            __syncwarp();
            const int line = t / p.t.tpl, pos = (t - line * p.t.tpl) * TM + half * 64;
            if (lane == 0 && pos < p.t.span) {      // the second token half may lie beyond the line's end: nothing to store
                for (int h = 0; h < 2; ++h) tma_store_4d(&map_v, stg + h * STG_WARP, pos, 0, line, h * 4 + quarter);
                bulk_commit();
            }
        }
        if (lane == 0) bulk_wait0();
    }
    if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------------------------------------------------------
// pair-weighted averaging: gate, output projection, residual
// ------------------------------------------------------------------------------------------------
namespace ou {
constexpr int SLOTS = 3, SLOT = 2 * BOX;                  // a slot: 128 channels (4 heads) x 128 tokens of o, two token halves
constexpr int WO_KB = 64 * 128;                           // [64 out][64 channels]
constexpr int OFF_WG = 0, OFF_WO = 2 * BOX, OFF_X = OFF_WO + 4 * WO_KB, OFF_O = OFF_X + 2 * X_BYTES, OFF_STG = OFF_O + SLOTS * SLOT;
constexpr int OFF_BAR = OFF_STG + 2 * BOX, SMEM = OFF_BAR + 256;          // 229,632
static_assert(SMEM <= 232448, "shared memory budget");
constexpr uint32_t COL_G = 0, COL_D2 = 256;                               // 2 x 128 | 2 x 64
struct Bars {
    uint64_t w_full, x_full[2], x_empty[2], g_full[2], g_empty[2], o_full[SLOTS], o_empty[SLOTS], val_full[2], d2_full[2], d2_empty[2];
    uint32_t tmem_slot;
    int abort_flag;
};
// MN-major A operand: K rows (channels) of 64 tokens (128 bytes), 128-byte swizzle; the two token halves BOX bytes apart.
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(BOX >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
}  // namespace ou

__global__ void __launch_bounds__(THREADS, 1)
pwa_output_kernel(const __grid_constant__ CUtensorMap map_wg, const __grid_constant__ CUtensorMap map_wo, const __grid_constant__ CUtensorMap map_o,
                  const __grid_constant__ CUtensorMap map_m, LnRows p, unsigned int* status) {
    using namespace sm100;
    using namespace ou;
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
        mbar_init(&B->w_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->x_full[i], PASSES); mbar_init(&B->x_empty[i], 1);
            mbar_init(&B->g_full[i], 1); mbar_init(&B->g_empty[i], EPI_WARPS);
            mbar_init(&B->val_full[i], EPI_WARPS);
            mbar_init(&B->d2_full[i], 1); mbar_init(&B->d2_empty[i], EPI_WARPS);
        }
        for (int i = 0; i < SLOTS; ++i) { mbar_init(&B->o_full[i], 1); mbar_init(&B->o_empty[i], 1); }
        B->abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == MMA_WARP) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    if (tid == 32) { tma_prefetch_desc(&map_wg); tma_prefetch_desc(&map_wo); tma_prefetch_desc(&map_o); tma_prefetch_desc(&map_m); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = B->tmem_slot;
    grid_dependency_wait();                 // behind the CTA's barrier: every warp goes to work by itself from here on
    grid_launch_dependents();

    bool ok = true;
    if (warp < LOAD_WARPS) {
        ok = load_loop(p, smem + OFF_X, B->x_full, B->x_empty, abort_flag, warp, lane);
    } else if (warp == TMA_WARP) {
        if (lane == 0) {
            uint32_t slot = 0, ph = 0;
            for (int t = blockIdx.x; t < p.t.tiles && ok; t += gridDim.x) {
                const int line = t / p.t.tpl, pos0 = (t - line * p.t.tpl) * TM;
                for (int h = 0; h < 2; ++h) {
                    ok = mbar_wait(&B->o_empty[slot], ph ^ 1, abort_flag);
                    if (!ok) break;
                    uint8_t* dst = smem + OFF_O + slot * SLOT;
                    mbar_arrive_expect_tx(&B->o_full[slot], SLOT);
                    tma_load_4d(dst, &map_o, &B->o_full[slot], pos0, 0, line, h * 4);
                    tma_load_4d(dst + BOX, &map_o, &B->o_full[slot], pos0 + 64, 0, line, h * 4);
                    if (++slot == SLOTS) { slot = 0; ph ^= 1; }
                }
            }
            if (!ok) {   // give copies in flight time to land before the CTA's shared memory goes away
                const uint64_t t0 = global_timer_ns();
                while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
            }
        }
    } else if (warp == MMA_WARP) {
        // per tile and channel half: D_g[half] = W_g[half] x^T, then D2 += (gated o of the half)^T W_o[:, half]^T; the gate of the
        // next tile is issued as soon as the epilogue has read this one's
        constexpr uint32_t idesc_g = make_idesc_bf16(128, TM), idesc_o = make_idesc_bf16(TM, 64) | (1u << 15);      // A MN-major
        const uint64_t d_wg = make_desc_k_sw128(smem_u32(smem + OFF_WG)), d_x = make_desc_k_sw128(smem_u32(smem + OFF_X)),
                       d_wo = make_desc_k_sw128(smem_u32(smem + OFF_WO)), d_o = desc_mn_sw128(smem_u32(smem + OFF_O));
        if (elect_one()) {
            mbar_arrive_expect_tx(&B->w_full, 2 * BOX + 4 * WO_KB);
            for (int h = 0; h < 2; ++h) tma_load_4d(smem + OFF_WG + h * BOX, &map_wg, &B->w_full, 0, h * 128, 0, 0);
            for (int k = 0; k < 4; ++k) tma_load_4d(smem + OFF_WO + k * WO_KB, &map_wo, &B->w_full, k * 64, 0, 0, 0);
        }
        __syncwarp();
        ok = mbar_wait_warp(&B->w_full, 0, abort_flag);
        auto gate = [&](uint32_t tile, int h) {           // tile: this CTA's running number
            const uint32_t stage = tile & 1;
            if (h == 0) ok = mbar_wait_warp(&B->x_full[stage], (tile >> 1) & 1, abort_flag);
            ok = ok && mbar_wait_warp(&B->g_empty[h], (tile & 1) ^ 1, abort_flag);
            if (!ok) return;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t dx = d_x + stage * (uint64_t)(X_BYTES >> 4);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    umma_bf16(tmem + COL_G + h * 128, d_wg + h * (uint64_t)(BOX >> 4) + 2 * k, dx + 2 * k, idesc_g, k ? 1u : 0u);
                umma_commit(&B->g_full[h]);
                if (h == 1) umma_commit(&B->x_empty[stage]);
            }
            __syncwarp();
        };
        uint32_t it = 0, slot = 0;
        for (int h = 0; h < 2 && ok; ++h) gate(0, h);
        for (int t = blockIdx.x; t < p.t.tiles && ok; t += gridDim.x, ++it) {
            const uint32_t acc = it & 1;
            for (int h = 0; h < 2 && ok; ++h) {
                ok = mbar_wait_warp(&B->val_full[h], it & 1, abort_flag);
                if (ok && h == 0) ok = mbar_wait_warp(&B->d2_empty[acc], ((it >> 1) & 1) ^ 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t da = d_o + slot * (uint64_t)(SLOT >> 4);
#pragma unroll
                    for (int k = 0; k < 8; ++k)           // 16 channels = 16 rows of 128 bytes per step
                        umma_bf16(tmem + COL_D2 + acc * 64, da + k * (uint64_t)(2048 >> 4),
                                  d_wo + (uint64_t)((h * 2 + (k >> 2)) * (WO_KB >> 4) + (k & 3) * 2), idesc_o, (h | k) ? 1u : 0u);
                    umma_commit(&B->o_empty[slot]);
                    if (h == 1) umma_commit(&B->d2_full[acc]);
                }
                __syncwarp();
                if (++slot == SLOTS) slot = 0;
                if (t + (int)gridDim.x < p.t.tiles) gate(it + 1, h);
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - EPI_WARP0) >> 2, lrow = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        auto update = [&](uint32_t tile, int t) {         // D2 of this CTA's tile number `tile` (global tile t) into m
            const uint32_t acc = tile & 1;
            ok = mbar_wait(&B->d2_full[acc], (tile >> 1) & 1, abort_flag);
            if (!ok) return;
            tc_fence_after();
            uint32_t d[32];
            tmem_ld_32x32(tmem + lane_off + COL_D2 + acc * 64 + half * 32, d);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->d2_empty[acc]);
            const int line = t / p.t.tpl, pos0 = (t - line * p.t.tpl) * TM;
            reduce_update(&map_m, smem + OFF_STG + (warp - EPI_WARP0) * STG_WARP, d, lane, half * 32, pos0 + quarter * 32, p.t.span, line);
        };
        uint32_t it = 0, slot = 0, ph = 0;
        int t = blockIdx.x;
        for (; t < p.t.tiles && ok; t += gridDim.x, ++it) {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                // thread = channel 128 h + lrow, the 64 tokens of its half: row lrow of box `half`
                ok = mbar_wait(&B->g_full[h], it & 1, abort_flag) && mbar_wait(&B->o_full[slot], ph, abort_flag);
                if (!ok) break;
                tc_fence_after();
                uint8_t* row = smem + OFF_O + slot * SLOT + half * BOX;
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    uint32_t g[32];
                    tmem_ld_32x32(tmem + lane_off + COL_G + h * 128 + half * 64 + b * 32, g);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint4* at = reinterpret_cast<uint4*>(row + sw128(lrow, b * 4 + j));
                        const uint4 ov = *at;
                        const uint32_t w[4] = {ov.x, ov.y, ov.z, ov.w};
                        uint32_t r[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float2 gate = sigmoids(make_float2(__uint_as_float(g[j * 8 + q * 2]), __uint_as_float(g[j * 8 + q * 2 + 1])));
                            const float2 u = mul2(make_float2(bf16_lo(w[q]), bf16_hi(w[q])), gate);
                            r[q] = pack_bf16x2(u.x, u.y);
                        }
                        *at = make_uint4(r[0], r[1], r[2], r[3]);
                    }
                }
                tc_fence_before();
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) { mbar_arrive(&B->g_empty[h]); mbar_arrive(&B->val_full[h]); }
                if (++slot == SLOTS) { slot = 0; ph ^= 1; }
            }
            if (ok && it > 0) update(it - 1, t - (int)gridDim.x);      // the tile before, whose product ran under this one's gate
        }
        if (ok) update(it - 1, t - (int)gridDim.x);
        if (lane == 0) bulk_wait0();
    }
    if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ---- host --------------------------------------------------------------------------------------
static int map_rows64(CUtensorMap* map, const void* w, int rows, int cols, int box_rows, const char* what) {      // [rows][cols] bf16, boxes of 64 columns
    cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)rows, 1, 1};
    cuuint64_t str[3] = {(cuuint64_t)cols * 2, (cuuint64_t)rows * cols * 2, (cuuint64_t)rows * cols * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
    return tmap_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, what);
}
static int map_update(CUtensorMap* map, const float* m, const Tiling& t) {
    cuuint64_t dims[4] = {CM, (cuuint64_t)t.span, (cuuint64_t)t.lines, 1};
    cuuint64_t str[3] = {CM * 4, (cuuint64_t)t.span * CM * 4, (cuuint64_t)t.span * t.lines * CM * 4};
    cuuint32_t box[4] = {32, 32, 1, 1};
    return tmap_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, m, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "m");
}
static int map_heads(CUtensorMap* map, const void* v, int s_len, int n, int np, int box_heads, const char* what) {      // [8][S][32][np] bf16
    cuuint64_t dims[4] = {(cuuint64_t)n, 32, (cuuint64_t)s_len, 8};
    cuuint64_t str[3] = {(cuuint64_t)np * 2, (cuuint64_t)np * 64, (cuuint64_t)np * 64 * s_len};
    cuuint32_t box[4] = {64, 32, 1, (cuuint32_t)box_heads};
    return tmap_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, v, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, what);
}
static Tiling tiling(int lines, int span) {
    const int tpl = (span + TM - 1) / TM;
    return Tiling{lines, span, tpl, lines * tpl};
}

}  // namespace msatc
}  // namespace b200pf

using namespace b200pf;
using namespace b200pf::msatc;

extern "C" int b200pf_msa_transition(float* m, const float* ln_gamma, const float* ln_beta, const b200pf_bf16* w12, const b200pf_bf16* w3,
                                     long long rows, void* stream) {
    B200PF_REQUIRE(m && ln_gamma && ln_beta && w12 && w3 && aligned16(m) && aligned16(ln_gamma) && aligned16(ln_beta) && aligned16(w12) && aligned16(w3),
                   B200PF_ERR_INVALID, "msa_transition: null or misaligned pointer");
    B200PF_REQUIRE(rows > 0 && rows < (1ll << 31) - TM, B200PF_ERR_UNSUPPORTED, "msa_transition: bad number of rows");
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "msa_transition: no device status word");
    const Tiling t = tiling(1, (int)rows);
    CUtensorMap m12, m3, mm;
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK || (rc = map_rows64(&m12, w12, 512, CM, 128, "w12")) != B200PF_OK ||
        (rc = map_rows64(&m3, w3, 64, 256, 64, "w3")) != B200PF_OK || (rc = map_update(&mm, m, t)) != B200PF_OK) return rc;
    B200PF_SMEM_ATTR_ONCE(msa_transition_kernel, tr::SMEM);
    return launch_pdl(msa_transition_kernel, dim3((unsigned)(t.tiles < sms ? t.tiles : sms)), dim3(THREADS), tr::SMEM, (cudaStream_t)stream, m12, m3, mm,
                      LnRows{m, ln_gamma, ln_beta, t}, status);
}

extern "C" int b200pf_pwa_value(const float* m, const float* ln_gamma, const float* ln_beta, const b200pf_bf16* w_m, b200pf_bf16* v, int s_len, int n,
                                int np, void* stream) {
    B200PF_REQUIRE(m && ln_gamma && ln_beta && w_m && v && aligned16(m) && aligned16(ln_gamma) && aligned16(ln_beta) && aligned16(w_m) && aligned16(v),
                   B200PF_ERR_INVALID, "pwa_value: null or misaligned pointer");
    B200PF_REQUIRE(s_len > 0 && n > 0 && np >= n && np % 8 == 0 && (long long)s_len * ((n + TM - 1) / TM) < (1ll << 31), B200PF_ERR_INVALID,
                   "pwa_value: np must be a multiple of 8 covering n");
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "pwa_value: no device status word");
    const Tiling t = tiling(s_len, n);
    CUtensorMap mw, mv;
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK || (rc = map_rows64(&mw, w_m, 256, CM, 128, "w_m")) != B200PF_OK ||
        (rc = map_heads(&mv, v, s_len, n, np, 1, "v")) != B200PF_OK) return rc;
    B200PF_SMEM_ATTR_ONCE(pwa_value_kernel, va::SMEM);
    return launch_pdl(pwa_value_kernel, dim3((unsigned)(t.tiles < sms ? t.tiles : sms)), dim3(THREADS), va::SMEM, (cudaStream_t)stream, mw, mv,
                      LnRows{m, ln_gamma, ln_beta, t}, status);
}

extern "C" int b200pf_pwa_output(float* m, const float* ln_gamma, const float* ln_beta, const b200pf_bf16* w_g, const b200pf_bf16* w_o,
                                 const b200pf_bf16* o, int s_len, int n, int np, void* stream) {
    B200PF_REQUIRE(m && ln_gamma && ln_beta && w_g && w_o && o && aligned16(m) && aligned16(ln_gamma) && aligned16(ln_beta) && aligned16(w_g) &&
                       aligned16(w_o) && aligned16(o), B200PF_ERR_INVALID, "pwa_output: null or misaligned pointer");
    B200PF_REQUIRE(s_len > 0 && n > 0 && np >= n && np % 8 == 0 && (long long)s_len * ((n + TM - 1) / TM) < (1ll << 31), B200PF_ERR_INVALID,
                   "pwa_output: np must be a multiple of 8 covering n");
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "pwa_output: no device status word");
    const Tiling t = tiling(s_len, n);
    CUtensorMap mg, mo, mov, mm;
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK || (rc = map_rows64(&mg, w_g, 256, CM, 128, "w_g")) != B200PF_OK ||
        (rc = map_rows64(&mo, w_o, 64, 256, 64, "w_o")) != B200PF_OK || (rc = map_heads(&mov, o, s_len, n, np, 4, "o")) != B200PF_OK ||
        (rc = map_update(&mm, m, t)) != B200PF_OK) return rc;
    B200PF_SMEM_ATTR_ONCE(pwa_output_kernel, ou::SMEM);
    return launch_pdl(pwa_output_kernel, dim3((unsigned)(t.tiles < sms ? t.tiles : sms)), dim3(THREADS), ou::SMEM, (cudaStream_t)stream, mg, mo, mov, mm,
                      LnRows{m, ln_gamma, ln_beta, t}, status);
}
