// Triangle-multiplication epilogue on tcgen05:
//   z += (LN_out(x) W_pout^T) * sigmoid(LN_in(z) W_gout^T)        per tile of 128 positions of one row.
//
// x arrives as channel-major planes x[d][row][pos].  A TMA load brings the [128 d][128 pos] block in
// as it lies (d rows, positions contiguous), which is exactly an MN-major A operand, so the first
// GEMM runs on the RAW x with W' = 0.5 * W_pout * gamma_out and the LayerNorm over d is applied
// afterwards per position:  p' = rstd * (acc - mean * wsum[c]) + wb[c],  wsum[c] = sum_d W'[c][d],
// wb = 0.5 * W_pout beta_out.  mean / rstd over d are taken from the same tile in shared memory.
// The gate GEMM uses LN_in(z) (affine applied by the loader warps) against 0.5 * W_gout, so that
// p * sigmoid(g) = p' + p' * tanh(g').  The fp32 update leaves through TMA reduce-add straight
// into z: the kernel never reads z for the residual.
// Roles (512 threads): warps 0-5 loaders (LN of z rows, 16 at a time, round robin), warp 6 TMA of the x tiles, warp 7 MMA issuer,
// warps 8-15 epilogue (x statistics, gate, update; each with a staging tile and reductions of its own, so that no warp waits for
// another).  A CTA's first tile is normalised by the epilogue warps, 16 rows each, which have nothing else to do before its
// accumulators exist; the loaders begin with the second.
// What bounded it was the chain x tile -> statistics -> accumulators -> update of ONE x buffer, whose copy could only start when the tile
// before had been read twice, and the statistics' 128 two-byte reads and 400 scalar instructions per thread.  With two x buffers,
// packed statistics of two positions per lane and six loader warps for four: 22.0 -> 14.0 us at 203 tokens, 65.8 -> 47.4 at 400,
// 288 -> 225 at 1024 (6.0 TB/s of its 10 E bytes, 0.91 of the copy rate).
#include "rowtc.cuh"
#include "tmap.cuh"

namespace b200pf {
namespace tme {

using namespace rtc;

constexpr int LOAD_WARPS = 6, X_WARP = 6, MMA_WARP = 7, EPI_WARP0 = 8, EPI_WARPS = 8, THREADS = 16 * 32;
constexpr int PASS_ROWS = 16, PASSES = TM / PASS_ROWS;   // a loader warp's unit of work
constexpr int W_TILE = 128 * 128 * 2;                    // 32 KB: two k-blocks of [128][128 B]
constexpr int OFF_WP = 0, OFF_WG = W_TILE;               // 0.5 * W_pout * gamma_out, 0.5 * W_gout
constexpr int OFF_AZ = 2 * W_TILE;                       // 2 stages
constexpr int OFF_XT = OFF_AZ + 2 * A_TILE_BYTES;        // 2 stages of 2 boxes of [128 d][64 pos]
constexpr int XT_BOX = 128 * 128;
constexpr int OFF_STG = OFF_XT + 4 * XT_BOX;             // staging: per epilogue warp [32 pos][32 fp32], 128-byte swizzle
constexpr int STG_BOX = 32 * 128;
constexpr int OFF_CONST = OFF_STG + EPI_WARPS * STG_BOX; // wsum[128], wb[128] fp32
constexpr int OFF_BAR = OFF_CONST + 1024;
constexpr int SMEM_BYTES = OFF_BAR + 128;                // 230,528; the dynamic window must start 1024-byte aligned
static_assert(SMEM_BYTES <= 232448, "shared memory budget");

struct Args {
    const float* z;                 // read for LN_in; the residual is added by TMA reduce
    const float* ln_in_gamma;
    const float* ln_in_beta;
    const float* wsum;              // [128] row sums of w_pout (as stored in bf16)
    const float* wb;                // [128] 0.5 * W_pout beta_out
    int rows, n;
};

struct Bars {
    uint64_t w_full, x_full[2], x_empty[2], in_full[2], in_empty[2], acc_full[2], acc_empty[2];
    uint32_t tmem_slot;
    int abort_flag;
};

// MN-major A operand: rows of the tile are K (d), 64 positions (128 bytes) per row, 128-byte swizzle;
// the two 64-position boxes are XT_BOX bytes apart (leading offset), 8-row K groups 1024 bytes (stride offset).
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(XT_BOX >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ float tanh_approx(float x) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
    return t;
}

// Two fp32 values in one 64-bit register for the packed instructions (one issue slot, two results).
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__global__ void __launch_bounds__(THREADS, 1)
trimul_epilogue_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_z,
                          const __grid_constant__ CUtensorMap map_wp, const __grid_constant__ CUtensorMap map_wg, Args p,
                          unsigned int* status) {
    using namespace sm100;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {
        grid_dependency_wait();
        if (threadIdx.x == 0) atomicOr(status, DEV_STATUS_BAD_INDEX);
        return;
    }
    Bars* B = reinterpret_cast<Bars*>(smem + OFF_BAR);
    volatile int* abort_flag = &B->abort_flag;
    float* wsum_s = reinterpret_cast<float*>(smem + OFF_CONST);
    float* wb_s = wsum_s + 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int tpl = (p.n + TM - 1) / TM;
    const long long tiles = (long long)p.rows * tpl;

    if (tid == 0) {
        mbar_init(&B->w_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->x_full[i], 1);
            mbar_init(&B->x_empty[i], 1 + EPI_WARPS);      // the MMAs and the epilogue warps' statistics pass both read the x tile
            mbar_init(&B->in_full[i], PASSES); mbar_init(&B->in_empty[i], 1);
            mbar_init(&B->acc_full[i], 1); mbar_init(&B->acc_empty[i], EPI_WARPS);
        }
        B->abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (tid == 32) { tma_prefetch_desc(&map_x); tma_prefetch_desc(&map_wp); tma_prefetch_desc(&map_wg); tma_prefetch_desc(&map_z); }
    if (warp == MMA_WARP) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    grid_dependency_wait();
    grid_launch_dependents();
    if (tid < 128) { wsum_s[tid] = p.wsum[tid]; wb_s[tid] = p.wb[tid]; }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = B->tmem_slot;

    // One warp's 16 rows of a tile, 8 lanes per row: fetched, and normalised into the A tile.  Positions beyond the row's end repeat
    // its first one: the reduce-add clips them (zeroing them cost the loaders registers: with spills the kernel took 297 us at
    // 1024 tokens, this way 270).
    const int sub = lane & 7, rq = lane >> 3;
    auto fetch16 = [&](int r, int pos0, int row0, float4 (&v)[4][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + row0 + i * 4 + rq;
            const float4* src = reinterpret_cast<const float4*>(p.z + ((long long)r * p.n + (pos < p.n ? pos : 0)) * KC);
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = src[j * 8 + sub];
        }
    };
    auto normalise16 = [&](int row0, float4 (&v)[4][4], uint8_t* a_tile, const float4 (&gam)[4], const float4 (&bet)[4]) {
        // the four rows of a pass stage by stage (sums, shuffles, variance, ...): instruction-level parallelism
        // for a warp that has its scheduler almost to itself
        float s4[4], ss4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 t = add2(low2(v[i][0]), high2(v[i][0]));
#pragma unroll
            for (int j = 1; j < 4; ++j) t = add2(t, add2(low2(v[i][j]), high2(v[i][j])));
            const float s = t.x + t.y;
            s4[i] = s;
        }
#pragma unroll
        for (int step = 1; step < 8; step <<= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) s4[i] += __shfl_xor_sync(0xffffffffu, s4[i], step);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float mean = s4[i] * (1.f / KC);
            float2 sq = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; ++j) centre4(v[i][j], make_float2(-mean, -mean), sq);
            const float ss = sq.x + sq.y;
            ss4[i] = ss;
        }
#pragma unroll
        for (int step = 1; step < 8; step <<= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) ss4[i] += __shfl_xor_sync(0xffffffffu, ss4[i], step);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = row0 + i * 4 + rq;
            const float rstd = rsqrtf(ss4[i] * (1.f / KC) + LN_EPS);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint2 o;
                const float4 y = affine4(v[i][j], make_float2(rstd, rstd), gam[j], bet[j]);
                o.x = pack_bf16x2(y.x, y.y);
                o.y = pack_bf16x2(y.z, y.w);
                const int chunk = (j & 1) * 4 + (sub >> 1);
                *reinterpret_cast<uint2*>(a_tile + (j >> 1) * A_KB_BYTES + sw128(row, chunk) + (sub & 1) * 8) = o;
            }
        }
    };
    auto load_affine = [&](float4 (&gam)[4], float4 (&bet)[4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            gam[j] = reinterpret_cast<const float4*>(p.ln_in_gamma)[j * 8 + sub];
            bet[j] = reinterpret_cast<const float4*>(p.ln_in_beta)[j * 8 + sub];
        }
    };
    if (warp < LOAD_WARPS) {
        // ---------------------------- loaders ----------------------------
        float4 gam[4], bet[4];
        load_affine(gam, bet);
        // Passes of 16 rows go round robin over the loader warps: pass u is rows 16 (u % 8) of tile 1 + u / 8 of this CTA
        // (the epilogue warps normalise its first).
        auto tile_of = [&](uint32_t u) { return (int)(blockIdx.x + (1 + u / PASSES) * gridDim.x); };
        bool ok = true;
        for (uint32_t u = warp; ok; u += LOAD_WARPS) {
            const int t = tile_of(u);
            if (t >= tiles) break;
            const int r = t / tpl, pos0 = (t - r * tpl) * TM, row0 = (int)(u % PASSES) * PASS_ROWS;
            const uint32_t it = 1 + u / PASSES, stage = it & 1, ph = (it >> 1) & 1;
            ok = mbar_wait(&B->in_empty[stage], ph ^ 1, abort_flag);
            if (!ok) break;
            {   // ask L2 for this warp's next 16 rows (two lanes per row, two 128-byte lines each)
                const int tn = tile_of(u + LOAD_WARPS), rn = tn / tpl;
                const int posn = (tn - rn * tpl) * TM + (int)((u + LOAD_WARPS) % PASSES) * PASS_ROWS + (lane & 15);
                if (tn < tiles && posn < p.n) {
                    const char* rowp = reinterpret_cast<const char*>(p.z + ((long long)rn * p.n + posn) * KC) + (lane >> 4) * 256;
#pragma unroll
                    for (int j = 0; j < 2; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(rowp + j * 128));
                }
            }
            float4 v[4][4];
            fetch16(r, pos0, row0, v);
            normalise16(row0, v, smem + OFF_AZ + stage * A_TILE_BYTES, gam, bet);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->in_full[stage]);
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else if (warp == X_WARP) {
        // ---------------------------- TMA of the x tiles ----------------------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
                const int r = t / tpl, pos0 = (t - r * tpl) * TM;
                const uint32_t stage = it & 1;
                ok = mbar_wait(&B->x_empty[stage], ((it >> 1) & 1) ^ 1, abort_flag);
                if (!ok) break;
                uint8_t* xt = smem + OFF_XT + stage * 2 * XT_BOX;
                mbar_arrive_expect_tx(&B->x_full[stage], 2 * XT_BOX);
                tma_load_4d(xt, &map_x, &B->x_full[stage], pos0, r, 0, 0);
                tma_load_4d(xt + XT_BOX, &map_x, &B->x_full[stage], pos0 + 64, r, 0, 0);
            }
            if (!ok) {
                atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
                uint64_t t0 = global_timer_ns();
                while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
            }
        }
    } else if (warp == MMA_WARP) {
        // ---------------------------- MMA issuer ----------------------------
        // The whole warp runs the loop and waits; one elected lane issues (see sm100::elect_one).
        constexpr uint32_t idesc_g = make_idesc_bf16(TM, 128);
        constexpr uint32_t idesc_p = make_idesc_bf16(TM, 128) | (1u << 15);      // A operand MN-major
        const uint32_t wp_addr = smem_u32(smem + OFF_WP), wg_addr = smem_u32(smem + OFF_WG), xt_addr = smem_u32(smem + OFF_XT);
        if (elect_one()) {
            mbar_arrive_expect_tx(&B->w_full, 2 * W_TILE);
            load_weights_tma(smem + OFF_WP, &map_wp, 128, &B->w_full);
            load_weights_tma(smem + OFF_WG, &map_wg, 128, &B->w_full);
        }
        __syncwarp();
        uint32_t it = 0;
        bool ok = mbar_wait_warp(&B->w_full, 0, abort_flag);
        for (long long t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++it) {
            const uint32_t stage = it & 1, ph = (it >> 1) & 1;
            ok = mbar_wait_warp(&B->in_full[stage], ph, abort_flag) && mbar_wait_warp(&B->x_full[stage], ph, abort_flag) &&
                 mbar_wait_warp(&B->acc_empty[stage], ph ^ 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t az_addr = smem_u32(smem + OFF_AZ + stage * A_TILE_BYTES), xs_addr = xt_addr + stage * 2 * XT_BOX;
                const uint32_t d = tmem_base + stage * 256;
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)      // D_p = x^T-tile (MN-major, 16 d rows per step) * W_pout'^T
                    umma_bf16(d, desc_mn_sw128(xs_addr + ks * 2048), make_desc_k_sw128(wp_addr + (ks >> 2) * (128 * 128) + (ks & 3) * 32),
                              idesc_p, ks ? 1u : 0u);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)      // D_g = LN_in(z) tile * W_gout'^T
                    umma_bf16(d + 128, make_desc_k_sw128(az_addr + (ks >> 2) * A_KB_BYTES + (ks & 3) * 32),
                              make_desc_k_sw128(wg_addr + (ks >> 2) * (128 * 128) + (ks & 3) * 32), idesc_g, ks ? 1u : 0u);
                umma_commit(&B->in_empty[stage]);
                umma_commit(&B->x_empty[stage]);
                umma_commit(&B->acc_full[stage]);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else {
        // ---------------------------- epilogue ----------------------------
        const int quarter = warp & 3, chalf = (warp - EPI_WARP0) >> 2;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        uint8_t* stg = smem + OFF_STG + (warp - EPI_WARP0) * STG_BOX;
        uint32_t it = 0;
        bool ok = true;
        if (blockIdx.x < tiles) {
            // the first tile's LayerNorm, 16 rows a warp.  At 45 tokens, one tile per CTA, four loader warps in two passes each
            // took 3.7 of the kernel's 7 us.
            const int r = (int)blockIdx.x / tpl, pos0 = ((int)blockIdx.x % tpl) * TM, row0 = (warp - EPI_WARP0) * PASS_ROWS;
            float4 v[4][4], gam[4], bet[4];
            fetch16(r, pos0, row0, v);
            load_affine(gam, bet);
            normalise16(row0, v, smem + OFF_AZ, gam, bet);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->in_full[0]);
        }
        for (long long t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++it) {
            const int r = (int)(t / tpl), pos0 = (int)(t % tpl) * TM;
            const uint32_t stage = it & 1, ph = (it >> 1) & 1;
            // LayerNorm statistics over the 128 channels of the raw x tile for this quarter's 32 positions (both warps of a lane
            // quarter compute them): a lane reads two positions of every other four channels.
            ok = mbar_wait(&B->x_full[stage], ph, abort_flag);
            if (!ok) break;
            float2 st;
            {
                const int pp = lane & 15, dg = lane >> 4;         // positions 2 pp and 2 pp + 1, channels 8 i + 4 dg + 0 .. 3
                const uint8_t* col = smem + OFF_XT + stage * 2 * XT_BOX + (quarter >> 1) * XT_BOX + (pp & 3) * 4 + dg * 512;
                const int pchunk = (quarter & 1) * 4 + (pp >> 2);
                uint64_t s2[2] = {0, 0}, q2[2] = {0, 0};
#pragma unroll 4
                for (int i = 0; i < 16; ++i)
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const uint32_t w = *reinterpret_cast<const uint32_t*>(col + i * 1024 + b * 128 + ((pchunk ^ (dg * 4 + b)) << 4));
                        const uint64_t x2 = f2_pack(bf16_lo(w), bf16_hi(w));
                        s2[b & 1] = f2_add(s2[b & 1], x2);
                        q2[b & 1] = f2_fma(x2, x2, q2[b & 1]);
                    }
                const uint64_t s = f2_add(s2[0], s2[1]), q = f2_add(q2[0], q2[1]);
                float sv[2], qv[2], mean[2], rstd[2];
                f2_unpack(s, sv[0], sv[1]);
                f2_unpack(q, qv[0], qv[1]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    sv[e] += __shfl_xor_sync(0xffffffffu, sv[e], 16);
                    qv[e] += __shfl_xor_sync(0xffffffffu, qv[e], 16);
                    mean[e] = sv[e] * (1.f / KC);
                    rstd[e] = rsqrtf(fmaxf(qv[e] * (1.f / KC) - mean[e] * mean[e], 0.f) + LN_EPS);
                    mean[e] = __shfl_sync(0xffffffffu, mean[e], lane >> 1);
                    rstd[e] = __shfl_sync(0xffffffffu, rstd[e], lane >> 1);
                }
                st = (lane & 1) ? make_float2(mean[1], rstd[1]) : make_float2(mean[0], rstd[0]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->x_empty[stage]);
            ok = mbar_wait(&B->acc_full[stage], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t tbase = tmem_base + lane_off + stage * 256;
#pragma unroll 1
            for (int rd = 0; rd < 2; ++rd) {
                const int c0 = rd * 64 + chalf * 32;
                uint32_t pr[32], gr[32];
                tmem_ld_32x32(tbase + c0, pr);
                tmem_ld_32x32(tbase + 128 + c0, gr);
                tmem_ld_wait();
                float4 o[8];
                float* of = reinterpret_cast<float*>(o);
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    const float2 ws = *reinterpret_cast<const float2*>(wsum_s + c0 + e), wb = *reinterpret_cast<const float2*>(wb_s + c0 + e);
                    const float2 centred = fma2(make_float2(-st.x, -st.x), ws, make_float2(__uint_as_float(pr[e]), __uint_as_float(pr[e + 1])));
                    const float2 ph2 = fma2(make_float2(st.y, st.y), centred, wb);
                    const float2 u = fma2(ph2, make_float2(tanh_approx(__uint_as_float(gr[e])), tanh_approx(__uint_as_float(gr[e + 1]))), ph2);
                    of[e] = u.x; of[e + 1] = u.y;
                }
                if (lane == 0) bulk_wait_read0();                  // this warp's previous reduction has read the staging tile
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j) *reinterpret_cast<float4*>(stg + sw128(lane, j)) = o[j];
                fence_proxy_async();
                __syncwarp();
                if (lane == 0 && pos0 + quarter * 32 < p.n) {
                    tma_reduce_add_4d(&map_z, stg, c0, pos0 + quarter * 32, r, 0);
                    bulk_commit();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->acc_empty[stage]);
        }
        if (lane == 0) bulk_wait0();
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

}  // namespace tme
}  // namespace b200pf

using namespace b200pf;

extern "C" int b200pf_trimul_epilogue_tc(float* z, const b200pf_bf16* x, long long x_plane_stride, int x_pitch,
                                         const float* ln_in_gamma, const float* ln_in_beta,
                                         const b200pf_bf16* w_pout, const b200pf_bf16* w_gout,
                                         const float* wsum, const float* wb, int rows, int n, void* stream) {
    using namespace tme;
    B200PF_REQUIRE(z && x && ln_in_gamma && ln_in_beta && w_pout && w_gout && wsum && wb, B200PF_ERR_INVALID,
                   "trimul_epilogue_tc: null pointer");
    B200PF_REQUIRE(rows > 0 && n > 0 && x_pitch % 8 == 0 && x_pitch >= n && x_plane_stride % 8 == 0 &&
                   x_plane_stride >= (long long)x_pitch * rows, B200PF_ERR_INVALID, "trimul_epilogue_tc: bad sizes");
    B200PF_REQUIRE(aligned16(z) && aligned16(x) && aligned16(w_pout) && aligned16(w_gout) && aligned16(ln_in_gamma) &&
                   aligned16(ln_in_beta), B200PF_ERR_INVALID, "trimul_epilogue_tc: pointers must be 16-byte aligned");
    CUtensorMap mx, mz, mwp, mwg;
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK || (rc = weight_map(&mwp, w_pout, 128, "w_pout")) != B200PF_OK ||
        (rc = weight_map(&mwg, w_gout, 128, "w_gout")) != B200PF_OK) return rc;
    {
        cuuint64_t dims[4] = {(cuuint64_t)n, (cuuint64_t)rows, 128, 1};
        cuuint64_t str[3] = {(cuuint64_t)x_pitch * 2, (cuuint64_t)x_plane_stride * 2, (cuuint64_t)x_plane_stride * 2 * 128};
        cuuint32_t box[4] = {64, 1, 128, 1};
        if ((rc = tmap_encode(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "x")) != B200PF_OK) return rc;
    }
    {
        cuuint64_t dims[4] = {128, (cuuint64_t)n, (cuuint64_t)rows, 1};
        cuuint64_t str[3] = {512, (cuuint64_t)n * 512, (cuuint64_t)n * 512 * rows};
        cuuint32_t box[4] = {32, 32, 1, 1};
        if ((rc = tmap_encode(&mz, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, z, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "z")) != B200PF_OK) return rc;
    }
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "trimul_epilogue_tc: no device status word");
    B200PF_SMEM_ATTR_ONCE(trimul_epilogue_tc_kernel, SMEM_BYTES);
    long long tiles = (long long)rows * ((n + TM - 1) / TM);
    Args a{z, ln_in_gamma, ln_in_beta, wsum, wb, rows, n};
    return launch_pdl(trimul_epilogue_tc_kernel, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream,
                      mx, mz, mwp, mwg, a, status);
}
