// The two "128 -> 512" producers on tcgen05: LayerNorm (with its affine) -> GEMMs of one tile of 128
// pair positions against 512 weight rows kept in shared memory -> thin epilogue out of TMEM.
//
// The orientation of each GEMM is chosen so that the epilogue thread already holds the values
// in the order they are stored, and nothing is transposed through shared memory:
//   MODE_TRIMUL : D[channel][position] = W x^T for the four groups p_a, g_a, p_b, g_b (M = 128
//                 channels, N = 128 positions): thread = channel, 32 consecutive positions per
//                 tcgen05.ld = 64 contiguous bytes of a plane row.  u = p*sigmoid(g) costs one
//                 MUFU and one FMA per element: the host halves W_p and W_g, so with
//                 p' = p/2, t = tanh(g/2):  p*sigmoid(g) = p' + p'*t.  Masked / out-of-range
//                 positions are zero rows of x, which makes p' (and u) exactly zero.
//   MODE_TRIATT : D[position][q|k] = x W^T and D[position][g] = x W_g^T (thread = position:
//                 64-byte head rows and z-layout gate rows), D[v-channel][position] = W_v x^T
//                 (thread = channel: rows of the transposed V).  The 4 triangle-bias heads are
//                 dotted by the epilogue warps (fp32 weights and accumulation) from the normalised
//                 bf16 rows of the A tile: on the loader warps, one per scheduler, the same work
//                 doubled the time of the whole kernel.
// Output goes TMEM -> registers -> a swizzled staging tile -> TMA stores, so that global memory
// only ever sees full, contiguous lines (thread-per-row 16-byte stores were 3x slower).  Every epilogue
// warp has a staging tile and stores of its own: no warp waits for another.
// Roles (480 threads): warps 0-5 LayerNorm loaders (16 rows at a time, round robin), warp 6 MMA issuer, warps 7-14
// epilogue (two warps per TMEM lane quarter, each taking half of the columns).  TMEM is used as
// two halves of 256 columns so the epilogue of one half overlaps the MMAs of the next, and the x
// tile is double buffered so the loaders run a tile ahead.  A CTA's first tile is normalised by the
// epilogue warps, 16 rows each, which have nothing else to do before its accumulators exist; the
// loaders begin with the second.
// The loaders bound it: a pass is one long chain (loads, two reductions, stores) with nothing to interleave, and four warps took
// some 9 k clocks for a tile.  Up to 16 warps cost no registers (four per scheduler, 128 a thread, as with 13).  Six loaders against
// four with 32 rows each: 269 / 290 -> 232 / 247 us (multiplication, outgoing / incoming) and 352 / 356 -> 326 / 330 (attention, rows /
// columns) at 1024 tokens, 47.8 -> 43.4 and 61.3 -> 60.2 at 400, the same at 203, where a CTA has three tiles; five are slower
// everywhere (252 / 273 and 334 / 333), seven no faster (238 / 251 and 324 / 334) and spill in the MXFP8 form.
// A pass's arithmetic goes two channels to an instruction: 43.7 / 46.4 -> 42.1 / 44.9 and 61.3 / 61.0 -> 58.8 / 59.2 at 400, the attention
// producer 347 / 360 -> 329 / 328 at 1024; the gates alike.
#include "mxfp8.cuh"
#include "row512_tc.h"
#include "rowtc.cuh"
#include "tmap.cuh"

namespace b200pf {
namespace r512 {

using namespace rtc;

constexpr int MODE_TRIMUL = 0, MODE_TRIATT = 1, MODE_TRIMUL_MX = 2;   // MX: e4m3 planes + e8m0 scales (mxfp8.cuh)
constexpr int LOAD_WARPS = 6, MMA_WARP = 6, EPI_WARP0 = 7, EPI_WARPS = 8, THREADS = 15 * 32;
constexpr int PASS_ROWS = 16, PASSES = TM / PASS_ROWS;  // a loader warp's unit of work
constexpr int W_BYTES = 512 * 128 * 2;                 // two k-blocks of [512][128 B]
constexpr int W_KB = 512 * 128;
constexpr int OFF_A = W_BYTES;                          // 2 stages x 32 KB
constexpr int OFF_STG = OFF_A + 2 * A_TILE_BYTES;       // output staging: per epilogue warp [32 rows][128 B], 128-byte swizzle
constexpr int STG_BOX = 32 * 128;
constexpr int OFF_WB = OFF_STG + EPI_WARPS * STG_BOX;           // triangle-bias rows [4][128] fp32
constexpr int OFF_BAR = OFF_WB + 4 * 128 * 4;
constexpr int SMEM_BYTES = OFF_BAR + 128;               // 231,552: the dynamic window must start 1024-byte aligned
constexpr int EPI_BAR_ID = 1;

struct Bars {
    uint64_t a_full[2], a_empty[2], acc_full[2], acc_empty[2], w_full;
    uint32_t tmem_slot;
    int abort_flag;
};

// D[tmem] = A (M = 128 rows) * B^T over K = 128: two k-blocks of 64, each four K = 16 steps.  Operands are given as
// ready descriptors of their first k-block (address field in 16-byte units) plus the k-block distance in the same
// units: the issuing thread must not spend longer per instruction than the ~64 cycles it occupies the tensor pipe.
__device__ __forceinline__ void gemm_k128(uint32_t tmem_d, uint64_t da, uint32_t a_kb16, uint64_t db, uint32_t b_kb16, uint32_t idesc) {
    using namespace sm100;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
        const uint32_t kb = ks >> 2, kk = ks & 3;
        umma_bf16(tmem_d, da + kb * a_kb16 + kk * 2, db + kb * b_kb16 + kk * 2, idesc, ks ? 1u : 0u);
    }
}

__device__ __forceinline__ float tanh_approx(float x) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
    return t;
}

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
row512_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1,
              const __grid_constant__ CUtensorMap map2, const __grid_constant__ CUtensorMap map3,
              const __grid_constant__ CUtensorMap map_w, Args p, unsigned int* status) {
    using namespace sm100;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {       // swizzled tiles need 1024-byte alignment; there is no slack to fix it up
        grid_dependency_wait();
        if (threadIdx.x == 0) atomicOr(status, DEV_STATUS_BAD_INDEX);
        return;
    }
    Bars* B = reinterpret_cast<Bars*>(smem + OFF_BAR);
    volatile int* abort_flag = &B->abort_flag;
    float* wb_s = reinterpret_cast<float*>(smem + OFF_WB);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;

    const int span = p.transposed ? p.rows : p.n;                 // positions along a line
    const int n_lines = p.transposed ? p.n : p.rows;
    const int tpl = (span + TM - 1) / TM;
    const int tiles = n_lines * tpl;                              // below 2^31: a row is at least 256 bytes of memory

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->a_full[i], PASSES); mbar_init(&B->a_empty[i], MODE == MODE_TRIATT ? 1 + EPI_WARPS : 1);
            mbar_init(&B->acc_full[i], 1); mbar_init(&B->acc_empty[i], EPI_WARPS);
        }
        mbar_init(&B->w_full, 1);
        B->abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    // Fetched by warp 1, the multiplication's producers spill in their loaders (at 1024 tokens outgoing 257 us for 242, incoming 326 for 289);
    // by the MMA warp, the attention's does (18.4 us for 17.8 at 203).
    if (MODE == MODE_TRIATT ? tid == 32 : warp == MMA_WARP && elect_one()) {
        tma_prefetch_desc(&map_w); tma_prefetch_desc(&map0); tma_prefetch_desc(&map1);
        if (MODE == MODE_TRIATT) { tma_prefetch_desc(&map2); tma_prefetch_desc(&map3); }
    }
    if (warp == MMA_WARP) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dependency_wait();                 // behind the CTA's barrier: every warp goes to work by itself from here on
    const uint32_t tmem_base = B->tmem_slot;

    auto flat_of = [&](int line, int pos) -> long long {   // flat (r * n + c) index, or -1 outside
        if (pos >= span) return -1;
        return p.transposed ? (long long)pos * p.n + line : (long long)line * p.n + pos;
    };

    // Mask byte of row `row` of tile `t`, 0 where there is none.  The bf16 multiplication's loaders ask for it a tile ahead, a lane per row:
    // eight lanes asking with the row itself, in a column each on a line of its own, took 293 us for 278 incoming at 1024 tokens.  The MXFP8
    // producer is slower that way (279 us for 260) and asks with the row.
    auto mask_of = [&](int t, int row) -> uint32_t {
        const int line = t / tpl;
        const long long f = t < tiles ? flat_of(line, (t - line * tpl) * TM + row) : -1;
        return f >= 0 ? p.mask[f] : 0u;
    };
    // One warp's 16 rows of a tile: LayerNorm of positions pos0 + row0 .. of line `line` into the A tile; 8 lanes per row.
    const int sub = lane & 7, rq = lane >> 3;
    auto normalise16 = [&](int line, int pos0, int row0, auto kept_bits, uint8_t* a_tile, const float4 (&gam)[4], const float4 (&bet)[4]) {
        float4 v[4][4];
        // rows 4 i of the pass: one flat index and a stride (positions of a column lie n rows apart)
        const int pos_b = pos0 + row0 + rq;
        const long long f0 = p.transposed ? (long long)pos_b * p.n + line : (long long)line * p.n + pos_b;
        const long long fstep = p.transposed ? 4LL * p.n : 4LL;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool valid = pos_b + i * 4 < span;
            if (MODE != MODE_TRIMUL && p.z_bf16) {          // warp-uniform: four bf16 channels per lane and j, widened on the fly
                const uint2* src = reinterpret_cast<const uint2*>(p.z_bf16 + (f0 + i * fstep) * KC) + sub;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint2 w = valid ? src[j * 8] : make_uint2(0u, 0u);
                    v[i][j] = make_float4(bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y));
                }
            } else {
                const float4* src = reinterpret_cast<const float4*>(p.z + (f0 + i * fstep) * KC) + sub;
#pragma unroll
                for (int j = 0; j < 4; ++j) v[i][j] = valid ? src[j * 8] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        // The four rows of a pass are worked on stage by stage (all sums, then all shuffles, ...), not row by
        // row: one loader warp per scheduler has nothing else to hide a dependent chain behind.
        const uint32_t kept = kept_bits();       // asked for behind the rows' loads: nothing waits for a mask ahead of them
        float kz[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            bool keep = pos_b + i * 4 < span;
            if (MODE == MODE_TRIMUL) keep = (kept >> (i * 4 + rq)) & 1u;
            if (MODE == MODE_TRIMUL_MX) keep = keep && p.mask[f0 + i * fstep] != 0;
            kz[i] = keep ? 1.f : 0.f;
        }
        float s4[4];
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
        float ss4[4];
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
                const float4 y = affine4(v[i][j], make_float2(rstd, rstd), gam[j], bet[j]);
                const float2 k2 = make_float2(kz[i], kz[i]), a = mul2(low2(y), k2), b = mul2(high2(y), k2);
                uint2 o;
                o.x = pack_bf16x2(a.x, a.y);
                o.y = pack_bf16x2(b.x, b.y);
                const int chunk = (j & 1) * 4 + (sub >> 1);
                *reinterpret_cast<uint2*>(a_tile + (j >> 1) * A_KB_BYTES + sw128(row, chunk) + (sub & 1) * 8) = o;
            }
        }
    };
    auto load_affine = [&](float4 (&gam)[4], float4 (&bet)[4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            gam[j] = reinterpret_cast<const float4*>(p.ln_gamma)[j * 8 + sub];
            bet[j] = reinterpret_cast<const float4*>(p.ln_beta)[j * 8 + sub];
        }
    };

    if (warp < LOAD_WARPS) {
        // ---------------------------- LayerNorm loaders ----------------------------
        float4 gam[4], bet[4];
        load_affine(gam, bet);
        // Passes of 16 rows go round robin over the loader warps: pass u is rows 16 (u % 8) of tile 1 + u / 8 of this CTA
        // (the epilogue warps normalise its first).
        auto tile_of = [&](uint32_t u) { return (int)(blockIdx.x + (1 + u / PASSES) * gridDim.x); };
        uint32_t mine = 0;                  // mask of this lane's row of the next pass
        if (MODE == MODE_TRIMUL) mine = mask_of(tile_of(warp), (warp % PASSES) * PASS_ROWS + (lane & 15));
        bool ok = true;
        for (uint32_t u = warp; ok; u += LOAD_WARPS) {
            const int t = tile_of(u);
            if (t >= tiles) break;
            const int line = t / tpl, pos0 = (t - line * tpl) * TM;
            const uint32_t it = 1 + u / PASSES, stage = it & 1, ph = (it >> 1) & 1;
            const int row0 = (int)(u % PASSES) * PASS_ROWS;
            ok = mbar_wait(&B->a_empty[stage], ph ^ 1, abort_flag);
            if (!ok) break;
            uint8_t* a_tile = smem + OFF_A + stage * A_TILE_BYTES;
            const uint32_t kept = MODE != MODE_TRIMUL ? 0u : __ballot_sync(0xffffffffu, mine != 0);
            if (MODE == MODE_TRIMUL) mine = 0;
            // this warp's NEXT 16 rows: two lanes per row ask L2 for its 128-byte lines, so the loads of the next pass find
            // them there instead of paying the DRAM latency
            {
                const int tn = tile_of(u + LOAD_WARPS), ln = tn / tpl;
                if (tn < tiles) {
                    const long long f = flat_of(ln, (tn - ln * tpl) * TM + (int)((u + LOAD_WARPS) % PASSES) * PASS_ROWS + (lane & 15));
                    if (f >= 0) {
                        if (MODE == MODE_TRIMUL) mine = p.mask[f];
                        if (MODE != MODE_TRIMUL && p.z_bf16) {
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p.z_bf16 + f * KC) + (lane >> 4) * 128));
                        } else {
                            const char* rowp = reinterpret_cast<const char*>(p.z + f * KC) + (lane >> 4) * 256;
#pragma unroll
                            for (int j = 0; j < 2; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(rowp + j * 128));
                        }
                    }
                }
            }
            normalise16(line, pos0, row0, [&] { return kept; }, a_tile, gam, bet);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->a_full[stage]);
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else if (warp == MMA_WARP) {
        // ---------------------------- MMA issuer ----------------------------
        // The whole warp runs the loop and waits; one elected lane issues (see sm100::elect_one).
        constexpr uint32_t idesc128 = make_idesc_bf16(TM, 128), idesc256 = make_idesc_bf16(TM, 256);
        const uint64_t d_w = make_desc_k_sw128(smem_u32(smem));            // weight row r starts 8 r units further
        const uint64_t d_x0 = make_desc_k_sw128(smem_u32(smem + OFF_A));
        constexpr uint32_t W_KB16 = W_KB >> 4, A_KB16 = A_KB_BYTES >> 4;
        if (elect_one()) {
            mbar_arrive_expect_tx(&B->w_full, W_BYTES);
            load_weights_tma(smem, &map_w, 512, &B->w_full);
        }
        __syncwarp();
        uint32_t it = 0, acc_cnt[2] = {0, 0};
        bool ok = mbar_wait_warp(&B->w_full, 0, abort_flag);
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++it) {
            const uint32_t stage = it & 1, ph = (it >> 1) & 1;
            ok = mbar_wait_warp(&B->a_full[stage], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint64_t d_x = d_x0 + stage * (uint64_t)(A_TILE_BYTES >> 4);
            for (int half = 0; half < 2 && ok; ++half) {
                ok = mbar_wait_warp(&B->acc_empty[half], (acc_cnt[half] & 1) ^ 1, abort_flag);
                if (!ok) break;
                ++acc_cnt[half];
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t d = tmem_base + half * 256;
                    if (MODE != MODE_TRIATT) {
                        // channels on the lanes: A = 128 weight rows, B = the x tile (positions)
                        gemm_k128(d, d_w + (half * 256) * 8, W_KB16, d_x, A_KB16, idesc128);
                        gemm_k128(d + 128, d_w + (half * 256 + 128) * 8, W_KB16, d_x, A_KB16, idesc128);
                    } else if (half == 0) {
                        gemm_k128(d, d_x, A_KB16, d_w, W_KB16, idesc256);                          // [q | k]
                    } else {
                        gemm_k128(d, d_x, A_KB16, d_w + 256 * 8, W_KB16, idesc128);                // g
                        gemm_k128(d + 128, d_w + 384 * 8, W_KB16, d_x, A_KB16, idesc128);          // v^T
                    }
                    umma_commit(&B->acc_full[half]);
                    if (half == 1) umma_commit(&B->a_empty[stage]);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else {
        // ---------------------------- epilogue ----------------------------
        // Each round moves one [128 x 128] bf16 block out: TMEM -> registers -> swizzled staging tile
        // -> a TMA store of [32 rows x 64 elements] per warp, so global memory only sees full lines.
        const int quarter = warp & 3, chalf = (warp - EPI_WARP0) >> 2;
        if ((int)blockIdx.x < tiles) {
            // the first tile's LayerNorm, 16 rows a warp.  At 45 tokens, one tile per CTA, four loader warps in two passes each
            // took 3.6 of the kernel's 9 us.
            if (MODE == MODE_TRIATT)
                for (int i = (int)threadIdx.x - EPI_WARP0 * 32; i < 4 * 128; i += EPI_WARPS * 32) wb_s[i] = p.w_bias_f32[i];
            float4 gam[4], bet[4];
            load_affine(gam, bet);
            const int line = (int)blockIdx.x / tpl;
            const int row0 = (warp - EPI_WARP0) * 16;
            const uint32_t mine = MODE != MODE_TRIMUL ? 0u : mask_of((int)blockIdx.x, row0 + (lane & 15));
            normalise16(line, ((int)blockIdx.x - line * tpl) * TM, row0, [&] { return MODE != MODE_TRIMUL ? 0u : __ballot_sync(0xffffffffu, mine != 0); },
                        smem + OFF_A, gam, bet);
            fence_proxy_async();
            if (MODE == MODE_TRIATT) named_bar_sync(EPI_BAR_ID, EPI_WARPS * 32);              // wb_s is there
            else __syncwarp();
            if (lane == 0) mbar_arrive(&B->a_full[0]);
        }
        const int lrow = quarter * 32 + lane;                     // TMEM lane of this thread = staging row
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        uint8_t* stg = smem + OFF_STG + (warp - EPI_WARP0) * STG_BOX;
        uint32_t acc_cnt = 0;
        bool ok = true;
        // tanh_mode: 0 = copy, 1 = p' + p' * tanh(g')  (gate columns at +128), 2 = 0.5 + 0.5 * tanh(x)
        auto load64 = [&](uint32_t taddr, int tanh_mode, uint4 (&o)[8]) {
            uint32_t r[2][32];
            tmem_ld_32x32(taddr, r[0]);
            tmem_ld_32x32(taddr + 32, r[1]);
            uint32_t gq[2][32];
            if (tanh_mode == 1) {
                tmem_ld_32x32(taddr + 128, gq[0]);
                tmem_ld_32x32(taddr + 160, gq[1]);
            }
            tmem_ld_wait();
            uint32_t* w = reinterpret_cast<uint32_t*>(o);
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                float2 v = make_float2(__uint_as_float(r[e >> 4][(2 * e) & 31]), __uint_as_float(r[e >> 4][(2 * e + 1) & 31]));
                if (tanh_mode == 1) {
                    const uint32_t* g = &gq[e >> 4][(2 * e) & 31];
                    v = fma2(v, make_float2(tanh_approx(__uint_as_float(g[0])), tanh_approx(__uint_as_float(g[1]))), v);
                } else if (tanh_mode == 2) {
                    v = fma2(make_float2(0.5f, 0.5f), make_float2(tanh_approx(v.x), tanh_approx(v.y)), make_float2(0.5f, 0.5f));
                }
                w[e] = pack_bf16x2(v.x, v.y);
            }
        };
        // This warp's 32 staging rows x 128 bytes; `inside`: the box is not wholly beyond the tensor's edge.
        auto store_round = [&](const uint4 (&o)[8], const CUtensorMap* map, bool inside, int c0, int c1, int c2, int c3) {
            if (lane == 0) bulk_wait_read0();                  // this warp's previous store has read the staging tile
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(stg + sw128(lane, j)) = o[j];
            fence_proxy_async();
            __syncwarp();
            if (lane == 0 && inside) {
                tma_store_4d(map, stg, c0, c1, c2, c3);
                bulk_commit();
            }
        };
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++acc_cnt) {
            // The next kernel's CTAs may come with this one's last tile and not before: they would hold the idle SMs that the single track,
            // beside, finds its slots on (eight confidence blocks at 45 tokens 911 -> 894 us, trunk blocks at 400 7860 -> 7802).
            if (t + (int)gridDim.x >= tiles) grid_launch_dependents();
            const int line = t / tpl, pos0 = (t - line * tpl) * TM, pos_w = pos0 + quarter * 32;
            for (int half = 0; half < 2 && ok; ++half) {
                ok = mbar_wait(&B->acc_full[half], acc_cnt & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint32_t tbase = tmem_base + lane_off + half * 256;
                uint4 o[8];
                if (MODE == MODE_TRIMUL_MX) {
                    // lane = channel of operand `half`; this warp's 64 positions are two scale blocks
                    uint32_t sc = 0;
#pragma unroll
                    for (int blk = 0; blk < 2; ++blk) {
                        uint32_t pr[32], gr[32];
                        tmem_ld_32x32(tbase + chalf * 64 + blk * 32, pr);
                        tmem_ld_32x32(tbase + 128 + chalf * 64 + blk * 32, gr);
                        tmem_ld_wait();
                        float amax = 0.f;
#pragma unroll
                        for (int e = 0; e < 32; ++e) {
                            const float pv = __uint_as_float(pr[e]);
                            const float u = fmaf(pv, tanh_approx(__uint_as_float(gr[e])), pv);
                            pr[e] = __float_as_uint(u);
                            amax = fmaxf(amax, fabsf(u));
                        }
                        const uint32_t eb = mx::scale_byte(amax);
                        const float inv = mx::inv_scale(eb);
                        sc |= eb << (8 * blk);
                        uint32_t* w = reinterpret_cast<uint32_t*>(&o[blk * 2]);
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            w[e] = mx::pack_e4m3x4(__uint_as_float(pr[4 * e]) * inv, __uint_as_float(pr[4 * e + 1]) * inv,
                                                   __uint_as_float(pr[4 * e + 2]) * inv, __uint_as_float(pr[4 * e + 3]) * inv);
                    }
                    *reinterpret_cast<uint16_t*>(p.scales[half] + mx::scale_offset(lrow, line, (pos0 >> 5) + chalf * 2,
                                                                                   p.sf_kgroups, p.sf_row_blocks)) = (uint16_t)sc;
                    if (lane == 0) bulk_wait_read0();
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 4; ++j)               // 64-byte rows, 64-byte swizzle
                        *reinterpret_cast<uint4*>(stg + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = o[j];
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0 && pos0 + chalf * 64 < p.pitch) {
                        tma_store_4d(half == 0 ? &map0 : &map1, stg, pos0 + chalf * 64, line, quarter * 32, 0);
                        bulk_commit();
                    }
                } else if (MODE == MODE_TRIMUL) {
                    // lane = channel of operand `half`, columns = positions; this warp's 64 positions = box `chalf`
                    load64(tbase + chalf * 64, 1, o);
                    const int rg = p.row_group[half];
                    const int c0 = pos0 + chalf * 64;
                    store_round(o, half == 0 ? &map0 : &map1, c0 < p.pitch, c0, line % rg, quarter * 32, line / rg);
                } else if (half == 0) {
                    {   // The 4 triangle-bias heads of this tile, from the normalised bf16 rows still in the A tile (the
                        // accumulator being ready means the loaders' writes are visible): thread = position `lrow`,
                        // this warp's two heads 2 chalf, 2 chalf + 1; fp32 weights, fp32 accumulation.
                        const uint32_t stage = acc_cnt & 1;
                        const uint8_t* a_row = smem + OFF_A + stage * A_TILE_BYTES + lrow * 128;
                        const float* w0 = wb_s + (2 * chalf) * 128;
                        float b0 = 0.f, b1 = 0.f;
#pragma unroll
                        for (int kb = 0; kb < 2; ++kb)
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                const uint4 xv = *reinterpret_cast<const uint4*>(a_row + kb * A_KB_BYTES + ((c ^ (lrow & 7)) << 4));
                                const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                                for (int q = 0; q < 2; ++q) {
                                    const float4 wa = *reinterpret_cast<const float4*>(w0 + kb * 64 + c * 8 + q * 4);
                                    const float4 wc = *reinterpret_cast<const float4*>(w0 + 128 + kb * 64 + c * 8 + q * 4);
                                    const float x0 = __uint_as_float(xw[2 * q] << 16), x1 = __uint_as_float(xw[2 * q] & 0xffff0000u);
                                    const float x2 = __uint_as_float(xw[2 * q + 1] << 16), x3 = __uint_as_float(xw[2 * q + 1] & 0xffff0000u);
                                    b0 = fmaf(x0, wa.x, fmaf(x1, wa.y, fmaf(x2, wa.z, fmaf(x3, wa.w, b0))));
                                    b1 = fmaf(x0, wc.x, fmaf(x1, wc.y, fmaf(x2, wc.z, fmaf(x3, wc.w, b1))));
                                }
                            }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&B->a_empty[stage]);          // the A tile may be overwritten
                        if (pos0 + lrow < span) {
                            __nv_bfloat16* bp = p.tri_bias + (long long)line * p.bias_qs + pos0 + lrow;
                            bp[(2 * chalf) * p.bias_hs] = __float2bfloat16(b0);
                            bp[(2 * chalf + 1) * p.bias_hs] = __float2bfloat16(b1);
                        }
                    }
                    // lane = position, columns = channels of q then k; box `chalf` = channels 64*chalf ..
                    load64(tbase + chalf * 64, 0, o);
                    store_round(o, &map0, pos_w < span, chalf * 64, pos_w, line, 0);
                    load64(tbase + 128 + chalf * 64, 0, o);
                    store_round(o, &map1, pos_w < span, chalf * 64, pos_w, line, 0);
                } else {
                    load64(tbase + chalf * 64, 2, o);                       // gate: sigmoid
                    if (p.transposed) store_round(o, &map2, pos_w < span, chalf * 64, line, pos_w, 0);
                    else store_round(o, &map2, pos_w < span, chalf * 64, pos_w, line, 0);
                    load64(tbase + 128 + chalf * 64, 0, o);                 // v^T: lane = v channel, columns = positions
                    store_round(o, &map3, pos0 + chalf * 64 < p.vt_pitch, pos0 + chalf * 64, quarter * 32, line, 0);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&B->acc_empty[half]);
            }
        }
        if (lane == 0) bulk_wait0();
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

static int make_maps(int mode, const Args& a, CUtensorMap (&m)[4]) {
    const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int span = a.transposed ? a.rows : a.n, lines = a.transposed ? a.n : a.rows;
    int rc;
    if (mode == MODE_TRIMUL_MX) {
        for (int i = 0; i < 2; ++i) {     // byte planes [d][line][pitch]
            cuuint64_t dims[4] = {(cuuint64_t)a.pitch, (cuuint64_t)lines, 128, 1};
            cuuint64_t str[3] = {(cuuint64_t)a.pitch, (cuuint64_t)a.plane_stride[i], (cuuint64_t)a.plane_stride[i] * 128};
            cuuint32_t box[4] = {64, 1, 32, 1};
            if ((rc = tmap_encode(&m[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, a.planes[i], 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_64B,
                                  "mx planes")) != B200PF_OK) return rc;
        }
        m[2] = m[0];
        m[3] = m[0];
        return B200PF_OK;
    }
    if (mode == MODE_TRIMUL) {
        for (int i = 0; i < 2; ++i) {
            const int rg = a.row_group[i], groups = (lines + rg - 1) / rg;
            cuuint64_t dims[4] = {(cuuint64_t)a.pitch, (cuuint64_t)(rg < lines ? rg : lines), 128, (cuuint64_t)groups};
            cuuint64_t str[3] = {(cuuint64_t)a.pitch * 2, (cuuint64_t)a.plane_stride[i] * 2,
                                 (cuuint64_t)(groups > 1 ? a.group_stride[i] : a.plane_stride[i] * 128) * 2};
            cuuint32_t box[4] = {64, 1, 32, 1};
            if ((rc = tmap_encode(&m[i], bf, a.planes[i], 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "planes")) != B200PF_OK) return rc;
        }
        m[2] = m[0];
        m[3] = m[0];
        return B200PF_OK;
    }
    {   // q, k: [line][pos][128]
        cuuint64_t dims[4] = {128, (cuuint64_t)span, (cuuint64_t)lines, 1};
        cuuint64_t str[3] = {256, (cuuint64_t)span * 256, (cuuint64_t)span * 256 * lines};
        cuuint32_t box[4] = {64, 32, 1, 1};
        if ((rc = tmap_encode(&m[0], bf, a.q, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "q")) != B200PF_OK) return rc;
        if ((rc = tmap_encode(&m[1], bf, a.k, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "k")) != B200PF_OK) return rc;
    }
    {   // g in the layout of the z view [rows][n][128]
        cuuint64_t dims[4] = {128, (cuuint64_t)a.n, (cuuint64_t)a.rows, 1};
        cuuint64_t str[3] = {256, (cuuint64_t)a.n * 256, (cuuint64_t)a.n * 256 * a.rows};
        cuuint32_t box_rows[4] = {64, 32, 1, 1}, box_cols[4] = {64, 1, 32, 1};
        if ((rc = tmap_encode(&m[2], bf, a.g, 4, dims, str, a.transposed ? box_cols : box_rows, CU_TENSOR_MAP_SWIZZLE_128B, "g")) != B200PF_OK) return rc;
    }
    {   // v transposed: [line][head*32 + d][vt_pitch]
        cuuint64_t dims[4] = {(cuuint64_t)a.vt_pitch, 128, (cuuint64_t)lines, 1};
        cuuint64_t str[3] = {(cuuint64_t)a.vt_pitch * 2, (cuuint64_t)a.vt_pitch * 256, (cuuint64_t)a.vt_pitch * 256 * lines};
        cuuint32_t box[4] = {64, 32, 1, 1};
        if ((rc = tmap_encode(&m[3], bf, a.v, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, "vt")) != B200PF_OK) return rc;
    }
    return B200PF_OK;
}

template <int MODE>
static int launch(const Args& a, cudaStream_t st) {
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "row512: no device status word");
    B200PF_REQUIRE(a.ln_gamma && a.ln_beta && aligned16(a.ln_gamma) && aligned16(a.ln_beta), B200PF_ERR_INVALID,
                   "row512: LayerNorm gain / offset must be given and 16-byte aligned");
    B200PF_SMEM_ATTR_ONCE(row512_kernel<MODE>, SMEM_BYTES);
    int span = a.transposed ? a.rows : a.n, lines = a.transposed ? a.n : a.rows;
    long long tiles = (long long)lines * ((span + TM - 1) / TM);
    CUtensorMap m[4], m_w;
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK || (rc = make_maps(MODE, a, m)) != B200PF_OK || (rc = weight_map(&m_w, a.w, 512, "w")) != B200PF_OK) return rc;
    return launch_pdl(row512_kernel<MODE>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(THREADS), SMEM_BYTES, st, m[0], m[1], m[2], m[3], m_w, a, status);
}

int launch_trimul(const Args& a, cudaStream_t st) { return launch<MODE_TRIMUL>(a, st); }
int launch_trimul_mx(const Args& a, cudaStream_t st) { return launch<MODE_TRIMUL_MX>(a, st); }
int launch_triatt(const Args& a, cudaStream_t st) { return launch<MODE_TRIATT>(a, st); }

}  // namespace r512
}  // namespace b200pf
