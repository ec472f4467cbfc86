// Triangle-attention epilogue on tcgen05:  z += (o * g) W_o^T, or the update itself as bf16, per tile of 128 positions.
//
// Loader warps multiply o and g into a bf16 A tile (K-major, 128-byte swizzle), one thread issues the products against W_o in shared
// memory, epilogue warps stage the fp32 update and reduce-add it into z by TMA (z is not read), or store it.  The staging tiles hold a whole
// update, so that one tile's reductions run under the next tile's products.
// Roles (480 threads): warps 0-5 loaders (16 rows at a time, round robin), warp 6 MMA issuer, warps 7-14 epilogue (two per TMEM lane
// quarter, 64 channels each).  A CTA's first tile is multiplied by the epilogue warps, which have nothing else to do before its accumulators
// exist; the loaders begin with the second.
// It is bound by memory: 253 us at 1024 tokens, 6.4 TB/s of its 12 E bytes (0.97 of the copy rate), where mma.sync warps with units of 32 rows
// and 8-byte red.global took 283; 39 for 52 us at 400, 13 for 24 at 300, 8.9 for 14 at 203, 5.3 for 8.9 at 117, 3.8 for 4.5 at 45.
#include "rowtc.cuh"
#include "tmap.cuh"
#include "triatt_epilogue_tc.h"

namespace b200pf {
namespace tae {

using namespace rtc;

constexpr int LOAD_WARPS = 6, MMA_WARP = 6, EPI_WARP0 = 7, EPI_WARPS = 8, THREADS = 15 * 32;
constexpr int PASS_ROWS = 16, PASSES = TM / PASS_ROWS, ST = 3, ACCS = 4;
constexpr int OFF_W = 0, OFF_A = 128 * 128 * 2;
constexpr int OFF_STG = OFF_A + ST * A_TILE_BYTES;        // per epilogue warp 2 boxes of [32 pos][32 fp32], 128-byte swizzle
constexpr int STG_BOX = 32 * 128;
constexpr int OFF_BAR = OFF_STG + EPI_WARPS * 2 * STG_BOX;
constexpr int SMEM_BYTES = OFF_BAR + 256;                 // 196,864

struct Args {
    const __nv_bfloat16 *o, *g;
    int rows, tiles, step;          // a tile's rows: 128, or with few rows 64 or 32, over more CTAs (the rest of the A tile is left as it is)
};
struct Bars {
    uint64_t w_full, a_full[ST], a_empty[ST], acc_full[ACCS], acc_empty[ACCS];
    uint32_t tmem_slot;
    int abort_flag;
};

// One warp's 16 rows: o * g, rounded to bf16, into the A tile; 16 lanes a row.  Rows past the last one are zero.
__device__ __forceinline__ void gather16(const Args& p, int row0, int row_in, uint8_t* a_tile) {
    if (row_in >= p.step) return;
    const int lane = threadIdx.x & 31, c = lane & 15, r = lane >> 4;
    uint4 ov[8], gv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int f = row0 + row_in + 2 * i + r;
        const bool in = f < p.rows;
        ov[i] = in ? reinterpret_cast<const uint4*>(p.o + (long long)f * KC)[c] : make_uint4(0u, 0u, 0u, 0u);
        gv[i] = in ? reinterpret_cast<const uint4*>(p.g + (long long)f * KC)[c] : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t a[4] = {ov[i].x, ov[i].y, ov[i].z, ov[i].w}, b[4] = {gv[i].x, gv[i].y, gv[i].z, gv[i].w};
        uint32_t d[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) d[e] = pack_bf16x2(bf16_lo(a[e]) * bf16_lo(b[e]), bf16_hi(a[e]) * bf16_hi(b[e]));
        *reinterpret_cast<uint4*>(a_tile + (c >> 3) * A_KB_BYTES + sw128(row_in + 2 * i + r, c & 7)) = make_uint4(d[0], d[1], d[2], d[3]);
    }
}

template <bool UPD>
__global__ void __launch_bounds__(THREADS, 1)
triatt_epilogue_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_out, Args p, unsigned int* status) {
    using namespace sm100;
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
        for (int i = 0; i < ST; ++i) { mbar_init(&B->a_full[i], PASSES); mbar_init(&B->a_empty[i], 1); }
        for (int i = 0; i < ACCS; ++i) { mbar_init(&B->acc_full[i], 1); mbar_init(&B->acc_empty[i], EPI_WARPS); }
        B->abort_flag = 0;
        fence_barrier_init();
    }
    if (tid == 32) { tma_prefetch_desc(&map_w); tma_prefetch_desc(&map_out); }
    if (warp == MMA_WARP) { tmem_alloc(&B->tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dependency_wait();                 // behind the CTA's barrier: every warp goes to work by itself from here on
    grid_launch_dependents();
    const uint32_t tmem_base = B->tmem_slot;

    if (warp < LOAD_WARPS) {
        // ---------------------------- loaders ----------------------------
        // Pass u is rows 16 (u % 8) of tile 1 + u / 8 of this CTA.
        bool ok = true;
        for (uint32_t u = warp; ok; u += LOAD_WARPS) {
            const uint32_t it = 1 + u / PASSES, st = it % ST;
            const int t = (int)(blockIdx.x + it * gridDim.x);
            if (t >= p.tiles) break;
            ok = mbar_wait(&B->a_empty[st], ((it / ST) & 1) ^ 1, abort_flag);
            if (!ok) break;
            gather16(p, t * p.step, (int)(u % PASSES) * PASS_ROWS, smem + OFF_A + st * A_TILE_BYTES);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->a_full[st]);
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else if (warp == MMA_WARP) {
        // ---------------------------- MMA issuer ----------------------------
        // The whole warp runs the loop and waits; one elected lane issues (see sm100::elect_one).
        constexpr uint32_t idesc = make_idesc_bf16(TM, 128);
        const uint64_t d_w = make_desc_k_sw128(smem_u32(smem + OFF_W)), d_a = make_desc_k_sw128(smem_u32(smem + OFF_A));
        if (elect_one()) {
            mbar_arrive_expect_tx(&B->w_full, 128 * 128 * 2);
            load_weights_tma(smem + OFF_W, &map_w, 128, &B->w_full);
        }
        __syncwarp();
        uint32_t it = 0;
        bool ok = mbar_wait_warp(&B->w_full, 0, abort_flag);
        for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++it) {
            const uint32_t st = it % ST, ab = it % ACCS;
            ok = mbar_wait_warp(&B->a_full[st], (it / ST) & 1, abort_flag) && mbar_wait_warp(&B->acc_empty[ab], ((it / ACCS) & 1) ^ 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t da = d_a + st * (uint64_t)(A_TILE_BYTES >> 4);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma_bf16(tmem_base + ab * 128, da + (ks >> 2) * (A_KB_BYTES >> 4) + (ks & 3) * 2, d_w + (ks >> 2) * ((128 * 128) >> 4) + (ks & 3) * 2, idesc, ks ? 1u : 0u);
                umma_commit(&B->a_empty[st]);
                umma_commit(&B->acc_full[ab]);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    } else {
        // ---------------------------- epilogue ----------------------------
        const int quarter = warp & 3, eh = (warp - EPI_WARP0) >> 2;
        uint8_t* stg = smem + OFF_STG + (warp - EPI_WARP0) * 2 * STG_BOX;
        uint32_t it = 0;
        bool ok = true;
        if ((int)blockIdx.x < p.tiles) {
            gather16(p, (int)blockIdx.x * p.step, (warp - EPI_WARP0) * PASS_ROWS, smem + OFF_A);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->a_full[0]);
        }
        for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++it) {
            const uint32_t ab = it % ACCS;
            ok = mbar_wait(&B->acc_full[ab], (it / ACCS) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            uint32_t d[2][32];
            tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + ab * 128 + eh * 64, d[0]);
            tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + ab * 128 + eh * 64 + 32, d[1]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&B->acc_empty[ab]); bulk_wait_read0(); }          // the tile before has left the staging tile
            __syncwarp();
            const int row = t * p.step + quarter * 32;
            if (UPD) {                                   // one box of [32 pos][64 bf16]
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t* e = &d[j >> 2][(j & 3) * 8];
                    uint4 v;
                    v.x = pack_bf16x2(__uint_as_float(e[0]), __uint_as_float(e[1]));
                    v.y = pack_bf16x2(__uint_as_float(e[2]), __uint_as_float(e[3]));
                    v.z = pack_bf16x2(__uint_as_float(e[4]), __uint_as_float(e[5]));
                    v.w = pack_bf16x2(__uint_as_float(e[6]), __uint_as_float(e[7]));
                    *reinterpret_cast<uint4*>(stg + sw128(lane, j)) = v;
                }
            } else {
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<uint4*>(stg + b * STG_BOX + sw128(lane, j)) = make_uint4(d[b][4 * j], d[b][4 * j + 1], d[b][4 * j + 2], d[b][4 * j + 3]);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0 && quarter * 32 < p.step && row < p.rows) {
                if (UPD) {
                    tma_store_4d(&map_out, stg, eh * 64, row, 0, 0);
                } else {
                    tma_reduce_add_4d(&map_out, stg, eh * 64, row, 0, 0);
                    tma_reduce_add_4d(&map_out, stg + STG_BOX, eh * 64 + 32, row, 0, 0);
                }
                bulk_commit();
            }
        }
        if (lane == 0) bulk_wait0();
        if (!ok && lane == 0) atomicOr(status, DEV_STATUS_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

int launch(float* z, __nv_bfloat16* upd, const __nv_bfloat16* o, const __nv_bfloat16* g, const __nv_bfloat16* w_o, int rows, int sms, cudaStream_t st) {
    unsigned int* status = device_status_word();
    B200PF_REQUIRE(status, B200PF_ERR_CUDA, "triatt_epilogue: no device status word");
    CUtensorMap mw, mo;
    int rc;
    if ((rc = weight_map(&mw, w_o, 128, "w_o")) != B200PF_OK) return rc;
    const unsigned es = z ? 4 : 2;
    cuuint64_t dims[4] = {128, (cuuint64_t)rows, 1, 1};
    cuuint64_t str[3] = {128 * es, (cuuint64_t)rows * 128 * es, (cuuint64_t)rows * 128 * es};
    cuuint32_t box[4] = {128 / es, 32, 1, 1};
    if ((rc = tmap_encode(&mo, z ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, z ? (void*)z : (void*)upd, 4, dims, str, box,
                          CU_TENSOR_MAP_SWIZZLE_128B, z ? "z" : "update")) != B200PF_OK) return rc;
    // few rows go over more CTAs: what a CTA reduces into z takes it some 2.4 clocks per 32 bytes (a tile of 128 rows 2.6 us)
    const int step = (rows + 31) / 32 <= sms ? 32 : (rows + 63) / 64 <= sms ? 64 : TM;
    const int tiles = (rows + step - 1) / step;
    const Args a{o, g, rows, tiles, step};
    const dim3 grid((unsigned)(tiles < sms ? tiles : sms));
    if (z) {
        B200PF_SMEM_ATTR_ONCE(triatt_epilogue_tc_kernel<false>, SMEM_BYTES);
        return launch_pdl(triatt_epilogue_tc_kernel<false>, grid, dim3(THREADS), SMEM_BYTES, st, mw, mo, a, status);
    }
    B200PF_SMEM_ATTR_ONCE(triatt_epilogue_tc_kernel<true>, SMEM_BYTES);
    return launch_pdl(triatt_epilogue_tc_kernel<true>, grid, dim3(THREADS), SMEM_BYTES, st, mw, mo, a, status);
}

}  // namespace tae
}  // namespace b200pf
