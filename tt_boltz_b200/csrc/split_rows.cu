// LayerNorm and conversion kernels in front of the split GEMM (split_gemm.cu): one pass over the fp32 rows, 16-bit part planes
// out.  Bound by HBM (or by launch latency for the single track's few hundred rows): a warp owns R rows at a time so that
// R rows' loads are in flight per warp, every access is a contiguous run of a row.
#include "split_rows.cuh"

namespace b200pf {
namespace split {

// Reduces V values per lane over groups of L lanes; a lane ends up with the totals of max(1, V / L) values from index
// reduced_base<V, L>(lane) on (powers of two; for V < L neighbouring lanes hold the same value).
template <int V, int L> __device__ __forceinline__ void lane_reduce(float (&v)[V], int lane) {
    int cnt = V;
#pragma unroll
    for (int bit = L / 2; bit >= 1; bit >>= 1) {
        if (cnt > 1) {
            const int half = cnt / 2;
            const bool upper = (lane & bit) != 0;
#pragma unroll
            for (int i = 0; i < V / 2; ++i)
                if (i < half) {
                    const float keep = upper ? v[i + half] : v[i], send = upper ? v[i] : v[i + half];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
                }
            cnt = half;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
        }
    }
}
template <int V, int L> __device__ __forceinline__ int reduced_base(int lane) {
    int base = 0, half = V / 2;
#pragma unroll
    for (int bit = L / 2; bit >= 1; bit >>= 1)
        if (half >= 1) { base += (lane & bit) ? half : 0; half /= 2; }
    return base;
}

// A row's channels lie over L lanes, V consecutive ones each and J times, so that a warp works on 32 / L rows at a step and on R steps' rows at
// a time.  With every row over the whole warp, ten shuffles a row and a 64-bit division per head sum bound the 64-wide rows: 10.4 -> 8.1 us
// at 292 tokens (85,264 rows), with four heads 15.0 -> 12.2; 256 wide with 16 heads, packed sums and a grid that is resident at once
// 55 -> 47 us for 65,536 rows.  256 and more channels keep four a lane: eight took 21.5 us for 19.5 there.
template <int C, int NH, int R>
__global__ void __launch_bounds__(256, NH > 0 ? 2 : 1) ln_split_kernel(LnArgs p) {
    constexpr int V = C >= 256 ? 4 : 8, L = C >= 256 ? 32 : C / V, J = C / (L * V), Q = V / 4, RW = 32 / L;
    static_assert(J * L * V == C, "width must be 64, 128, 256 or 384");
    extern __shared__ __align__(16) float head_s[];                  // [NH][J][Q][L] four channels each
    const int lane = threadIdx.x & 31, sub = lane % L, rsub = lane / L;
    grid_dependency_wait();
    grid_launch_dependents();
    const long long warp = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    if (NH > 0) {
        for (int i = threadIdx.x; i < NH * C; i += blockDim.x) {
            const int c = i % C, h = i / C, j = c / (L * V), l = c % (L * V) / V, q = c % V / 4;
            head_s[(((h * J + j) * Q + q) * L + l) * 4 + c % 4] = *(p.head_w + i);
        }
        __syncthreads();
    }
    float2 gam[J][V / 2], bet[J][V / 2];
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 0; e < V / 2; ++e) {
            const int c = (j * L + sub) * V + 2 * e;
            gam[j][e] = make_float2(*(p.gamma + c), *(p.gamma + c + 1));
            bet[j][e] = make_float2(*(p.beta + c), *(p.beta + c + 1));
        }
    for (long long base = warp * (R * RW); base < p.rows; base += nwarps * (R * RW)) {
        float2 x[R][J][V / 2];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long long mine = base + r * RW + rsub, row = mine < p.rows ? mine : p.rows - 1;
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const float4 t = *reinterpret_cast<const float4*>(p.x + row * C + (j * L + sub) * V + 4 * q);
                    x[r][j][2 * q] = make_float2(t.x, t.y);
                    x[r][j][2 * q + 1] = make_float2(t.z, t.w);
                }
        }
        float s[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float2 a = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int e = 0; e < V / 2; ++e) a = add2(a, x[r][j][e]);
            s[r] = a.x + a.y;
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float mean = s[r] * (1.f / C);
            const float2 neg = make_float2(-mean, -mean);
            float2 a = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int e = 0; e < V / 2; ++e) { x[r][j][e] = add2(x[r][j][e], neg); a = fma2(x[r][j][e], x[r][j][e], a); }
            s[r] = a.x + a.y;
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float rstd = rsqrtf(s[r] * (1.f / C) + LN_EPS);
            const float2 r2 = make_float2(rstd, rstd);
            const long long row = base + r * RW + rsub;
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int e = 0; e < V / 2; ++e) x[r][j][e] = fma2(mul2(x[r][j][e], r2), gam[j][e], bet[j][e]);
            if (p.planes && row < p.rows) {
                __half* dst = p.planes + row * C + sub * V;
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    uint32_t h[V / 2], l[V / 2];
#pragma unroll
                    for (int e = 0; e < V / 2; ++e) split_f16x2(x[r][j][e].x, x[r][j][e].y, h[e], l[e]);
                    if constexpr (V == 8) {
                        *reinterpret_cast<uint4*>(dst + j * L * V) = make_uint4(h[0], h[1], h[2], h[3]);
                        *reinterpret_cast<uint4*>(dst + p.part_stride + j * L * V) = make_uint4(l[0], l[1], l[2], l[3]);
                    } else {
                        *reinterpret_cast<uint2*>(dst + j * L * V) = make_uint2(h[0], h[1]);
                        *reinterpret_cast<uint2*>(dst + p.part_stride + j * L * V) = make_uint2(l[0], l[1]);
                    }
                }
            }
        }
        if constexpr (NH > 0) {
            constexpr int NV = R * NH;                               // a lane's partial sums, [head][step]
            float acc[NV];
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                float2 a[R];
#pragma unroll
                for (int r = 0; r < R; ++r) a[r] = make_float2(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < J; ++j)
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const float4 w = reinterpret_cast<const float4*>(head_s)[((h * J + j) * Q + q) * L + sub];
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            a[r] = fma2(x[r][j][2 * q], make_float2(w.x, w.y), a[r]);
                            a[r] = fma2(x[r][j][2 * q + 1], make_float2(w.z, w.w), a[r]);
                        }
                    }
#pragma unroll
                for (int r = 0; r < R; ++r) acc[h * R + r] = a[r].x + a[r].y;
            }
            lane_reduce<NV, L>(acc, lane);
            const int b0 = reduced_base<NV, L>(lane);
            constexpr int PER = NV >= L ? NV / L : 1, DUP = NV >= L ? 1 : L / NV;
            if (sub % DUP == 0) {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int idx = b0 + i, h = idx / R;
                    const long long row = base + idx % R * RW + rsub;
                    if (row < p.rows) {
                        long long line, pos;
                        if (p.rows <= 0x7fffffffLL) { line = (unsigned)row / (unsigned)p.n; pos = (unsigned)row - (unsigned)line * (unsigned)p.n; }
                        else { line = row / p.n; pos = row - line * p.n; }
                        p.head_out[h * p.head_stride + (p.transposed ? pos * p.head_pitch + line : line * p.head_pitch + pos)] = acc[i];
                    }
                }
            }
        }
    }
}

bool ln_supported(int c) { return c == 64 || c == 128 || c == 256 || c == 384; }

template <int C, int NH> static int ln_go(const LnArgs& a, cudaStream_t st) {
    constexpr int R = NH > 0 && C >= 256 ? 4 : 2, RW = C >= 256 ? 1 : 256 / C;
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK) return rc;
    // few rows: one warp pass per block of fewer warps, so that every SM gets some
    const int warps = a.rows >= (long long)sms * 8 * R * RW ? 8 : 2;
    const long long need = (a.rows + (long long)warps * R * RW - 1) / ((long long)warps * R * RW);
    const long long most = (long long)sms * (NH > 0 ? 2 : 8);
    return launch_pdl(ln_split_kernel<C, NH, R>, dim3((unsigned)(need < most ? need : most)), dim3(warps * 32), (size_t)NH * C * 4, st, a);
}
template <int C> static int ln_heads(const LnArgs& a, int heads, cudaStream_t st) {
    switch (heads) {
        case 0: return ln_go<C, 0>(a, st);
        case 4: return ln_go<C, 4>(a, st);
        case 8: return ln_go<C, 8>(a, st);
        case 16: return ln_go<C, 16>(a, st);
    }
    B200PF_REQUIRE(false, B200PF_ERR_UNSUPPORTED, "layernorm: 0, 4, 8 or 16 head projections (got %d)", heads);
}
int launch_ln(const LnArgs& a, int c, int heads, cudaStream_t st) {
    B200PF_REQUIRE(a.x && a.gamma && a.beta && aligned16(a.x) && (a.planes == nullptr || aligned16(a.planes)) && a.rows > 0, B200PF_ERR_INVALID,
                   "layernorm: null or misaligned pointer");
    switch (c) {
        case 64: return ln_heads<64>(a, heads, st);
        case 128: return ln_heads<128>(a, heads, st);
        case 256: return ln_heads<256>(a, heads, st);
        case 384: B200PF_REQUIRE(heads == 0, B200PF_ERR_UNSUPPORTED, "layernorm: no head projections at width 384"); return ln_go<384, 0>(a, st);
    }
    B200PF_REQUIRE(false, B200PF_ERR_UNSUPPORTED, "layernorm: width %d is not built", c);
}

// t[d][i][j] -> planes[(i, j)][d]: a block takes 32 positions of one row through shared memory ([D][33]: both the row-wise
// fill and the column-wise reads are conflict free) and its warps normalise four positions each.
template <int D>
__global__ void __launch_bounds__(256, D <= 256 ? 4 : 2) ln_channels_kernel(const float* t, long long plane_stride, int pitch, const float* gamma,
                                                          const float* beta, __half* planes, long long part_stride, int n) {
    extern __shared__ float ts[];
    constexpr int E = D / 64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    grid_dependency_wait();
    grid_launch_dependents();
    const int i = blockIdx.y, j0 = blockIdx.x * 32;
    const float* src = t + (long long)i * pitch + j0 + lane;
    const bool in = j0 + lane < n;
#pragma unroll
    for (int d0 = 0; d0 < D; d0 += 64) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = in ? *(src + (long long)(d0 + e * 8 + warp) * plane_stride) : 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) ts[(d0 + e * 8 + warp) * 33 + lane] = v[e];
    }
    __syncthreads();
    // lane: channels 2 lane + 64 e, 2 lane + 1 + 64 e
    float2 g[E], b[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int c = 2 * lane + 64 * e;
        g[e] = make_float2(*(gamma + c), *(gamma + c + 1));
        b[e] = make_float2(*(beta + c), *(beta + c + 1));
    }
    float2 x[4][E];
    float s[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float2 a = make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float* at = ts + (2 * lane + 64 * e) * 33 + warp * 4 + r;
            x[r][e] = make_float2(at[0], at[33]);
            a = add2(a, x[r][e]);
        }
        s[r] = a.x + a.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float mean = s[r] * (1.f / D);
        float2 a = make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < E; ++e) { x[r][e] = add2(x[r][e], make_float2(-mean, -mean)); a = fma2(x[r][e], x[r][e], a); }
        s[r] = a.x + a.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int j = j0 + warp * 4 + r;
        if (j >= n) break;
        const float rstd = rsqrtf(s[r] * (1.f / D) + LN_EPS);
        __half* dst = planes + ((long long)i * n + j) * D + 2 * lane;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float2 u = fma2(mul2(x[r][e], make_float2(rstd, rstd)), g[e], b[e]);
            uint32_t h, l;
            split_f16x2(u.x, u.y, h, l);
            *reinterpret_cast<uint32_t*>(dst + 64 * e) = h;
            *reinterpret_cast<uint32_t*>(dst + part_stride + 64 * e) = l;
        }
    }
}

template <int D> static int ln_channels_go(const float* t, long long plane_stride, int pitch, const float* gamma, const float* beta, __half* planes,
                                           int n, cudaStream_t st) {
    constexpr int smem = D * 33 * 4;
    B200PF_SMEM_ATTR_ONCE(ln_channels_kernel<D>, smem);
    return launch_pdl(ln_channels_kernel<D>, dim3((unsigned)((n + 31) / 32), (unsigned)n), dim3(256), smem, st, t, plane_stride, pitch, gamma, beta, planes,
                      (long long)n * n * D, n);
}
int launch_ln_channels(const float* t, long long plane_stride, int pitch, const float* gamma, const float* beta, __half* planes, int n, int d,
                       cudaStream_t st) {
    switch (d) {
        case 64: return ln_channels_go<64>(t, plane_stride, pitch, gamma, beta, planes, n, st);
        case 128: return ln_channels_go<128>(t, plane_stride, pitch, gamma, beta, planes, n, st);
        case 256: return ln_channels_go<256>(t, plane_stride, pitch, gamma, beta, planes, n, st);
        case 384: return ln_channels_go<384>(t, plane_stride, pitch, gamma, beta, planes, n, st);
    }
    B200PF_REQUIRE(false, B200PF_ERR_UNSUPPORTED, "channel layernorm: width %d is not built", d);
}

__global__ void __launch_bounds__(256) parts_kernel(const float4* x, uint2* planes, long long count4) {
    grid_dependency_wait();
    grid_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count4; i += (long long)gridDim.x * blockDim.x) {
        const float4 v = *(x + i);
        uint2 h, m, l;
        split_bf16x3(v.x, v.y, h.x, m.x, l.x);
        split_bf16x3(v.z, v.w, h.y, m.y, l.y);
        planes[i] = h; planes[count4 + i] = m; planes[2 * count4 + i] = l;
    }
}
int launch_parts(const float* x, __nv_bfloat16* planes, long long count, cudaStream_t st) {
    B200PF_REQUIRE(x && planes && aligned16(x) && aligned16(planes) && count > 0 && count % 8 == 0, B200PF_ERR_INVALID, "parts: bad arguments");
    int sms, rc;
    if ((rc = multiprocessors(&sms)) != B200PF_OK) return rc;
    const long long need = (count / 4 + 255) / 256, most = 16LL * sms;
    return launch_pdl(parts_kernel, dim3((unsigned)(need < most ? need : most)), dim3(256), 0, st, reinterpret_cast<const float4*>(x),
                      reinterpret_cast<uint2*>(planes), count / 4);
}

__global__ void __launch_bounds__(256) add_partials_kernel(float4* x, const float4* partial, int n_partial, long long count4) {
    grid_dependency_wait();
    grid_launch_dependents();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count4) return;
    float4 v = x[i];
    for (int q = 0; q < n_partial; ++q) {
        const float4 t = *(partial + q * count4 + i);
        v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
    }
    x[i] = v;
}
int launch_add_partials(float* x, const float* partial, int n_partial, long long count, cudaStream_t st) {
    B200PF_REQUIRE(x && partial && aligned16(x) && aligned16(partial) && count > 0 && count % 4 == 0, B200PF_ERR_INVALID, "add_partials: bad arguments");
    return launch_pdl(add_partials_kernel, dim3((unsigned)((count / 4 + 255) / 256)), dim3(256), 0, st, reinterpret_cast<float4*>(x),
                      reinterpret_cast<const float4*>(partial), n_partial, count / 4);
}

}  // namespace split
}  // namespace b200pf
