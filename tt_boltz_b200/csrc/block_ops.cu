// A block's kernels enqueued by one call: the pair track of the bf16 tier and the single track.  Only the order of the launches
// is kept here; the work is behind the entry points of the sub-operations.  A block is some 23 launches: enqueued one by one from
// an interpreter they cost the host 7.8 us each, 180 us a block, more than a block of 45 tokens keeps the GPU busy.
#include "rowtc.cuh"

using namespace b200pf;

#define B200PF_TRY(call)                    \
    do {                                    \
        const int rc__ = (call);            \
        if (rc__ != B200PF_OK) return rc__; \
    } while (0)

static int tri_mul(float* z, const b200pf_trimul_weights& w, const b200pf_pair_scratch& k, int incoming, void* st) {
    const int n = k.n;
    const long long plane = (long long)n * k.pitch;
    const b200pf_plane_out oa{k.buf[0], plane, 0, 0}, ob{k.buf[1], plane, 0, 0};
    B200PF_TRY(b200pf_trimul_producer(z, k.mask, w.ln_in_gamma, w.ln_in_beta, w.w_pg, &oa, &ob, k.pitch, n, n, incoming, st));
    const b200pf_planes pa{k.buf[0], plane, 0, k.pitch, n, n, 1, 0}, pb{k.buf[1], plane, 0, k.pitch, n, n, 1, 0};
    B200PF_TRY(b200pf_trimul_contract(&pa, &pb, nullptr, nullptr, k.buf[2], plane, k.pitch, 0, 0, 128, 0, st));
    return b200pf_trimul_epilogue_tc(z, k.buf[2], plane, k.pitch, w.ln_in_gamma, w.ln_in_beta, w.w_pout, w.w_gout, w.wsum, w.wb, n, n, st);
}

static int tri_att(float* z, const b200pf_triatt_weights& w, const b200pf_pair_scratch& k, int ending, void* st) {
    const int n = k.n;
    const long long hs = k.pitch, qs = 4LL * k.pitch, nc = 128LL * n;        // triangle bias [query][head][key]
    B200PF_TRY(b200pf_triatt_producer(z, w.ln_gamma, w.ln_beta, w.w_bias, w.w_qkgv, k.buf[0], k.buf[1], k.buf[2], k.buf[3], k.tri_bias, hs, qs, k.pitch, n, n,
                                      ending, st));
    B200PF_TRY(b200pf_triatt_core_tc4(k.buf[0], k.buf[1], k.buf[2], k.pitch, k.tri_bias, hs, qs, ending ? k.mask_cols : k.mask_rows, k.mask_pitch, k.buf[4],
                                      ending ? 128 : nc, ending ? nc : 128, n, n, st));
    return b200pf_triatt_epilogue(z, k.buf[4], k.buf[3], w.w_o, (long long)n * n, st);
}

extern "C" int b200pf_pair_block(float* z, const b200pf_pair_weights* w, const b200pf_pair_scratch* k, void* stream) {
    B200PF_REQUIRE(z && w && k && k->mask && k->mask_rows && k->mask_cols && k->tri_bias && k->n > 0 && k->pitch >= k->n && k->pitch % 8 == 0,
                   B200PF_ERR_INVALID, "pair_block: bad argument");
    B200PF_TRY(tri_mul(z, w->tri_mul_out, *k, 0, stream));
    B200PF_TRY(tri_mul(z, w->tri_mul_in, *k, 1, stream));
    B200PF_TRY(tri_att(z, w->tri_att_start, *k, 0, stream));
    B200PF_TRY(tri_att(z, w->tri_att_end, *k, 1, stream));
    const b200pf_transition_weights& t = w->transition;
    return b200pf_transition_z_tc(z, t.ln_gamma, t.ln_beta, t.w12, t.w3, (long long)k->n * k->n, stream);
}

extern "C" long long b200pf_single_track_rows_workspace(int n, int cs, int hidden) {
    return ((long long)n * cs * 4 + 255) / 256 * 256 + b200pf_single_track_workspace(n, cs, hidden);
}

extern "C" int b200pf_single_track_rows(float* s, const b200pf_single_track_weights* w, const float* bias, const uint8_t* mask, int n, void* workspace,
                                        void* stream) {
    B200PF_REQUIRE(s && w && bias && workspace && aligned16(workspace) && n > 0, B200PF_ERR_INVALID, "single_track_rows: null or misaligned pointer");
    char* rest = static_cast<char*>(workspace) + ((long long)n * w->cs * 4 + 255) / 256 * 256;       // behind the gated output's two part planes
    B200PF_TRY(b200pf_single_track_attention(s, w, bias, mask, workspace, n, 0, n, rest, stream));
    return b200pf_single_track_finish(s, w, workspace, n, rest, stream);
}

extern "C" int b200pf_single_track_beside(float* s, const float* z, const b200pf_pair_bias_weights* wb, const b200pf_single_track_weights* w, float* bias,
                                          const uint8_t* mask, int n, void* workspace, void* pair_stream, void* side_stream, void* ready, void* done,
                                          int wait_done) {
    B200PF_REQUIRE(s && z && wb && w && bias && workspace && ready && done && n > 0, B200PF_ERR_INVALID, "single_track_beside: bad argument");
    cudaStream_t pair = (cudaStream_t)pair_stream, side = (cudaStream_t)side_stream;
    const long long nn = (long long)n * n;
    if (wait_done) B200PF_CUDA(cudaStreamWaitEvent(pair, (cudaEvent_t)done, 0));
    if (wb->cz == 128 && (wb->heads == 4 || wb->heads == 16))
        B200PF_TRY(b200pf_ln_proj_heads(z, wb->gamma, wb->beta, wb->w, bias, nn, nn, wb->cz, wb->heads, pair));
    else
        B200PF_TRY(b200pf_ln_heads(z, wb->gamma, wb->beta, wb->w, bias, nn, nn, wb->cz, wb->heads, pair));
    B200PF_CUDA(cudaEventRecord((cudaEvent_t)ready, pair));
    B200PF_CUDA(cudaStreamWaitEvent(side, (cudaEvent_t)ready, 0));
    {
        // Up to one tile of positions per line, the producers and the tri-mul epilogue of a 128-wide pair track have a CTA per line and
        // leave the other SMs idle most of the time.  The single track's GEMMs, whose CTAs take an SM each, are sized for those: spread
        // over the whole chip they hold SMs that the pair track's next kernel then waits for.  (Its LayerNorms, attention and partial sums
        // are small CTAs that fit beside others.)  Eight blocks at 128 tokens 1199 -> 1136 us, at 117 1158 -> 1151, at 90 1035 -> 1025.
        // With 12, 16 or 20 SMs it is the same at 128, with 8 the single track becomes the longer one (1161; 1168 at 117).  The GEMMs of a
        // 256-wide pair track fill the chip at any size: four of its blocks at 110 tokens lose by the limit (1604 -> 1610 us).
        constexpr int LEAST_SMS = 12;
        int sms;
        B200PF_TRY(device_multiprocessors(&sms));
        const CtaLimit limit(wb->cz == rtc::KC && n <= rtc::TM && sms - n >= LEAST_SMS ? sms - n : 0);
        B200PF_TRY(b200pf_single_track_rows(s, w, bias, mask, n, workspace, side));
    }
    B200PF_CUDA(cudaEventRecord((cudaEvent_t)done, side));
    return B200PF_OK;
}
