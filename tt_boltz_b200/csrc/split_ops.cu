// The sub-operations of the fp32-accurate path as single calls: LayerNorm to part planes, GEMMs with their epilogues
// (split_gemm.cu), attention (split_attn.cu).  The single track of every tier and the pair track of the fp32 tier run here.
#include "split_attn.cuh"
#include "split_rows.cuh"

namespace b200pf {
namespace split {

struct Arena {          // carves a caller's workspace; with a null base it only counts
    char* base;
    long long used = 0;
    explicit Arena(void* p) : base(static_cast<char*>(p)) {}
    template <class T> T* take(long long count) {
        char* at = base ? base + used : nullptr;
        used += (count * (long long)sizeof(T) + 255) / 256 * 256;
        return reinterpret_cast<T*>(at);
    }
};

static Operand matrix(const void* p, long long rows, int cols) {
    return Operand{p, (int)rows, cols, 1, cols, 0, rows * cols};
}
static Output dense(void* p, long long rows, int cols, int parts) {
    return Output{p, (int)rows, cols, 1, parts, cols, 0, rows * cols, false};
}
static int round_up(int x, int m) { return (x + m - 1) / m * m; }

// How many K splits a GEMM of few rows takes: enough CTAs to use the chip's bandwidth for its weights, at least three
// k-blocks each, never more than eight partial sums for the reader to add.
static int k_splits_for(int rows, int n, int k, int sms) {
    const int kb = (k + 63) / 64;
    const int tiles = ((rows + 127) / 128) * ((n + 31) / 32);
    int want = sms / (tiles > 0 ? tiles : 1);
    if (want > 8) want = 8;
    if (want > kb / 3) want = kb / 3;
    if (want < 2) return 1;
    const int per = (kb + want - 1) / want;
    return (kb + per - 1) / per;
}

// y[rows][n] (fp32) += planes[rows][k] w[n][k]^T; few rows: K-split partial sums, added in a fixed order
static int residual_gemm(float* y, const void* planes, const b200pf_split_weight& w, long long rows, int k, int n, float* partial, cudaStream_t st) {
    Gemm g;
    g.a[0] = matrix(planes, rows, k);
    g.b[0] = matrix(w.w, n, k);
    g.m_rows = (int)rows; g.n_rows = n; g.k[0] = k; g.alpha[0] = w.alpha;
    int sms, rc = device_multiprocessors(&sms);       // not the launch's share: the sums' order must not depend on it
    if (rc != B200PF_OK) return rc;
    const int ks = partial ? k_splits_for((int)rows, n, k, sms) : 1;
    if (ks == 1) {
        g.epi = EPI_ADD;
        g.out[0] = dense(y, rows, n, 1);
        return launch_gemm(g, st);
    }
    g.epi = EPI_STORE;
    g.k_splits = ks;
    g.out[0] = Output{partial, (int)rows, n, ks, 1, n, rows * n, 0, false};
    if ((rc = launch_gemm(g, st)) != B200PF_OK) return rc;
    return launch_add_partials(y, partial, ks, rows * n, st);
}

// x += fc3(silu(fc1 LN x) * fc2 LN x)
// Up to PARTIAL_ROWS rows may take partial sums.  Their room is in every workspace, so that one for more rows serves fewer.
constexpr long long PARTIAL_ROWS = 2048;
struct TransWs { __half *x, *h; float* partial; long long bytes; };
static TransWs transition_ws(void* ws, long long rows, int c, int hidden) {
    Arena a(ws);
    TransWs w;
    w.x = a.take<__half>(2 * rows * c);
    w.h = a.take<__half>(2 * rows * hidden);
    float* partial = a.take<float>(8 * (rows < PARTIAL_ROWS ? rows : PARTIAL_ROWS) * c);
    w.partial = rows <= PARTIAL_ROWS ? partial : nullptr;
    w.bytes = a.used;
    return w;
}
static int transition(float* x, long long rows, const float* gamma, const float* beta, const b200pf_split_weight& fc12, float hidden_scale,
                      const b200pf_split_weight& fc3, int c, int hidden, void* ws, cudaStream_t st) {
    const TransWs w = transition_ws(ws, rows, c, hidden);
    LnArgs ln = {};
    ln.x = x; ln.gamma = gamma; ln.beta = beta; ln.planes = w.x; ln.part_stride = rows * c; ln.rows = rows;
    int rc;
    if ((rc = launch_ln(ln, c, 0, st)) != B200PF_OK) return rc;
    Gemm g;
    g.epi = EPI_SWIGLU;
    g.a[0] = matrix(w.x, rows, c);
    g.b[0] = matrix(fc12.w, 2 * hidden, c);
    g.m_rows = (int)rows; g.n_rows = 2 * hidden; g.k[0] = c; g.alpha[0] = fc12.alpha; g.out_scale = hidden_scale;
    g.out[0] = dense(w.h, rows, hidden, 2);
    if ((rc = launch_gemm(g, st)) != B200PF_OK) return rc;
    return residual_gemm(x, w.h, fc3, rows, hidden, c, w.partial, st);
}
constexpr long long TRANSITION_ROWS = 1 << 17;        // rows whose hidden activations are held at a time

struct SingleWs { __half *x, *qkv; float* gate; long long bytes; };
static SingleWs single_ws(void* ws, int n, int cs) {
    Arena a(ws);
    SingleWs w;
    w.x = a.take<__half>(2LL * n * cs);
    w.qkv = a.take<__half>(2LL * n * 3 * cs);
    w.gate = a.take<float>((long long)n * cs);
    w.bytes = a.used;
    return w;
}

struct TriMulWs { __half *x, *tn, *ab; float* t; int pitch, tpitch; long long bytes; };
static TriMulWs trimul_ws(void* ws, int n, int c) {
    Arena a(ws);
    TriMulWs w;
    w.pitch = round_up(n, 32);                         // rows of both on 64-byte boundaries: no store or box of one splits a sector
    w.tpitch = round_up(n, 16);
    w.x = a.take<__half>(2LL * n * n * c);
    w.ab = a.take<__half>(2LL * 2 * c * n * w.pitch);
    w.tn = w.ab;                                       // the operands are spent when the normalised product is written
    w.t = a.take<float>((long long)c * n * w.tpitch);
    w.bytes = a.used;
    return w;
}
struct TriAttWs { __half *x, *og, *qkv; float *gate, *bias; int bpitch; long long bytes; };
static TriAttWs triatt_ws(void* ws, int n, int c, int heads, int hd) {
    Arena a(ws);
    const long long nn = (long long)n * n;
    const int ht = heads * hd;
    TriAttWs w;
    w.x = a.take<__half>(2 * nn * (c > ht ? c : ht));
    w.og = w.x;                                        // x is spent once q, k, v, g exist
    w.qkv = a.take<__half>(2 * nn * 3 * ht);
    w.gate = a.take<float>(nn * ht);
    w.bpitch = round_up(n, 16);                        // bias rows start on 64-byte boundaries
    w.bias = a.take<float>((long long)n * w.bpitch * heads);
    w.bytes = a.used;
    return w;
}

}  // namespace split
}  // namespace b200pf

using namespace b200pf;
using namespace b200pf::split;

extern "C" {

long long b200pf_single_track_workspace(int n, int cs, int hidden) {
    const long long a = single_ws(nullptr, n, cs).bytes, b = transition_ws(nullptr, n, cs, hidden).bytes;
    return a > b ? a : b;
}

int b200pf_single_track_attention(const float* s, const b200pf_single_track_weights* w, const float* bias, const uint8_t* mask, void* og, int n, int q0,
                                  int nq, void* workspace, void* stream) {
    B200PF_REQUIRE(s && w && bias && og && workspace && aligned16(s) && aligned16(og) && aligned16(workspace), B200PF_ERR_INVALID,
                   "single_track_attention: null or misaligned pointer");
    B200PF_REQUIRE(n > 0 && q0 >= 0 && nq > 0 && q0 + nq <= n && w->heads > 0 && w->cs % w->heads == 0, B200PF_ERR_INVALID,
                   "single_track_attention: bad sizes");
    const int cs = w->cs, hd = cs / w->heads;
    cudaStream_t st = (cudaStream_t)stream;
    const SingleWs k = single_ws(workspace, n, cs);
    LnArgs ln = {};
    ln.x = s; ln.gamma = w->ln_gamma; ln.beta = w->ln_beta; ln.planes = k.x; ln.part_stride = (long long)n * cs; ln.rows = n;
    int rc;
    if ((rc = launch_ln(ln, cs, 0, st)) != B200PF_OK) return rc;
    Gemm g;
    g.epi = EPI_QKVG;
    g.a[0] = matrix(k.x, n, cs);
    g.b[0] = matrix(w->qkvg.w, 4 * cs, cs);
    g.m_rows = n; g.n_rows = 4 * cs; g.k[0] = cs; g.alpha[0] = w->qkvg.alpha; g.bias = w->qkvg_bias; g.n_split = 3 * cs;
    g.qkv_scale[0] = w->q_scale; g.qkv_scale[1] = w->k_scale; g.qkv_scale[2] = w->o_scale;
    g.out[0] = dense(k.qkv, n, 3 * cs, 2);
    g.out[1] = dense(k.gate, n, cs, 1);
    if ((rc = launch_gemm(g, st)) != B200PF_OK) return rc;
    AttnArgs a = {};
    a.qkv = k.qkv; a.part_stride = (long long)n * 3 * cs; a.ld = 3 * cs; a.line_rows = 0; a.pos_rows = 1;
    a.gate = k.gate; a.bias = bias; a.bias_hs = (long long)nq * n; a.bias_qs = n;
    a.mask = mask; a.mask_ls = 0; a.mask_ks = 1; a.mask_add = -1e6f * 1.4426950408889634f;
    a.out = (__half*)og; a.out_part_stride = (long long)nq * cs; a.out_row0 = q0; a.qk_scale = w->q_scale * w->k_scale;
    a.lines = 1; a.heads = w->heads; a.q0 = q0; a.n_q = nq; a.n_k = n;
    return launch_attention(a, hd, st);
}

int b200pf_single_track_finish(float* s, const b200pf_single_track_weights* w, const void* og, int rows, void* workspace, void* stream) {
    B200PF_REQUIRE(s && w && og && workspace && aligned16(s) && aligned16(og) && aligned16(workspace) && rows > 0, B200PF_ERR_INVALID,
                   "single_track_finish: null or misaligned pointer");
    cudaStream_t st = (cudaStream_t)stream;
    int rc;
    if ((rc = residual_gemm(s, og, w->o, rows, w->cs, w->cs, nullptr, st)) != B200PF_OK) return rc;
    return transition(s, rows, w->ln2_gamma, w->ln2_beta, w->fc12, w->hidden_scale, w->fc3, w->cs, w->hidden, workspace, st);
}

long long b200pf_split_pair_workspace(int n, int c, int heads, int hd, int hidden) {
    const long long nn = (long long)n * n, rows = nn < TRANSITION_ROWS ? nn : TRANSITION_ROWS;
    long long b = trimul_ws(nullptr, n, c).bytes;
    const long long t = transition_ws(nullptr, rows, c, hidden).bytes;
    const long long a = heads > 0 ? triatt_ws(nullptr, n, c, heads, hd).bytes : 0;
    if (t > b) b = t;
    return a > b ? a : b;
}

int b200pf_split_tri_mul(float* z, const uint8_t* mask, const b200pf_split_trimul_weights* w, int n, int incoming, void* workspace, void* stream) {
    B200PF_REQUIRE(z && mask && w && workspace && aligned16(z) && aligned16(workspace) && n > 0, B200PF_ERR_INVALID,
                   "split_tri_mul: null or misaligned pointer");
    const int c = w->c;
    B200PF_REQUIRE(c % 64 == 0 && ln_supported(c), B200PF_ERR_UNSUPPORTED, "split_tri_mul: width %d is not built", c);
    cudaStream_t st = (cudaStream_t)stream;
    const TriMulWs k = trimul_ws(workspace, n, c);
    const long long nn = (long long)n * n;
    int rc;
    LnArgs ln = {};
    ln.x = z; ln.gamma = w->ln_in_gamma; ln.beta = w->ln_in_beta; ln.planes = k.x; ln.part_stride = nn * c; ln.rows = nn;
    if ((rc = launch_ln(ln, c, 0, st)) != B200PF_OK) return rc;
    {   // u[channel][line][k] = p * sigmoid(g) * mask, line = row (outgoing) or column (incoming) of z
        Gemm g;
        g.epi = EPI_GATE_PLANES;
        g.a[0] = matrix(w->in.w, 4 * c, c);
        g.a_second_row = 2 * c;
        g.b[0] = incoming ? Operand{k.x, n, c, n, (long long)n * c, c, nn * c} : Operand{k.x, n, c, n, c, (long long)n * c, nn * c};
        g.b_batched = true;
        g.m_rows = 2 * c; g.n_rows = n; g.batches = n; g.k[0] = c; g.alpha[0] = w->in.alpha;
        g.mask = mask; g.mask_bs = incoming ? 1 : n; g.mask_cs = incoming ? n : 1;
        g.out_scale = w->u_scale;
        g.out[0] = Output{k.ab, 2 * c, n, n, 2, (long long)n * k.pitch, k.pitch, 2LL * c * n * k.pitch, true};
        if ((rc = launch_gemm(g, st)) != B200PF_OK) return rc;
    }
    {   // t[channel][i][j] = sum_k a[channel][i][k] b[channel][j][k]
        Gemm g;
        g.epi = EPI_CONTRACT;
        g.alpha[0] = 1.f / (w->u_scale * w->u_scale);
        g.a[0] = Operand{k.ab, n, n, c, k.pitch, (long long)n * k.pitch, 2LL * c * n * k.pitch};
        g.b[0] = Operand{k.ab + (long long)c * n * k.pitch, n, n, c, k.pitch, (long long)n * k.pitch, 2LL * c * n * k.pitch};
        g.a_batched = g.b_batched = true;
        g.m_rows = n; g.n_rows = n; g.batches = c; g.k[0] = n;
        g.out[0] = Output{k.t, n, n, c, 1, k.tpitch, (long long)n * k.tpitch, 0, false};
        if ((rc = launch_gemm(g, st)) != B200PF_OK) return rc;
    }
    if ((rc = launch_ln_channels(k.t, (long long)n * k.tpitch, k.tpitch, w->ln_out_gamma, w->ln_out_beta, k.tn, n, c, st)) != B200PF_OK) return rc;
    Gemm g;      // z += (LN(t) W_p^T) * sigmoid(LN(z) W_g^T)
    g.epi = EPI_GATE_ADD;
    g.a[0] = matrix(k.tn, nn, c);
    g.b[0] = matrix(w->p_out.w, c, c);
    g.a[1] = matrix(k.x, nn, c);
    g.b[1] = matrix(w->g_out.w, c, c);
    g.m_rows = (int)nn; g.n_rows = c; g.k[0] = g.k[1] = c; g.alpha[0] = w->p_out.alpha; g.alpha[1] = w->g_out.alpha;
    g.out[0] = dense(z, nn, c, 1);
    return launch_gemm(g, st);
}

int b200pf_split_tri_att(float* z, const uint8_t* mask, const b200pf_split_triatt_weights* w, int n, int ending, void* workspace, void* stream) {
    B200PF_REQUIRE(z && mask && w && workspace && aligned16(z) && aligned16(workspace) && n > 0, B200PF_ERR_INVALID,
                   "split_tri_att: null or misaligned pointer");
    const int c = w->c, heads = w->heads, hd = w->hd, ht = heads * hd;
    B200PF_REQUIRE(c % 64 == 0 && ln_supported(c) && ht % 64 == 0, B200PF_ERR_UNSUPPORTED, "split_tri_att: width %d with %d x %d heads is not built", c, heads, hd);
    cudaStream_t st = (cudaStream_t)stream;
    const TriAttWs k = triatt_ws(workspace, n, c, heads, hd);
    const long long nn = (long long)n * n;
    int rc;
    LnArgs ln = {};
    ln.x = z; ln.gamma = w->ln_gamma; ln.beta = w->ln_beta; ln.planes = k.x; ln.part_stride = nn * c; ln.rows = nn;
    ln.head_w = w->head_w; ln.head_out = k.bias; ln.head_stride = (long long)n * k.bpitch; ln.n = n; ln.transposed = ending; ln.head_pitch = k.bpitch;
    if ((rc = launch_ln(ln, c, heads, st)) != B200PF_OK) return rc;
    {
        Gemm g;
        g.epi = EPI_QKVG;
        g.a[0] = matrix(k.x, nn, c);
        g.b[0] = matrix(w->qkvg.w, 4 * ht, c);
        g.m_rows = (int)nn; g.n_rows = 4 * ht; g.k[0] = c; g.alpha[0] = w->qkvg.alpha; g.n_split = 3 * ht;
        g.qkv_scale[0] = w->q_scale; g.qkv_scale[1] = w->k_scale; g.qkv_scale[2] = w->o_scale;
        g.out[0] = dense(k.qkv, nn, 3 * ht, 2);
        g.out[1] = dense(k.gate, nn, ht, 1);
        if ((rc = launch_gemm(g, st)) != B200PF_OK) return rc;
    }
    AttnArgs a = {};
    a.qkv = k.qkv; a.part_stride = nn * 3 * ht; a.ld = 3 * ht;
    a.line_rows = ending ? 1 : n; a.pos_rows = ending ? n : 1;       // a line is a row of z, or a column
    a.gate = k.gate; a.bias = k.bias; a.bias_hs = (long long)n * k.bpitch; a.bias_qs = k.bpitch;
    a.mask = mask; a.mask_ls = ending ? 1 : n; a.mask_ks = ending ? n : 1; a.mask_add = -1e9f * 1.4426950408889634f;
    a.out = k.og; a.out_part_stride = nn * ht; a.out_row0 = 0; a.qk_scale = w->q_scale * w->k_scale;
    a.lines = n; a.heads = heads; a.q0 = 0; a.n_q = n; a.n_k = n;
    if ((rc = launch_attention(a, hd, st)) != B200PF_OK) return rc;
    return residual_gemm(z, k.og, w->o, nn, ht, c, nullptr, st);
}

long long b200pf_split_transition_workspace(long long rows, int c, int hidden) {
    return transition_ws(nullptr, rows < TRANSITION_ROWS ? rows : TRANSITION_ROWS, c, hidden).bytes;
}

int b200pf_split_transition(float* x, long long rows, const b200pf_split_transition_weights* w, void* workspace, long long workspace_bytes, void* stream) {
    B200PF_REQUIRE(x && w && workspace && aligned16(x) && aligned16(workspace) && rows > 0, B200PF_ERR_INVALID,
                   "split_transition: null or misaligned pointer");
    B200PF_REQUIRE(w->c % 64 == 0 && ln_supported(w->c) && w->hidden % 64 == 0, B200PF_ERR_UNSUPPORTED, "split_transition: %d -> %d is not built", w->c, w->hidden);
    B200PF_REQUIRE(workspace_bytes >= b200pf_split_transition_workspace(rows, w->c, w->hidden), B200PF_ERR_INVALID,
                   "split_transition: %lld bytes of workspace are too few for %lld rows", workspace_bytes, rows);
    for (long long r = 0; r < rows; r += TRANSITION_ROWS) {
        const long long m = rows - r < TRANSITION_ROWS ? rows - r : TRANSITION_ROWS;
        const int rc = transition(x + r * w->c, m, w->ln_gamma, w->ln_beta, w->fc12, w->hidden_scale, w->fc3, w->c, w->hidden, workspace, (cudaStream_t)stream);
        if (rc != B200PF_OK) return rc;
    }
    return B200PF_OK;
}

int b200pf_ln_heads(const float* x, const float* gamma, const float* beta, const float* w, float* out, long long head_stride, long long rows, int c,
                    int heads, void* stream) {
    B200PF_REQUIRE(x && gamma && beta && w && out && rows >= 0, B200PF_ERR_INVALID, "ln_heads: null pointer");
    B200PF_REQUIRE(heads == 4 || heads == 8 || heads == 16, B200PF_ERR_UNSUPPORTED, "ln_heads: 4, 8 or 16 heads (got %d)", heads);
    if (rows == 0) return B200PF_OK;
    LnArgs ln = {};
    ln.x = x; ln.gamma = gamma; ln.beta = beta; ln.rows = rows; ln.head_w = w; ln.head_out = out; ln.head_stride = head_stride; ln.n = 1; ln.head_pitch = 1;
    return launch_ln(ln, c, heads, (cudaStream_t)stream);
}

/* y[rows][n] (+)= x[rows][k] w[n][k]^T (+ bias) for any fp32 x: both operands as three bf16 parts */
long long b200pf_split_linear_workspace(long long rows, int k) { return 6 * rows * k; }

int b200pf_split_linear(const float* x, const void* w, const float* bias, float* y, long long rows, int k, int n, int accumulate, void* workspace,
                        void* stream) {
    B200PF_REQUIRE(x && w && y && workspace && aligned16(x) && aligned16(w) && aligned16(y) && aligned16(workspace), B200PF_ERR_INVALID,
                   "split_linear: null or misaligned pointer");
    B200PF_REQUIRE(rows > 0 && rows <= 0x7fffffffLL && k > 0 && k % 8 == 0 && n > 0 && n % 4 == 0, B200PF_ERR_UNSUPPORTED, "split_linear: bad sizes");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = launch_parts(x, (__nv_bfloat16*)workspace, rows * k, st);
    if (rc != B200PF_OK) return rc;
    Gemm g;
    g.parts = 3;
    g.epi = accumulate ? EPI_ADD : EPI_STORE;
    g.a[0] = matrix(workspace, rows, k);
    g.b[0] = matrix(w, n, k);
    g.m_rows = (int)rows; g.n_rows = n; g.k[0] = k; g.bias = bias;
    g.out[0] = dense(y, rows, n, 1);
    return launch_gemm(g, st);
}

}  // extern "C"
