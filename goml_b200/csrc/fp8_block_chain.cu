// fp8_block_chain.cu — the calls of a decoder block in native code (fp8_block_run, include/fp8_block.h).
//
// A block over a few tokens is 10 to 16 launches of a few microseconds each.  Issued one by one from the host language they cost
// it 7 us apiece (argument conversion, checks, the launch), more than the GPU needs; here they cost the launch.  The maxima of
// all quantisers of the block are cleared once, by its first kernel, where every larger op had a clearing kernel in front.
//
// A step of one or two sequences has its quantisers inside the products that read their codes (fp8_gemm_rows): six calls in the
// place of ten.  Each of the four that this saved took 2 to 5 us with its hand-over, and the product behind it began to stream its
// weight only then.
#include "../../include/fp8_gemm.h"   // the argument block of fp8_gemm_rows; nothing of that library is linked
#include "fp8_block_glue.h"

namespace {

constexpr size_t ALIGN = 256;
size_t up(size_t n) { return (n + ALIGN - 1) & ~(ALIGN - 1); }

// maxima (one word each, cleared together) and scales, in the order of the block
enum { NORM1 = 0, Q, K, V, O, NORM2, HIDDEN, N_WORDS };

// code of a failed call: its place in the chain << 16 | what it returned
int at(int place, int rc) { return rc == 0 ? 0 : (place << 16) | (rc & 0xffff); }

using GemmRows = int (*)(const fp8_gemm_rows_args_t*);
// Most values that such a product goes over for their maximum, in every thread block, and most of those whose maximum is known, of which
// a block takes its slice.  Steps with a quantiser ahead of each product / as here / with all four products quantising for themselves,
// us, calls queued ahead: d = 4096, F = 11008, one sequence 73.5 / 65.3 / 65.3, two 75.6 / 73.2 / 73.2; 5120, 13824, one 92.8 / 87.6 / 87.6, two
// 95.7 / 93.4 / 97.8; 8192, 28672, one 212 / 210 / 210, two 205 / 205 / 210 (208 with the last product alone).
constexpr size_t ROWS_SWEPT = 8192, ROWS_KNOWN = 32768;
enum { ROWS_QKV = 11, ROWS_O, ROWS_GATE_UP, ROWS_DOWN };   // places of the products that quantise for themselves

}  // namespace

extern "C" {

size_t fp8_block_region_bytes(int rows, int d_model, int ffn_hidden) {
    if (rows < 0 || d_model <= 0 || ffn_hidden <= 0) return 0;
    const size_t n = (size_t)rows * d_model, f = (size_t)rows * ffn_hidden;
    const size_t attention = up(6 * n) + up(n) + up(2 * n) + up(n), feed_forward = up(2 * f) + up(f);
    return attention > feed_forward ? attention : feed_forward;
}

int fp8_block_run(const fp8_block_run_args_t* a) { return fp8_block_run_rows(a, nullptr); }

int fp8_block_run_rows(const fp8_block_run_args_t* a, GemmRows gemm_rows) {
    if (!a || !a->gemm_scaled || !a->gemm_accumulate_f32 || !a->gemm_swiglu_raise || !a->attention_raise || !a->attention_decode || !a->attention_ctx) return (int)cudaErrorInvalidValue;
    if (!a->x || !a->h || !a->wqkv || !a->wo || !a->wgate_up || !a->wdown || !a->words || !a->rstd || !a->codes || !a->region)
        return (int)cudaErrorInvalidValue;
    const bool decode = a->decode != 0;
    if (a->batch <= 0 || a->heads <= 0 || a->d_model <= 0 || a->d_model % a->heads != 0 || a->ffn_hidden <= 0) return (int)cudaErrorInvalidValue;
    // a prompt's positions are 0 .. seq_len - 1, each of which must have its row of the tables (a step looks at rope_rows itself)
    if (decode ? a->seq_len != 1 || !a->k_cache : a->seq_len <= 0 || a->rope_rows < a->seq_len || !a->k_codes || !a->v_codes) return (int)cudaErrorInvalidValue;
    if (a->k_cache && (!a->v_cache || !a->cache_scales || !a->cache_lens || a->s_max < a->seq_len)) return (int)cudaErrorInvalidValue;
    if ((long long)a->batch * a->seq_len > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
    const int T = a->batch * a->seq_len, d = a->d_model, H = a->heads, hd = d / H, F = a->ffn_hidden;
    const size_t n = (size_t)T * d;
    if (a->region_bytes < fp8_block_region_bytes(T, d, F)) return (int)cudaErrorInvalidValue;
    uint8_t* qkv = a->region;                       // [T, 3, H, hd] bf16
    uint8_t* qc = qkv + up(6 * n);
    uint8_t* o = qc + up(n);                        // fp16
    uint8_t* oc = o + up(2 * n);
    uint8_t* hb = a->region;                        // [T, F] bf16: the attention half is done with the region by then
    uint8_t* hc = hb + up(2 * (size_t)T * F);
    float* amax = a->words;
    float* scale = a->words + 16;
    void* stream = a->stream;
    cudaStream_t s = (cudaStream_t)stream;
    int rc;
    // a product of a step's rows as values; done: it has been launched
    bool done = false;
    auto rows = [&](int place, int source, const void* values, const float* gamma, const uint8_t* w, const float* w_scale, int n_out, int k, auto more) -> int {
        done = false;
        if (!decode || !gemm_rows || (size_t)T * k > (source == FP8_ROWS_BF16 ? ROWS_KNOWN : ROWS_SWEPT)) return 0;
        fp8_gemm_rows_args_t g{};
        g.rows = values; g.gamma = gamma; g.eps = a->eps; g.b = w; g.scale_b = w_scale;
        g.m = T; g.n = n_out; g.k = k; g.source = source; g.stream = stream;
        // every kernel of the chain lets the next one start after its own wait, so behind the first one the weights are complete
        g.b_complete = place != ROWS_QKV;
        more(g);
        const int r = gemm_rows(&g);
        if (r == (int)cudaErrorNotSupported) return 0;
        done = r == 0;
        return at(place, r);
    };
    // attention half
    const float* stream_in = a->h;   // the residual stream that the attention's projection is added to
    if ((rc = rows(ROWS_QKV, FP8_ROWS_RMSNORM_F32, a->x, a->norm1, a->wqkv, a->wqkv_scale, 3 * d, d,
                   [&](fp8_gemm_rows_args_t& g) { g.c = qkv; g.zero = amax; g.zeros = N_WORDS; }))) return rc;
    if (done) {
        stream_in = a->x;
    } else {
        if ((rc = at(1, fp8_block::rmsnorm(a->x, nullptr, a->h, a->h != a->x, a->norm1, a->codes, scale + NORM1, amax + NORM1, a->rstd,
                                           {amax, N_WORDS, true}, T, d, a->eps, s)))) return rc;
        if ((rc = at(2, a->gemm_scaled(T, 3 * d, d, a->codes, a->wqkv, qkv, 1.0f, scale + NORM1, a->wqkv_scale, 1, stream)))) return rc;
    }
    if (decode) {
        fp8_decode_append_args_t g{};
        g.qkv_bf16 = qkv; g.cos_tab = a->cos_tab; g.sin_tab = a->sin_tab; g.positions = a->cache_lens;
        g.q_out = qc; g.q_scale_out = scale + Q; g.q_amax_out = amax + Q;
        g.k_cache = a->k_cache; g.v_cache = a->v_cache; g.k_scale = a->cache_scales; g.v_scale = a->cache_scales + 1;
        g.seq_lens_out = a->cache_lens;   // the lengths advance in place: the step can be replayed from a CUDA graph
        g.batch = a->batch; g.q_heads = g.kv_heads = H; g.head_dim = hd; g.s_max = a->s_max; g.rope_rows = a->rope_rows;
        g.stream = stream;
        if ((rc = at(3, fp8_block::append(&g, true)))) return rc;
        fa_decode_args_t t{};
        t.q = qc; t.k_cache = a->k_cache; t.v_cache = a->v_cache; t.o = o; t.seq_lens = a->cache_lens;
        t.batch = a->batch; t.q_heads = t.kv_heads = H; t.head_dim = hd; t.s_max = a->s_max;
        t.scale = a->softmax_scale; t.v_descale = 1.0f;
        t.scale_q_dev = scale + Q; t.scale_k_dev = a->cache_scales; t.scale_v_dev = a->cache_scales + 1;
        t.stream = (fa_stream_t)stream;
        if ((rc = at(4, a->attention_decode(a->attention_ctx, &t)))) return rc;
    } else {
        fp8_block::Rope r{};
        r.qkv_bf16 = qkv; r.cos_tab = a->cos_tab; r.sin_tab = a->sin_tab;
        r.q_out = qc; r.k_out = a->k_codes; r.v_out = a->v_codes; r.scales = scale + Q; r.amaxes = amax + Q;
        r.k_cache = a->k_cache; r.v_cache = a->v_cache; r.cache_scales = a->cache_scales; r.cache_lens = a->cache_lens;
        r.batch = a->batch; r.seq_len = a->seq_len; r.s_max = a->s_max; r.heads = H; r.head_dim = hd;
        if ((rc = at(3, fp8_block::rope_qkv(r, true, s)))) return rc;
        fa_forward_args_t t{};
        t.q = qc; t.k = a->k_codes; t.v = a->v_codes; t.o = o;
        t.batch_heads = a->batch * H; t.seq_len = a->seq_len; t.head_dim = hd; t.causal = 1;
        t.scale = a->softmax_scale; t.v_descale = 1.0f;
        t.scale_q_dev = scale + Q; t.scale_k_dev = scale + K; t.scale_v_dev = scale + V;
        t.stream = (fa_stream_t)stream;
        if ((rc = at(4, a->attention_raise(a->attention_ctx, &t, amax + O)))) return rc;
    }
    // h += attention projection, in the GEMM epilogue (a step's attention output lies as the projection reads it)
    if ((rc = rows(ROWS_O, FP8_ROWS_F16, o, nullptr, a->wo, a->wo_scale, d, d, [&](fp8_gemm_rows_args_t& g) { g.x = a->h; g.x_in = stream_in; }))) return rc;
    if (!done) {
        if (stream_in != a->h && (rc = at(6, (int)cudaMemcpyAsync(a->h, stream_in, n * sizeof(float), cudaMemcpyDeviceToDevice, s)))) return rc;
        const fp8_block::Max known = decode ? fp8_block::Max::ZERO : fp8_block::Max::KNOWN;
        if ((rc = at(5, fp8_block::permute_heads(o, oc, scale + O, amax + O, a->batch, a->seq_len, H, hd, known, s)))) return rc;
        if ((rc = at(6, a->gemm_accumulate_f32(T, d, d, oc, a->wo, a->h, 1.0f, scale + O, a->wo_scale, stream)))) return rc;
    }
    // feed-forward half: gate/up projections with silu(gate) * up and max|.| in the GEMM epilogue
    if ((rc = rows(ROWS_GATE_UP, FP8_ROWS_RMSNORM_F32, a->h, a->norm2, a->wgate_up, a->wgate_up_scale, F, d,
                   [&](fp8_gemm_rows_args_t& g) { g.h = hb; g.h_amax = amax + HIDDEN; }))) return rc;
    if (!done) {
        if ((rc = at(7, fp8_block::rmsnorm(a->h, nullptr, nullptr, false, a->norm2, a->codes, scale + NORM2, amax + NORM2, a->rstd,
                                           {nullptr, 0, true}, T, d, a->eps, s)))) return rc;
        if ((rc = at(8, a->gemm_swiglu_raise(T, F, d, a->codes, a->wgate_up, hb, 1.0f, scale + NORM2, a->wgate_up_scale, amax + HIDDEN, stream)))) return rc;
    }
    if ((rc = rows(ROWS_DOWN, FP8_ROWS_BF16, hb, nullptr, a->wdown, a->wdown_scale, d, F,
                   [&](fp8_gemm_rows_args_t& g) { g.amax = amax + HIDDEN; g.x = a->h; g.x_in = a->h; }))) return rc;
    if (!done) {
        if ((rc = at(9, fp8_quantize_bf16(hb, hc, scale + HIDDEN, amax + HIDDEN, (size_t)T * F, stream)))) return rc;
        if ((rc = at(10, a->gemm_accumulate_f32(T, d, F, hc, a->wdown, a->h, 1.0f, scale + HIDDEN, a->wdown_scale, stream)))) return rc;
    }
    return 0;
}

}  // extern "C"
