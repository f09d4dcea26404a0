// The launches of a run of equal decoder layers (norm, q|k|v, attention, output, norm, gate/up, down) from one call.
//
// A layer is five kernels in steps of few tokens and eight to ten otherwise, of 3 to 10 us each at small sizes, and called
// one by one from Python each costs the host 13 to 25 us: a prompt portion of 25 tokens at Qwen3-0.6B sizes took 3.2 ms to
// launch and 1.0 ms to run.  From here a launch costs 2 to 3 us.  The kernels, their order and their arguments are those of the parts
// (parts/attention.py, parts/feedforward.py, parts/norm.py); what depends on the step alone (which attention kernel, K
// splits, which product) the caller has decided once for all layers.  Nothing is kept between calls.
#include "entry_points.cuh"

extern "C" {
// One layer's tensors, in the order that csrc/ops.py fills in.
struct TkDenseLayer {
  const void *w_qkv, *w_o, *w_gate_up, *w_down;
  const float *norm1_w, *norm2_w, *next_norm_w, *q_norm_w, *k_norm_w;
  void *k_cache, *v_cache;
  const int* block_table;
};

// What all layers of a step share; mirrored field by field in csrc/ops.py.
struct TkDenseStep {
  // inputs of the first layer: its normed rows x (or, with x_sumsq, rows whose norm is still owed); cleared fields are null
  const void* x;
  const float* x_sumsq;
  float* resid;
  const int *positions, *tok_req, *req_slot, *req_q_len, *req_kv_len;
  const float* rope_table;
  int* err;
  const int *dec_items, *records, *plain_items;
  float* dec_scratch;
  int *dec_counters, *sched, *part_count;
  float *part_o, *part_ml;
  // buffers: queries, attention rows, q|k|v rows, normed rows, output rows, gate and up rows, activations, down rows; rows
  // and sums of squares for an owed norm behind the output and behind the down product
  void *q, *att, *qkv, *h, *o, *gate_up, *act, *down;
  void* xb_mid;
  float* sumsq_mid;
  void* xb_end;
  float* sumsq_end;
  cudaStream_t side;                 // null: single tokens and prompt portions one after the other
  cudaEvent_t fork, join;
  long long n_plain;
  int mode;                          // 0: bf16, few tokens; 1: bf16, more; 2: float32
  int n_tokens, n_reqs, hidden, inter, n_q_heads, n_kv_heads, head_dim, rotary_dim, page_size, max_pages, num_pages, window;
  int glu_act, glu_block;
  int n_dec, dec_kind, dec_n;        // dec_kind 0: none, 1: equal splits (dec_n of them), 2: balanced (dec_n blocks)
  int n_records;
  int bn;
  int splits[4], stages[4];          // mode 0: q|k|v, output, gate/up, down
  int product[4];                    // mode 1: 1 = gemm_tokens, 2 = gemm_pair
  float scale, eps1, eps2, next_eps, qk_eps, x_eps;
  int launches;                      // out: kernels launched
};
}

namespace tk {

#define TK_LAUNCH(call)               \
  do {                                \
    const int rc_ = (call);           \
    if (rc_ != 0) return rc_;         \
    ++s.launches;                     \
  } while (0)

static int dense_product(TkDenseStep& s, int which, const void* x, const void* w, void* out, int n_out, int k, bool glu,
                         cudaStream_t stream) {
  const int mode = glu ? 1 + s.glu_act : 0, width = glu ? n_out / 2 : n_out;
  if (s.product[which] == 1) {
    return tk_gemm_bf16_tokens(x, w, out, s.err, s.n_tokens, n_out, k, k, k, width, mode, 0, 0, &s.launches, stream);
  } else {
    TK_LAUNCH(tk_gemm_bf16_pair(x, w, out, s.err, s.n_tokens, n_out, k, k, k, width, mode, stream));
  }
  return 0;
}

static int dense_decode(TkDenseStep& s, const TkDenseLayer& l, cudaStream_t stream) {
  if (s.dec_kind == 1) {
    TK_LAUNCH(tk_attention_decode(s.q, s.att, l.k_cache, l.v_cache, s.dec_scratch, s.dec_counters, s.dec_items, s.positions,
                                  s.tok_req, s.req_slot, l.block_table, s.err, s.n_dec, s.n_reqs, s.n_q_heads, s.n_kv_heads,
                                  s.head_dim, s.page_size, s.max_pages, s.num_pages, s.window, s.dec_n, s.scale, 0.0f,
                                  nullptr, 0, nullptr, nullptr, 0, stream));
  } else if (s.dec_kind == 2) {
    TK_LAUNCH(tk_attention_decode_balanced(s.q, s.att, l.k_cache, l.v_cache, s.dec_scratch, s.dec_counters, s.dec_items,
                                           s.positions, s.tok_req, s.req_slot, l.block_table, s.err, s.n_dec, s.n_reqs,
                                           s.n_q_heads, s.n_kv_heads, s.head_dim, s.page_size, s.max_pages, s.num_pages,
                                           s.window, s.dec_n, s.scale, 0.0f, nullptr, 0, nullptr, nullptr, 0, stream));
  }
  return 0;
}

static int dense_prompts(TkDenseStep& s, const TkDenseLayer& l, cudaStream_t stream) {
  if (s.n_records > 0) {
    TK_LAUNCH(tk_attention_prefill_tc(s.q, s.att, l.k_cache, l.v_cache, s.records, l.block_table, s.err, s.sched, s.part_o,
                                      s.part_ml, s.part_count, s.n_tokens, s.n_records, s.n_q_heads, s.n_kv_heads,
                                      s.head_dim, s.page_size, s.max_pages, s.num_pages, s.window, s.scale, 0.0f, nullptr, 0,
                                      nullptr, nullptr, 0, stream));
  }
  return 0;
}

static int dense_attention(TkDenseStep& s, const TkDenseLayer& l, cudaStream_t stream) {
  if (s.mode == 2) {
    const int kv_row = s.head_dim;
    TK_LAUNCH(tk_attention_plain(s.q, s.att, l.k_cache, l.v_cache, s.positions, s.tok_req, s.req_slot, l.block_table,
                                 s.plain_items, s.err, (int)s.n_plain, s.n_reqs, s.n_q_heads, s.n_kv_heads, s.head_dim,
                                 s.page_size, s.max_pages, s.num_pages, s.window, s.scale, kF32, s.head_dim, 0.0f, nullptr,
                                 kF32, (long long)s.n_q_heads * s.head_dim, s.head_dim, kv_row, kv_row, 0, nullptr, nullptr, 0,
                                 stream));
    return 0;
  }
  if (s.side == nullptr) {
    const int rc = dense_decode(s, l, stream);
    return rc != 0 ? rc : dense_prompts(s, l, stream);
  }
  // the decode kernel runs beside the prompt portions'; the side stream is joined whatever a launch says
  cudaError_t e = cudaEventRecord(s.fork, stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(s.side, s.fork, 0);
  if (e != cudaSuccess) return (int)e;
  int rc = dense_decode(s, l, s.side);
  const cudaError_t e1 = cudaEventRecord(s.join, s.side);
  if (rc == 0) rc = dense_prompts(s, l, stream);
  const cudaError_t e2 = cudaStreamWaitEvent(stream, s.join, 0);
  if (rc == 0) rc = (int)(e1 != cudaSuccess ? e1 : e2);
  return rc;
}

// Few tokens: norm, rotation and page write, activation, residual sums and the next norm's input ride in the products.
static int dense_layer_few(TkDenseStep& s, const TkDenseLayer& l, const void*& x, const float*& x_sumsq, float& x_eps,
                           cudaStream_t stream) {
  const int tiles = s.hidden / 128;
  const float inv = 1.0f / (float)s.hidden;
  TK_LAUNCH(tk_gemm_qkv_rope(l.w_qkv, x, s.err, s.n_tokens, s.hidden, s.hidden, s.hidden, s.bn, s.splits[0], s.stages[0],
                             x_sumsq, x_sumsq != nullptr ? tiles : 0, x_sumsq != nullptr ? inv : 0.0f,
                             x_sumsq != nullptr ? x_eps : 0.0f, s.q, l.k_cache, l.v_cache, s.positions, s.tok_req, s.req_slot,
                             l.block_table, s.req_q_len, s.req_kv_len, l.q_norm_w, l.k_norm_w, s.rope_table, s.n_reqs,
                             s.n_q_heads, s.n_kv_heads, s.page_size, s.max_pages, s.num_pages, s.qk_eps, stream));
  const int rc = dense_attention(s, l, stream);
  if (rc != 0) return rc;
  const int width = s.n_q_heads * s.head_dim;
  TK_LAUNCH(tk_gemm_bf16_tcgen05(l.w_o, s.att, nullptr, s.err, s.hidden, s.n_tokens, width, width, width, s.bn, s.splits[1],
                                 s.stages[1], s.splits[1] > 1 ? s.splits[1] : 0, 2, nullptr, 0, 0.0f, 0.0f, s.resid, l.norm2_w,
                                 s.xb_mid, s.sumsq_mid, stream));
  TK_LAUNCH(tk_gemm_bf16_tcgen05(l.w_gate_up, s.xb_mid, s.act, s.err, 2 * s.inter, s.n_tokens, s.hidden, s.hidden, s.hidden, s.bn,
                                 s.splits[2], s.stages[2], s.splits[2] > 1 ? s.splits[2] : 0, s.glu_act == 0 ? 1 : 4,
                                 s.sumsq_mid, tiles, inv, s.eps2, nullptr, nullptr, nullptr, nullptr, stream));
  TK_LAUNCH(tk_gemm_bf16_tcgen05(l.w_down, s.act, nullptr, s.err, s.hidden, s.n_tokens, s.inter, s.inter, s.inter, s.bn,
                                 s.splits[3], s.stages[3], s.splits[3] > 1 ? s.splits[3] : 0, 2, nullptr, 0, 0.0f, 0.0f, s.resid,
                                 l.next_norm_w, s.xb_end, s.sumsq_end, stream));
  x = s.xb_end;
  x_sumsq = s.sumsq_end;
  x_eps = s.next_eps;
  return 0;
}

static int dense_layer_many(TkDenseStep& s, const TkDenseLayer& l, const void* x, cudaStream_t stream) {
  const int dtype = s.mode == 2 ? kF32 : kBF16;
  const int width = s.n_q_heads * s.head_dim, qkv = (s.n_q_heads + 2 * s.n_kv_heads) * s.head_dim;
  if (x == nullptr) {
    TK_LAUNCH(tk_add_rmsnorm(s.resid, s.down, nullptr, 0, 0, l.norm1_w, s.h, nullptr, s.n_tokens, s.hidden, s.eps1, dtype, stream));
    x = s.h;
  }
  const auto product = [&](int which, const void* in, const void* w, void* out, int n_out, int k) -> int {
    if (s.mode == 1) return dense_product(s, which, in, w, out, n_out, k, false, stream);
    TK_LAUNCH(tk_gemm_f32((const float*)in, (const float*)w, (float*)out, s.n_tokens, n_out, k, k, k, n_out, 1, 0, 0, 0, 0, stream));
    return 0;
  };
  int rc = product(0, x, l.w_qkv, s.qkv, qkv, s.hidden);
  if (rc != 0) return rc;
  TK_LAUNCH(tk_rope_kv(s.qkv, nullptr, 0, s.q, l.k_cache, l.v_cache, s.positions, s.tok_req, s.req_slot, l.block_table,
                       s.req_q_len, s.req_kv_len, l.q_norm_w, l.k_norm_w, s.rope_table, s.err, s.n_tokens, s.n_reqs,
                       s.n_q_heads, s.n_kv_heads, s.head_dim, s.rotary_dim, qkv, s.page_size, s.max_pages, s.num_pages, 1,
                       s.qk_eps, dtype, stream));
  rc = dense_attention(s, l, stream);
  if (rc != 0) return rc;
  rc = product(1, s.att, l.w_o, s.o, s.hidden, width);
  if (rc != 0) return rc;
  TK_LAUNCH(tk_add_rmsnorm(s.resid, s.o, nullptr, 0, 0, l.norm2_w, s.h, nullptr, s.n_tokens, s.hidden, s.eps2, dtype, stream));
  if (s.mode == 1) {
    rc = dense_product(s, 2, s.h, l.w_gate_up, s.act, 2 * s.inter, s.hidden, true, stream);
  } else {
    rc = product(2, s.h, l.w_gate_up, s.gate_up, 2 * s.inter, s.hidden);
    if (rc == 0) {
      TK_LAUNCH(tk_swiglu(s.gate_up, nullptr, 0, 0, s.act, s.n_tokens, s.inter, s.glu_block, dtype, s.glu_act, stream));
    }
  }
  if (rc != 0) return rc;
  return product(3, s.act, l.w_down, s.down, s.hidden, s.inter);
}

}  // namespace tk

// Launches `n_layers` layers.  Mode 0 leaves the rows for the norm behind the last layer, whose scaling is owed, in xb_end and
// sumsq_end, which the next call takes as x and x_sumsq; the other modes leave the last branch in `down`, and a call with x
// null begins by adding it.
TK_API int tk_dense_layers(const TkDenseLayer* layers, int n_layers, TkDenseStep* step, cudaStream_t stream) {
  TkDenseStep& s = *step;
  const void* x = s.x;
  const float* x_sumsq = s.x_sumsq;
  float x_eps = s.x_eps;
  for (int i = 0; i < n_layers; ++i) {
    const int rc = s.mode == 0 ? tk::dense_layer_few(s, layers[i], x, x_sumsq, x_eps, stream)
                               : tk::dense_layer_many(s, layers[i], i == 0 ? x : nullptr, stream);
    if (rc != 0) return rc;
  }
  return 0;
}

// The sizes of the two records, for a caller that lays them out in another language.
TK_API int tk_dense_step_bytes(void) { return (int)sizeof(TkDenseStep); }
TK_API int tk_dense_layer_bytes(void) { return (int)sizeof(TkDenseLayer); }
