// One layer's share of a training step as a whole: the activation buffer of the forward pass and the
// backward with everything between the tensors a framework hands over and the gradients it gets back.
// These entry points choose how the intermediates are stored and which kernels run, so that a binding
// makes one call per direction; hot_hlq_backward is the reference extension's call on top of them.
//
// Quantisers of the backward, by configuration:
//   bf16, order-16 transforms, basis of 8 of 16 rows, one scale: the tensor-core pair (go_dual_tc.cu), the weight inside
//   otherwise: the tiled pair (quant_tiles.cu), grad_out and the weight as two jobs; a scale per token on the g_x side
//              is the one-launch kernel of row_ht_quant, which holds a whole row in registers
//   what neither covers (explicit noise, orders above 16, odd widths): row_ht_quant and col_ht_quant, one operand after
//              the other
#include <cstdlib>
#include <cstring>

#include "layer.cuh"
#include "quant_tiles.cuh"

namespace hot {

int gemm_i8_dual_ws(const hot_gemm_problem_t* main_problem, const hot_gemm_problem_t* rider_problem, void* workspace,
                    size_t workspace_bytes, uint32_t* counters, size_t clear_words, uint32_t* status_word, hot_stream_t stream);

int gemm_i8_grouped(const void* a, int64_t lda, const void* b, int64_t ldb, int64_t M, int64_t N, int64_t groups, int64_t group_k,
                    int64_t len, const float* scale_a, int scale_a_per_row, const float* scale_b, float post, void* out, int out_dtype,
                    int64_t ldo, uint32_t* status_word, hot_stream_t stream);

namespace {

constexpr size_t kAlign = 256;
constexpr int kRiderCounters = 160;  // one word per g_w tile that the dual GEMM may cut along K
inline size_t up(size_t v, size_t a) { return (v + a - 1) / a * a; }
inline int64_t code_pitch(int64_t len, int storage) { return (int64_t)up((size_t)(storage == HOT_STORE_INT4 ? (len + 1) / 2 : len), 16); }
// a sample's codes take whole 128-byte k-blocks of the grouped GEMM
inline int64_t sample_pitch(int64_t out_len) { return (out_len + 127) / 128 * 128; }

// The workspace of a backward.
struct Plan {
  int64_t batch, rows;      // samples (1 in a plain call) and rows of grad_out over all of them
  int64_t lp, pitch;        // codes per sample on the token side; bytes from sample to sample (0: plain)
  int64_t ld_qgo, ld_qw, ld_qgw;
  size_t off_qgo, off_sgo, off_qw, off_sw, off_qgw, off_sgw, off_words, w_words, off_tiles, tiles_bytes, off_gemm, gemm_bytes, total;
};

// The jobs of a backward on the tiled quantisers (pointers that are not known yet may be null: sizes do not depend on them).
void backward_jobs(const hot_layer_t& l, const Plan& p, const void* go, int64_t ldgo, const void* w, int64_t ldw, uint8_t* base, bool row,
                   bool col, void* sum, TileJob& jgo, TileJob& jw) {
  const hot_linear_cfg_t& c = l.cfg;
  jgo = TileJob();
  jgo.x = go;
  jgo.ldx = ldgo;
  jgo.batch = p.batch;
  jgo.rows = l.L;
  jgo.channels = l.O;
  jgo.row = row;
  jgo.order_row = c.order_o;
  jgo.q_row = c.q_gx;
  jgo.codes_row = base + p.off_qgo;
  jgo.ld_row = p.ld_qgo;
  jgo.scale_row = (float*)(base + p.off_sgo);
  jgo.col = col;
  jgo.order_col = c.order_l;
  jgo.rank = c.rank_l;
  jgo.sel = c.sel_l;
  jgo.q_col = c.q_gw;
  jgo.codes_col = base + p.off_qgw;
  jgo.ld_col = p.ld_qgw;
  jgo.sample_pitch = p.pitch;
  jgo.scale_col = (float*)(base + p.off_sgw);
  jgo.sum = sum;
  jw = TileJob();
  jw.x = w;
  jw.ldx = ldw;
  jw.rows = l.O;
  jw.channels = l.I;
  jw.col = true;
  jw.order_col = jw.rank = c.order_o;
  jw.q_col = c.q_w;
  jw.q_col.storage = HOT_STORE_INT8;  // the B operand of every CTA of the g_x product: reaches the tensor core by TMA alone
  jw.codes_col = base + p.off_qw;
  jw.ld_col = p.ld_qw;
  jw.scale_col = (float*)(base + p.off_sw);
}

int make_plan(const hot_layer_t& l, Plan& p) {
  const hot_linear_cfg_t& c = l.cfg;
  if (c.order_l < 1 || c.rank_l < 1 || c.rank_l > c.order_l || l.L % c.order_l != 0)
    HOT_FAIL(HOT_ERR_ARG, "hot_linear: tokens %lld not a multiple of the low-rank order %d (rank %d)", (long long)l.L, c.order_l, c.rank_l);
  const bool batched = l.batch > 0;
  p.batch = batched ? l.batch : 1;
  p.rows = p.batch * l.L;
  p.lp = l.L / c.order_l * c.rank_l;
  p.pitch = batched ? sample_pitch(p.lp) : 0;
  p.ld_qgo = code_pitch(l.O, c.q_gx.storage);
  p.ld_qw = code_pitch(l.O, HOT_STORE_INT8);
  p.ld_qgw = batched ? p.batch * p.pitch : code_pitch(p.lp, c.q_gw.storage);
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += up(bytes, kAlign);
    return at;
  };
  const bool gw_row = c.q_gw.scale_mode == HOT_SCALE_ROW;
  p.off_qgo = take((size_t)p.rows * p.ld_qgo);
  p.off_sgo = take((size_t)(c.q_gx.scale_mode == HOT_SCALE_ROW ? p.rows : p.batch) * sizeof(float));
  p.off_qw = take((size_t)l.I * p.ld_qw);
  p.off_sw = take(sizeof(float));
  p.off_qgw = take((size_t)l.O * p.ld_qgw);
  p.off_sgw = take((size_t)p.batch * (gw_row ? l.O : 1) * sizeof(float));
  // scratch words: abs-max of grad_out per token (plain) or per sample, and per channel or per sample and channel; two tile
  // counters of the tensor-core pair; kRiderCounters of the GEMM; the weight quantiser's own
  const size_t front = (size_t)(batched ? p.batch : l.L) + (size_t)p.batch * (batched && !gw_row ? 1 : l.O) + 2 + kRiderCounters;
  p.w_words = (front + 1) / 2 * 2;
  p.off_words = take((p.w_words + hot_col_ht_quant_scratch_words(c.dtype, l.O, l.I, c.order_o, c.order_o, c.q_w.scale_mode) + 64) * sizeof(uint32_t));
  TileJob jobs[2];
  backward_jobs(l, p, nullptr, l.O, nullptr, l.I, nullptr, true, true, nullptr, jobs[0], jobs[1]);
  jobs[0].sum = &p;  // (any non-null: only its presence matters here)
  p.tiles_bytes = tile_scratch_bytes(jobs, 2);
  if (!batched && c.dtype == HOT_BF16 && c.order_l == 16) {  // the tensor-core pair's sums for the bias gradient take the same place
    const size_t sums = tc_sum_bytes(l.L, l.O);
    if (sums > p.tiles_bytes) p.tiles_bytes = sums;
  }
  p.off_tiles = take(p.tiles_bytes);
  p.gemm_bytes = 0;
  if (!batched) {  // the two products run one after the other, or in one launch, and share it
    const size_t g1 = hot_gemm_i8_workspace_bytes(l.L, l.I), g2 = hot_gemm_i8_workspace_bytes(l.O, l.I);
    p.gemm_bytes = g1 > g2 ? g1 : g2;
  }
  p.off_gemm = take(p.gemm_bytes);
  p.total = o;
  return HOT_OK;
}

int check_layer(const hot_layer_t* l, const char* who) {
  if (!l) HOT_FAIL(HOT_ERR_ARG, "%s: null pointer", who);
  if (l->batch < 0 || l->batch > 65535 || l->L <= 0 || l->O <= 0 || l->I <= 0) HOT_FAIL(HOT_ERR_ARG, "%s: bad shape", who);
  return HOT_OK;
}

// The activation buffer as a job of the tiled quantisers.
TileJob compress_job(const hot_layer_t& l, const void* x, int64_t ldx, void* x_q_t, float* scale_x) {
  const hot_linear_cfg_t& c = l.cfg;
  TileJob j;
  j.x = x;
  j.ldx = ldx;
  j.batch = l.batch ? l.batch : 1;
  j.rows = l.L;
  j.channels = l.I;
  j.col = true;
  j.order_col = c.order_l;
  j.rank = c.rank_l;
  j.sel = c.sel_l;
  j.q_col = c.q_x;
  if (l.batch) {
    j.q_col.storage = HOT_STORE_INT8;
    j.sample_pitch = sample_pitch(l.L / c.order_l * c.rank_l);
    j.ld_col = l.batch * j.sample_pitch;
  } else {
    j.ld_col = code_pitch(l.L / c.order_l * c.rank_l, c.q_x.storage);
  }
  j.codes_col = x_q_t;
  j.scale_col = scale_x;
  return j;
}

// The separate kernels, one operand after the other (the configurations the tiled pair does not cover).
int quantise_row_side(const hot_layer_t& l, const Plan& p, const void* go, int64_t ldgo, uint8_t* base, hot_stream_t stream) {
  const hot_linear_cfg_t& c = l.cfg;
  uint32_t* words = (uint32_t*)(base + p.off_words);
  float* s_go = (float*)(base + p.off_sgo);
  if (l.batch && c.q_gx.scale_mode == HOT_SCALE_TENSOR)
    return hot_row_ht_quant_batched(go, c.dtype, p.batch, l.L, l.O, ldgo, c.order_o, &c.q_gx, base + p.off_qgo, p.ld_qgo, s_go, words, stream);
  return hot_row_ht_quant(go, c.dtype, p.rows, l.O, ldgo, c.order_o, &c.q_gx, base + p.off_qgo, p.ld_qgo, s_go, words, stream);
}
int quantise_col_side(const hot_layer_t& l, const Plan& p, const void* go, int64_t ldgo, uint8_t* base, hot_stream_t stream) {
  const hot_linear_cfg_t& c = l.cfg;
  uint32_t* words = (uint32_t*)(base + p.off_words) + (l.batch ? p.batch : l.L);
  float* s_gw = (float*)(base + p.off_sgw);
  if (!l.batch)
    return hot_col_ht_quant(go, c.dtype, l.L, l.O, ldgo, c.order_l, c.sel_l, c.rank_l, &c.q_gw, HOT_LAYOUT_TRANSPOSED, base + p.off_qgw, p.ld_qgw,
                            s_gw, words, stream);
  hot_quant_t q = c.q_gw;
  q.storage = HOT_STORE_INT8;
  return hot_col_ht_quant_batched(go, c.dtype, p.batch, l.L, l.O, ldgo, c.order_l, c.sel_l, c.rank_l, &q, HOT_LAYOUT_TRANSPOSED, base + p.off_qgw,
                                  p.ld_qgw, p.pitch, s_gw, words, stream);
}
int quantise_weight(const hot_layer_t& l, const Plan& p, const void* w, int64_t ldw, uint8_t* base, hot_stream_t stream) {
  const hot_linear_cfg_t& c = l.cfg;
  int32_t ident[64];
  for (int i = 0; i < 64; ++i) ident[i] = i;
  hot_quant_t q = c.q_w;
  q.storage = HOT_STORE_INT8;
  return hot_col_ht_quant(w, c.dtype, l.O, l.I, ldw, c.order_o, ident, c.order_o, &q, HOT_LAYOUT_NATURAL, base + p.off_qw, p.ld_qw,
                          (float*)(base + p.off_sw), (uint32_t*)(base + p.off_words) + p.w_words, stream);
}

}  // namespace

int layer_backward(const hot_layer_t& l, const void* go, int64_t ldgo, const void* w, int64_t ldw, const void* x_q_t,
                   const float* scale_x, void* grad_x, int64_t ldgx, void* grad_w, int64_t ldgw, void* grad_b, void* workspace,
                   size_t workspace_bytes, uint32_t* status, cudaEvent_t quantised, hot_stream_t stream, const CompressArgs* compress,
                   const hot_conv_t* fold) {
  if (!go || !w || !x_q_t || !scale_x || !workspace) HOT_FAIL(HOT_ERR_ARG, "hot_linear_backward: null pointer");
  if (!grad_x && !grad_w) HOT_FAIL(HOT_ERR_ARG, "hot_linear_backward: no output requested");
  if (int rc = check_layer(&l, "hot_linear_backward")) return rc;
  const hot_linear_cfg_t& c = l.cfg;
  Plan p;
  if (int rc = make_plan(l, p)) return rc;
  if (workspace_bytes < p.total) HOT_FAIL(HOT_ERR_WORKSPACE, "hot_linear_backward: workspace %zu < %zu bytes", workspace_bytes, p.total);
  if (((uintptr_t)workspace) % kAlign != 0) HOT_FAIL(HOT_ERR_ARG, "hot_linear_backward: workspace must be 256-byte aligned");
  if (c.order_o < 1 || c.order_o > 64 || l.O % c.order_o != 0)
    HOT_FAIL(HOT_ERR_ARG, "hot_linear_backward: order_o %d does not divide O = %lld", c.order_o, (long long)l.O);
  // the two-moment clip is what the reference offers for the weight and the activation only
  if (c.q_gx.scale_mode == HOT_SCALE_SAWB || c.q_gw.scale_mode == HOT_SCALE_SAWB)
    HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_linear_backward: HOT_SCALE_SAWB is for the weight and the activation buffer, not for grad_out");
  if (grad_x && c.q_w.scale_mode == HOT_SCALE_ROW) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_linear_backward: the weight takes one scale");
  if (int rc = validate_quant(&c.q_gx, "hot_linear_backward")) return rc;
  if (int rc = validate_quant(&c.q_gw, "hot_linear_backward")) return rc;
  if (int rc = validate_quant(&c.q_w, "hot_linear_backward")) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* base = (uint8_t*)workspace;
  uint32_t* words = (uint32_t*)(base + p.off_words);
  float *s_go = (float*)(base + p.off_sgo), *s_w = (float*)(base + p.off_sw), *s_gw = (float*)(base + p.off_sgw);
  const bool gx_row = c.q_gx.scale_mode == HOT_SCALE_ROW;
  hot_quant_t q_w8 = c.q_w;
  q_w8.storage = HOT_STORE_INT8;
  bool counters_cleared = false;

  auto compress_alone = [&]() {
    return compress ? hot_layer_compress(&l, compress->x, compress->ldx, compress->x_q_t, compress->scale_x, compress->workspace,
                                         compress->workspace_bytes, stream)
                    : HOT_OK;
  };
  const bool tc = !l.batch && grad_x && grad_w && use_tc(l.L, l.O, ldgo, c) && ((uintptr_t)go) % 16 == 0;
  if (tc) {
    if (int rc = compress_alone()) return rc;
    // HOT_WEIGHT_QUANT=separate keeps the weight out of these launches (the parity tests compare the two)
    const char* env = getenv("HOT_WEIGHT_QUANT");
    const bool rides = c.q_w.scale_mode == HOT_SCALE_TENSOR && tc_weight_job_supported(l.O, l.I, ldw, q_w8) && !(env && env[0] == 's');
    const TcWeightJob wj = {w, ldw, l.I, q_w8, base + p.off_qw, p.ld_qw, s_w, words + p.w_words};
    if (!rides)
      if (int rc = quantise_weight(l, p, w, ldw, base, stream)) return rc;
    // counters: two for the tile hand-out, and the GEMM's behind them, cleared along
    if (int rc = go_dual_quant_tc(go, l.L, l.O, ldgo, c.q_gx, c.q_gw, base + p.off_qgo, p.ld_qgo, s_go, base + p.off_qgw, p.ld_qgw, s_gw, words,
                                  words + l.L, words + l.L + l.O, 2 + kRiderCounters, status, st, rides ? &wj : nullptr, false,
                                  grad_b ? (float*)(base + p.off_tiles) : nullptr, grad_b))
      return rc;
    counters_cleared = true;
  } else {
    TileJob jgo, jw, jobs[2];
    int count = 0;
    bool row = grad_x && !gx_row, col = grad_w != nullptr;
    auto covered = [&](bool r, bool k) {
      TileJob a, b;
      backward_jobs(l, p, go, ldgo, w, ldw, base, r, k, nullptr, a, b);
      return tile_job_covered(a, c.dtype);
    };
    if (row && !covered(true, false)) row = false;
    if (col && !covered(false, true)) col = false;
    backward_jobs(l, p, go, ldgo, w, ldw, base, row, col, grad_b, jgo, jw);
    const bool sum_only = grad_b && !row && !col;
    jgo.times16 = row && c.q_gx.bits == 4 && c.q_gx.rounding == HOT_ROUND_STOCH_PHILOX && c.q_gx.storage == HOT_STORE_INT8;
    if (row || col || sum_only) {
      if (!tile_job_covered(jgo, c.dtype)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_layer_backward: grad_b is not made for this grad_out (see hot_layer_sums_rows)");
      jobs[count++] = jgo;
    }
    const bool weight = grad_x && tile_job_covered(jw, c.dtype);
    if (weight) jobs[count++] = jw;
    // the activation buffer shares the launches of a grad_out job of its kind: a small call is launches more than work
    TileJob jx;
    bool shared = false;
    if (compress && col) {
      jx = compress_job(l, compress->x, compress->ldx, compress->x_q_t, compress->scale_x);
      shared = c.q_x.scale_mode != HOT_SCALE_ROW && tile_job_covered(jx, c.dtype) && tile_jobs_alike(jgo, jx) &&
               tile_scratch_bytes(&jx, 1) <= compress->workspace_bytes && validate_quant(&c.q_x, "hot_hlq_backward") == HOT_OK;
    }
    if (!shared)
      if (int rc = compress_alone()) return rc;
    if (count)
      if (int rc = launch_tile_jobs(jobs, count, c.dtype, base + p.off_tiles, p.tiles_bytes, st, shared ? &jx : nullptr,
                                    shared ? compress->workspace : nullptr))
        return rc;
    if (grad_x && !row)
      if (int rc = quantise_row_side(l, p, go, ldgo, base, stream)) return rc;
    if (grad_x && !weight)
      if (int rc = quantise_weight(l, p, w, ldw, base, stream)) return rc;
    if (grad_w && !col)
      if (int rc = quantise_col_side(l, p, go, ldgo, base, stream)) return rc;
  }
  if (quantised) HOT_CUDA(cudaEventRecord(quantised, st));

  const float post_x = 1.0f / (float)c.order_o, post_w = 1.0f / (float)c.order_l;
  const int rows_per_scale = gx_row ? 1 : (l.batch ? (int)l.L : 0);
  if (fold && grad_x) {
    if (int rc = conv_grad_input(l, *fold, base + p.off_qgo, p.ld_qgo, s_go, base + p.off_qw, p.ld_qw, s_w, post_x, grad_x, status, st)) return rc;
    grad_x = nullptr;
  }
  if (l.batch) {
    if (grad_x)
      if (int rc = hot_gemm_i8(base + p.off_qgo, c.q_gx.storage, p.ld_qgo, base + p.off_qw, HOT_STORE_INT8, p.ld_qw, p.rows, l.I, l.O, s_go,
                               rows_per_scale, s_w, 0, post_x, grad_x, c.dtype, ldgx, status, stream))
        return rc;
    if (grad_w)
      return gemm_i8_grouped(base + p.off_qgw, p.ld_qgw, x_q_t, p.ld_qgw, l.O, l.I, l.batch, p.pitch, p.lp, s_gw,
                             c.q_gw.scale_mode == HOT_SCALE_ROW, scale_x, post_w, grad_w, c.dtype, ldgw, status, stream);
    return HOT_OK;
  }
  const int gw_row = c.q_gw.scale_mode == HOT_SCALE_ROW;
  const int64_t ld_xq = hot_abc_pitch(l.L, &c);
  void* gemm_ws = p.gemm_bytes ? base + p.off_gemm : nullptr;
  if (grad_x && grad_w && c.q_gw.storage == HOT_STORE_INT8 && c.q_x.storage == HOT_STORE_INT8) {
    // both products in one launch: the few long g_w tiles run in the SMs that the last wave of g_x tiles leaves idle
    hot_gemm_problem_t gx = {base + p.off_qgo, c.q_gx.storage, p.ld_qgo, base + p.off_qw, p.ld_qw, l.L, l.I, l.O, s_go, gx_row,
                             s_w, 0, post_x, grad_x, c.dtype, ldgx};
    hot_gemm_problem_t gw = {base + p.off_qgw, HOT_STORE_INT8, p.ld_qgw, x_q_t, ld_xq, l.O, l.I, p.lp, s_gw, gw_row,
                             scale_x, 0, post_w, grad_w, c.dtype, ldgw};
    return gemm_i8_dual_ws(&gx, &gw, gemm_ws, p.gemm_bytes, words + l.L + l.O + 2, counters_cleared ? 0 : kRiderCounters, status, stream);
  }
  if (grad_x)
    if (int rc = hot_gemm_i8_ws(base + p.off_qgo, c.q_gx.storage, p.ld_qgo, base + p.off_qw, HOT_STORE_INT8, p.ld_qw, l.L, l.I, l.O, s_go, gx_row,
                                s_w, 0, post_x, grad_x, c.dtype, ldgx, gemm_ws, p.gemm_bytes, status, stream))
      return rc;
  if (grad_w)
    if (int rc = hot_gemm_i8_ws(base + p.off_qgw, c.q_gw.storage, p.ld_qgw, x_q_t, c.q_x.storage, ld_xq, l.O, l.I, p.lp, s_gw, gw_row, scale_x, 0,
                                post_w, grad_w, c.dtype, ldgw, gemm_ws, p.gemm_bytes, status, stream))
      return rc;
  return HOT_OK;
}

namespace {

// Events and the status word of hot_hlq_backward, one set per host thread and device, made on first use and
// given back when the thread ends.  The word lies in pinned host memory that the kernels can reach: it is only ever
// written when a bounded wait runs out, and reading it after the stream has drained costs no copy.
struct CallKit {
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  uint32_t* status = nullptr;
};
struct CallKits {
  CallKit kit[kMaxDevices];
  ~CallKits() {
    for (CallKit& k : kit) {
      for (cudaEvent_t e : k.ev)
        if (e) cudaEventDestroy(e);
      if (k.status) cudaFreeHost(k.status);
    }
  }
};

int call_kit(CallKit** out) {
  static thread_local CallKits kits;
  int dev = -1;
  HOT_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_hlq_backward: device ordinal %d", dev);
  CallKit& k = kits.kit[dev];
  for (cudaEvent_t& e : k.ev)
    if (!e) HOT_CUDA(cudaEventCreate(&e));
  if (!k.status) {
    HOT_CUDA(cudaHostAlloc((void**)&k.status, sizeof(uint32_t), cudaHostAllocMapped | cudaHostAllocPortable));
    *k.status = 0;
  }
  *out = &k;
  return HOT_OK;
}

}  // namespace
}  // namespace hot

extern "C" int64_t hot_layer_buffer_pitch(const hot_layer_t* layer) {
  using namespace hot;
  if (check_layer(layer, "hot_layer_buffer_pitch")) return 0;
  const hot_linear_cfg_t& c = layer->cfg;
  if (c.order_l < 1 || layer->L % c.order_l != 0) return 0;
  return layer->batch ? layer->batch * sample_pitch(layer->L / c.order_l * c.rank_l) : hot_abc_pitch(layer->L, &c);
}

extern "C" size_t hot_layer_compress_workspace_bytes(const hot_layer_t* layer) {
  using namespace hot;
  if (check_layer(layer, "hot_layer_compress_workspace_bytes")) return 0;
  const hot_linear_cfg_t& c = layer->cfg;
  const size_t words = hot_col_ht_quant_scratch_words(c.dtype, layer->L, layer->I, c.order_l, c.rank_l, c.q_x.scale_mode);
  if (words == 0) return 0;
  const TileJob job = compress_job(*layer, nullptr, layer->I, nullptr, nullptr);
  const size_t tiles = tile_scratch_bytes(&job, 1), plain = sizeof(uint32_t) * (words * (size_t)(layer->batch ? layer->batch : 1) + 16);
  return up(tiles > plain ? tiles : plain, kAlign);
}

extern "C" int hot_layer_compress(const hot_layer_t* layer, const void* x, int64_t ldx, void* x_q_t, float* scale_x, void* workspace,
                                  size_t workspace_bytes, hot_stream_t stream) {
  using namespace hot;
  if (int rc = check_layer(layer, "hot_layer_compress")) return rc;
  if (!x || !x_q_t || !scale_x || !workspace) HOT_FAIL(HOT_ERR_ARG, "hot_layer_compress: null pointer");
  const hot_linear_cfg_t& c = layer->cfg;
  const size_t need = hot_layer_compress_workspace_bytes(layer);
  if (need == 0 || workspace_bytes < need) HOT_FAIL(HOT_ERR_WORKSPACE, "hot_layer_compress: workspace %zu < %zu bytes", workspace_bytes, need);
  if (int rc = validate_quant(&c.q_x, "hot_layer_compress")) return rc;
  const bool tc = !layer->batch && abc_tc_supported(layer->L, layer->I, ldx, c.dtype, c.order_l, c.rank_l, c.sel_l, c.q_x);
  const TileJob job = compress_job(*layer, x, ldx, x_q_t, scale_x);
  if (!tc && c.q_x.scale_mode != HOT_SCALE_ROW && tile_job_covered(job, c.dtype))
    return launch_tile_jobs(&job, 1, c.dtype, workspace, workspace_bytes, (cudaStream_t)stream);
  if (!layer->batch) return hot_abc_compress(x, layer->L, layer->I, ldx, &c, x_q_t, scale_x, workspace, workspace_bytes, stream);
  return hot_col_ht_quant_batched(x, c.dtype, layer->batch, layer->L, layer->I, ldx, c.order_l, c.sel_l, c.rank_l, &job.q_col,
                                  HOT_LAYOUT_NATURAL, x_q_t, job.ld_col, job.sample_pitch, scale_x, (uint32_t*)workspace, stream);
}

extern "C" size_t hot_layer_backward_workspace_bytes(const hot_layer_t* layer) {
  using namespace hot;
  if (check_layer(layer, "hot_layer_backward_workspace_bytes")) return 0;
  Plan p;
  return make_plan(*layer, p) ? 0 : p.total;
}

extern "C" int hot_layer_sums_rows(const hot_layer_t* layer, const void* go) {
  using namespace hot;
  Plan p;
  if (check_layer(layer, "hot_layer_sums_rows") || make_plan(*layer, p)) return 0;
  TileJob jgo, jw;
  backward_jobs(*layer, p, go, layer->O, nullptr, layer->I, nullptr, false, false, &p, jgo, jw);  // (any non-null sum)
  return tile_job_covered(jgo, layer->cfg.dtype) ? 1 : 0;
}

extern "C" int hot_layer_backward(const hot_layer_t* layer, const void* go, const void* w, int64_t ldw, const void* x_q_t,
                                  const float* scale_x, void* grad_x, int64_t ldgx, void* grad_w, int64_t ldgw, void* grad_b, void* workspace,
                                  size_t workspace_bytes, uint32_t* status_word, hot_stream_t stream) {
  using namespace hot;
  if (!layer) HOT_FAIL(HOT_ERR_ARG, "hot_layer_backward: null pointer");
  return layer_backward(*layer, go, layer->O, w, ldw, x_q_t, scale_x, grad_x, ldgx, grad_w, ldgw, grad_b, workspace, workspace_bytes,
                        status_word, nullptr, stream);
}

extern "C" int hot_layer_backward_conv(const hot_layer_t* layer, const hot_conv_t* conv, const void* go, const void* w, int64_t ldw,
                                       const void* x_q_t, const float* scale_x, void* grad_x, void* grad_w, int64_t ldgw, void* grad_b,
                                       void* workspace, size_t workspace_bytes, uint32_t* status_word, hot_stream_t stream) {
  using namespace hot;
  if (!layer || !conv) HOT_FAIL(HOT_ERR_ARG, "hot_layer_backward_conv: null pointer");
  if (!conv_fold_covered(*layer, *conv)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_layer_backward_conv: not covered (see hot_conv_folds)");
  return layer_backward(*layer, go, layer->O, w, ldw, x_q_t, scale_x, grad_x, layer->I, grad_w, ldgw, grad_b, workspace, workspace_bytes,
                        status_word, nullptr, stream, nullptr, conv);
}

namespace hot {
namespace {
// workspace of hot_hlq_backward: activation buffer | its scale | compression scratch | backward
struct HlqPlan {
  hot_layer_t layer;
  int64_t pitch;
  size_t off_sx, off_cws, cws, off_bws, bws, total;
};
int hlq_plan(int64_t L, int64_t O, int64_t I, const hot_linear_cfg_t* cfg, HlqPlan& p) {
  p.layer = hot_layer_t{0, L, O, I, *cfg};
  p.pitch = hot_layer_buffer_pitch(&p.layer);
  p.bws = hot_layer_backward_workspace_bytes(&p.layer);
  p.cws = hot_layer_compress_workspace_bytes(&p.layer);
  if (p.pitch <= 0 || p.bws == 0 || p.cws == 0)
    HOT_FAIL(HOT_ERR_ARG, "hot_hlq_backward: unsupported sizes L=%lld O=%lld I=%lld for this configuration", (long long)L, (long long)O, (long long)I);
  p.off_sx = up((size_t)I * p.pitch, kAlign);
  p.off_cws = p.off_sx + kAlign;
  p.off_bws = p.off_cws + p.cws;
  p.total = p.off_bws + p.bws;
  return HOT_OK;
}
}  // namespace
}  // namespace hot

extern "C" size_t hot_hlq_workspace_bytes(int64_t L, int64_t O, int64_t I, const hot_linear_cfg_t* cfg) {
  hot::HlqPlan p;
  if (!cfg || L <= 0 || O <= 0 || I <= 0 || hot::hlq_plan(L, O, I, cfg, p)) return 0;
  return p.total;
}

extern "C" int hot_hlq_backward(const void* go, const void* w, const void* x, int64_t L, int64_t O, int64_t I,
                                const hot_linear_cfg_t* cfg, void* grad_x, void* grad_w, void* workspace, size_t workspace_bytes,
                                float* stage_ms, hot_stream_t stream) {
  using namespace hot;
  if (!go || !w || !x || !cfg || !grad_x || !grad_w || !workspace || !stage_ms) HOT_FAIL(HOT_ERR_ARG, "hot_hlq_backward: null pointer");
  HlqPlan p;
  if (int rc = hlq_plan(L, O, I, cfg, p)) return rc;
  if (workspace_bytes < p.total || ((uintptr_t)workspace) % kAlign != 0)
    HOT_FAIL(HOT_ERR_WORKSPACE, "hot_hlq_backward: workspace needs %zu bytes, 256-byte aligned (got %zu)", p.total, workspace_bytes);
  CallKit* kit = nullptr;
  if (int rc = call_kit(&kit)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* base = (uint8_t*)workspace;
  HOT_CUDA(cudaEventRecord(kit->ev[0], st));
  float* const scale_x = (float*)(base + p.off_sx);
  const CompressArgs compress = {x, I, base, scale_x, base + p.off_cws, p.cws};
  const int rc = layer_backward(p.layer, go, O, w, I, base, scale_x, grad_x, I, grad_w, I, nullptr, base + p.off_bws, p.bws, kit->status, kit->ev[1],
                                stream, &compress);
  if (rc) {  // refused after launches perhaps: they may still write the status word, which the thread's next call reads
    cudaStreamSynchronize(st);
    *kit->status = 0;
    return rc;
  }
  HOT_CUDA(cudaEventRecord(kit->ev[2], st));
  HOT_CUDA(cudaStreamSynchronize(st));
  const uint32_t status = *kit->status;
  *kit->status = 0;
  if (status) return hot_check_status(status);
  HOT_CUDA(cudaEventElapsedTime(&stage_ms[0], kit->ev[0], kit->ev[1]));
  HOT_CUDA(cudaEventElapsedTime(&stage_ms[1], kit->ev[1], kit->ev[2]));
  return HOT_OK;
}
