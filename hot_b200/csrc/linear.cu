// The C entry points of one linear layer on plain (2-D) tensors: activation-buffer compression, the fused grad_out
// quantisers, and the backward, which layer.cu composes.  All intermediates live in a caller-owned workspace; nothing here
// allocates or synchronises.
#include <cstdlib>

#include "layer.cuh"

namespace hot {

bool go_dual_supported(int64_t L, int64_t O, int64_t ldgo, int dtype, int order_o, int order_l, int rank_l,
                       const int32_t* sel_l, const hot_quant_t& q_gx, const hot_quant_t& q_gw);
int go_dual_quant(const void* go, int dtype, int64_t L, int64_t O, int64_t ldgo, int order_o, const int32_t* sel_l,
                  const hot_quant_t& q_gx, const hot_quant_t& q_gw, void* q_go, int64_t ld_qgo, float* s_gx, void* q_gw_t,
                  int64_t ld_qgw, float* s_gw, uint32_t* max_x, uint32_t* max_w, uint32_t* status, cudaStream_t st);

// Which fused grad_out kernels serve a call: the tensor-core pair where it covers the configuration,
// else the butterfly pair.  HOT_GO_DUAL=butterfly keeps the tensor-core pair out (the parity tests
// compare the two).
bool use_tc(int64_t L, int64_t O, int64_t ldgo, const hot_linear_cfg_t& c) {
  const char* env = getenv("HOT_GO_DUAL");
  if (env && env[0] == 'b') return false;
  return go_dual_tc_supported(L, O, ldgo, c.dtype, c.order_o, c.order_l, c.rank_l, c.sel_l, c.q_gx, c.q_gw);
}

}  // namespace hot

extern "C" size_t hot_linear_workspace_bytes(int64_t L, int64_t O, int64_t I, const hot_linear_cfg_t* cfg) {
  if (!cfg || L <= 0 || O <= 0 || I <= 0) return 0;
  const hot_layer_t layer = {0, L, O, I, *cfg};
  return hot_layer_backward_workspace_bytes(&layer);
}

extern "C" int64_t hot_abc_pitch(int64_t L, const hot_linear_cfg_t* cfg) {
  if (!cfg || cfg->order_l < 1 || L % cfg->order_l != 0) return 0;
  const int64_t codes = L / cfg->order_l * cfg->rank_l;
  return ((cfg->q_x.storage == HOT_STORE_INT4 ? (codes + 1) / 2 : codes) + 15) / 16 * 16;
}

extern "C" int hot_abc_compress(const void* x, int64_t L, int64_t I, int64_t ldx, const hot_linear_cfg_t* cfg,
                                void* x_q_t, float* scale_x, void* workspace, size_t workspace_bytes,
                                hot_stream_t stream) {
  using namespace hot;
  if (!x || !cfg || !x_q_t || !scale_x || !workspace) HOT_FAIL(HOT_ERR_ARG, "hot_abc_compress: null pointer");
  if (cfg->q_x.scale_mode == HOT_SCALE_ROW) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_abc_compress: the activation buffer takes one scale");
  const size_t need = 4 * hot_col_ht_quant_scratch_words(cfg->dtype, L, I, cfg->order_l, cfg->rank_l, cfg->q_x.scale_mode);
  if (need == 0 || workspace_bytes < need || ((uintptr_t)workspace) % 8 != 0)
    HOT_FAIL(HOT_ERR_WORKSPACE, "hot_abc_compress: workspace needs %zu bytes, 8-byte aligned (got %zu)", need, workspace_bytes);
  const int64_t pitch = hot_abc_pitch(L, cfg);
  if (pitch == 0) HOT_FAIL(HOT_ERR_ARG, "hot_abc_compress: tokens %lld not a multiple of the low-rank order %d", (long long)L, cfg->order_l);
  // bf16 with the order-16 token basis: the token side of the tensor-core grad_out kernels on its own (same codes as
  // the butterfly kernel below unless a 16-term sum is inexact in fp32; HOT_ABC=butterfly keeps that kernel).
  // Workspace words: 0 abs-max, 1-2 tile counters, 3 status (non-zero afterwards: a device-side wait ran out).
  const char* abc_env = getenv("HOT_ABC");
  if (workspace_bytes >= 16 && !(abc_env && abc_env[0] == 'b') && pitch % 16 == 0 && ((uintptr_t)x_q_t) % 16 == 0 &&
      ((uintptr_t)x) % 16 == 0 && abc_tc_supported(L, I, ldx, cfg->dtype, cfg->order_l, cfg->rank_l, cfg->sel_l, cfg->q_x)) {
    if (int rc = validate_quant(&cfg->q_x, "hot_abc_compress")) return rc;
    uint32_t* wsw = (uint32_t*)workspace;
    return go_dual_quant_tc(x, L, I, ldx, cfg->q_x, cfg->q_x, nullptr, 0, nullptr, x_q_t, pitch, scale_x, nullptr, wsw, wsw + 1, 3, wsw + 3,
                            (cudaStream_t)stream, nullptr, true);
  }
  return hot_col_ht_quant(x, cfg->dtype, L, I, ldx, cfg->order_l, cfg->sel_l, cfg->rank_l, &cfg->q_x, HOT_LAYOUT_NATURAL,
                          x_q_t, pitch, scale_x, (uint32_t*)workspace, stream);
}

extern "C" int hot_go_dual_quant(const void* go, int64_t L, int64_t O, int64_t ldgo, const hot_linear_cfg_t* cfg, void* q_go,
                                 int64_t ld_qgo, float* s_gx, void* q_gw_t, int64_t ld_qgw, float* s_gw,
                                 uint32_t* scratch, uint32_t* status_word, hot_stream_t stream) {
  using namespace hot;
  if (!go || !cfg || !q_go || !s_gx || !q_gw_t || !s_gw || !scratch) HOT_FAIL(HOT_ERR_ARG, "hot_go_dual_quant: null pointer");
  if (L <= 0 || O <= 0) HOT_FAIL(HOT_ERR_ARG, "hot_go_dual_quant: bad shape");
  if (int rc = validate_quant(&cfg->q_gx, "hot_go_dual_quant")) return rc;
  if (int rc = validate_quant(&cfg->q_gw, "hot_go_dual_quant")) return rc;
  if (!go_dual_supported(L, O, ldgo, cfg->dtype, cfg->order_o, cfg->order_l, cfg->rank_l, cfg->sel_l, cfg->q_gx, cfg->q_gw))
    HOT_FAIL(HOT_ERR_UNSUPPORTED,
             "hot_go_dual_quant covers: low-rank basis = 8 lowest-sequency rows of H_16, tokens %% 32 == 0, channels %% 64 == 0, "
             "INT8 storage on the g_w side, nearest or Philox rounding");
  const int64_t need_x = cfg->q_gx.storage == HOT_STORE_INT4 ? O / 2 : O;
  if (ld_qgo < need_x || ld_qgo % 16 || ld_qgw < L / 2 || ld_qgw % 16 || ((uintptr_t)q_go) % 16 || ((uintptr_t)q_gw_t) % 16 ||
      ((uintptr_t)go) % 16)
    HOT_FAIL(HOT_ERR_ARG, "hot_go_dual_quant: buffers and pitches must be 16-byte aligned and cover the codes");
  if (use_tc(L, O, ldgo, *cfg))
    return go_dual_quant_tc(go, L, O, ldgo, cfg->q_gx, cfg->q_gw, q_go, ld_qgo, s_gx, q_gw_t, ld_qgw, s_gw, scratch, scratch + L, scratch + L + O, 2,
                            status_word, (cudaStream_t)stream, nullptr, false);
  return go_dual_quant(go, cfg->dtype, L, O, ldgo, cfg->order_o, cfg->sel_l, cfg->q_gx, cfg->q_gw, q_go, ld_qgo, s_gx, q_gw_t, ld_qgw, s_gw, scratch,
                       scratch + L, status_word, (cudaStream_t)stream);
}

extern "C" int hot_linear_backward(const void* go, int64_t ldgo, const void* w, int64_t ldw, const void* x_q_t,
                                   const float* scale_x, int64_t L, int64_t O, int64_t I, const hot_linear_cfg_t* cfg,
                                   void* grad_x, int64_t ldgx, void* grad_w, int64_t ldgw, void* workspace,
                                   size_t workspace_bytes, uint32_t* status_word, hot_stream_t stream) {
  using namespace hot;
  if (!cfg) HOT_FAIL(HOT_ERR_ARG, "hot_linear_backward: null pointer");
  if (cfg->order_o > 16) HOT_FAIL(HOT_ERR_ARG, "hot_linear_backward: order_o %d outside [1, 16]", cfg->order_o);  // (the extension call takes up to 64)
  const hot_layer_t layer = {0, L, O, I, *cfg};
  return layer_backward(layer, go, ldgo, w, ldw, x_q_t, scale_x, grad_x, ldgx, grad_w, ldgw, nullptr, workspace, workspace_bytes, status_word,
                        nullptr, stream);
}
