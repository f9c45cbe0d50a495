// What linear.cu and layer.cu share.
#pragma once

#include "common.cuh"

namespace hot {

// Whether the tensor-core grad_out kernels serve a call (HOT_GO_DUAL=butterfly keeps them out, for the parity tests).
bool use_tc(int64_t L, int64_t O, int64_t ldgo, const hot_linear_cfg_t& c);
bool tc_weight_job_supported(int64_t O, int64_t I, int64_t ldw, const hot_quant_t& q_w);
int go_dual_quant_tc(const void* go, int64_t L, int64_t O, int64_t ldgo, const hot_quant_t& q_gx, const hot_quant_t& q_gw,
                     void* q_go, int64_t ld_qgo, float* s_gx, void* q_gw_t, int64_t ld_qgw, float* s_gw, uint32_t* max_x,
                     uint32_t* max_w, uint32_t* counters, size_t counter_words, uint32_t* status, cudaStream_t st,
                     const TcWeightJob* wj, bool col_only, float* part_sum = nullptr, void* sum = nullptr);
// sum (nullable, bf16): the sum of grad_out over its rows; part_sum is scratch for it of this size.
size_t tc_sum_bytes(int64_t L, int64_t O);
bool abc_tc_supported(int64_t L, int64_t I, int64_t ldx, int dtype, int order_l, int rank_l, const int32_t* sel_l,
                      const hot_quant_t& q_x);
bool go_dual_tc_supported(int64_t L, int64_t O, int64_t ldgo, int dtype, int order_o, int order_l, int rank_l,
                          const int32_t* sel_l, const hot_quant_t& q_gx, const hot_quant_t& q_gw);

// The activation buffer as part of a backward that has x at hand: what hot_layer_compress takes.
struct CompressArgs {
  const void* x;
  int64_t ldx;
  void* x_q_t;
  float* scale_x;
  void* workspace;
  size_t workspace_bytes;
};

// The input gradient of a convolution, folded by the product that makes it (gemm_conv.cu).
bool conv_fold_covered(const hot_layer_t& layer, const hot_conv_t& conv);
int conv_grad_input(const hot_layer_t& layer, const hot_conv_t& conv, const void* q_go, int64_t ld_go, const float* s_go, const void* q_w, int64_t ld_w,
                    const float* s_w, float post, void* out, uint32_t* status, cudaStream_t st);

// The backward of one layer.  fold (nullable): grad_x is that convolution's input gradient, not the rows'.  compress (nullable): the buffer (x_q_t, scale_x) is made first.  grad_b (nullable): the sum of go over its rows, in the tensors' type.  quantised
// (nullable): an event recorded between the quantisers and the products.
int layer_backward(const hot_layer_t& layer, const void* go, int64_t ldgo, const void* w, int64_t ldw, const void* x_q_t,
                   const float* scale_x, void* grad_x, int64_t ldgx, void* grad_w, int64_t ldgw, void* grad_b, void* workspace,
                   size_t workspace_bytes, uint32_t* status_word, cudaEvent_t quantised, hot_stream_t stream,
                   const CompressArgs* compress = nullptr, const hot_conv_t* fold = nullptr);

}  // namespace hot
