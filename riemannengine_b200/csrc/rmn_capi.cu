// C-ABI entry points of the convolution passes: argument checks and dispatch
// between the tensor-core (tcgen05, bf16) and SIMT (fp32 / odd shapes) kernels.
#include "rmn_common.cuh"

namespace rmn {
int simt_conv_forward(const void* feats, int c_in, const void* w, int K, int c_out,
                      const int32_t* nbr, uint32_t n_dst, void* out, int dtype, const float* ep_scale,
                      const float* ep_shift, int ep_relu, cudaStream_t stream);
int simt_conv_backward_input(const void* grad_out, int c_out, const void* w, int K, int c_in,
                             const int32_t* nbr_t, uint32_t n_src, void* grad_feats, int dtype,
                             cudaStream_t stream);
size_t simt_wgrad_workspace_bytes(uint32_t n_dst, int K, int c_in, int c_out);
int simt_conv_backward_weight(const void* feats, int c_in, const void* grad_out, uint32_t n_dst,
                              int c_out, const int32_t* nbr, int K, float* dw, int dtype,
                              void* workspace, cudaStream_t stream);
int tc_conv(const void* src, uint32_t n_src, const void* w, const int32_t* nbr, uint32_t n_dst, int K, int c_red,
            int c_col, bool transposed_weights, void* out, const float* ep_scale, const float* ep_shift, int ep_relu,
            cudaStream_t stream, const void* plan);
size_t ta_image_bytes(int K, int c_red, int c_col);
int ta_weight_image(const void* w, int K, int w_red, int w_col, int c_red, int c_col, int transpose, int reverse,
                    const rmn_bn_fold& fold, void* image, cudaStream_t stream);
int ta_conv(const void* src, const void* image, const int32_t* nbr, uint32_t n_dst, int K, int c_red, int c_col, void* out,
            const float* ep_scale, const float* ep_shift, const void* ep_add, int ep_relu, float* stats_partial,
            uint32_t* n_partials, cudaStream_t stream, const void* plan, const int32_t* order);
int ta_weight_images(const rmn_weight_job* jobs, int n_jobs, cudaStream_t stream);
int tc_read_status(cudaStream_t stream, uint32_t* status);
unsigned long long tc_launch_count();
int tc_conv_wgrad(const void* feats, const void* grad_out, const int32_t* nbr, uint32_t n_dst, int K, int c_in,
                  int c_out, float* dw, void* workspace, size_t workspace_bytes, size_t* need,
                  cudaStream_t stream);
}  // namespace rmn

#include <atomic>
#include <cstdlib>

namespace rmn {
static std::atomic<unsigned long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
}  // namespace rmn

using namespace rmn;

extern "C" unsigned long long rmn_launch_count(void) {
  return g_launches.load(std::memory_order_relaxed);
}

extern "C" unsigned long long rmn_tensor_core_launch_count(void) { return tc_launch_count(); }

extern "C" int rmn_version(void) { return 100; }

extern "C" const char* rmn_status_string(int status) {
  switch (status) {
    case RMN_OK: return "ok";
    case RMN_ERR_BAD_ARG: return "bad argument";
    case RMN_ERR_ALLOC: return "caller-provided buffer too small";
    case RMN_ERR_PROBE_LIMIT: return "hash probe limit reached (table full)";
    case RMN_ERR_TIMEOUT: return "bounded device wait ran out";
    case RMN_ERR_CUDA: return "CUDA runtime error";
    case RMN_ERR_RANGE: return "coordinate bounding box does not pack into 63 bits";
    case RMN_ERR_UNSUPPORTED: return "unsupported shape or dtype";
    case RMN_ERR_TOO_LARGE: return "size exceeds the fixed capacity of the allocation-free entry point";
    default: return "unknown status";
  }
}


extern "C" int rmn_device_status(void* stream_) {
  uint32_t st = 0;
  const int rc = tc_read_status((cudaStream_t)stream_, &st);
  return rc != RMN_OK ? rc : (int)st;
}

static bool conv_args_ok(const void* a, const void* w, const int32_t* nbr, const void* out, int K,
                         int c_in, int c_out, int dtype) {
  return a && w && nbr && out && K >= 1 && K <= 65535 && c_in >= 1 && c_out >= 1 &&
         c_in <= 65536 && c_out <= 65536 && (dtype == RMN_F32 || dtype == RMN_BF16);
}

extern "C" int rmn_conv_forward_fused(const void* d_feats, uint32_t n_src, int c_in, const void* d_weights, int K,
                                      int c_out, const int32_t* d_nbr, uint32_t n_dst, void* d_out, int dtype,
                                      const float* d_scale, const float* d_shift, int relu, void* stream_) {
  return rmn_conv_forward_planned(d_feats, n_src, c_in, d_weights, K, c_out, d_nbr, nullptr, n_dst, d_out, dtype,
                                  d_scale, d_shift, relu, stream_);
}

extern "C" int rmn_conv_forward_planned(const void* d_feats, uint32_t n_src, int c_in, const void* d_weights, int K,
                                        int c_out, const int32_t* d_nbr, const void* d_plan, uint32_t n_dst,
                                        void* d_out, int dtype, const float* d_scale, const float* d_shift, int relu,
                                        void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n_dst == 0) return RMN_OK;
  if (!conv_args_ok(n_src ? d_feats : d_out, d_weights, d_nbr, d_out, K, c_in, c_out, dtype)) return RMN_ERR_BAD_ARG;
  if (dtype == RMN_BF16 && n_src > 0) {
    const int st = tc_conv(d_feats, n_src, d_weights, d_nbr, n_dst, K, c_in, c_out, false, d_out, d_scale, d_shift,
                           relu, stream, d_plan);
    if (st != RMN_ERR_UNSUPPORTED) return st;
  }
  // (with no source rows every neighbour entry is -1: the SIMT kernel then writes act(shift))
  return simt_conv_forward(d_feats, c_in, d_weights, K, c_out, d_nbr, n_dst, d_out, dtype, d_scale, d_shift, relu,
                           stream);
}

extern "C" int rmn_conv_forward(const void* d_feats, uint32_t n_src, int c_in,
                                const void* d_weights, int K, int c_out, const int32_t* d_nbr,
                                uint32_t n_dst, void* d_out, int dtype, void* stream_) {
  return rmn_conv_forward_fused(d_feats, n_src, c_in, d_weights, K, c_out, d_nbr, n_dst, d_out, dtype, nullptr,
                                nullptr, 0, stream_);
}

extern "C" size_t rmn_conv_weight_image_bytes(int K, int c_in, int c_out, int dtype) {
  if (K < 1 || K > 65535 || dtype != RMN_BF16) return 0;
  const size_t plain = ta_image_bytes(K, c_in, c_out), transposed = ta_image_bytes(K, c_out, c_in);
  return plain > transposed ? plain : transposed;  // (both orders of every pair have a kernel)
}

extern "C" int rmn_conv_weight_image(const void* d_weights, int K, int w_in, int w_out, int c_in, int c_out, int dtype,
                                     int transpose, int reverse, const rmn_bn_fold* fold, void* d_image, void* stream_) {
  if (!d_weights || !d_image || K < 1 || K > 65535 || ((uintptr_t)d_image & 15)) return RMN_ERR_BAD_ARG;
  if (w_in < 1 || w_in > c_in || w_out < 1 || w_out > c_out) return RMN_ERR_BAD_ARG;
  rmn_bn_fold f = {};
  if (fold) {
    f = *fold;
    if (transpose || !f.scale || !f.shift || (f.param_dtype != RMN_F32 && f.param_dtype != RMN_BF16)) return RMN_ERR_BAD_ARG;
  }
  if (rmn_conv_weight_image_bytes(K, c_in, c_out, dtype) == 0) return RMN_ERR_UNSUPPORTED;
  return transpose ? ta_weight_image(d_weights, K, w_out, w_in, c_out, c_in, 1, reverse, f, d_image, (cudaStream_t)stream_)
                   : ta_weight_image(d_weights, K, w_in, w_out, c_in, c_out, 0, reverse, f, d_image, (cudaStream_t)stream_);
}

extern "C" int rmn_conv_weight_images(const rmn_weight_job* jobs, int n_jobs, void* stream_) {
  if (n_jobs < 0 || (n_jobs > 0 && !jobs)) return RMN_ERR_BAD_ARG;
  for (int j = 0; j < n_jobs; ++j) {
    const rmn_weight_job& a = jobs[j];
    if (!a.weights || !a.image || a.K < 1 || a.K > 65535 || ((uintptr_t)a.image & 15)) return RMN_ERR_BAD_ARG;
    if (a.w_in < 1 || a.w_in > a.c_in || a.w_out < 1 || a.w_out > a.c_out) return RMN_ERR_BAD_ARG;
    if (a.fold.scale && (!a.fold.shift || (a.fold.param_dtype != RMN_F32 && a.fold.param_dtype != RMN_BF16))) return RMN_ERR_BAD_ARG;
    if (rmn_conv_weight_image_bytes(a.K, a.c_in, a.c_out, RMN_BF16) == 0) return RMN_ERR_UNSUPPORTED;
  }
  return ta_weight_images(jobs, n_jobs, (cudaStream_t)stream_);
}

extern "C" int rmn_conv_forward_image(const void* d_feats, uint32_t n_src, int c_in, const void* d_image, int K, int c_out,
                                      const int32_t* d_nbr, const void* d_plan, uint32_t n_dst, void* d_out,
                                      const float* d_scale, const float* d_shift, const void* d_add, int relu,
                                      void* stream_) {
  if (n_dst == 0) return RMN_OK;
  // (with no source rows every table entry is -1 and nothing is read through d_feats)
  if (!d_image || !d_nbr || !d_out || (n_src > 0 && !d_feats) || K < 1 || K > 65535) return RMN_ERR_BAD_ARG;
  if (((uintptr_t)d_feats & 31) || ((uintptr_t)d_image & 15) || ((uintptr_t)d_out & 15) || ((uintptr_t)d_add & 15))
    return RMN_ERR_BAD_ARG;
  return ta_conv(d_feats, d_image, d_nbr, n_dst, K, c_in, c_out, d_out, d_scale, d_shift, d_add, relu, nullptr, nullptr,
                 (cudaStream_t)stream_, d_plan, nullptr);
}

extern "C" int rmn_conv_forward_ordered(const void* d_feats, uint32_t n_src, int c_in, const void* d_image, int K, int c_out,
                                        const int32_t* d_nbr, const int32_t* d_order, uint32_t n_dst, void* d_out,
                                        const float* d_scale, const float* d_shift, const void* d_add, int relu,
                                        void* stream_) {
  if (n_dst == 0) return RMN_OK;
  if (!d_image || !d_nbr || !d_order || !d_out || (n_src > 0 && !d_feats) || K < 1 || K > 65535) return RMN_ERR_BAD_ARG;
  if (((uintptr_t)d_feats & 31) || ((uintptr_t)d_image & 15) || ((uintptr_t)d_out & 15) || ((uintptr_t)d_add & 15))
    return RMN_ERR_BAD_ARG;
  return ta_conv(d_feats, d_image, d_nbr, n_dst, K, c_in, c_out, d_out, d_scale, d_shift, d_add, relu, nullptr, nullptr,
                 (cudaStream_t)stream_, nullptr, d_order);
}

extern "C" int rmn_conv_backward_input(const void* d_grad_out, uint32_t n_dst, int c_out,
                                       const void* d_weights, int K, int c_in,
                                       const int32_t* d_nbr_t, uint32_t n_src, void* d_grad_feats,
                                       int dtype, void* stream_) {
  return rmn_conv_backward_input_planned(d_grad_out, n_dst, c_out, d_weights, K, c_in, d_nbr_t, nullptr, n_src,
                                         d_grad_feats, dtype, stream_);
}

extern "C" int rmn_conv_backward_input_planned(const void* d_grad_out, uint32_t n_dst, int c_out,
                                               const void* d_weights, int K, int c_in, const int32_t* d_nbr_t,
                                               const void* d_plan_t, uint32_t n_src, void* d_grad_feats, int dtype,
                                               void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n_src == 0) return RMN_OK;
  if (n_dst == 0) {
    if (!d_grad_feats || (dtype != RMN_F32 && dtype != RMN_BF16)) return RMN_ERR_BAD_ARG;
    RMN_CUDA_TRY(cudaMemsetAsync(d_grad_feats, 0, (size_t)n_src * c_in * (dtype == RMN_F32 ? 4 : 2), stream));
    return RMN_OK;
  }
  if (!conv_args_ok(d_grad_out, d_weights, d_nbr_t, d_grad_feats, K, c_in, c_out, dtype))
    return RMN_ERR_BAD_ARG;
  if (dtype == RMN_BF16) {
    const int st = tc_conv(d_grad_out, n_dst, d_weights, d_nbr_t, n_src, K, c_out, c_in, true, d_grad_feats, nullptr, nullptr, 0,
                           stream, d_plan_t);
    if (st != RMN_ERR_UNSUPPORTED) return st;
  }
  return simt_conv_backward_input(d_grad_out, c_out, d_weights, K, c_in, d_nbr_t, n_src,
                                  d_grad_feats, dtype, stream);
}

extern "C" size_t rmn_conv_backward_weight_workspace_bytes(uint32_t n_dst, int K, int c_in,
                                                           int c_out, int dtype) {
  if (K < 1 || c_in < 1 || c_out < 1) return 0;
  size_t need = 0;
  if (dtype == RMN_BF16 &&
      tc_conv_wgrad(nullptr, nullptr, nullptr, n_dst, K, c_in, c_out, nullptr, nullptr, 0, &need, nullptr) == RMN_OK)
    return need;
  return simt_wgrad_workspace_bytes(n_dst, K, c_in, c_out);
}

extern "C" int rmn_conv_backward_weight(const void* d_feats, uint32_t n_src, int c_in,
                                        const void* d_grad_out, uint32_t n_dst, int c_out,
                                        const int32_t* d_nbr, int K, float* d_grad_weights,
                                        int dtype, void* d_workspace, size_t workspace_bytes,
                                        void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!d_grad_weights || K < 1 || c_in < 1 || c_out < 1) return RMN_ERR_BAD_ARG;
  if (n_dst == 0 || n_src == 0) {
    RMN_CUDA_TRY(cudaMemsetAsync(d_grad_weights, 0, (size_t)K * c_in * c_out * sizeof(float), stream));
    return RMN_OK;
  }
  if (!conv_args_ok(d_feats, d_grad_out, d_nbr, d_grad_weights, K, c_in, c_out, dtype) || !d_workspace)
    return RMN_ERR_BAD_ARG;
  if (workspace_bytes < rmn_conv_backward_weight_workspace_bytes(n_dst, K, c_in, c_out, dtype))
    return RMN_ERR_ALLOC;
  if (dtype == RMN_BF16) {
    size_t need = 0;
    const int st = tc_conv_wgrad(d_feats, d_grad_out, d_nbr, n_dst, K, c_in, c_out, d_grad_weights, d_workspace,
                                 workspace_bytes, &need, stream);
    if (st != RMN_ERR_UNSUPPORTED) return st;
  }
  return simt_conv_backward_weight(d_feats, c_in, d_grad_out, n_dst, c_out, d_nbr, K,
                                   d_grad_weights, dtype, d_workspace, stream);
}
