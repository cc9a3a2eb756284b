// Native host side of the operators: what stands between a Python call and the C ABI of
// libturbot5_b200.so.  Argument checks, output allocation, the argument blocks, the per-stream
// scratch and the autograd nodes live here; a call costs a few microseconds of host time (the
// same steps in Python with ctypes cost fifteen to twenty, more than the kernel of a short call).
#pragma once

#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <optional>
#include <vector>

#include "../../../include/turbot5_b200.h"

namespace t5b_host {

using at::Tensor;

// ---- small helpers -----------------------------------------------------------------
inline int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return T5B_F32;
    case at::kHalf: return T5B_F16;
    case at::kBFloat16: return T5B_BF16;
    default: break;
  }
  TORCH_CHECK_TYPE(false, "turbot5_b200 supports float32, float16 and bfloat16, got ", c10::toString(t));
  return -1;
}
inline void require_cuda(const Tensor& t) {
  TORCH_CHECK(!t.defined() || t.is_cuda(), "turbot5_b200 operators need CUDA tensors: there is no CPU path");
}
inline void check_status(int status, const char* what) {
  TORCH_CHECK(status == T5B_OK, what, ": ", t5b_status_string(status), " (t5b_status ", status, ")");
}
inline bool is_half_type(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }
inline Tensor empty_like_dense(at::IntArrayRef sizes, at::ScalarType dtype, at::Device dev) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, dev, std::nullopt));
}
inline Tensor empty_strided(at::IntArrayRef sizes, at::IntArrayRef strides, at::ScalarType dtype, at::Device dev) {
  return Tensor(at::detail::empty_strided_cuda(sizes, strides, dtype, dev));
}
inline bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline cudaStream_t stream_of(at::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
inline Tensor unit_stride_last(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
inline void zero_async(const Tensor& t) {
  TORCH_CHECK(cudaMemsetAsync(t.data_ptr(), 0, t.nbytes(), stream_of(t.device())) == cudaSuccess, "memset failed");
}

// Per-device int32 word the kernels write to when a bounded wait runs out.
Tensor device_status(int index);
// Zero-initialised scratch, one buffer per (device, stream, kind); kernels leave it ready for the next call.
enum ScratchKind { SCRATCH_ATTN = 0, SCRATCH_ATTN_BWD = 1, SCRATCH_DECODE = 2, SCRATCH_KINDS = 3 };
Tensor scratch(at::Device dev, int kind, int64_t nbytes);

// ---- attention ---------------------------------------------------------------------
struct AttnOptions {
  bool causal = false;
  double sm_scale = 1.0;
  int num_buckets = 32, max_distance = 128;
  std::optional<int64_t> q_pos_offset;
  int kernel = T5B_KERNEL_AUTO;
  bool balance_last_wave = true;
  int local_block = 0, window = 0;
  bool out_f32 = false;
  int64_t max_q = 0, max_k = 0;     // packed calls: the caller's bounds
};
// One forward call: the argument block and the tensors that it points to.
struct AttnCall {
  t5b_attn_args args;
  Tensor q, k, v, table, cu_q, cu_k, out, lse;
  bool packed = false;
};
// Raises NotImplementedError for a request no kernel takes.
void dense_forward(AttnCall& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias,
                   const AttnOptions& o, bool want_lse, const Tensor& out = Tensor());
void packed_forward(AttnCall& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias,
                    const Tensor& cu_q, const Tensor& cu_k, const AttnOptions& o, bool want_lse,
                    const Tensor& out = Tensor());
// dq, dk, dv are written (strides of q, k, v); dtable: float32 [buckets, H], ADDED to, or undefined.
void attention_backward(AttnCall& c, const Tensor& dout, const Tensor& dq, const Tensor& dk, const Tensor& dv,
                        const Tensor& dtable);

// ---- token-wise operators ----------------------------------------------------------
Tensor rmsnorm(const Tensor& x, const Tensor& w, double eps, Tensor* rstd = nullptr);
void rmsnorm_backward(const Tensor& x, const Tensor& w, const Tensor& dy, const Tensor& dx, const Tensor& dw, double eps);
// (hidden + branch, norm of it); both outputs fresh unless `inplace`, which overwrites hidden
std::pair<Tensor, Tensor> add_rmsnorm(const Tensor& hidden, const Tensor& branch, const Tensor& w, double eps, bool inplace);
Tensor gated_gelu(const Tensor& x);

struct UnpadPlan { Tensor seqlens, cu, dest; int64_t batch = 0, seqlen = 0; };
UnpadPlan unpad_plan(Tensor mask);
Tensor gather_rows(const Tensor& x, const Tensor& dest, int64_t n_rows);       // (n, ...) -> packed (n, row)
Tensor scatter_rows(const Tensor& packed, const Tensor& dest, int64_t n_rows); // packed -> (n, row), zeros where dropped


}  // namespace t5b_host
