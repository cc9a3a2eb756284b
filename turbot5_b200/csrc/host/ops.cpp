// Operators: forward calls, their backward nodes and the Python bindings.
#include "host.h"

#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <map>
#include <mutex>
#include <tuple>

#include "bindings.h"

namespace t5b_host {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ------------------------------------------------------------------ per-device and per-stream state
namespace {
std::mutex g_mutex;
Tensor g_status[64];
std::map<std::tuple<int, int, cudaStream_t>, Tensor>& scratch_map() {
  static auto* m = new std::map<std::tuple<int, int, cudaStream_t>, Tensor>();   // outlives the interpreter's teardown
  return *m;
}
const char* const kScratchNames[SCRATCH_KINDS] = {"attn", "attn_bwd", "decode"};
}  // namespace

Tensor device_status(int index) {
  TORCH_CHECK(index >= 0 && index < 64, "bad device index");
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_status[index].defined())
    g_status[index] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, index));
  return g_status[index];
}

Tensor scratch(at::Device dev, int kind, int64_t nbytes) {
  const auto key = std::make_tuple(kind, (int)dev.index(), stream_of(dev));
  std::lock_guard<std::mutex> lock(g_mutex);
  Tensor& t = scratch_map()[key];
  if (!t.defined() || t.numel() < nbytes)
    t = at::zeros({std::max<int64_t>(nbytes, 1 << 20)}, at::TensorOptions().dtype(at::kByte).device(dev));
  return t;
}

// ------------------------------------------------------------------ attention
namespace {

[[noreturn]] void raise_assertion(const char* msg) {
  PyErr_SetString(PyExc_AssertionError, msg);
  throw python_error();
}

void check_qkv(const Tensor& q, const Tensor& k, const Tensor& v, int rank) {
  const int64_t D = q.size(-1);
  if (k.size(-1) != D || v.size(-1) != D) raise_assertion("q, k and v must share a head dim");
  if (D != 16 && D != 32 && D != 64 && D != 128) raise_assertion("head dim must be 16, 32, 64 or 128");
  TORCH_CHECK_TYPE(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "q, k and v must share a dtype");
  require_cuda(q); require_cuda(k); require_cuda(v);
  TORCH_CHECK_VALUE(q.dim() == rank, rank == 4 ? "q must be (B, H, M, D)" : "q must be (Tq, H, D)");
}

// the bias table, its dtype code and its row stride
void set_table(AttnCall& c, const Tensor& bias, int64_t H) {
  c.args.table = nullptr; c.args.table_dtype = T5B_F32; c.args.table_stride0 = 0;
  if (!bias.defined()) return;
  require_cuda(bias);
  TORCH_CHECK_VALUE(bias.dim() == 2 && bias.size(1) == H, "bias table must be [NUM_BUCKETS, ", H, "], got ", bias.sizes());
  c.table = bias.stride(1) == 1 ? bias : bias.contiguous();
  c.args.table = c.table.data_ptr();
  c.args.table_dtype = dtype_code(c.table.scalar_type());
  c.args.table_stride0 = c.table.stride(0);
}

void set_common(AttnCall& c, const AttnOptions& o, double sm_scale) {
  t5b_attn_args& a = c.args;
  a.device_status = (int32_t*)device_status(c.q.device().index()).data_ptr();
  a.dtype = dtype_code(c.q.scalar_type());
  a.causal = o.causal;
  a.num_buckets = o.num_buckets; a.max_distance = o.max_distance;
  a.kernel = o.kernel;
  a.sm_scale = (float)sm_scale;
  a.workspace = nullptr; a.workspace_bytes = 0;
  a.local_block = o.local_block;
  a.out_f32 = o.out_f32;
  a.window = o.window;
}

// Pointers and strides of the argument block, from the call's tensors.
void set_operands(AttnCall& c) {
  t5b_attn_args& a = c.args;
  const int row = c.packed ? 0 : 2;                 // packed (rows, H, D); dense (B, H, rows, D)
  auto batch = [&](const Tensor& t) { return c.packed ? 0 : t.stride(0); };
  a.q = c.q.data_ptr(); a.k = c.k.data_ptr(); a.v = c.v.data_ptr(); a.out = c.out.data_ptr();
  a.lse = (float*)ptr(c.lse);
  a.q_stride_b = batch(c.q); a.q_stride_h = c.q.stride(1); a.q_stride_m = c.q.stride(row);
  a.k_stride_b = batch(c.k); a.k_stride_h = c.k.stride(1); a.k_stride_n = c.k.stride(row);
  a.v_stride_b = batch(c.v); a.v_stride_h = c.v.stride(1); a.v_stride_n = c.v.stride(row);
  a.o_stride_b = batch(c.out); a.o_stride_h = c.out.stride(1); a.o_stride_m = c.out.stride(row);
}

}  // namespace

// softmax(sm_scale * Q K^T + T5 bias(n - m) [+ causal mask]) V; the query at row m sits at key
// position q_pos_offset + m (default N - M: the cached-decoding alignment of the reference's `basic` path).
void dense_forward(AttnCall& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias,
                   const AttnOptions& o, bool want_lse, const Tensor& out) {
  check_qkv(q, k, v, 4);
  const int64_t B = q.size(0), H = q.size(1), M = q.size(2), D = q.size(3);
  TORCH_CHECK_VALUE(k.dim() == 4 && k.size(0) == B && k.size(1) == H && v.sizes() == k.sizes(),
                    "k/v must be (B, H, N, D) with q's batch and heads");
  const int64_t N = k.size(2);
  c.packed = false;
  c.q = unit_stride_last(q); c.k = unit_stride_last(k); c.v = unit_stride_last(v);
  set_table(c, bias, H);
  const at::ScalarType ot = o.out_f32 ? at::kFloat : q.scalar_type();
  if (out.defined()) {
    c.out = out;
  } else if (c.q.stride(1) == D && c.q.stride(2) >= H * D) {
    // q is a (B,H,M,D) view of token-major rows (a projection output, possibly one slice of a stacked
    // q|k|v projection): the result is laid out (B,M,H,D) so that merging the heads afterwards is free
    c.out = empty_strided({B, H, M, D}, {M * H * D, D, H * D, 1}, ot, q.device());
  } else {
    c.out = at::empty_like(c.q, c.q.options().dtype(ot));
    if (c.out.stride(-1) != 1) c.out = empty_like_dense({B, H, M, D}, ot, q.device());
  }
  c.lse = want_lse ? empty_like_dense({B, H, M}, at::kFloat, q.device()) : Tensor();
  t5b_attn_args& a = c.args;
  set_operands(c);
  a.cu_seqlens_q = a.cu_seqlens_k = nullptr;
  a.B = (int32_t)B; a.H = (int32_t)H; a.M = (int32_t)M; a.N = (int32_t)N; a.D = (int32_t)D;
  a.total_q = a.total_k = 0;
  a.q_pos_offset = (int32_t)o.q_pos_offset.value_or(N - M);
  set_common(c, o, o.sm_scale);
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor ws;
  if (o.balance_last_wave) {
    const int64_t need = t5b_attention_workspace_bytes(&a);
    if (need > 0) {
      ws = scratch(q.device(), SCRATCH_ATTN, need);
      a.workspace = ws.data_ptr(); a.workspace_bytes = ws.numel();
    }
  }
  const int st = t5b_attention_fwd(&a, stream_of(q.device()));
  TORCH_CHECK_NOT_IMPLEMENTED(!(st == T5B_ERR_UNSUPPORTED && (o.out_f32 || o.window)),
                              "float32 partial outputs and sliding windows need the tensor-core forward kernel "
                              "(bf16/fp16, 16-byte aligned rows)");
  check_status(st, "flash_attention_with_fusing_bias");
}

// Packed sequences: q (Tq,H,D), k/v (Tk,H,D), int32 cu_seqlens on the device.  Positions are relative to
// each sequence; tiles are scheduled on the device from cu_seqlens.
void packed_forward(AttnCall& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias,
                    const Tensor& cu_q, const Tensor& cu_k, const AttnOptions& o, bool want_lse, const Tensor& out) {
  check_qkv(q, k, v, 3);
  const int64_t Tq = q.size(0), H = q.size(1), D = q.size(2);
  TORCH_CHECK_VALUE(k.dim() == 3 && k.size(1) == H && v.sizes() == k.sizes(), "k/v must be (Tk, H, D) with q's heads");
  require_cuda(cu_q); require_cuda(cu_k);
  TORCH_CHECK_TYPE(cu_q.scalar_type() == at::kInt && cu_k.scalar_type() == at::kInt, "cu_seqlens must be int32");
  TORCH_CHECK_VALUE(cu_q.numel() == cu_k.numel() && cu_q.numel() >= 1, "cu_seqlens_q and cu_seqlens_k must both hold batch+1 entries");
  c.packed = true;
  c.cu_q = cu_q.contiguous(); c.cu_k = cu_k.contiguous();
  c.q = unit_stride_last(q); c.k = unit_stride_last(k); c.v = unit_stride_last(v);
  set_table(c, bias, H);
  if (out.defined()) {
    c.out = out;
  } else {
    c.out = at::empty_like(c.q);
    if (c.out.stride(-1) != 1) c.out = empty_like_dense({Tq, H, D}, q.scalar_type(), q.device());
  }
  const c10::cuda::CUDAGuard guard(q.device());
  c.lse = Tensor();
  if (want_lse) {
    c.lse = empty_like_dense({Tq, H}, at::kFloat, q.device());
    zero_async(c.lse);
  }
  t5b_attn_args& a = c.args;
  set_operands(c);
  a.cu_seqlens_q = (const int32_t*)c.cu_q.data_ptr(); a.cu_seqlens_k = (const int32_t*)c.cu_k.data_ptr();
  a.B = (int32_t)(cu_q.numel() - 1); a.H = (int32_t)H; a.M = (int32_t)o.max_q; a.N = (int32_t)o.max_k; a.D = (int32_t)D;
  a.total_q = (int32_t)Tq; a.total_k = (int32_t)k.size(0);
  a.q_pos_offset = 0;
  set_common(c, o, o.sm_scale);
  const int st = t5b_attention_fwd(&a, stream_of(q.device()));
  TORCH_CHECK_NOT_IMPLEMENTED(!(st == T5B_ERR_UNSUPPORTED && o.window),
                              "sliding windows need the tensor-core forward kernel (bf16/fp16, head dim 64 or 128, "
                              "16-byte aligned rows)");
  check_status(st, "flash_attention_with_fusing_bias_varlen");
}

// Mirrors flash_attn_v2_bwd_bias (src/turbot5/ops/fused_bias_attention.py:62-147): delta, then the k/v
// and q kernels.
void attention_backward(AttnCall& c, const Tensor& dout_in, const Tensor& dq, const Tensor& dk, const Tensor& dv,
                        const Tensor& dtable) {
  Tensor dout = dout_in.scalar_type() == c.out.scalar_type() ? dout_in : dout_in.to(c.out.scalar_type());
  bool aligned = dout.stride(-1) == 1 && ((uintptr_t)dout.data_ptr() % 16) == 0;
  for (int64_t i = 0; i + 1 < dout.dim(); ++i) aligned = aligned && dout.stride(i) % 8 == 0;
  if (!aligned) dout = dout.contiguous();
  t5b_attn_bwd_args g;
  g.fwd = c.args;
  t5b_attn_args& a = g.fwd;
  a.workspace = nullptr; a.workspace_bytes = 0;
  g.dout = dout.data_ptr();
  g.do_stride_h = dout.stride(1);
  g.do_stride_b = c.packed ? 0 : dout.stride(0);
  g.do_stride_m = c.packed ? dout.stride(0) : dout.stride(2);
  g.dq = dq.data_ptr(); g.dk = dk.data_ptr(); g.dv = dv.data_ptr();
  g.dtable = (float*)ptr(dtable);
  const Tensor delta = empty_like_dense(c.lse.sizes(), at::kFloat, c.q.device());
  g.delta = (float*)delta.data_ptr();
  g.workspace = nullptr; g.workspace_bytes = 0;
  const c10::cuda::CUDAGuard guard(c.q.device());
  Tensor ws;
  const int64_t need = t5b_attention_bwd_workspace_bytes(&g);
  if (need > 0) {
    ws = scratch(c.q.device(), SCRATCH_ATTN_BWD, need);      // all zero at rest (the kernels restore it)
    g.workspace = ws.data_ptr(); g.workspace_bytes = ws.numel();
  }
  const int st = t5b_attention_bwd(&g, stream_of(c.q.device()));
  TORCH_CHECK_NOT_IMPLEMENTED(st != T5B_ERR_UNSUPPORTED,
                              "no backward kernel for this call (max_distance above 2048, a sliding window or "
                              "kernel='tcgen05' on a shape the tensor-core backward does not take: bf16/fp16, "
                              "16-byte aligned rows)");
  check_status(st, "flash_attention_with_fusing_bias (backward)");
}

namespace {

// An input kept for the backward pass.  Inference tensors (frozen states computed once) cannot be saved variables; they
// are kept as they are.
struct KeptInput {
  SavedVariable saved;
  Tensor inference;
  void keep(const Tensor& t) {
    if (t.is_inference()) inference = t;
    else saved = SavedVariable(t, false);
  }
  Tensor unpack() const { return inference.defined() ? inference : saved.unpack(); }
  void reset() { saved.reset_data(); inference = Tensor(); }
};

// Backward of one attention call, as FlashAttentionBias (src/turbot5/ops/fused_bias_attention.py:822-873).
struct AttentionNode : public Node {
  AttnCall call;                                  // argument block; its tensors are kept by the saved variables
  KeptInput q, k, v, table;
  SavedVariable out, lse;
  bool has_table = false;

  variable_list apply(variable_list&& grads) override {
    variable_list r(4);
    if (!grads[0].defined()) return r;
    std::lock_guard<std::mutex> lock(mutex_);
    AttnCall c = call;
    c.q = q.unpack(); c.k = k.unpack(); c.v = v.unpack();
    c.out = out.unpack(shared_from_this()); c.lse = lse.unpack(shared_from_this());
    if (has_table) c.table = table.unpack();
    // A saved-tensor hook may have given back any layout (or, by mistake, another tensor): the argument block is
    // made anew from what was unpacked.
    const t5b_attn_args& a = c.args;
    auto is = [&](const Tensor& t, int64_t rows, int dtype) {
      return t.is_cuda() && dtype_code(t.scalar_type()) == dtype &&
             (c.packed ? t.sizes() == at::IntArrayRef({rows, a.H, a.D}) : t.sizes() == at::IntArrayRef({a.B, a.H, rows, a.D}));
    };
    const int64_t M = c.packed ? a.total_q : a.M, N = c.packed ? a.total_k : a.N;
    TORCH_CHECK(is(c.q, M, a.dtype) && is(c.k, N, a.dtype) && is(c.v, N, a.dtype) && is(c.out, M, a.dtype) && c.lse.is_cuda() &&
                    c.lse.scalar_type() == at::kFloat && c.lse.numel() == (c.packed ? M * a.H : a.B * a.H * M),
                "a saved tensor of an attention call came back with another shape, type or device");
    c.q = unit_stride_last(c.q); c.k = unit_stride_last(c.k); c.v = unit_stride_last(c.v);
    c.out = unit_stride_last(c.out); c.lse = c.lse.contiguous();
    const at::Device dev = c.q.device();
    const c10::cuda::CUDAGuard guard(dev);
    set_table(c, has_table ? c.table : Tensor(), a.H);
    set_operands(c);
    const Tensor dq = empty_strided(c.q.sizes(), c.q.strides(), c.q.scalar_type(), dev);
    const Tensor dk = empty_strided(c.k.sizes(), c.k.strides(), c.k.scalar_type(), dev);
    const Tensor dv = empty_strided(c.v.sizes(), c.v.strides(), c.v.scalar_type(), dev);
    const int row_dim = c.packed ? 0 : 2;
    Tensor dtable;
    if (has_table) {
      dtable = empty_like_dense({std::max<int64_t>(c.args.num_buckets, c.table.size(0)), c.q.size(1)}, at::kFloat, dev);
      zero_async(dtable);
    }
    if (c.k.size(row_dim) == 0 || c.q.size(row_dim) == 0) {
      dq.zero_(); dk.zero_(); dv.zero_();
    } else {
      attention_backward(c, grads[0], dq, dk, dv, dtable);
    }
    r[0] = dq; r[1] = dk; r[2] = dv;
    if (has_table && task_should_compute_output(3)) {
      if (dtable.size(0) != c.table.size(0)) dtable = dtable.slice(0, 0, c.table.size(0));
      r[3] = dtable.to(c.table.scalar_type());
    }
    return r;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    q.reset(); k.reset(); v.reset(); table.reset(); out.reset_data(); lse.reset_data();
    call.q = call.k = call.v = call.table = call.out = call.lse = Tensor();
  }
  std::string name() const override { return "T5FusedBiasAttentionBackward"; }
};

// Whether a call is recorded.  The nodes have no forward-mode derivative: a tangent would be dropped.
bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  bool grad = false, tangent = false;
  for (const Tensor* t : ts)
    if (t->defined()) {
      grad = grad || t->requires_grad();
      tangent = tangent || has_tangent(*t);
    }
  TORCH_CHECK_NOT_IMPLEMENTED(!grad || !tangent, "turbot5_b200 operators have no forward-mode derivative");
  return grad;
}

// (out, lse) of a call, recorded for autograd when an input asks for it
void run_attention(AttnCall& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias,
                   const Tensor* cu_q, const Tensor* cu_k, const AttnOptions& o, bool want_lse) {
  const bool grad = wants_grad({&q, &k, &v, &bias});
  {
    at::AutoGradMode no_grad(false);
    if (cu_q) packed_forward(c, q, k, v, bias, *cu_q, *cu_k, o, want_lse || grad);
    else dense_forward(c, q, k, v, bias, o, want_lse || grad);
  }
  if (!grad) return;
  auto node = std::make_shared<AttentionNode>();
  node->set_next_edges(torch::autograd::collect_next_edges(q, k, v, bias));
  // inputs that were copied for the kernels are copied again in the backward pass: what is saved is the input
  node->q.keep(q); node->k.keep(k); node->v.keep(v);
  node->has_table = bias.defined();
  if (bias.defined()) node->table.keep(bias);
  torch::autograd::set_history(c.out, node);
  node->out = SavedVariable(c.out, true);
  node->lse = SavedVariable(c.lse, false);
  node->call = c;
  node->call.q = node->call.k = node->call.v = node->call.table = node->call.out = node->call.lse = Tensor();
}

// ------------------------------------------------------------------ decoding
Tensor decode(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& bias, bool causal,
              std::optional<double> sm_scale, int nb, int md, std::optional<int64_t> kv_len, Tensor seqlens_k,
              std::optional<int64_t> q_pos_offset, int64_t num_splits, Tensor workspace) {
  check_qkv(q_in, k_in, v_in, 4);
  const int64_t B = q_in.size(0), H = q_in.size(1), M = q_in.size(2), D = q_in.size(3);
  const int64_t cap = k_in.size(2), N = kv_len.value_or(cap);
  TORCH_CHECK_VALUE(N <= cap && N >= 0, "kv_len exceeds the cache capacity");
  const Tensor q = unit_stride_last(q_in), k = unit_stride_last(k_in), v = unit_stride_last(v_in);
  AttnCall c;
  set_table(c, bias, H);
  const Tensor out = empty_like_dense({B, H, M, D}, q.scalar_type(), q.device());
  const c10::cuda::CUDAGuard guard(q.device());
  const int splits = num_splits ? (int)num_splits : t5b_decode_num_splits((int)B, (int)H, (int)N);
  const int64_t need = splits > 1 ? t5b_decode_workspace_bytes((int)B, (int)H, (int)M, (int)D, splits) : 0;
  if (!workspace.defined() && need) workspace = scratch(q.device(), SCRATCH_DECODE, need);
  t5b_decode_args a;
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.out = out.data_ptr();
  a.table = c.args.table;
  if (seqlens_k.defined()) {
    require_cuda(seqlens_k);
    TORCH_CHECK_TYPE(seqlens_k.scalar_type() == at::kInt && seqlens_k.numel() == B,
                     "seqlens_k must be int32 with one entry per batch row");
    seqlens_k = seqlens_k.contiguous();
  }
  a.seqlens_k = (const int32_t*)ptr(seqlens_k);
  a.workspace = ptr(workspace);
  a.workspace_bytes = workspace.defined() ? (int64_t)workspace.nbytes() : 0;
  a.q_stride_b = q.stride(0); a.q_stride_h = q.stride(1); a.q_stride_m = q.stride(2);
  a.k_stride_b = k.stride(0); a.k_stride_h = k.stride(1); a.k_stride_n = k.stride(2);
  a.v_stride_b = v.stride(0); a.v_stride_h = v.stride(1); a.v_stride_n = v.stride(2);
  a.o_stride_b = out.stride(0); a.o_stride_h = out.stride(1); a.o_stride_m = out.stride(2);
  a.table_stride0 = c.args.table_stride0;
  a.dtype = dtype_code(q.scalar_type()); a.table_dtype = c.args.table_dtype;
  a.B = (int32_t)B; a.H = (int32_t)H; a.M = (int32_t)M; a.N = (int32_t)N; a.D = (int32_t)D;
  a.causal = causal; a.num_buckets = nb; a.max_distance = md;
  a.q_pos_offset = (int32_t)q_pos_offset.value_or(-1);
  a.num_splits = splits;
  a.sm_scale = (float)sm_scale.value_or(1.0 / std::sqrt((double)D));
  check_status(t5b_decode_fwd(&a, stream_of(q.device())), "flash_decoding_with_fusing_bias");
  return out;
}

// ------------------------------------------------------------------ merge of partial results
std::pair<Tensor, Tensor> merge(const std::vector<Tensor>& outs_in, const std::vector<Tensor>& lses_in, at::ScalarType dtype,
                                bool want_lse) {
  const size_t n = outs_in.size();
  TORCH_CHECK_VALUE(n >= 1 && n <= T5B_MERGE_MAX_PARTS, "between 1 and ", T5B_MERGE_MAX_PARTS, " partial results can be merged");
  const Tensor& o0 = outs_in[0];
  require_cuda(o0);
  TORCH_CHECK_VALUE(o0.dim() == 4, "partials must be float32 (B,H,M,D) outputs with float32 (B,H,M) log-sum-exps");
  const int64_t B = o0.size(0), H = o0.size(1), M = o0.size(2), D = o0.size(3);
  const c10::cuda::CUDAGuard guard(o0.device());
  std::vector<Tensor> outs, lses;
  t5b_merge_args a;
  for (size_t i = 0; i < n; ++i) {
    const Tensor &o = outs_in[i], &l = lses_in[i];
    TORCH_CHECK_VALUE(o.scalar_type() == at::kFloat && l.scalar_type() == at::kFloat && o.sizes() == o0.sizes() &&
                          l.sizes() == at::IntArrayRef({B, H, M}),
                      "partials must be float32 (B,H,M,D) outputs with float32 (B,H,M) log-sum-exps");
    outs.push_back(o.strides() == o0.strides() ? o : o0.is_contiguous() ? o.contiguous() : at::empty_like(o0).copy_(o));
    lses.push_back(l.contiguous());
    a.part_out[i] = (const float*)outs.back().data_ptr();
    a.part_lse[i] = (const float*)lses.back().data_ptr();
  }
  const Tensor out = at::empty_like(o0, o0.options().dtype(dtype));
  const Tensor lse = want_lse ? empty_like_dense({B, H, M}, at::kFloat, o0.device()) : Tensor();
  a.out = out.data_ptr(); a.lse_out = (float*)ptr(lse);
  a.part_stride_b = o0.stride(0); a.part_stride_h = o0.stride(1); a.part_stride_m = o0.stride(2);
  a.o_stride_b = out.stride(0); a.o_stride_h = out.stride(1); a.o_stride_m = out.stride(2);
  a.n_parts = (int32_t)n; a.out_dtype = dtype_code(dtype);
  a.B = (int32_t)B; a.H = (int32_t)H; a.M = (int32_t)M; a.D = (int32_t)D;
  check_status(t5b_attention_merge(&a, stream_of(o0.device())), "merge_attention_partials");
  return {out, lse};
}

// rows of the last dim, with a unit stride
Tensor as_rows(const Tensor& x) {
  Tensor r = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  return r.stride(-1) == 1 ? r : r.contiguous();
}

}  // namespace

// ------------------------------------------------------------------ token-wise operators
// T5 RMSNorm (replaces RMSLayerNorm.apply, src/turbot5/ops/rms_norm.py:129-185)
Tensor rmsnorm(const Tensor& x, const Tensor& w, double eps, Tensor* rstd) {
  require_cuda(x); require_cuda(w);
  const int64_t d = x.size(-1);
  TORCH_CHECK_VALUE(w.dim() == 1 && w.size(0) == d, "weight must have the size of the last dimension");
  const Tensor x2 = as_rows(x), wc = w.contiguous();
  const at::ScalarType ot = is_half_type(w.scalar_type()) ? w.scalar_type() : at::kFloat;
  const Tensor y = empty_like_dense(x.sizes(), ot, x.device());
  if (rstd) *rstd = empty_like_dense({x2.size(0)}, at::kFloat, x.device());
  const c10::cuda::CUDAGuard guard(x.device());
  check_status(t5b_rmsnorm_fwd(x2.data_ptr(), wc.data_ptr(), y.data_ptr(), rstd ? (float*)rstd->data_ptr() : nullptr,
                               x2.size(0), (int32_t)d, x2.stride(0), d, dtype_code(x.scalar_type()),
                               dtype_code(wc.scalar_type()), (float)eps, stream_of(x.device())), "rms_layer_norm");
  return y;
}

// dx is written, the weight gradient is ADDED to dw (float32)
void rmsnorm_backward(const Tensor& x, const Tensor& w, const Tensor& dy, const Tensor& dx, const Tensor& dw, double eps) {
  const int64_t d = x.size(-1);
  const at::ScalarType ot = is_half_type(w.scalar_type()) ? w.scalar_type() : at::kFloat;
  const Tensor x2 = as_rows(x), g2 = as_rows(dy.scalar_type() == ot ? dy : dy.to(ot)), wc = w.contiguous();
  const c10::cuda::CUDAGuard guard(x.device());
  check_status(t5b_rmsnorm_bwd(x2.data_ptr(), wc.data_ptr(), g2.data_ptr(), dx.data_ptr(), (float*)dw.data_ptr(), x2.size(0),
                               (int32_t)d, x2.stride(0), g2.stride(0), d, dtype_code(x.scalar_type()),
                               dtype_code(wc.scalar_type()), (float)eps, stream_of(x.device())), "rms_layer_norm (backward)");
}

std::pair<Tensor, Tensor> add_rmsnorm(const Tensor& hidden, const Tensor& branch, const Tensor& w, double eps, bool inplace) {
  require_cuda(hidden); require_cuda(branch); require_cuda(w);
  const int64_t d = hidden.size(-1);
  TORCH_CHECK_VALUE(branch.sizes() == hidden.sizes() && branch.scalar_type() == hidden.scalar_type() && w.dim() == 1 && w.size(0) == d,
                    "hidden and branch must match; weight must have the size of the last dimension");
  const Tensor h2 = as_rows(hidden), b2 = as_rows(branch), wc = w.contiguous();
  const bool same = inplace && h2.data_ptr() == hidden.data_ptr();
  const Tensor h_out = same ? hidden : empty_like_dense(hidden.sizes(), hidden.scalar_type(), hidden.device());
  const Tensor normed = empty_like_dense(hidden.sizes(), hidden.scalar_type(), hidden.device());
  const c10::cuda::CUDAGuard guard(hidden.device());
  check_status(t5b_add_rmsnorm_fwd(h2.data_ptr(), b2.data_ptr(), wc.data_ptr(), h_out.data_ptr(), normed.data_ptr(), h2.size(0),
                                   (int32_t)d, h2.stride(0), b2.stride(0), same ? h2.stride(0) : d, d,
                                   dtype_code(hidden.scalar_type()), dtype_code(wc.scalar_type()), (float)eps,
                                   stream_of(hidden.device())), "add_rms_layer_norm");
  return {h_out, normed};
}

Tensor gated_gelu(const Tensor& x) {
  require_cuda(x);
  const int64_t f2 = x.size(-1);
  TORCH_CHECK_VALUE(f2 % 2 == 0, "the last dimension holds the two projections side by side");
  const Tensor x2 = as_rows(x);
  auto sizes = x.sizes().vec();
  sizes.back() = f2 / 2;
  const Tensor out = empty_like_dense(sizes, x.scalar_type(), x.device());
  const c10::cuda::CUDAGuard guard(x.device());
  check_status(t5b_gated_gelu_fwd(x2.data_ptr(), out.data_ptr(), x2.size(0), (int32_t)(f2 / 2), x2.stride(0), f2 / 2,
                                  dtype_code(x.scalar_type()), stream_of(x.device())), "gated_gelu");
  return out;
}

// ------------------------------------------------------------------ unpad / pad
UnpadPlan unpad_plan(Tensor mask) {
  require_cuda(mask);
  TORCH_CHECK_VALUE(mask.dim() == 2, "attention_mask must be (batch, seqlen)");
  if (mask.is_floating_point()) mask = mask.ne(0);
  const Tensor m = mask.contiguous();
  UnpadPlan p;
  p.batch = m.size(0); p.seqlen = m.size(1);
  p.seqlens = empty_like_dense({p.batch}, at::kInt, m.device());
  p.cu = empty_like_dense({p.batch + 1}, at::kInt, m.device());
  p.dest = empty_like_dense({p.batch * p.seqlen}, at::kInt, m.device());
  const c10::cuda::CUDAGuard guard(m.device());
  if (p.batch == 0) zero_async(p.cu);
  check_status(t5b_unpad_plan(m.data_ptr(), (int32_t)m.element_size(), (int32_t)p.batch, (int32_t)p.seqlen,
                              (int32_t*)p.seqlens.data_ptr(), (int32_t*)p.cu.data_ptr(), (int32_t*)p.dest.data_ptr(),
                              stream_of(m.device())), "get_unpad_plan");
  return p;
}

namespace {
Tensor plain_rows(const Tensor& t, int64_t n_rows) {
  Tensor r = t.reshape({n_rows, -1});
  if (r.stride(-1) != 1 || (r.stride(0) * r.element_size()) % 16 || (uintptr_t)r.data_ptr() % 16) r = r.contiguous();
  TORCH_CHECK_VALUE((r.size(1) * r.element_size()) % 16 == 0, "row size must be a multiple of 16 bytes");
  return r;
}
}  // namespace

Tensor gather_rows(const Tensor& x, const Tensor& dest, int64_t n) {
  require_cuda(x);
  const Tensor src = plain_rows(x, n);
  const int64_t row_bytes = src.size(1) * src.element_size();
  const Tensor out = empty_like_dense({n, src.size(1)}, x.scalar_type(), x.device());
  const c10::cuda::CUDAGuard guard(x.device());
  check_status(t5b_gather_rows(src.data_ptr(), src.stride(0) * src.element_size(), out.data_ptr(), row_bytes,
                               (const int32_t*)dest.data_ptr(), n, (int32_t)row_bytes, stream_of(x.device())), "unpad_rows");
  return out;
}

Tensor scatter_rows(const Tensor& packed, const Tensor& dest, int64_t n) {
  require_cuda(packed);
  const Tensor src = plain_rows(packed, packed.size(0));
  const int64_t row_bytes = src.size(1) * src.element_size();
  const Tensor out = empty_like_dense({n, src.size(1)}, packed.scalar_type(), packed.device());
  const c10::cuda::CUDAGuard guard(packed.device());
  check_status(t5b_scatter_rows(src.data_ptr(), src.stride(0) * src.element_size(), out.data_ptr(), row_bytes,
                                (const int32_t*)dest.data_ptr(), n, (int32_t)row_bytes, stream_of(packed.device())), "pad_rows");
  return out;
}

namespace {

struct RMSNormNode : public Node {
  SavedVariable x, w;
  double eps = 0;
  variable_list apply(variable_list&& grads) override {
    variable_list r(2);
    if (!grads[0].defined()) return r;
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor xv = x.unpack(), wv = w.unpack();
    const c10::cuda::CUDAGuard guard(xv.device());
    const Tensor dx = empty_like_dense(xv.sizes(), xv.scalar_type(), xv.device());
    const Tensor dw = empty_like_dense({xv.size(-1)}, at::kFloat, xv.device());
    zero_async(dw);
    rmsnorm_backward(xv, wv, grads[0], dx, dw, eps);
    r[0] = dx;
    if (task_should_compute_output(1)) r[1] = dw.to(wv.scalar_type());
    return r;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data(); w.reset_data();
  }
  std::string name() const override { return "T5RMSNormBackward"; }
};

// padded rows -> packed rows and back; the gradient of one is the other
struct RowsNode : public Node {
  Tensor dest;
  std::vector<int64_t> in_sizes;       // of the forward's input
  int64_t n = 0;
  bool gather = true;                  // the forward was the gather (unpad)
  variable_list apply(variable_list&& grads) override {
    variable_list r(1);
    if (!grads[0].defined()) return r;
    if (gather) {
      r[0] = scatter_rows(grads[0], dest, n).view(in_sizes);
    } else {
      Tensor g = gather_rows(grads[0], dest, n);           // kept tokens first, zero tail
      const int64_t rows = in_sizes[0];
      if (g.size(0) > rows) g = g.slice(0, 0, rows);
      else if (g.size(0) < rows) g = at::cat({g, at::zeros({rows - g.size(0), g.size(1)}, g.options())});
      r[0] = g.reshape(in_sizes);
    }
    return r;
  }
  std::string name() const override { return gather ? "T5UnpadBackward" : "T5PadBackward"; }
};

Tensor rows_op(const Tensor& x, const Tensor& dest, int64_t batch, int64_t seqlen, bool gather) {
  const bool grad = wants_grad({&x});
  const int64_t n = batch * seqlen;
  std::vector<int64_t> sizes;
  Tensor y;
  {
    at::AutoGradMode no_grad(false);
    if (gather) {
      sizes.push_back(n);
      for (int64_t i = 2; i < x.dim(); ++i) sizes.push_back(x.size(i));
      y = at::_unsafe_view(gather_rows(x, dest, n), sizes);
    } else {
      sizes = {batch, seqlen};
      for (int64_t i = 1; i < x.dim(); ++i) sizes.push_back(x.size(i));
      y = at::_unsafe_view(scatter_rows(x, dest, n), sizes);
    }
  }
  if (grad) {
    auto node = std::make_shared<RowsNode>();
    node->set_next_edges(torch::autograd::collect_next_edges(x));
    node->dest = dest; node->in_sizes = x.sizes().vec(); node->n = n; node->gather = gather;
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ------------------------------------------------------------------ Python bindings
// attention(q, k, v, bias, causal, sm_scale, nb, md, q_pos_offset, return_lse, kernel, balance, local_block, window, out_f32)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 15);
  const Tensor q = tensor_arg(a[0]), k = tensor_arg(a[1]), v = tensor_arg(a[2]), bias = tensor_arg(a[3]);
  AttnOptions o;
  o.causal = bool_arg(a[4]);
  o.sm_scale = a[5] == Py_None ? 1.0 / std::sqrt((double)q.size(-1)) : float_arg(a[5]);
  o.num_buckets = (int)int_arg(a[6]); o.max_distance = (int)int_arg(a[7]);
  o.q_pos_offset = opt_int(a[8]);
  const bool want_lse = bool_arg(a[9]);
  o.kernel = (int)int_arg(a[10]);
  o.balance_last_wave = bool_arg(a[11]);
  o.local_block = a[12] == Py_None ? 0 : (int)int_arg(a[12]);
  o.window = a[13] == Py_None ? 0 : (int)int_arg(a[13]);
  o.out_f32 = bool_arg(a[14]);
  if (o.local_block || o.window) o.balance_last_wave = false;
  if (o.local_block) o.q_pos_offset = 0;
  AttnCall c;
  run_attention(c, q, k, v, bias, nullptr, nullptr, o, want_lse);
  return want_lse ? wrap2(c.out, c.lse) : wrap(c.out);
  END_HANDLE_TH_ERRORS
}

// attention_packed(q, k, v, bias, cu_q, cu_k, max_q, max_k, causal, sm_scale, nb, md, return_lse, kernel, window)
PyObject* py_attention_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 15);
  const Tensor q = tensor_arg(a[0]), k = tensor_arg(a[1]), v = tensor_arg(a[2]), bias = tensor_arg(a[3]);
  const Tensor cu_q = tensor_arg(a[4]), cu_k = tensor_arg(a[5]);
  AttnOptions o;
  o.max_q = a[6] == Py_None ? 0 : int_arg(a[6]);
  o.max_k = a[7] == Py_None ? 0 : int_arg(a[7]);
  o.causal = bool_arg(a[8]);
  o.sm_scale = a[9] == Py_None ? 1.0 / std::sqrt((double)q.size(-1)) : float_arg(a[9]);
  o.num_buckets = (int)int_arg(a[10]); o.max_distance = (int)int_arg(a[11]);
  const bool want_lse = bool_arg(a[12]);
  o.kernel = (int)int_arg(a[13]);
  o.window = a[14] == Py_None ? 0 : (int)int_arg(a[14]);
  AttnCall c;
  run_attention(c, q, k, v, bias, &cu_q, &cu_k, o, want_lse);
  return want_lse ? wrap2(c.out, c.lse) : wrap(c.out);
  END_HANDLE_TH_ERRORS
}

// decode(q, k, v, bias, causal, sm_scale, nb, md, kv_len, seqlens_k, q_pos_offset, num_splits, workspace)
PyObject* py_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 13);
  std::optional<double> scale;
  if (a[5] != Py_None) scale = float_arg(a[5]);
  return wrap(decode(tensor_arg(a[0]), tensor_arg(a[1]), tensor_arg(a[2]), tensor_arg(a[3]), bool_arg(a[4]), scale,
                     (int)int_arg(a[6]), (int)int_arg(a[7]), opt_int(a[8]), tensor_arg(a[9]), opt_int(a[10]),
                     a[11] == Py_None ? 0 : int_arg(a[11]), tensor_arg(a[12])));
  END_HANDLE_TH_ERRORS
}

// merge(outs, lses, dtype, return_lse)
PyObject* py_merge(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 4);
  auto list = [](PyObject* o) {
    std::vector<Tensor> r;
    PyObject* seq = PySequence_Fast(o, "expected a sequence of tensors");
    if (!seq) throw python_error();
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) r.push_back(tensor_arg(PySequence_Fast_GET_ITEM(seq, i)));
    Py_DECREF(seq);
    return r;
  };
  TORCH_CHECK_TYPE(THPDtype_Check(a[2]), "expected a dtype");
  const bool want_lse = bool_arg(a[3]);
  auto r = merge(list(a[0]), list(a[1]), reinterpret_cast<THPDtype*>(a[2])->scalar_type, want_lse);
  return want_lse ? wrap2(r.first, r.second) : wrap(r.first);
  END_HANDLE_TH_ERRORS
}

// rmsnorm(x, w, eps, return_rstd)
PyObject* py_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 4);
  const Tensor x = tensor_arg(a[0]), w = tensor_arg(a[1]);
  const double eps = float_arg(a[2]);
  const bool want_rstd = bool_arg(a[3]);
  const bool grad = !want_rstd && wants_grad({&x, &w});
  Tensor y, rstd;
  {
    at::AutoGradMode no_grad(false);
    y = rmsnorm(x, w, eps, want_rstd ? &rstd : nullptr);
  }
  if (want_rstd) return wrap2(y, rstd);
  if (grad) {
    auto node = std::make_shared<RMSNormNode>();
    node->set_next_edges(torch::autograd::collect_next_edges(x, w));
    node->x = SavedVariable(x, false); node->w = SavedVariable(w, false); node->eps = eps;
    torch::autograd::set_history(y, node);
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// add_rmsnorm(hidden, branch, w, eps, inplace) -> (hidden', normed)
PyObject* py_add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 5);
  at::AutoGradMode no_grad(false);
  auto r = add_rmsnorm(tensor_arg(a[0]), tensor_arg(a[1]), tensor_arg(a[2]), float_arg(a[3]), bool_arg(a[4]));
  return wrap2(r.first, r.second);
  END_HANDLE_TH_ERRORS
}

PyObject* py_gated_gelu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 1);
  at::AutoGradMode no_grad(false);
  return wrap(gated_gelu(tensor_arg(a[0])));
  END_HANDLE_TH_ERRORS
}

// unpad_plan(mask) -> (seqlens, cu_seqlens, dest)
PyObject* py_unpad_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 1);
  at::AutoGradMode no_grad(false);
  const UnpadPlan p = unpad_plan(tensor_arg(a[0]));
  PyObject* r = PyTuple_New(3);
  PyTuple_SET_ITEM(r, 0, wrap(p.seqlens));
  PyTuple_SET_ITEM(r, 1, wrap(p.cu));
  PyTuple_SET_ITEM(r, 2, wrap(p.dest));
  return r;
  END_HANDLE_TH_ERRORS
}

// rows(x, dest, batch, seqlen, gather)
PyObject* py_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 5);
  return wrap(rows_op(tensor_arg(a[0]), tensor_arg(a[1]), int_arg(a[2]), int_arg(a[3]), bool_arg(a[4])));
  END_HANDLE_TH_ERRORS
}

PyObject* py_device_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 1);
  return wrap(device_status((int)int_arg(a[0])));
  END_HANDLE_TH_ERRORS
}

// every scratch buffer alive, as ((kind, device index, stream), tensor)
PyObject* py_scratch_items(PyObject*, PyObject* const*, Py_ssize_t) {
  HANDLE_TH_ERRORS
  std::lock_guard<std::mutex> lock(g_mutex);
  PyObject* r = PyList_New(0);
  for (auto& kv : scratch_map()) {
    PyObject* item = Py_BuildValue("((siK)N)", kScratchNames[std::get<0>(kv.first)], std::get<1>(kv.first),
                                   (unsigned long long)std::get<2>(kv.first), wrap(kv.second));
    PyList_Append(r, item);
    Py_DECREF(item);
  }
  return r;
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    T5B_METHOD("attention", py_attention), T5B_METHOD("attention_packed", py_attention_packed),
    T5B_METHOD("decode", py_decode), T5B_METHOD("merge", py_merge), T5B_METHOD("rmsnorm", py_rmsnorm),
    T5B_METHOD("add_rmsnorm", py_add_rmsnorm), T5B_METHOD("gated_gelu", py_gated_gelu),
    T5B_METHOD("unpad_plan", py_unpad_plan), T5B_METHOD("rows", py_rows),
    T5B_METHOD("device_status", py_device_status), T5B_METHOD("scratch_items", py_scratch_items),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "Native host side of the operators.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace t5b_host

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&t5b_host::kModule);
  if (m && PyModule_AddFunctions(m, t5b_host::stack_methods) < 0) { Py_DECREF(m); return nullptr; }
  return m;
}
