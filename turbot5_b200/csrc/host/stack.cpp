// Whole passes of a T5 stack as one native launch sequence: inference (token-wise work fused around the
// attention path, buffers reused from layer to layer) and training (the same forward pass recorded as ONE
// autograd node, whose backward issues every product and kernel of all layers itself).
//
// Block structure: T5LayerSelfAttention / T5LayerCrossAttention / T5LayerFF
// (src/turbot5/model/modeling.py:63-342).  Per encoder block eight launches: stacked q|k|v projection, attention,
// output projection, residual add + RMSNorm, stacked wi_0|wi_1 projection, gated GELU, wo projection, residual
// add + RMSNorm; five more per decoder block.  Driven from Python the same sequence costs 8-15 us of host time
// per launch, more than most of the kernels of a batch of short sequences; here it costs 2-4 us.
#include "host.h"

#include <ATen/SavedTensorHooks.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDACachingAllocator.h>
#include <cublas_v2.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>

#include <pybind11/pybind11.h>

#include <mutex>

#include "bindings.h"

namespace t5b_host {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// ------------------------------------------------------------------ matrix products (cuBLAS)
cudaDataType_t cuda_type(at::ScalarType t) { return t == at::kBFloat16 ? CUDA_R_16BF : CUDA_R_16F; }

void gemm(cublasOperation_t ta, cublasOperation_t tb, int64_t m, int64_t n, int64_t k, const Tensor& a, int64_t lda,
          const Tensor& b, int64_t ldb, const Tensor& c, int64_t ldc, float beta) {
  if (m == 0 || n == 0) return;
  const float alpha = 1.f;
  const cudaDataType_t t = cuda_type(c.scalar_type());
  const auto st = cublasGemmEx(at::cuda::getCurrentCUDABlasHandle(), ta, tb, (int)m, (int)n, (int)k, &alpha, a.data_ptr(), t,
                               (int)lda, b.data_ptr(), t, (int)ldb, &beta, c.data_ptr(), t, (int)ldc, CUBLAS_COMPUTE_32F,
                               CUBLAS_GEMM_DEFAULT_TENSOR_OP);
  TORCH_CHECK(st == CUBLAS_STATUS_SUCCESS, "cuBLAS failed with status ", (int)st);
}
// y[R, N] = x[R, K] w[N, K]^T
void linear(const Tensor& x, const Tensor& w, const Tensor& y) {
  gemm(CUBLAS_OP_T, CUBLAS_OP_N, w.size(0), x.size(0), w.size(1), w, w.stride(0), x, x.stride(0), y, y.stride(0), 0.f);
}
// dx[R, K] (+)= dy[R, N] w[N, K]
void linear_dx(const Tensor& dy, const Tensor& w, const Tensor& dx, bool add = false) {
  gemm(CUBLAS_OP_N, CUBLAS_OP_N, w.size(1), dy.size(0), w.size(0), w, w.stride(0), dy, dy.stride(0), dx, dx.stride(0), add ? 1.f : 0.f);
}
// dw[N, K] = dy[R, N]^T x[R, K]
void linear_dw(const Tensor& dy, const Tensor& x, const Tensor& dw) {
  gemm(CUBLAS_OP_N, CUBLAS_OP_T, x.size(1), dy.size(1), x.size(0), x, x.stride(0), dy, dy.stride(0), dw, dw.stride(0), 0.f);
}

// ------------------------------------------------------------------ parameters of a stack
struct Layer {
  Tensor ln_self, q, k, v, o;
  Tensor ln_cross, cq, ck, cv, co;       // decoder blocks
  Tensor ln_ff, wi0, wi1, wo;            // wi1 undefined: not gated (relu)
};
struct Stack {
  std::vector<Layer> layers;
  Tensor final_ln, table;
  bool decoder = false, gated = true;
  int64_t H = 0, D = 0, d = 0, F = 0;
  int nb = 32, md = 128;
  double eps = 1e-6;
  bool plain = true;                     // every module is of the expected class and has no hooks
  bool flash = true;                     // every attention module is the full-attention one
  bool plain_ff = true;                  // `plain` of the feed-forward layers alone
  bool complete = true;                  // every module and weight was found
};

struct Names {
  PyObject *modules, *parameters, *forward, *eps, *hooks[4], *attention[4];
  Names() {
    auto intern = PyUnicode_InternFromString;
    modules = intern("_modules"); parameters = intern("_parameters"); forward = intern("forward"); eps = intern("eps");
    hooks[0] = intern("_forward_hooks"); hooks[1] = intern("_forward_pre_hooks");
    hooks[2] = intern("_backward_hooks"); hooks[3] = intern("_backward_pre_hooks");
    attention[0] = intern("n_heads"); attention[1] = intern("key_value_proj_dim");
    attention[2] = intern("relative_attention_num_buckets"); attention[3] = intern("relative_attention_max_distance");
  }
};
const Names& names() { static const Names* n = new Names(); return *n; }

// Walks the module tree.  `types`: the classes a plain stack is made of, in the order of enum Kind.  A module that is
// not plain (another class, hooks, a `forward` in the instance, other settings than the stack's) is for the
// caller to run; one that has not the children or weights looked for makes the walk incomplete.
enum Kind { K_BLOCK = 0, K_LIST, K_SELF, K_CROSS, K_FF, K_ATTENTION, K_NORM, K_LINEAR, K_GATED, K_RELU, K_EMBEDDING };
#define T5B_KEY(name) ([] { static PyObject* const k = PyUnicode_InternFromString(name); return k; }())

// A module's own dicts, looked up once (borrowed: the module keeps them alive); null where there is none.
struct Module {
  PyObject *self = nullptr, *dict = nullptr, *modules = nullptr, *parameters = nullptr;
  Module() = default;
  explicit Module(PyObject* m) : self(m) {
    PyObject* d = m ? PyObject_GenericGetDict(m, nullptr) : nullptr;
    if (!d) { PyErr_Clear(); return; }
    Py_DECREF(d);
    if (!PyDict_Check(d)) return;
    dict = d;
    modules = PyDict_GetItem(d, names().modules);
    parameters = PyDict_GetItem(d, names().parameters);
    if (modules && !PyDict_Check(modules)) modules = nullptr;
    if (parameters && !PyDict_Check(parameters)) parameters = nullptr;
  }
  Module find(PyObject* key) const {
    PyObject* c = modules ? PyDict_GetItem(modules, key) : nullptr;
    return c && c != Py_None ? Module(c) : Module();
  }
};

struct Walker {
  PyObject* types;
  const Stack* s;
  bool plain = true, flash = true, complete = true;

  Module child(const Module& m, PyObject* key, int kind) {
    const Module c = m.find(key);
    if (c.self) look(c, kind);
    else complete = plain = false;
    return c;
  }
  bool has_int(PyObject* dict, PyObject* name, int64_t want) {
    PyObject* v = PyDict_GetItem(dict, name);
    if (!v || !PyLong_Check(v)) return false;
    const long long got = PyLong_AsLongLong(v);
    if (got == -1 && PyErr_Occurred()) PyErr_Clear();
    return got == want;
  }
  void look(const Module& c, int kind) {
    const bool exact = (PyObject*)Py_TYPE(c.self) == PyTuple_GET_ITEM(types, kind);
    if (kind == K_ATTENTION && !exact) flash = false;
    if (!plain) return;
    if (!exact || !c.dict || PyDict_GetItem(c.dict, names().forward)) { plain = false; return; }
    for (PyObject* h : names().hooks) {
      PyObject* t = PyDict_GetItem(c.dict, h);
      if (!t || !PyDict_Check(t) || PyDict_Size(t) != 0) { plain = false; return; }
    }
    if (kind == K_NORM) {
      PyObject* e = PyDict_GetItem(c.dict, names().eps);
      const double v = e ? PyFloat_AsDouble(e) : -1.0;
      if (v == -1.0 && PyErr_Occurred()) PyErr_Clear();
      plain = v == s->eps;
    } else if (kind == K_ATTENTION) {
      const int64_t want[4] = {s->H, s->D, s->nb, s->md};
      for (int i = 0; i < 4; ++i) plain = plain && has_int(c.dict, names().attention[i], want[i]);
    }
  }
  Tensor parameter(const Module& m) {                       // its weight
    if (!m.self) { complete = false; return Tensor(); }
    PyObject* p = m.parameters ? PyDict_GetItem(m.parameters, T5B_KEY("weight")) : nullptr;
    if (p && THPVariable_Check(p)) return THPVariable_Unpack(p);
    plain = false;                                          // a parametrised weight: ask the module for it
    PyObject* a = PyObject_GetAttr(m.self, T5B_KEY("weight"));
    if (!a || !THPVariable_Check(a)) {
      PyErr_Clear();
      Py_XDECREF(a);
      complete = false;
      return Tensor();
    }
    Tensor w = THPVariable_Unpack(a);
    Py_DECREF(a);
    return w;
  }
  Tensor weight(const Module& m, PyObject* key, int kind) {
    const Module c = child(m, key, kind);
    if (kind == K_LINEAR && plain) {                        // a bias is not part of these blocks
      PyObject* b = c.parameters ? PyDict_GetItem(c.parameters, T5B_KEY("bias")) : nullptr;
      if (b && b != Py_None) plain = false;
    }
    return parameter(c);
  }
};

// dims: (heads, head dim, buckets, max distance, eps)
Stack collect(PyObject* stack, PyObject* types, bool decoder, int64_t H, int64_t D, int nb, int md, double eps) {
  Stack s;
  Walker w{types, &s}, wf{types, &s};    // feed-forward layers are looked at apart
  s.decoder = decoder; s.H = H; s.D = D; s.nb = nb; s.md = md; s.eps = eps;
  const Module top(stack);
  PyObject* blocks = top.find(T5B_KEY("block")).modules;
  PyObject *key, *blk;
  Py_ssize_t pos = 0;
  while (blocks && w.complete && wf.complete && PyDict_Next(blocks, &pos, &key, &blk)) {
    const Module block(blk);
    w.look(block, K_BLOCK);
    const Module list = w.child(block, T5B_KEY("layer"), K_LIST);
    Layer l;
    const Module sa = w.child(list, T5B_KEY("0"), K_SELF);
    const Module att = w.child(sa, T5B_KEY("SelfAttention"), K_ATTENTION);
    l.ln_self = w.weight(sa, T5B_KEY("layer_norm"), K_NORM);
    l.q = w.weight(att, T5B_KEY("q"), K_LINEAR); l.k = w.weight(att, T5B_KEY("k"), K_LINEAR);
    l.v = w.weight(att, T5B_KEY("v"), K_LINEAR); l.o = w.weight(att, T5B_KEY("o"), K_LINEAR);
    if (s.layers.empty()) s.table = w.weight(att, T5B_KEY("relative_attention_bias"), K_EMBEDDING);
    if (decoder) {
      const Module ca = w.child(list, T5B_KEY("1"), K_CROSS);
      const Module catt = w.child(ca, T5B_KEY("EncDecAttention"), K_ATTENTION);
      l.ln_cross = w.weight(ca, T5B_KEY("layer_norm"), K_NORM);
      l.cq = w.weight(catt, T5B_KEY("q"), K_LINEAR); l.ck = w.weight(catt, T5B_KEY("k"), K_LINEAR);
      l.cv = w.weight(catt, T5B_KEY("v"), K_LINEAR); l.co = w.weight(catt, T5B_KEY("o"), K_LINEAR);
    }
    const Module ffl = w.child(list, decoder ? T5B_KEY("2") : T5B_KEY("1"), K_FF);
    l.ln_ff = w.weight(ffl, T5B_KEY("layer_norm"), K_NORM);
    const Module ff = ffl.find(T5B_KEY("DenseReluDense"));
    if (!ff.self) { s.complete = false; return s; }
    const bool gated = ff.find(T5B_KEY("wi_0")).self != nullptr;
    if (!s.layers.empty() && gated != s.gated) wf.plain = false;
    s.gated = gated;
    wf.look(ff, s.gated ? K_GATED : K_RELU);
    l.wi0 = wf.weight(ff, s.gated ? T5B_KEY("wi_0") : T5B_KEY("wi"), K_LINEAR);
    if (s.gated) l.wi1 = wf.weight(ff, T5B_KEY("wi_1"), K_LINEAR);
    l.wo = wf.weight(ff, T5B_KEY("wo"), K_LINEAR);
    s.layers.push_back(std::move(l));
  }
  s.final_ln = w.weight(top, T5B_KEY("final_layer_norm"), K_NORM);
  s.complete = w.complete && wf.complete && !s.layers.empty();
  if (!s.complete) return s;
  s.d = s.final_ln.dim() == 1 ? s.final_ln.size(0) : 0;
  s.F = s.layers[0].wi0.dim() == 2 ? s.layers[0].wi0.size(0) : 0;
  s.plain = w.plain && wf.plain;
  s.plain_ff = wf.plain;
  s.flash = w.flash;
  return s;
}

// Whether the native passes take this stack: 16-bit weights of one type throughout, on the rows' device, contiguous, of
// the sizes that the products assume (a layer may have been replaced or pruned) and plain tensors (a subclass
// keeps its data elsewhere); d_model of whole 16-byte vectors and at most 2048 (the norm kernels keep a row in
// registers).
bool plain_tensor(const Tensor& t) { return t.is_cuda() && !t.unsafeGetTensorImpl()->is_python_dispatch(); }
bool supported(const Stack& s, const Tensor& x) {
  const at::ScalarType dtype = x.scalar_type();
  if (!is_half_type(dtype) || s.d <= 0 || s.d % 8 || s.d > 2048 || s.F <= 0 || s.F % 8) return false;
  auto ok = [&](const Tensor& t, at::IntArrayRef sizes) {
    return plain_tensor(t) && t.device() == x.device() && t.scalar_type() == dtype && t.sizes() == sizes && t.is_contiguous();
  };
  const int64_t HD = s.H * s.D;
  const int64_t in[] = {HD, s.d}, out[] = {s.d, HD}, up[] = {s.F, s.d}, down[] = {s.d, s.F}, norm[] = {s.d}, table[] = {s.nb, s.H};
  for (const Layer& l : s.layers) {
    if (!ok(l.ln_self, norm) || !ok(l.q, in) || !ok(l.k, in) || !ok(l.v, in) || !ok(l.o, out)) return false;
    if (s.decoder && (!ok(l.ln_cross, norm) || !ok(l.cq, in) || !ok(l.ck, in) || !ok(l.cv, in) || !ok(l.co, out))) return false;
    if (!ok(l.ln_ff, norm) || !ok(l.wi0, up) || !ok(l.wo, down) || (s.gated && !ok(l.wi1, up))) return false;
  }
  return plain_tensor(x) && ok(s.final_ln, norm) && ok(s.table, table);
}

// Stacked weights: [q; k; v], the cross attention's [k; v] and [wi_0; wi_1] of every layer, so that each group
// is one matrix product.  All layers of a group are concatenated by one launch.
struct Stacked {
  Tensor qkv, ckv, wi;
  int64_t HD = 0, F2 = 0;
  Tensor qkv_of(size_t i) const { return qkv.narrow(0, (int64_t)i * 3 * HD, 3 * HD); }
  Tensor ckv_of(size_t i) const { return ckv.narrow(0, (int64_t)i * 2 * HD, 2 * HD); }
  Tensor wi_of(size_t i, const Stack& s) const { return s.gated ? wi.narrow(0, (int64_t)i * F2, F2) : s.layers[i].wi0; }
};
Stacked stack_weights(const Stack& s) {
  at::AutoGradMode no_grad(false);
  std::vector<Tensor> qkv, ckv, wi;
  for (const Layer& l : s.layers) {
    qkv.push_back(l.q); qkv.push_back(l.k); qkv.push_back(l.v);
    if (s.decoder) { ckv.push_back(l.ck); ckv.push_back(l.cv); }
    if (s.gated) { wi.push_back(l.wi0); wi.push_back(l.wi1); }
  }
  Stacked r;
  r.HD = s.H * s.D; r.F2 = 2 * s.F;
  r.qkv = at::cat(qkv);
  if (s.decoder) r.ckv = at::cat(ckv);
  if (s.gated) r.wi = at::cat(wi);
  return r;
}

// Kept with the module for `forward_fused`: the stacked weights of its last pass, rebuilt when a parameter has been
// modified in place or replaced.  Inference tensors have no version that would show a change: weights that hold
// one are stacked anew by every pass, as they are wherever the modules used to read the weights themselves (the
// module interface, a decoding session): those see changes through `p.data` too, which no version shows.
// A pass on another stream waits for the copies and keeps their memory from being given out while it reads.  A
// captured pass stacks inside its graph: eager passes must not read what only a replay would write, a replay
// must not read what a later update has freed, and so a replay sees updated weights.
struct StackCache {
  std::mutex mu;
  // (storage, first element, version) of every stacked parameter; a storage that has been freed never matches
  // again, even where the allocator hands out its address anew
  struct Entry { c10::weak_intrusive_ptr<c10::StorageImpl> storage; const void* data; uint32_t version; };
  std::vector<Entry> key;
  std::shared_ptr<Stacked> weights;
  at::cuda::CUDAEvent ready;             // the copies are written
  std::optional<c10::cuda::CUDAStream> stream;   // ... on this stream
};
std::shared_ptr<Stacked> cached_weights(StackCache* cache, const Stack& s) {
  auto fresh = [&]() { return std::make_shared<Stacked>(stack_weights(s)); };
  if (!cache || at::cuda::currentStreamCaptureStatus() != at::cuda::CaptureStatus::None) return fresh();
  StackCache& c = *cache;
  std::vector<const Tensor*> ts;
  for (const Layer& l : s.layers)
    for (const Tensor* t : {&l.q, &l.k, &l.v, &l.ck, &l.cv, &l.wi0, &l.wi1})
      if (t->defined()) {
        if (t->is_inference()) return fresh();
        ts.push_back(t);
      }
  auto version = [](const Tensor& t) { return (uint32_t)t._version(); };
  std::lock_guard<std::mutex> lock(c.mu);
  bool same = c.weights && c.key.size() == ts.size();
  for (size_t i = 0; same && i < ts.size(); ++i) {
    const auto& e = c.key[i];
    same = e.data == ts[i]->data_ptr() && e.version == version(*ts[i]) &&
           e.storage._unsafe_get_target() == ts[i]->storage().unsafeGetStorageImpl() && !e.storage.expired();
  }
  const auto stream = c10::cuda::getCurrentCUDAStream();
  if (!same) {
    c.weights = fresh();
    c.ready = at::cuda::CUDAEvent();   // (of this device)
    c.ready.record(stream);
    c.stream = stream;
    c.key.clear();
    for (const Tensor* t : ts)
      c.key.push_back({c10::weak_intrusive_ptr<c10::StorageImpl>(t->storage().getWeakStorageImpl()), t->data_ptr(), version(*t)});
  } else if (stream != *c.stream) {
    c.ready.block(stream);
    for (const Tensor* t : {&c.weights->qkv, &c.weights->ckv, &c.weights->wi})
      if (t->defined()) c10::cuda::CUDACachingAllocator::recordStream(t->storage().data_ptr(), stream);
  }
  return c.weights;
}

// What a pass is given besides the weights.
struct PassInputs {
  Tensor x;                    // (B, S, d) rows of this call; packed passes: (1, T, d)
  bool packed = false;         // rows are packed tokens of the sequences in `cu`
  bool padded = false;         // rows are padded; attention packs and pads around itself (cu, dest)
  bool zero_tail = false;      // packed rows past the last token may exist: keep them zero after attention
  Tensor cu, dest;
  int64_t max_len = 0;         // longest sequence of cu (a bound)
  Tensor enc;                  // decoder: (B, L, d), or packed (Te, d) with enc_cu
  Tensor enc_cu, enc_dest;     // packed keys, or (with enc_dest) a padded memory with a mask
  int64_t enc_max = 0;
};

AttnOptions self_options(const Stack& s) {
  AttnOptions o;
  o.causal = s.decoder;
  o.num_buckets = s.nb; o.max_distance = s.md;
  return o;
}
Tensor heads4(const Tensor& t, int64_t B, int64_t S, int64_t H, int64_t D, int64_t col) {      // (R, ld) rows -> (B, H, S, D)
  const int64_t ld = t.stride(0);
  return t.as_strided({B, H, S, D}, {S * ld, D, ld, 1}, t.storage_offset() + col);
}
Tensor heads3(const Tensor& t, int64_t H, int64_t D, int64_t col) {                             // (R, ld) rows -> (R, H, D)
  return t.as_strided({t.size(0), H, D}, {t.stride(0), D, 1}, t.storage_offset() + col);
}

// The self-attention call of a layer: qkv rows -> attn rows (both (R, .)).
void self_attention(AttnCall& c, const Stack& s, const PassInputs& in, const Tensor& qkv, const Tensor& attn, int64_t B, int64_t S,
                    bool want_lse) {
  const int64_t HD = s.H * s.D;
  AttnOptions o = self_options(s);
  if (in.packed || in.padded) {
    o.max_q = o.max_k = in.max_len;
    packed_forward(c, heads3(qkv, s.H, s.D, 0), heads3(qkv, s.H, s.D, HD), heads3(qkv, s.H, s.D, 2 * HD), s.table, in.cu, in.cu, o,
                   want_lse, heads3(attn, s.H, s.D, 0));
  } else {
    dense_forward(c, heads4(qkv, B, S, s.H, s.D, 0), heads4(qkv, B, S, s.H, s.D, HD), heads4(qkv, B, S, s.H, s.D, 2 * HD), s.table, o,
                  want_lse, heads4(attn, B, S, s.H, s.D, 0));
  }
}
void cross_attention(AttnCall& c, const Stack& s, const PassInputs& in, const Tensor& q, const Tensor& ckv, const Tensor& attn,
                     const Tensor& cu_dec, int64_t B, int64_t S, bool want_lse) {
  const int64_t HD = s.H * s.D;
  AttnOptions o;
  o.q_pos_offset = 0;
  if (in.enc_cu.defined()) {
    o.max_q = S; o.max_k = in.enc_max;
    packed_forward(c, heads3(q, s.H, s.D, 0), heads3(ckv, s.H, s.D, 0), heads3(ckv, s.H, s.D, HD), Tensor(), cu_dec, in.enc_cu, o,
                   want_lse, heads3(attn, s.H, s.D, 0));
  } else {
    const int64_t L = in.enc.size(1);
    dense_forward(c, heads4(q, B, S, s.H, s.D, 0), heads4(ckv, B, L, s.H, s.D, 0), heads4(ckv, B, L, s.H, s.D, HD), Tensor(), o, want_lse,
                  heads4(attn, B, S, s.H, s.D, 0));
  }
}

Tensor rows_of(const Tensor& t) { return t.view({-1, t.size(-1)}); }
Tensor new_rows(const Tensor& like, int64_t rows, int64_t cols) { return empty_like_dense({rows, cols}, like.scalar_type(), like.device()); }
Tensor decoder_offsets(const PassInputs& in, int64_t B, int64_t S) {
  return in.enc_cu.defined() ? at::arange(0, (B + 1) * S, S, at::TensorOptions().dtype(at::kInt).device(in.x.device())) : Tensor();
}
// memory rows the cross attention projects keys and values from
Tensor memory_rows(const PassInputs& in) { return in.enc.defined() ? rows_of(in.enc) : Tensor(); }

// Whether the rows, the memory and the plans of their masks belong together.  The gathers and scatters walk a plan's
// destinations for as many rows as there are, and the attention calls take the batch from the rows, so nothing
// else may get here; what the modules make of other sizes (an error, mostly) is theirs to say.
bool matching(const PassInputs& in, bool decoder) {
  const int64_t B = in.x.size(0), R = B * in.x.size(1);
  if (in.packed && !in.cu.defined()) return false;
  if (in.padded && (!in.cu.defined() || in.cu.numel() != B + 1 || !in.dest.defined() || in.dest.numel() != R)) return false;
  if (!decoder) return !in.enc.defined();
  if (!in.enc.defined() || in.packed || in.padded) return false;
  if (in.enc_cu.defined() && in.enc_cu.numel() != B + 1) return false;
  if (in.enc.dim() == 3) {
    if (in.enc.size(0) != B) return false;
    return !in.enc_cu.defined() || (in.enc_dest.defined() && in.enc_dest.numel() == B * in.enc.size(1));
  }
  return in.enc.dim() == 2 && in.enc_cu.defined() && !in.enc_dest.defined();
}

// ------------------------------------------------------------------ inference
Tensor infer(const Stack& s, const Stacked& w, const PassInputs& in) {
  const int64_t B = in.x.size(0), S = in.x.size(1), R = B * S, HD = s.H * s.D;
  // the residual stream is updated in place, in a copy of the caller's rows
  Tensor x = in.x.clone(at::MemoryFormat::Contiguous).view({R, s.d});
  const Tensor normed = new_rows(x, R, s.d), branch = new_rows(x, R, s.d), qkv = new_rows(x, R, 3 * HD), attn = new_rows(x, R, HD);
  const Tensor up = new_rows(x, R, s.gated ? 2 * s.F : s.F), act = s.gated ? new_rows(x, R, s.F) : up;
  if (in.zero_tail) zero_async(attn);        // rows past the last token are never written: zero for every layer
  const Tensor mem = memory_rows(in), cu_dec = decoder_offsets(in, B, S);
  const Tensor ckv = s.decoder ? new_rows(x, mem.size(0), 2 * HD) : Tensor();
  auto norm_into = [&](const Tensor& w_ln) {
    check_status(t5b_rmsnorm_fwd(x.data_ptr(), w_ln.data_ptr(), normed.data_ptr(), nullptr, R, (int32_t)s.d, s.d, s.d,
                                 dtype_code(x.scalar_type()), dtype_code(w_ln.scalar_type()), (float)s.eps, stream_of(x.device())), "rms_layer_norm");
  };
  auto add_norm = [&](const Tensor& w_ln) {
    check_status(t5b_add_rmsnorm_fwd(x.data_ptr(), branch.data_ptr(), w_ln.data_ptr(), x.data_ptr(), normed.data_ptr(), R, (int32_t)s.d,
                                     s.d, s.d, s.d, s.d, dtype_code(x.scalar_type()), dtype_code(w_ln.scalar_type()), (float)s.eps,
                                     stream_of(x.device())), "add_rms_layer_norm");
  };
  norm_into(s.layers[0].ln_self);
  for (size_t i = 0; i < s.layers.size(); ++i) {
    const Layer& l = s.layers[i];
    AttnCall c;
    linear(normed, w.qkv_of(i), qkv);
    if (in.padded) {
      const Tensor packed = gather_rows(qkv, in.dest, R), out = new_rows(x, R, HD);
      self_attention(c, s, in, packed, out, B, S, false);
      linear(scatter_rows(out, in.dest, R), l.o, branch);
    } else {
      self_attention(c, s, in, qkv, attn, B, S, false);
      linear(attn, l.o, branch);
    }
    if (s.decoder) {
      add_norm(l.ln_cross);
      linear(mem, w.ckv_of(i), ckv);
      const Tensor q = qkv.view({-1}).narrow(0, 0, R * HD).view({R, HD});        // the q|k|v rows are done with
      linear(normed, l.cq, q);
      const Tensor keys = in.enc_dest.defined() ? gather_rows(ckv, in.enc_dest, ckv.size(0)) : ckv;
      cross_attention(c, s, in, q, keys, attn, cu_dec, B, S, false);
      linear(attn, l.co, branch);
    }
    add_norm(l.ln_ff);
    linear(normed, w.wi_of(i, s), up);
    if (s.gated)
      check_status(t5b_gated_gelu_fwd(up.data_ptr(), act.data_ptr(), R, (int32_t)s.F, 2 * s.F, s.F, dtype_code(x.scalar_type()),
                                      stream_of(x.device())), "gated_gelu");
    else
      up.relu_();
    linear(act, l.wo, branch);
    add_norm(i + 1 < s.layers.size() ? s.layers[i + 1].ln_self : s.final_ln);
  }
  return normed.view(in.x.sizes());
}

// ------------------------------------------------------------------ training
// What the backward pass of one layer needs from its forward pass.
struct LayerState {
  Tensor x0, n0, qkv, attn;            // residual stream and norm before self attention
  Tensor x1, n1, cq, ckv, cattn;       // ... before cross attention (decoder)
  Tensor x2, n2, up, act;              // ... before the feed-forward layer
  AttnCall self, cross;
};

struct StackNode : public Node {
  Stack s;                             // weights are unpacked from `params` (checked for in-place changes)
  Stacked w;
  PassInputs in;
  std::vector<LayerState> st;
  std::vector<SavedVariable> params;   // in the order of param_list
  SavedVariable saved_x, saved_enc;    // inputs (the rows are read through `in` and `st`)
  Tensor x_final, cu_dec;
  bool alive = true;

  variable_list apply(variable_list&& grads) override;
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto& p : params) p.reset_data();
    saved_x.reset_data(); saved_enc.reset_data();
    st.clear();
    w = Stacked();
    in = PassInputs();
    x_final = cu_dec = Tensor();
    alive = false;
  }
  std::string name() const override { return "T5StackBackward"; }
};

// every parameter of the stack, in a fixed order
std::vector<Tensor*> param_list(Stack& s) {
  std::vector<Tensor*> r = {&s.table, &s.final_ln};
  for (Layer& l : s.layers) {
    for (Tensor* t : {&l.ln_self, &l.q, &l.k, &l.v, &l.o}) r.push_back(t);
    if (s.decoder) for (Tensor* t : {&l.ln_cross, &l.cq, &l.ck, &l.cv, &l.co}) r.push_back(t);
    r.push_back(&l.ln_ff); r.push_back(&l.wi0);
    if (s.gated) r.push_back(&l.wi1);
    r.push_back(&l.wo);
  }
  return r;
}

Tensor train_forward(StackNode& n) {
  const Stack& s = n.s;
  const PassInputs& in = n.in;
  const int64_t B = in.x.size(0), S = in.x.size(1), R = B * S, HD = s.H * s.D;
  Tensor x = in.x.contiguous().view({R, s.d});
  if ((uintptr_t)x.data_ptr() & 15) x = x.clone();           // a view of the caller's; the residual adds read vectors
  const Tensor mem = memory_rows(in);
  n.cu_dec = decoder_offsets(in, B, S);
  const Tensor branch = new_rows(x, R, s.d);
  Tensor normed = rmsnorm(x, s.layers[0].ln_self, s.eps);
  auto add_norm = [&](const Tensor& ln) {
    auto r = add_rmsnorm(x, branch, ln, s.eps, false);
    x = r.first; normed = r.second;
  };
  n.st.resize(s.layers.size());
  for (size_t i = 0; i < s.layers.size(); ++i) {
    const Layer& l = s.layers[i];
    LayerState& t = n.st[i];
    t.x0 = x; t.n0 = normed;
    t.qkv = new_rows(x, R, 3 * HD); t.attn = new_rows(x, R, HD);
    linear(normed, n.w.qkv_of(i), t.qkv);
    if (in.padded) {
      t.qkv = gather_rows(t.qkv, in.dest, R);              // packed from here on; the tail rows are zero
      self_attention(t.self, s, in, t.qkv, t.attn, B, S, true);
      const Tensor padded = scatter_rows(t.attn, in.dest, R);
      linear(padded, l.o, branch);
    } else {
      self_attention(t.self, s, in, t.qkv, t.attn, B, S, true);
      linear(t.attn, l.o, branch);
    }
    if (s.decoder) {
      add_norm(l.ln_cross);
      t.x1 = x; t.n1 = normed;
      t.cq = new_rows(x, R, HD); t.ckv = new_rows(x, mem.size(0), 2 * HD); t.cattn = new_rows(x, R, HD);
      linear(normed, l.cq, t.cq);
      linear(mem, n.w.ckv_of(i), t.ckv);
      if (in.enc_dest.defined()) t.ckv = gather_rows(t.ckv, in.enc_dest, t.ckv.size(0));
      cross_attention(t.cross, s, in, t.cq, t.ckv, t.cattn, n.cu_dec, B, S, true);
      linear(t.cattn, l.co, branch);
    }
    add_norm(l.ln_ff);
    t.x2 = x; t.n2 = normed;
    t.up = new_rows(x, R, s.gated ? 2 * s.F : s.F);
    linear(normed, n.w.wi_of(i, s), t.up);
    if (s.gated) t.act = gated_gelu(t.up);
    else t.act = t.up.relu_();
    linear(t.act, l.wo, branch);
    add_norm(i + 1 < s.layers.size() ? s.layers[i + 1].ln_self : s.final_ln);
  }
  n.x_final = x;
  return normed.view(in.x.sizes());
}

variable_list StackNode::apply(variable_list&& grads) {
  std::lock_guard<std::mutex> lock(mutex_);
  TORCH_CHECK(alive, "Trying to backward through the graph a second time (or directly access saved tensors after they have "
                     "already been freed).");
  const size_t n_params = params.size();
  variable_list out(2 + n_params);                          // x, encoder states, parameters
  if (!grads[0].defined()) return out;
  at::AutoGradMode no_grad(false);
  const c10::cuda::CUDAGuard guard(x_final.device());
  saved_x.unpack();                                         // raises if the rows were changed in place
  // the weights, as saved
  Stack sw = s;
  auto plist = param_list(sw);
  for (size_t i = 0; i < n_params; ++i) *plist[i] = params[i].unpack();
  auto wants = [&](size_t i) { return task_should_compute_output(2 + i); };
  const at::ScalarType dt = x_final.scalar_type();
  const at::Device dev = x_final.device();
  const int64_t R = x_final.size(0), HD = s.H * s.D, d = s.d, F = s.F;
  const size_t nl = sw.layers.size();
  // float32 sums: every norm weight's gradient and the bias table's, cleared by one memset, rounded by one cast
  const int64_t n_norms = (int64_t)nl * (s.decoder ? 3 : 2) + 1;
  const Tensor sums = empty_like_dense({n_norms * d + s.nb * s.H}, at::kFloat, dev);
  zero_async(sums);
  const Tensor dtable = sums.narrow(0, n_norms * d, s.nb * s.H).view({s.nb, s.H});
  int64_t next_norm = 0;
  std::vector<std::pair<size_t, int64_t>> norm_slots;        // (parameter, slot)
  // dx = add + gradient through the norm of x
  auto norm_bwd = [&](size_t param, const Tensor& ln, const Tensor& x, const Tensor& dy, const Tensor& add, const Tensor& dx) {
    const int64_t slot = next_norm++;
    norm_slots.emplace_back(param, slot);
    check_status(t5b_rmsnorm_bwd_add(x.data_ptr(), ln.data_ptr(), dy.data_ptr(), ptr(add), dx.data_ptr(),
                                     (float*)sums.data_ptr() + slot * d, R, (int32_t)d, d, d, d, dtype_code(dt), dtype_code(dt),
                                     (float)s.eps, stream_of(dev)), "rms_layer_norm (backward)");
  };
  auto weight_grad = [&](size_t param, const Tensor& dy, const Tensor& x, int64_t rows, int64_t cols) {
    if (!wants(param)) return;
    out[2 + param] = new_rows(x_final, rows, cols);
    linear_dw(dy, x, out[2 + param]);
  };
  // one product for the gradients of a group of stacked weights
  auto group_grad = [&](size_t first, int count, const Tensor& dy, const Tensor& x, int64_t rows_each) {
    bool any = false;
    for (int k = 0; k < count; ++k) any = any || wants(first + k);
    if (!any) return;
    const Tensor g = new_rows(x_final, rows_each * count, x.size(1));
    linear_dw(dy, x, g);
    for (int k = 0; k < count; ++k) out[2 + first + k] = g.narrow(0, k * rows_each, rows_each);
  };
  const Tensor mem = s.decoder ? rows_of(saved_enc.unpack().contiguous()) : Tensor();
  const bool want_enc = s.decoder && task_should_compute_output(1);
  Tensor denc;
  Tensor dx = new_rows(x_final, R, d);
  const Tensor dn = new_rows(x_final, R, d), dattn = new_rows(x_final, R, HD), dqkv = new_rows(x_final, R, 3 * HD);
  Tensor dact = new_rows(x_final, R, F), dup = s.gated ? new_rows(x_final, R, 2 * F) : dact;
  Tensor dy = grads[0].scalar_type() == dt ? grads[0] : grads[0].to(dt);
  dy = dy.contiguous().view({R, d});
  norm_bwd(1, sw.final_ln, x_final, dy, Tensor(), dx);
  const size_t per_layer = 5 + (s.decoder ? 5 : 0) + (s.gated ? 4 : 3);
  for (size_t i = nl; i-- > 0;) {
    const Layer& l = sw.layers[i];
    LayerState& t = st[i];
    const size_t p0 = 2 + i * per_layer, pc = p0 + 5, pf = p0 + (s.decoder ? 10 : 5);
    // feed-forward layer
    weight_grad(pf + (s.gated ? 3 : 2), dx, t.act, d, F);
    linear_dx(dx, l.wo, dact);
    if (s.gated)
      check_status(t5b_gated_gelu_bwd(t.up.data_ptr(), dact.data_ptr(), dup.data_ptr(), R, (int32_t)F, 2 * F, F, 2 * F, dtype_code(dt),
                                      stream_of(dev)), "gated_gelu (backward)");
    else
      at::threshold_backward_out(dup, dact, t.act, 0);
    group_grad(pf + 1, s.gated ? 2 : 1, dup, t.n2, F);
    linear_dx(dup, w.wi_of(i, sw), dn);
    norm_bwd(pf, l.ln_ff, t.x2, dn, dx, dx);
    // cross attention
    if (s.decoder) {
      weight_grad(pc + 4, dx, t.cattn, d, HD);
      linear_dx(dx, l.co, dattn);
      const Tensor dcq = dqkv.view({-1}).narrow(0, 0, R * HD).view({R, HD});
      Tensor dckv = new_rows(x_final, t.ckv.size(0), 2 * HD);
      AttnCall& c = t.cross;
      if (in.enc_cu.defined()) {
        if (in.zero_tail || in.enc_dest.defined()) zero_async(dckv);         // rows no sequence owns
        attention_backward(c, heads3(dattn, s.H, s.D, 0), heads3(dcq, s.H, s.D, 0), heads3(dckv, s.H, s.D, 0), heads3(dckv, s.H, s.D, HD), Tensor());
        if (in.enc_dest.defined()) dckv = scatter_rows(dckv, in.enc_dest, dckv.size(0));
      } else {
        const int64_t B = in.enc.size(0), L = in.enc.size(1), S = R / B;
        attention_backward(c, heads4(dattn, B, S, s.H, s.D, 0), heads4(dcq, B, S, s.H, s.D, 0), heads4(dckv, B, L, s.H, s.D, 0),
                           heads4(dckv, B, L, s.H, s.D, HD), Tensor());
      }
      weight_grad(pc + 1, dcq, t.n1, HD, d);
      linear_dx(dcq, l.cq, dn);
      group_grad(pc + 2, 2, dckv, mem, HD);
      if (want_enc) {
        const bool first = !denc.defined();
        if (first) denc = new_rows(x_final, mem.size(0), d);
        linear_dx(dckv, w.ckv_of(i), denc, !first);
      }
      norm_bwd(pc, l.ln_cross, t.x1, dn, dx, dx);
    }
    // self attention
    AttnCall& c = t.self;
    linear_dx(dx, l.o, dattn);
    Tensor dq_rows = dqkv;
    if (in.padded) {
      weight_grad(p0 + 4, dx, scatter_rows(t.attn, in.dest, R), d, HD);
      const Tensor da = gather_rows(dattn, in.dest, R), packed = new_rows(x_final, R, 3 * HD);
      zero_async(packed);
      attention_backward(c, heads3(da, s.H, s.D, 0), heads3(packed, s.H, s.D, 0), heads3(packed, s.H, s.D, HD), heads3(packed, s.H, s.D, 2 * HD), dtable);
      dq_rows = scatter_rows(packed, in.dest, R);
    } else {
      weight_grad(p0 + 4, dx, t.attn, d, HD);
      if (in.packed) {
        attention_backward(c, heads3(dattn, s.H, s.D, 0), heads3(dqkv, s.H, s.D, 0), heads3(dqkv, s.H, s.D, HD), heads3(dqkv, s.H, s.D, 2 * HD), dtable);
      } else {
        const int64_t B = c.out.size(0), S = c.out.size(2);
        attention_backward(c, heads4(dattn, B, S, s.H, s.D, 0), heads4(dqkv, B, S, s.H, s.D, 0), heads4(dqkv, B, S, s.H, s.D, HD),
                           heads4(dqkv, B, S, s.H, s.D, 2 * HD), dtable);
      }
    }
    group_grad(p0 + 1, 3, dq_rows, t.n0, HD);
    linear_dx(dq_rows, w.qkv_of(i), dn);
    norm_bwd(p0, l.ln_self, t.x0, dn, dx, dx);
  }
  const Tensor rounded = sums.to(dt);
  for (auto& ns : norm_slots)
    if (wants(ns.first)) out[2 + ns.first] = rounded.narrow(0, ns.second * d, d);
  if (wants(0)) {
    Tensor g = rounded.narrow(0, n_norms * d, s.nb * s.H).view({s.nb, s.H});
    out[2] = g.slice(0, 0, sw.table.size(0));
  }
  if (task_should_compute_output(0)) out[0] = dx.view(in.x.sizes());
  if (want_enc) out[1] = denc.view(in.enc.sizes());
  return out;
}

void free_cache(PyObject* capsule) { delete (StackCache*)PyCapsule_GetPointer(capsule, "t5b_stack_cache"); }

PyObject* py_new_stack_cache(PyObject*, PyObject* const*, Py_ssize_t) {
  HANDLE_TH_ERRORS
  return PyCapsule_New(new StackCache(), "t5b_stack_cache", free_cache);
  END_HANDLE_TH_ERRORS
}

// stack_forward(stack, types, cache or None, decoder, heads, d_kv, buckets, max_distance, eps, need_plain,
//               x, mode, cu, dest, max_len, zero_tail, enc, enc_cu, enc_dest, enc_max)
// mode: 0 plain rows, 1 packed rows (cu), 2 padded rows with a mask (cu, dest).
// Returns None when the pass is not one of the native ones (types, sizes, missing modules, a feed-forward layer of
// another class or with hooks; with `need_plain` or in training also when any other module of the stack is): the caller then runs the
// modules or operators.
PyObject* py_stack_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 20);
  Stack s = collect(a[0], a[1], bool_arg(a[3]), int_arg(a[4]), int_arg(a[5]), (int)int_arg(a[6]), (int)int_arg(a[7]), float_arg(a[8]));
  PassInputs in;
  in.x = tensor_arg(a[10]);
  const int64_t mode = int_arg(a[11]);
  in.packed = mode == 1; in.padded = mode == 2;
  in.cu = tensor_arg(a[12]); in.dest = tensor_arg(a[13]); in.max_len = int_arg(a[14]); in.zero_tail = bool_arg(a[15]);
  in.enc = tensor_arg(a[16]); in.enc_cu = tensor_arg(a[17]); in.enc_dest = tensor_arg(a[18]); in.enc_max = int_arg(a[19]);
  if (!s.complete || !s.flash || (s.D != 16 && s.D != 32 && s.D != 64 && s.D != 128) || s.md > 2048) Py_RETURN_NONE;
  // (a feed-forward layer is always the caller's module: what it computes shows in its class and nowhere else)
  if (!s.plain_ff || (bool_arg(a[9]) && !s.plain)) Py_RETURN_NONE;
  if (!in.x.is_cuda() || in.x.dim() != 3 || in.x.size(2) != s.d || !supported(s, in.x)) Py_RETURN_NONE;
  if (in.enc.defined() && (!plain_tensor(in.enc) || in.enc.device() != in.x.device() || in.enc.scalar_type() != in.x.scalar_type() ||
                           in.enc.size(-1) != s.d)) Py_RETURN_NONE;
  if (in.x.numel() == 0 || (in.enc.defined() && in.enc.numel() == 0)) Py_RETURN_NONE;
  if (!matching(in, s.decoder)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(in.x.device());
  bool grad = false;
  auto plist = param_list(s);
  if (at::GradMode::is_enabled()) {
    grad = in.x.requires_grad() || (in.enc.defined() && in.enc.requires_grad());
    for (Tensor* t : plist) grad = grad || t->requires_grad();
  }
  if (!grad) {
    auto* cache = a[2] == Py_None ? nullptr : (StackCache*)PyCapsule_GetPointer(a[2], "t5b_stack_cache");
    if (!cache && a[2] != Py_None) throw python_error();
    at::AutoGradMode no_grad(false);
    if (in.enc.defined()) in.enc = in.enc.contiguous();
    Tensor r;
    {
      pybind11::gil_scoped_release nogil;
      r = infer(s, *cached_weights(cache, s), in);
    }
    return wrap(r);
  }
  if (!s.plain) Py_RETURN_NONE;
  // Hooks on what is saved (offloading, checkpointing) have to see the activations: the modules save them one by
  // one, where the node keeps them to itself.
  if (at::SavedTensorDefaultHooks::get_hooks().has_value()) Py_RETURN_NONE;
  // (the operators refuse forward-mode inputs)
  if (has_tangent(in.x) || has_tangent(in.enc)) Py_RETURN_NONE;
  for (Tensor* t : plist)
    if (has_tangent(*t)) Py_RETURN_NONE;
  auto node = std::make_shared<StackNode>();
  Tensor y;
  {
    pybind11::gil_scoped_release nogil;
    torch::autograd::edge_list edges;
    auto edge = [&](const Tensor& t) {
      edges.push_back(t.defined() && t.requires_grad() ? torch::autograd::impl::gradient_edge(t) : torch::autograd::Edge());
    };
    edge(in.x); edge(in.enc);
    for (Tensor* t : plist) { edge(*t); node->params.emplace_back(*t, false); }
    node->set_next_edges(std::move(edges));
    node->saved_x = SavedVariable(in.x, false);
    if (in.enc.defined()) node->saved_enc = SavedVariable(in.enc, false);
    at::AutoGradMode no_grad(false);
    in.x = in.x.detach();
    if (in.enc.defined()) in.enc = in.enc.detach().contiguous();
    node->w = stack_weights(s);
    for (Tensor* t : plist) *t = t->detach();
    node->s = s;
    node->in = in;
    y = train_forward(*node);
    // only sizes are needed from here on: the weights come from the saved variables
    for (Tensor* t : param_list(node->s)) *t = Tensor();
    torch::autograd::set_history(y, node);
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------ greedy decoding
// One generation: caches, weights and the argument block of t5b_decoder_step.
struct DecodeSession {
  Stack s;
  Stacked w;
  Tensor head, embedding, hidden, logits, tokens, seqlens, enc_seqlens, workspace;
  std::vector<Tensor> self_kv, ckv;
  std::vector<t5b_decoder_layer> layers;
  t5b_decoder_step_args a = {};
  int64_t start_token = 0;

  void rewind() {
    hidden.copy_(embedding.select(0, start_token).expand_as(hidden));
    seqlens.fill_(1);
  }
  void step() { check_status(t5b_decoder_step(&a, stream_of(hidden.device())), "decoder step"); }

  // `n` steps.  A step is a chain of one to two hundred launches of 2-4 us each, about what the host needs to issue
  // one; from a few steps on the chain is recorded once (a CUDA graph on a stream of its own: nothing in it
  // depends on the step) and launched n times.
  void run(int64_t n) {
    const cudaStream_t stream = stream_of(hidden.device());
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess) cudaGetLastError();
    if (n < kGraphSteps || capturing != cudaStreamCaptureStatusNone) {
      for (int64_t i = 0; i < n; ++i) step();
      return;
    }
    step();                            // kernel attributes are set by a kernel's first launch, outside a capture
    cudaStream_t side = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int st = T5B_ERR_LAUNCH;
    if (cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking) == cudaSuccess &&
        cudaStreamBeginCapture(side, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      st = t5b_decoder_step(&a, side);
      if (cudaStreamEndCapture(side, &graph) != cudaSuccess) st = T5B_ERR_LAUNCH;
    }
    if (st == T5B_OK && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) st = T5B_ERR_LAUNCH;
    for (int64_t i = 1; st == T5B_OK && i < n; ++i)
      if (cudaGraphLaunch(exec, stream) != cudaSuccess) st = T5B_ERR_LAUNCH;
    // an executable graph may be destroyed while its launches are still running: it is freed when they are done
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (side) cudaStreamDestroy(side);
    if (st != T5B_OK) cudaGetLastError();
    check_status(st, "decoder step");
  }
  static constexpr int64_t kGraphSteps = 6;
};

DecodeSession& session_arg(PyObject* o) {
  auto* p = (DecodeSession*)PyCapsule_GetPointer(o, "t5b_decode_session");
  if (!p) throw python_error();
  return *p;
}
void free_session(PyObject* o) { delete (DecodeSession*)PyCapsule_GetPointer(o, "t5b_decode_session"); }

// new_decode_session(stack, types, heads, d_kv, buckets, max_distance, eps,
//                    memory, enc_seqlens, max_len, lm_head weight, embedding weight, lm_scale, start_token)
// None when the step kernels do not cover this decoder (types, sizes, replaced modules or hooks).
PyObject* py_new_decode_session(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 14);
  auto ses = std::make_unique<DecodeSession>();
  DecodeSession& d = *ses;
  d.s = collect(a[0], a[1], true, int_arg(a[2]), int_arg(a[3]), (int)int_arg(a[4]), (int)int_arg(a[5]), float_arg(a[6]));
  const Tensor memory = tensor_arg(a[7]);
  d.enc_seqlens = tensor_arg(a[8]);
  const int64_t max_len = int_arg(a[9]);
  d.head = tensor_arg(a[10]); d.embedding = tensor_arg(a[11]);
  d.start_token = int_arg(a[13]);
  const Stack& s = d.s;
  if (!s.complete || !s.plain || !memory.is_cuda() || memory.dim() != 3 || memory.size(2) != s.d || memory.numel() == 0 || max_len <= 0) Py_RETURN_NONE;
  const at::ScalarType dt = memory.scalar_type();
  auto plain = [&](const Tensor& t) {
    return plain_tensor(t) && t.device() == memory.device() && t.scalar_type() == dt && t.is_contiguous() && t.dim() == 2 && t.size(1) == s.d;
  };
  if (!supported(s, memory) || !plain(d.head) || !plain(d.embedding)) Py_RETURN_NONE;
  // what the step kernels fetch with 16-byte loads and bulk copies (the stacked copies are allocations of their own)
  auto aligned = [](const Tensor& t) { return !t.defined() || ((uintptr_t)t.data_ptr() & 15) == 0; };
  if (!aligned(d.head) || !aligned(d.embedding) || !aligned(s.final_ln)) Py_RETURN_NONE;
  for (const Layer& l : s.layers)
    if (!aligned(l.ln_self) || !aligned(l.o) || !aligned(l.ln_cross) || !aligned(l.cq) || !aligned(l.co) || !aligned(l.ln_ff) ||
        !aligned(l.wi0) || !aligned(l.wo)) Py_RETURN_NONE;
  if (d.start_token < 0 || d.start_token >= d.embedding.size(0) || d.head.size(0) > d.embedding.size(0)) Py_RETURN_NONE;
  const int64_t B = memory.size(0), L = memory.size(1), HD = s.H * s.D;
  if (d.enc_seqlens.defined()) {
    if (!plain_tensor(d.enc_seqlens) || d.enc_seqlens.device() != memory.device() || d.enc_seqlens.scalar_type() != at::kInt ||
        d.enc_seqlens.numel() != B) Py_RETURN_NONE;
    d.enc_seqlens = d.enc_seqlens.contiguous();
  }
  const at::Device dev = memory.device();
  const c10::cuda::CUDAGuard guard(dev);
  at::AutoGradMode no_grad(false);
  t5b_decoder_step_args& k = d.a;
  k.dtype = dtype_code(dt); k.table_dtype = dtype_code(s.table.scalar_type());
  k.device_status = device_status(dev.index()).data_ptr<int32_t>();
  k.n_layers = (int32_t)s.layers.size(); k.B = (int32_t)B; k.H = (int32_t)s.H; k.D = (int32_t)s.D;
  k.d_model = (int32_t)s.d; k.d_ff = (int32_t)s.F; k.gated = s.gated; k.vocab = (int32_t)d.head.size(0);
  k.max_len = (int32_t)max_len; k.enc_len = (int32_t)L;
  k.num_buckets = s.nb; k.max_distance = s.md;
  k.eps = (float)s.eps; k.lm_scale = (float)float_arg(a[12]);
  k.cross_stride_b = L * 2 * HD; k.cross_stride_n = 2 * HD; k.cross_stride_h = s.D;
  d.workspace = empty_like_dense({t5b_decoder_step_workspace_bytes(&k)}, at::kByte, dev);
  k.workspace = d.workspace.data_ptr(); k.workspace_bytes = d.workspace.numel();
  k.table = s.table.data_ptr(); k.table_stride0 = s.table.stride(0);
  d.layers.resize(s.layers.size());
  k.layers = d.layers.data();
  // sizes, bucket settings and head dims no step kernel takes show here, before anything is computed
  const int st = t5b_decoder_step_prepare(&k, stream_of(dev));
  if (st == T5B_ERR_UNSUPPORTED) Py_RETURN_NONE;
  check_status(st, "decoder step");
  {
    pybind11::gil_scoped_release nogil;
    d.w = stack_weights(s);
    d.hidden = empty_like_dense({B, s.d}, dt, dev);
    d.logits = empty_like_dense({B, 1, d.head.size(0)}, dt, dev);
    d.tokens = empty_like_dense({B, max_len}, at::kLong, dev);
    zero_async(d.tokens);
    d.seqlens = empty_like_dense({B}, at::kInt, dev);
    k.hidden = d.hidden.data_ptr(); k.logits = d.logits.data_ptr(); k.tokens = d.tokens.data_ptr<int64_t>();
    k.tokens_stride = max_len; k.seqlens = d.seqlens.data_ptr<int32_t>();
    k.enc_seqlens = (const int32_t*)ptr(d.enc_seqlens);
    k.final_ln = s.final_ln.data_ptr(); k.lm_head = d.head.data_ptr(); k.embedding = d.embedding.data_ptr();
    const Tensor mem = memory.contiguous().view({B * L, s.d});
    for (size_t i = 0; i < s.layers.size(); ++i) {
      // cross keys and values of the layer, projected once: rows of k | v per memory token
      d.ckv.push_back(new_rows(mem, B * L, 2 * HD));
      linear(mem, d.w.ckv_of(i), d.ckv.back());
      d.self_kv.push_back(empty_like_dense({2, B, s.H, max_len, s.D}, dt, dev));
      const Layer& l = s.layers[i];
      t5b_decoder_layer& o = d.layers[i];
      o.ln_self = l.ln_self.data_ptr(); o.wqkv = d.w.qkv_of(i).data_ptr(); o.wo = l.o.data_ptr();
      o.ln_cross = l.ln_cross.data_ptr(); o.wcq = l.cq.data_ptr(); o.wco = l.co.data_ptr();
      o.ln_ff = l.ln_ff.data_ptr(); o.wi = d.w.wi_of(i, s).data_ptr(); o.wff = l.wo.data_ptr();
      o.self_kv = d.self_kv.back().data_ptr();
      o.cross_k = d.ckv.back().data_ptr();
      o.cross_v = (const char*)d.ckv.back().data_ptr() + HD * 2;
    }
    d.rewind();
  }
  return PyCapsule_New(ses.release(), "t5b_decode_session", free_session);
  END_HANDLE_TH_ERRORS
}

// decode_session_run(session, steps)
PyObject* py_decode_session_run(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 2);
  DecodeSession& d = session_arg(a[0]);
  const int64_t steps = int_arg(a[1]);
  const c10::cuda::CUDAGuard guard(d.hidden.device());
  {
    pybind11::gil_scoped_release nogil;
    d.run(steps);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* py_decode_session_rewind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 1);
  at::AutoGradMode no_grad(false);
  session_arg(a[0]).rewind();
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// (tokens, logits) of the last step
PyObject* py_decode_session_tensors(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 1);
  DecodeSession& d = session_arg(a[0]);
  return wrap2(d.tokens, d.logits);
  END_HANDLE_TH_ERRORS
}

}  // namespace

PyMethodDef stack_methods[] = {T5B_METHOD("stack_forward", py_stack_forward), T5B_METHOD("new_stack_cache", py_new_stack_cache),
                               T5B_METHOD("new_decode_session", py_new_decode_session),
                               T5B_METHOD("decode_session_run", py_decode_session_run),
                               T5B_METHOD("decode_session_rewind", py_decode_session_rewind),
                               T5B_METHOD("decode_session_tensors", py_decode_session_tensors),
                               {nullptr, nullptr, 0, nullptr}};

}  // namespace t5b_host
