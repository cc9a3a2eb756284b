// One cached decoding step of a T5 decoder for a batch of up to 64 rows: all layers, the LM head, the greedy
// choice and the next token's embedding, as a chain of small kernels.
//
// A step reads every weight once and every cached key and value once, and computes almost nothing: at 16 rows
// the weights of a large-shaped layer (29 MB) and its 1024 cross keys (67 MB) take 15 us of HBM time, but spread
// over thirteen library calls they took 70 us, because each of those starts cold (launch, descriptor set-up, first
// loads) after the one before it has drained.  Here a layer is eight kernels, each fused with what surrounds its
// matrix product (norm before it; cache append, residual add, activation or argmax after it), and they are
// launched with programmatic dependencies: a block first requests its whole slice of the weights -- which no
// earlier kernel writes -- into shared memory, and only then waits for its predecessor.
//
//   [norm, q|k|v, append]  [self attention]  [o, residual]
//   [norm, cross q]        [cross attention] [o, residual]
//   [norm, wi, activation] [wo, residual]          ... per layer
//   [norm, LM head, argmax] [choice, append token, embedding]
//
// Every kernel lets its successor start (launch_dependents) only AFTER its own wait, so whatever ran two kernels
// earlier has completed, memory included, when a block starts: weights, cross keys and the cached keys of
// earlier steps may be read before the wait; activations and the newest key may not.
//
// Semantics: the cached step of the decoder stack (src/turbot5/model/modeling.py:166-219 per block,
// src/turbot5/model/attentions.py:198,229-234), rounding points as the separate operators.
#include "t5b_common.cuh"

#include <atomic>

namespace t5b {
namespace step {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 r;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a));
  return r;
}
__device__ __forceinline__ void sts128(uint32_t a, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// activations: written by an earlier kernel of the chain, so not through the non-coherent path
__device__ __forceinline__ uint4 ld_act(const void* p) {
  uint4 r;
  asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
  return r;
}

template <typename T> __device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                                uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                                    uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma16816<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                             uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <typename T> __device__ __forceinline__ T round_to(float x) { return from_float<T>(x); }
template <typename T> __device__ __forceinline__ float rounded(float x) { return to_float<T>(from_float<T>(x)); }

// ---------------------------------------------------------------- skinny matrix products
// y[B, N] = f(x)[B, K] w[N, K]^T for B <= 64.  A block owns NT * 8 rows of w (all of K), its warps take the
// 32-wide pieces of K in turn, sixteen rows of x at a time, and meet in shared memory.  mma.m16n8k16: these
// products are a stream of weights (16 flop per byte at 16 rows); the tensor unit is idle either way, and a
// tcgen05 tile of 128 rows would be seven eighths padding.
//
// Operands are read with 16-byte loads: a lane takes eight consecutive k of its row where the instruction's
// layout asks for four pairs eight apart; the order of k inside a 32-wide piece is the same for both operands,
// so the products meet.  Row pitch K * 2 + 64 bytes: the rows of a quarter warp's load fall into different banks.
enum Epilogue { E_STORE = 0, E_QKV, E_RESIDUAL, E_GATED, E_RELU, E_LOGITS };

struct GemmParams {
  const void* x; const void* w; const void* ln; void* out;
  const void* residual;            // E_RESIDUAL: hidden (out is hidden too)
  void* kv;                        // E_QKV: cache (2, B, H, max_len, D)
  const int32_t* seqlens;          // E_QKV: cached keys of each row, the new one included
  float2* cand;                    // E_LOGITS: (value, index bits) of each row and block
  int32_t B, N, K, F;              // F: E_GATED: rows of wi_0 (w holds wi_0 | wi_1)
  int32_t H, D, max_len, x_stride;
  float eps, x_scale;              // x_scale: multiplies the normed rows (tied embeddings), 1 = off
};

__device__ __forceinline__ float gelu_tanh(float a) {
  const float u2 = 1.5957691216057308f * a * fmaf(0.044715f * a, a, 1.f);
  return a * __frcp_rn(1.f + fast_exp2(-u2 * kLog2e));
}
// whether (a, ia) comes before (b, ib) in an argmax: larger value, NaN above all, ties to the lower index
__device__ __forceinline__ bool argmax_before(float a, int ia, float b, int ib) {
  const bool na = isnan(a), nb = isnan(b);
  if (na != nb) return na;
  if (!na && a != b) return a > b;
  return ia < ib;
}

// kNorm: 0 no norm; 1: rows of up to 1024 (four 16-byte vectors per lane, all of a warp's rows at once);
// 2: up to 2048 (eight vectors, one row at a time).  Registers are held to what lets three blocks share an SM:
// the successor's blocks have to find room beside the running ones.
template <typename T, int WARPS, int NT, int kNorm, int kEpi>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 3 : 2)
step_gemm_kernel(const __grid_constant__ GemmParams p) {
  constexpr int THREADS = WARPS * 32;
  constexpr int COLS = NT * 8;                               // accumulator columns of the block
  constexpr int OUT_COLS = kEpi == E_GATED ? COLS / 2 : COLS;
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = p.K, nvec = K >> 3;
  const uint32_t pitch = (uint32_t)K * 2 + 64;
  const uint32_t sW = smem_u32(smem);
  const uint32_t sLn = sW + COLS * pitch;
  const uint32_t sX = sLn + (kNorm ? (uint32_t)K * 2 : 0u);
  float* red = reinterpret_cast<float*>(smem + COLS * pitch + (kNorm ? (uint32_t)K * 2 + 16 * pitch : 0u));
  const int n0 = blockIdx.x * OUT_COLS;

  // the block's weights, before anything that depends on an earlier kernel
  for (int r = warp; r < COLS; r += WARPS) {
    int n;
    if (kEpi == E_GATED) n = r < COLS / 2 ? n0 + r : p.F + n0 + r - COLS / 2;
    else n = n0 + r;
    const bool ok = kEpi == E_GATED ? n0 + (r % (COLS / 2)) < p.F : n < p.N;
    const char* src = (const char*)p.w + (int64_t)n * K * 2;
    for (int c = lane; c < nvec; c += 32) {
      if (ok) cp_async16(sW + r * pitch + c * 16, src + c * 16);
      else sts128(sW + r * pitch + c * 16, make_uint4(0, 0, 0, 0));
    }
  }
  if (kNorm)
    for (int c = tid; c < nvec; c += THREADS) cp_async16(sLn + c * 16, (const char*)p.ln + c * 16);
  cp_async_commit();
  grid_wait();
  grid_launch_dependents();

  const int g = lane >> 2, t = lane & 3;
  for (int m0 = 0; m0 < p.B; m0 += 16) {
    if (kNorm) {
      constexpr int ROWS = 16 / WARPS;                       // rows per warp
      constexpr int VECS = kNorm == 2 ? 8 : 4, AT_ONCE = kNorm == 2 ? 1 : ROWS;
      #pragma unroll 1
      for (int q0 = 0; q0 < ROWS; q0 += AT_ONCE) {
        uint4 xv[AT_ONCE][VECS];
        #pragma unroll
        for (int q = 0; q < AT_ONCE; ++q) {
          const int row = m0 + warp + (q0 + q) * WARPS;
          #pragma unroll
          for (int i = 0; i < VECS; ++i) {
            const int c = lane + i * 32;
            xv[q][i] = make_uint4(0, 0, 0, 0);
            if (row < p.B && c < nvec) xv[q][i] = ld_act((const char*)p.x + (int64_t)row * p.x_stride * 2 + c * 16);
          }
        }
        if (q0 == 0) {
          cp_async_wait_all();
          __syncthreads();                                   // ln is in shared memory; the rows of the last round are done with
        }
        #pragma unroll
        for (int q = 0; q < AT_ONCE; ++q) {
          float ss = 0.f;
          #pragma unroll
          for (int i = 0; i < VECS; ++i) {
            const T* e = reinterpret_cast<const T*>(&xv[q][i]);
            #pragma unroll
            for (int k = 0; k < 8; ++k) { const float f = to_float<T>(e[k]); ss = fmaf(f, f, ss); }
          }
          #pragma unroll
          for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
          const float rstd = rsqrtf(ss / (float)K + p.eps);
          #pragma unroll
          for (int i = 0; i < VECS; ++i) {
            const int c = lane + i * 32;
            if (c < nvec) {
              const uint4 wv = lds128(sLn + c * 16);
              const T* e = reinterpret_cast<const T*>(&xv[q][i]);
              const T* we = reinterpret_cast<const T*>(&wv);
              uint4 o4;
              T* oe = reinterpret_cast<T*>(&o4);
              #pragma unroll
              for (int k = 0; k < 8; ++k) {
                float y = rounded<T>(to_float<T>(we[k]) * rounded<T>(to_float<T>(e[k]) * rstd));
                if (kEpi == E_LOGITS && p.x_scale != 1.f) y = rounded<T>(y * p.x_scale);
                oe[k] = round_to<T>(y);
              }
              sts128(sX + (warp + (q0 + q) * WARPS) * pitch + c * 16, o4);
            }
          }
        }
      }
    } else {
      cp_async_wait_all();
    }
    __syncthreads();

    float acc[NT][4];
    #pragma unroll
    for (int j = 0; j < NT; ++j)
      #pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    const char* xlo = (const char*)p.x + (int64_t)(m0 + g) * p.x_stride * 2 + t * 16;
    const char* xhi = xlo + (int64_t)8 * p.x_stride * 2;
    const bool lo_ok = m0 + g < p.B, hi_ok = m0 + g + 8 < p.B;
    #pragma unroll 4
    for (int kb = warp; kb < (K >> 5); kb += WARPS) {
      uint4 a = make_uint4(0, 0, 0, 0), b = make_uint4(0, 0, 0, 0);     // rows g and g + 8
      if (kNorm) {
        a = lds128(sX + g * pitch + kb * 64 + t * 16);
        b = lds128(sX + (g + 8) * pitch + kb * 64 + t * 16);
      } else {
        if (lo_ok) a = ld_act(xlo + kb * 64);
        if (hi_ok) b = ld_act(xhi + kb * 64);
      }
      #pragma unroll
      for (int j = 0; j < NT; ++j) {
        const uint4 w4 = lds128(sW + (j * 8 + g) * pitch + kb * 64 + t * 16);
        mma16816<T>(acc[j], a.x, b.x, a.y, b.y, w4.x, w4.y);
        mma16816<T>(acc[j], a.z, b.z, a.w, b.w, w4.z, w4.w);
      }
    }
    // ---- the warps' partial sums meet: red[warp][row][column]
    #pragma unroll
    for (int j = 0; j < NT; ++j) {
      float* r0 = red + (warp * 16 + g) * COLS + j * 8 + 2 * t;
      *reinterpret_cast<float2*>(r0) = make_float2(acc[j][0], acc[j][1]);
      *reinterpret_cast<float2*>(r0 + 8 * COLS) = make_float2(acc[j][2], acc[j][3]);
    }
    __syncthreads();
    for (int idx = tid; idx < 16 * OUT_COLS; idx += THREADS) {
      const int r = idx / OUT_COLS, c = idx % OUT_COLS;
      const int row = m0 + r, n = n0 + c;
      float s = 0.f, s2 = 0.f;
      #pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        s += red[(w * 16 + r) * COLS + c];
        if (kEpi == E_GATED) s2 += red[(w * 16 + r) * COLS + COLS / 2 + c];
      }
      const bool ok = row < p.B && n < (kEpi == E_GATED ? p.F : p.N);
      if (kEpi == E_STORE) {
        if (ok) ((T*)p.out)[(int64_t)row * p.N + n] = round_to<T>(s);
      } else if (kEpi == E_RELU) {
        if (ok) ((T*)p.out)[(int64_t)row * p.N + n] = round_to<T>(fmaxf(s, 0.f));
      } else if (kEpi == E_GATED) {
        if (ok) ((T*)p.out)[(int64_t)row * p.F + n] = round_to<T>(rounded<T>(gelu_tanh(rounded<T>(s))) * rounded<T>(s2));
      } else if (kEpi == E_RESIDUAL) {
        if (ok) {
          T* o = (T*)p.out + (int64_t)row * p.N + n;
          *o = round_to<T>(to_float<T>(*o) + rounded<T>(s));
        }
      } else if (kEpi == E_QKV) {
        if (ok) {
          const int HD = p.H * p.D;
          if (n < HD) ((T*)p.out)[(int64_t)row * HD + n] = round_to<T>(s);
          else {
            const int kv = n >= 2 * HD ? 1 : 0, m = n - HD - kv * HD, h = m / p.D, d = m - h * p.D;
            const int pos = p.seqlens[row] - 1;
            if (pos >= 0 && pos < p.max_len)
              ((T*)p.kv)[((((int64_t)kv * p.B + row) * p.H + h) * p.max_len + pos) * p.D + d] = round_to<T>(s);
          }
        }
      } else {     // E_LOGITS: a warp holds the 32 columns of one row (NT = 4)
        const float v = rounded<T>(s);
        if (ok) ((T*)p.out)[(int64_t)row * p.N + n] = round_to<T>(s);
        float bv = ok ? v : -INFINITY;
        int bi = ok ? n : 0x7fffffff;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (argmax_before(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0 && row < p.B) p.cand[(int64_t)row * gridDim.x + blockIdx.x] = make_float2(bv, __int_as_float(bi));
      }
    }
    if (m0 + 16 < p.B) __syncthreads();                       // `red` is written again
  }
}

// ---------------------------------------------------------------- attention of one query row per (batch, head)
// grid = (splits, H, B).  D / 8 lanes own a key row (16 bytes of it each), so a warp load covers 32 / (D / 8) keys;
// four loads of K and four of V per lane are in flight, the next four requested before the current ones are used.
// Cross keys are constant, so the first of them are requested before the wait.
struct AttnStepParams {
  const void* q; const void* k; const void* v; void* out;      // q, out (B, H * D)
  int64_t k_stride_b, k_stride_h, k_stride_n;                  // elements; v has the same
  const int32_t* lens;             // keys of each row (self: the new one included), or NULL: N
  const float* bias;               // self: [H][md + 1], log2 domain, by distance; NULL: none
  int32_t* counters; float* part_ml; float* part_o;
  int32_t B, H, N, md, splits;
};

template <typename T, int D, int WARPS, bool kSelf>
__global__ void __launch_bounds__(WARPS * 32)
step_attention_kernel(const __grid_constant__ AttnStepParams p) {
  constexpr int LPK = D / 8, KPW = 32 / LPK, UNROLL = 4, KPI = KPW * UNROLL;
  __shared__ float sm_m[WARPS], sm_l[WARPS];
  __shared__ float sm_o[WARPS][D];
  __shared__ int is_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = lane / LPK, gl = lane % LPK;
  const int split = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const char* kbase = (const char*)p.k + 2 * ((int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h + gl * 8);
  const char* vbase = (const char*)p.v + 2 * ((int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h + gl * 8);
  const int64_t kstep = 2 * p.k_stride_n;
  uint4 kr[2][UNROLL], vr[2][UNROLL];
  int n_begin = 0, n_end = 0;
  auto range = [&]() {
    const int len = p.lens ? min(p.lens[b], p.N) : p.N;
    int chunk = (len + p.splits - 1) / p.splits;
    chunk = (chunk + WARPS * KPI - 1) / (WARPS * KPI) * (WARPS * KPI);
    n_begin = min(split * chunk, len);
    n_end = min(n_begin + chunk, len);
    return len;
  };
  auto load = [&](int it, uint4 (&k4)[UNROLL], uint4 (&v4)[UNROLL]) {
    #pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int n = it + u * KPW + grp;
      k4[u] = make_uint4(0, 0, 0, 0); v4[u] = make_uint4(0, 0, 0, 0);
      if (n < n_end) {
        if (kSelf) { k4[u] = ld_act(kbase + n * kstep); v4[u] = ld_act(vbase + n * kstep); }
        else {
          asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(k4[u].x), "=r"(k4[u].y), "=r"(k4[u].z), "=r"(k4[u].w) : "l"(kbase + n * kstep));
          asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(v4[u].x), "=r"(v4[u].y), "=r"(v4[u].z), "=r"(v4[u].w) : "l"(vbase + n * kstep));
        }
      }
    }
  };
  int len = 0;
  if (!kSelf) {                      // the lengths of the memory are constant too
    len = range();
    load(n_begin + warp * KPI, kr[0], vr[0]);
  }
  grid_wait();
  grid_launch_dependents();
  const uint4 q4 = ld_act((const char*)p.q + 2 * (((int64_t)b * p.H + h) * D + gl * 8));
  if (kSelf) {
    len = range();
    load(n_begin + warp * KPI, kr[0], vr[0]);
  }
  float q[8], acc[8];
  {
    const T* e = reinterpret_cast<const T*>(&q4);
    #pragma unroll
    for (int i = 0; i < 8; ++i) { q[i] = to_float<T>(e[i]) * kLog2e; acc[i] = 0.f; }
  }
  float m_run = -INFINITY, l_run = 0.f;
  const float* brow = kSelf ? p.bias + (int64_t)h * (p.md + 1) : nullptr;

  auto consume = [&](int it, const uint4 (&k4)[UNROLL], const uint4 (&v4)[UNROLL]) {
    float s[UNROLL];
    #pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int n = it + u * KPW + grp;
      float bias = 0.f;
      if (kSelf && n < n_end) bias = __ldg(brow + min(len - 1 - n, p.md));
      const T* e = reinterpret_cast<const T*>(&k4[u]);
      float d = 0.f;
      #pragma unroll
      for (int i = 0; i < 8; ++i) d = fmaf(q[i], to_float<T>(e[i]), d);
      #pragma unroll
      for (int o = 1; o < LPK; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      s[u] = n < n_end ? d + bias : -INFINITY;
    }
    float mx = s[0];
    #pragma unroll
    for (int u = 1; u < UNROLL; ++u) mx = fmaxf(mx, s[u]);
    const float m_new = fmaxf(m_run, mx);
    const float m_safe = m_new == -INFINITY ? 0.f : m_new;
    const float alpha = fast_exp2(m_run - m_safe);
    m_run = m_new;
    l_run *= alpha;
    #pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= alpha;
    #pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const float pr = fast_exp2(s[u] - m_safe);
      l_run += pr;
      const T* e = reinterpret_cast<const T*>(&v4[u]);
      #pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(pr, to_float<T>(e[i]), acc[i]);
    }
  };
  int it = n_begin + warp * KPI;
  while (it < n_end) {
    load(it + WARPS * KPI, kr[1], vr[1]);
    consume(it, kr[0], vr[0]);
    it += WARPS * KPI;
    if (it >= n_end) break;
    load(it + WARPS * KPI, kr[0], vr[0]);
    consume(it, kr[1], vr[1]);
    it += WARPS * KPI;
  }

  // ---- merge lane groups, then warps
  #pragma unroll
  for (int o = LPK; o < 32; o <<= 1) {
    const float m_o = __shfl_xor_sync(0xffffffffu, m_run, o), l_o = __shfl_xor_sync(0xffffffffu, l_run, o);
    const float m_new = fmaxf(m_run, m_o), m_safe = m_new == -INFINITY ? 0.f : m_new;
    const float a = fast_exp2(m_run - m_safe), c = fast_exp2(m_o - m_safe);
    l_run = l_run * a + l_o * c;
    #pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = acc[i] * a + __shfl_xor_sync(0xffffffffu, acc[i], o) * c;
    m_run = m_new;
  }
  if (grp == 0) {
    #pragma unroll
    for (int i = 0; i < 8; ++i) sm_o[warp][gl * 8 + i] = acc[i];
    if (gl == 0) { sm_m[warp] = m_run; sm_l[warp] = l_run; }
  }
  __syncthreads();
  const int64_t bh = (int64_t)b * p.H + h;
  float mm = -INFINITY, l = 0.f, o = 0.f;
  if (tid < D) {
    #pragma unroll
    for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, sm_m[w]);
    const float m_safe = mm == -INFINITY ? 0.f : mm;
    #pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float sc = fast_exp2(sm_m[w] - m_safe);
      l += sm_l[w] * sc;
      o += sm_o[w][tid] * sc;
    }
  }
  T* out = (T*)p.out + bh * D;
  if (p.splits == 1) {
    if (tid < D) out[tid] = round_to<T>(l > 0.f ? o / l : 0.f);
    return;
  }
  if (tid < D) {
    const int64_t slot = bh * p.splits + split;
    p.part_o[slot * D + tid] = o;
    if (tid == 0) { p.part_ml[2 * slot] = mm; p.part_ml[2 * slot + 1] = l; }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) is_last = atomicAdd(&p.counters[bh], 1) == p.splits - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  if (tid < D) {
    mm = -INFINITY;
    for (int s = 0; s < p.splits; ++s) mm = fmaxf(mm, __ldcg(&p.part_ml[2 * (bh * p.splits + s)]));
    const float m_safe = mm == -INFINITY ? 0.f : mm;
    l = 0.f; o = 0.f;
    for (int s = 0; s < p.splits; ++s) {
      const int64_t slot = bh * p.splits + s;
      const float sc = fast_exp2(__ldcg(&p.part_ml[2 * slot]) - m_safe);
      l += __ldcg(&p.part_ml[2 * slot + 1]) * sc;
      o += __ldcg(&p.part_o[slot * D + tid]) * sc;
    }
    out[tid] = round_to<T>(l > 0.f ? o / l : 0.f);
  }
  if (tid == 0) p.counters[bh] = 0;
}

// ---------------------------------------------------------------- choice, token append, next embedding
// One block per row: the best candidate of the LM head's blocks, its embedding row, the row's position.
template <typename T>
__global__ void __launch_bounds__(256)
step_choose_kernel(const float2* cand, int n_cand, int64_t* tokens, int64_t tokens_stride, int32_t* seqlens, const T* embedding,
                   T* hidden, int d, int max_len) {
  __shared__ float sv[8];
  __shared__ int si[8];
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  grid_wait();
  grid_launch_dependents();
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = tid; i < n_cand; i += 256) {
    const float2 c = __ldcg(cand + (int64_t)row * n_cand + i);
    if (argmax_before(c.x, __float_as_int(c.y), bv, bi)) { bv = c.x; bi = __float_as_int(c.y); }
  }
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (argmax_before(ov, oi, bv, bi)) { bv = ov; bi = oi; }
  }
  if (lane == 0) { sv[tid >> 5] = bv; si[tid >> 5] = bi; }
  __syncthreads();
  bv = sv[0]; bi = si[0];
  for (int w = 1; w < 8; ++w)
    if (argmax_before(sv[w], si[w], bv, bi)) { bv = sv[w]; bi = si[w]; }
  const uint4* src = reinterpret_cast<const uint4*>(embedding + (int64_t)bi * d);
  uint4* dst = reinterpret_cast<uint4*>(hidden + (int64_t)row * d);
  for (int i = tid; i < d / 8; i += 256) dst[i] = src[i];
  if (tid == 0) {
    const int n = seqlens[row];
    if (n >= 1 && n <= max_len) tokens[(int64_t)row * tokens_stride + n - 1] = bi;
    seqlens[row] = n + 1;
  }
}

// distance -> bias of each head in the log2 domain (causal buckets), and the counters of the split attention cleared
__global__ void step_prepare_kernel(float* bias, const void* table, int table_dtype, int64_t stride0, int H, int32_t* counters,
                                    int n_counters, const __grid_constant__ BucketSpec spec) {
  const int n = H * (spec.max_distance + 1);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int h = i / (spec.max_distance + 1), dist = i - h * (spec.max_distance + 1);
    bias[i] = load_table(table, table_dtype, (int64_t)bucket_of_delta_counted(spec, -dist) * stride0 + h) * kLog2e;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_counters; i += gridDim.x * blockDim.x) counters[i] = 0;
}

// ------------------------------------------------------------------ host side
struct Launcher {
  cudaStream_t stream;
  int status = T5B_OK;
  template <typename... P, typename... A>
  void operator()(void (*kern)(P...), dim3 grid, int threads, size_t smem, A... args) {
    if (status != T5B_OK) return;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(threads, 1, 1); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, P(args)...) != cudaSuccess) { cudaGetLastError(); status = T5B_ERR_LAUNCH; }
  }
};

template <typename T, int WARPS, int NT, int kNorm, int kEpi>
static void launch_gemm(Launcher& go, const GemmParams& p) {
  auto kern = step_gemm_kernel<T, WARPS, NT, kNorm, kEpi>;
  const size_t pitch = (size_t)p.K * 2 + 64;
  const size_t smem = NT * 8 * pitch + (kNorm ? (size_t)p.K * 2 + 16 * pitch : 0) + (size_t)WARPS * 16 * NT * 8 * 4;
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) {
      cudaGetLastError();
      go.status = T5B_ERR_LAUNCH;
      return;
    }
    if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
  }
  if (smem > 227 * 1024) { go.status = T5B_ERR_UNSUPPORTED; return; }
  const int cols = kEpi == E_GATED ? NT * 4 : NT * 8, n = kEpi == E_GATED ? p.F : p.N;
  go(kern, dim3((unsigned)((n + cols - 1) / cols), 1, 1), WARPS * 32, smem, p);
}

// Rows of w per block: one tensor-core tile (8 rows) while that gives at most two blocks per SM, so that all SMs
// pull weights and the successor's blocks still find room; two or four tiles beyond.
template <typename T, int kNorm, int kEpi>
static void gemm_sized(Launcher& go, const GemmParams& p) {
  const int tiles = ((kEpi == E_GATED ? p.F : p.N) + 7) / 8;
  if constexpr (kEpi == E_GATED) {
    if (tiles <= 592) launch_gemm<T, 8, 2, kNorm, kEpi>(go, p);       // one tile of wi_0 and of wi_1 is four rows of each
    else launch_gemm<T, 8, 4, kNorm, kEpi>(go, p);
  } else if constexpr (kEpi == E_RESIDUAL) {
    // K = d_ff can be long: sixteen warps keep twice as many rows of x in flight
    if (p.K >= 2048) launch_gemm<T, 16, 1, kNorm, kEpi>(go, p);
    else launch_gemm<T, 8, 1, kNorm, kEpi>(go, p);
  } else if constexpr (kEpi == E_LOGITS) {
    launch_gemm<T, 8, 4, kNorm, kEpi>(go, p);
  } else {
    if (tiles <= 296) launch_gemm<T, 8, 1, kNorm, kEpi>(go, p);
    else if (tiles <= 592) launch_gemm<T, 8, 2, kNorm, kEpi>(go, p);
    else launch_gemm<T, 8, 4, kNorm, kEpi>(go, p);
  }
}
template <typename T, bool kNorm, int kEpi>
static void gemm(Launcher& go, const GemmParams& p) {
  if constexpr (!kNorm) gemm_sized<T, 0, kEpi>(go, p);
  else if (p.K <= 1024) gemm_sized<T, 1, kEpi>(go, p);
  else gemm_sized<T, 2, kEpi>(go, p);
}

template <typename T, bool kSelf>
static void attention(Launcher& go, const AttnStepParams& p, int D) {
  const dim3 grid((unsigned)p.splits, (unsigned)p.H, (unsigned)p.B);
  // a self-attention cache holds the tokens generated so far, mostly a few loads: four warps; the memory: eight
  constexpr int W = kSelf ? 4 : 8;
  switch (D) {
    case 16: go(step_attention_kernel<T, 16, W, kSelf>, grid, W * 32, 0, p); break;
    case 32: go(step_attention_kernel<T, 32, W, kSelf>, grid, W * 32, 0, p); break;
    case 64: go(step_attention_kernel<T, 64, W, kSelf>, grid, W * 32, 0, p); break;
    case 128: go(step_attention_kernel<T, 128, 8, kSelf>, grid, 256, 0, p); break;
    default: go.status = T5B_ERR_HEAD_DIM;
  }
}

// Splits of the keys: enough blocks for two per SM, at least 128 keys per split.
static int splits_for(int B, int H, int N) {
  const long long bh = (long long)B * H;
  long long want = (296 + bh - 1) / bh, cap = (N + 127) / 128;
  long long s = want < cap ? want : cap;
  return (int)(s < 1 ? 1 : (s > 64 ? 64 : s));
}

struct Layout { int64_t q, attn, act, bias, cand, counters, ml, o, total; int self_splits, cross_splits, n_cand; };
static Layout layout(const t5b_decoder_step_args& a) {
  Layout l;
  int64_t at = 0;
  auto take = [&](int64_t bytes) { const int64_t r = at; at += (bytes + 255) / 256 * 256; return r; };
  const int64_t HD = (int64_t)a.H * a.D, bh = (int64_t)a.B * a.H;
  l.self_splits = splits_for(a.B, a.H, a.max_len);
  l.cross_splits = splits_for(a.B, a.H, a.enc_len);
  const int s = l.self_splits > l.cross_splits ? l.self_splits : l.cross_splits;
  l.n_cand = (a.vocab + 31) / 32;
  l.q = take(a.B * HD * 2);
  l.attn = take(a.B * HD * 2);
  l.act = take((int64_t)a.B * a.d_ff * 2);
  l.bias = take((int64_t)a.H * (a.max_distance + 1) * 4);
  l.cand = take((int64_t)a.B * l.n_cand * 8);
  l.counters = take(bh * 4);
  l.ml = take(bh * s * 2 * 4);
  l.o = take(bh * s * a.D * 4);
  l.total = at;
  return l;
}

template <typename T>
static int run_step(const t5b_decoder_step_args& a, cudaStream_t stream) {
  const Layout l = layout(a);
  char* ws = (char*)a.workspace;
  Launcher go{stream};
  const int HD = a.H * a.D;
  for (int i = 0; i < a.n_layers; ++i) {
    const t5b_decoder_layer& w = a.layers[i];
    GemmParams g = {};
    g.B = a.B; g.eps = a.eps; g.x_scale = 1.f; g.H = a.H; g.D = a.D; g.max_len = a.max_len; g.F = a.d_ff;
    auto project = [&](const void* x, int K, const void* weight, const void* ln, void* out, int N) {
      g.x = x; g.K = K; g.x_stride = K; g.w = weight; g.ln = ln; g.out = out; g.N = N;
    };
    project(a.hidden, a.d_model, w.wqkv, w.ln_self, ws + l.q, 3 * HD);
    g.kv = w.self_kv; g.seqlens = a.seqlens;
    gemm<T, true, E_QKV>(go, g);
    AttnStepParams s = {};
    s.B = a.B; s.H = a.H; s.q = ws + l.q; s.out = ws + l.attn;
    s.counters = (int32_t*)(ws + l.counters); s.part_ml = (float*)(ws + l.ml); s.part_o = (float*)(ws + l.o);
    s.k = w.self_kv; s.v = (const char*)w.self_kv + (int64_t)a.B * a.H * a.max_len * a.D * 2;
    s.k_stride_b = (int64_t)a.H * a.max_len * a.D; s.k_stride_h = (int64_t)a.max_len * a.D; s.k_stride_n = a.D;
    s.lens = a.seqlens; s.bias = (const float*)(ws + l.bias); s.md = a.max_distance; s.N = a.max_len; s.splits = l.self_splits;
    attention<T, true>(go, s, a.D);
    project(ws + l.attn, HD, w.wo, nullptr, a.hidden, a.d_model);
    gemm<T, false, E_RESIDUAL>(go, g);

    project(a.hidden, a.d_model, w.wcq, w.ln_cross, ws + l.q, HD);
    gemm<T, true, E_STORE>(go, g);
    s.k = w.cross_k; s.v = w.cross_v;
    s.k_stride_b = a.cross_stride_b; s.k_stride_h = a.cross_stride_h; s.k_stride_n = a.cross_stride_n;
    s.lens = a.enc_seqlens; s.bias = nullptr; s.N = a.enc_len; s.splits = l.cross_splits;
    attention<T, false>(go, s, a.D);
    project(ws + l.attn, HD, w.wco, nullptr, a.hidden, a.d_model);
    gemm<T, false, E_RESIDUAL>(go, g);

    project(a.hidden, a.d_model, w.wi, w.ln_ff, ws + l.act, a.gated ? 2 * a.d_ff : a.d_ff);
    if (a.gated) gemm<T, true, E_GATED>(go, g);
    else gemm<T, true, E_RELU>(go, g);
    project(ws + l.act, a.d_ff, w.wff, nullptr, a.hidden, a.d_model);
    gemm<T, false, E_RESIDUAL>(go, g);
  }
  GemmParams g = {};
  g.B = a.B; g.eps = a.eps; g.x_scale = a.lm_scale; g.x = a.hidden; g.K = a.d_model; g.x_stride = a.d_model;
  g.w = a.lm_head; g.ln = a.final_ln; g.out = a.logits; g.N = a.vocab; g.cand = (float2*)(ws + l.cand);
  gemm<T, true, E_LOGITS>(go, g);
  go(step_choose_kernel<T>, dim3((unsigned)a.B, 1, 1), 256, 0, (const float2*)(ws + l.cand), l.n_cand, a.tokens, a.tokens_stride,
     a.seqlens, (const T*)a.embedding, (T*)a.hidden, a.d_model, a.max_len);
  return go.status;
}

static int validate(const t5b_decoder_step_args* a) {
  if (!a || !a->layers || a->n_layers <= 0) return T5B_ERR_ARG;
  if (a->dtype != T5B_BF16 && a->dtype != T5B_F16) return T5B_ERR_DTYPE;
  if (a->D != 16 && a->D != 32 && a->D != 64 && a->D != 128) return T5B_ERR_HEAD_DIM;
  if (a->B <= 0 || a->H <= 0 || a->d_model <= 0 || a->d_ff <= 0 || a->vocab <= 0 || a->max_len <= 0 || a->enc_len <= 0) return T5B_ERR_SHAPE;
  // 32-wide pieces of every contraction; a norm's row in registers; the weights of a block in shared memory
  if (a->B > 64 || a->d_model % 32 || (a->H * a->D) % 32 || a->d_ff % 32 || a->d_model > 2048 || a->H * a->D > 4096 ||
      a->d_ff > 8192 || a->max_distance > 2048)
    return T5B_ERR_UNSUPPORTED;
  if (((uintptr_t)a->workspace & 255) != 0 || !a->workspace || a->workspace_bytes < layout(*a).total) return T5B_ERR_WORKSPACE;
  return T5B_OK;
}

}  // namespace step
}  // namespace t5b

using namespace t5b;

extern "C" int64_t t5b_decoder_step_workspace_bytes(const t5b_decoder_step_args* a) {
  if (!a || a->B <= 0 || a->H <= 0 || a->D <= 0 || a->max_len <= 0 || a->enc_len <= 0 || a->vocab <= 0) return 0;
  return step::layout(*a).total;
}

extern "C" int t5b_decoder_step_prepare(const t5b_decoder_step_args* a, void* stream) {
  const int vst = step::validate(a);
  if (vst != T5B_OK) return vst;
  if (!a->table) return T5B_ERR_ARG;
  BucketSpec spec;
  const int st = make_bucket_spec(a->num_buckets, a->max_distance, 0, &spec);
  if (st != T5B_OK) return st;
  const step::Layout l = step::layout(*a);
  char* ws = (char*)a->workspace;
  step::step_prepare_kernel<<<16, 256, 0, (cudaStream_t)stream>>>((float*)(ws + l.bias), a->table, a->table_dtype, a->table_stride0,
                                                                  a->H, (int32_t*)(ws + l.counters), a->B * a->H, spec);
  return cudaGetLastError() == cudaSuccess ? T5B_OK : T5B_ERR_LAUNCH;
}

extern "C" int t5b_decoder_step(const t5b_decoder_step_args* a, void* stream) {
  const int vst = step::validate(a);
  if (vst != T5B_OK) return vst;
  if (!a->hidden || !a->logits || !a->tokens || !a->seqlens || !a->lm_head || !a->embedding || !a->final_ln) return T5B_ERR_ARG;
  return a->dtype == T5B_BF16 ? step::run_step<__nv_bfloat16>(*a, (cudaStream_t)stream)
                              : step::run_step<__half>(*a, (cudaStream_t)stream);
}
