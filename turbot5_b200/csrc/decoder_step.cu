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
// Every kernel lets its successor start at once, so two or three kernels of the chain sit on the SMs with their
// weights loaded while one computes.  What a block reads before its wait is therefore only what no kernel of the
// chain writes: weights, cross keys and values, their lengths.  Every kernel waits, and a wait ends when the
// predecessor has completed, its own wait included: after it everything earlier in the chain is visible.
//
// Semantics: the cached step of the decoder stack (src/turbot5/model/modeling.py:166-219 per block,
// src/turbot5/model/attentions.py:198,229-234).  Rounding points as the separate operators, except for the norm that
// opens a product in bf16: there the raw row times the norm weight is rounded once and rstd multiplies the float32 sum
// (step_gemm_kernel), where the operators round the normed row and then its product with the weight.
#include "t5b_common.cuh"

#include <atomic>

namespace t5b {
namespace step {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// untiled bulk copy, global -> shared, completion on an mbarrier (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
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

template <typename T> constexpr bool kIsBf16 = false;
template <> constexpr bool kIsBf16<__nv_bfloat16> = true;
template <typename T> __device__ __forceinline__ T round_to(float x) { return from_float<T>(x); }
template <typename T> __device__ __forceinline__ float rounded(float x) { return to_float<T>(from_float<T>(x)); }

// two elements of the 16-bit type, as float32 and back
template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t v);
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t v) {
  return __half22float2(*reinterpret_cast<const __half2*>(&v));
}
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// products of two pairs, each rounded once (the float32 product of two 16-bit values is exact)
template <typename T> __device__ __forceinline__ uint32_t mul2h(uint32_t a, uint32_t b);
template <> __device__ __forceinline__ uint32_t mul2h<__nv_bfloat16>(uint32_t a, uint32_t b) {
  const __nv_bfloat162 h = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t mul2h<__half>(uint32_t a, uint32_t b) {
  const __half2 h = __hmul2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&h);
}

// ---------------------------------------------------------------- skinny matrix products
// y[B, N] = f(x)[B, K] w[N, K]^T for B <= 64.  A block owns NT * 8 rows of w, its eight warps take the 32-wide pieces
// of K in turn, sixteen rows of x at a time, and meet in shared memory.  mma.m16n8k16: these products are a
// stream of weights (16 flop per byte at 16 rows); the tensor unit is idle either way, and a tcgen05 tile of 128
// rows would be seven eighths padding.
//
// Operands are read with 16-byte loads: a lane takes eight consecutive k of its row where the instruction's
// layout asks for four pairs eight apart; the order of k inside a 32-wide piece is the same for both operands,
// so the products meet.  Row pitch K * 2 + 64 bytes: the rows of a quarter warp's load fall into different banks.
// Rows of x past B and rows of w past N hold whatever was there: an output depends on its own row and column only.
enum Epilogue { E_STORE = 0, E_QKV, E_RESIDUAL, E_GATED, E_RELU };

struct GemmParams {
  const void* x; const void* w; const void* ln; void* out;
  void* kv;                        // E_QKV: cache (2, B, H, max_len, D)
  const int32_t* seqlens;          // E_QKV: cached keys of each row, the new one included
  float2* cand;                    // LM head: (value, index bits) of each row and block
  int32_t B, N, K, F;              // F: E_GATED: rows of wi_0 (w holds wi_0 | wi_1)
  int32_t H, D, max_len;
  float eps, x_scale;              // x_scale: multiplies the normed rows (tied embeddings), 1 = off
  int32_t* status;                 // device_status: a wait that gave up (see close_waits), or NULL
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

// Last act of a kernel with bounded waits, by one thread, after a block barrier that follows every wait: a wait that gave
// up has left wrong numbers, which the status word tells the host, and a copy may still be on its way into this
// block's shared memory, which the block must not leave before.  `flags[0]` was raised by the wait; the two
// barriers are the block's (phase 0).
__device__ __noinline__ void close_waits(volatile int* flags, int32_t* status, int code, uint32_t bar_a, uint32_t bar_b,
                                         long long limit) {
  if (status != nullptr) atomicCAS(status, 0, code);
  flags[1] = 0;
  mbar_wait_bounded(bar_a, 0, flags + 1, limit);
  flags[1] = 0;
  mbar_wait_bounded(bar_b, 0, flags + 1, limit);
}

constexpr int WARPS = 8, THREADS = WARPS * 32;

// RMSNorm of up to sixteen rows of x into shared memory (rows of `pitch` bytes), with the rounding points of
// t5b_rmsnorm_fwd.  The block's threads are dealt to the rows that exist (a power of two of them each): at one row the
// whole block shares it.  VECS: 16-byte vectors of a thread, K <= 4 * W * VECS * 4.  Uses part[W]; ends with the rows written, not yet synchronised.
template <typename T, int VECS, int W>
__device__ __forceinline__ void norm_rows(const GemmParams& p, int m0, uint32_t sLn, uint32_t sX, uint32_t pitch, float* part,
                                          uint32_t ln_bar, volatile int* abort_flag, float scale) {
  const int tid = threadIdx.x, nvec = p.K >> 3;
  const int rows = min(16, p.B - m0);
  constexpr int kAll = W == 16 ? 9 : 8;                                                // log2(threads)
  const int shift = rows > 8 ? kAll - 4 : rows > 4 ? kAll - 3 : rows > 2 ? kAll - 2 : rows > 1 ? kAll - 1 : kAll;
  const int tpr = 1 << shift, r = tid >> shift, c0 = tid & (tpr - 1);
  const bool mine = r < rows;
  uint4 xv[VECS];
  #pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const int c = c0 + i * tpr;
    xv[i] = make_uint4(0, 0, 0, 0);
    if (mine && c < nvec) xv[i] = ld_act((const char*)p.x + ((int64_t)(m0 + r) * p.K + c * 8) * 2);
  }
  float s0 = 0.f, s1 = 0.f;
  #pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const uint32_t w[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
    #pragma unroll
    for (int k = 0; k < 4; ++k) { const float2 f = unpack2<T>(w[k]); s0 = fmaf(f.x, f.x, s0); s1 = fmaf(f.y, f.y, s1); }
  }
  float ss = s0 + s1;
  #pragma unroll
  for (int o = 1; o < 32; o <<= 1)
    if (o < tpr) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (tpr > 32) {                                            // (uniform)
    if ((tid & 31) == 0) part[tid >> 5] = ss;
    __syncthreads();
    const int w0 = (tid >> shift) << (shift - 5);
    ss = 0.f;
    for (int w = 0; w < (tpr >> 5); ++w) ss += part[w0 + w];
  }
  const float rstd = rsqrtf(ss / (float)p.K + p.eps);
  mbar_wait_bounded(ln_bar, 0, abort_flag);
  if (mine) {
    #pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int c = c0 + i * tpr;
      if (c < nvec) {
        const uint4 wv = lds128(sLn + c * 16);
        const uint32_t x[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w}, w[4] = {wv.x, wv.y, wv.z, wv.w};
        uint32_t y[4];
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = unpack2<T>(x[k]);
          y[k] = mul2h<T>(w[k], pack2<T>(f.x * rstd, f.y * rstd));
          if (scale != 1.f) {                                 // the scale is a float32 factor of the rounded value
            const float2 n = unpack2<T>(y[k]);
            y[k] = pack2<T>(n.x * scale, n.y * scale);
          }
        }
        sts128(sX + r * pitch + c * 16, make_uint4(y[0], y[1], y[2], y[3]));
      }
    }
  }
}

// the warps' sums for one output element
template <int W, int COLS>
__device__ __forceinline__ float warp_sums(const float* red, int r, int c) {
  float s = 0.f;
  #pragma unroll
  for (int w = 0; w < W; ++w) s += red[(w * 16 + r) * COLS + c];
  return s;
}

// kNorm: the product is of the normed rows.  bf16: y = rstd * sum_k (x w_ln)[k] w[n, k] -- the norm weight goes onto the
// operand as it is loaded (one rounding where the separate norm has two), every warp sums the squares of its share
// of the row beside its products, and rstd multiplies the finished sum, so the norm adds no phase to the kernel
// (as a pass of its own, rows into shared memory and two barriers, it took 1.0 of 2.5 us at one row and 1.8 of 3.1
// at sixteen).  fp16 has not the range for unnormed products: its rows are normed first (norm_rows).
// W warps per block; registers are held to what lets the successor's blocks find room beside the running ones.
template <typename T, int W, int NT, bool kNorm, int kEpi>
__global__ void __launch_bounds__(W * 32, kNorm && !kIsBf16<T> ? 1 : 2)
step_gemm_kernel(const __grid_constant__ GemmParams p) {
  constexpr bool kFold = kNorm && sizeof(T) == 2 && kIsBf16<T>;
  constexpr bool kRows = kNorm && !kFold;
  constexpr int COLS = NT * 8;                               // accumulator columns of the block
  constexpr int OUT_COLS = kEpi == E_GATED ? COLS / 2 : COLS;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) unsigned long long bar_words[2];
  __shared__ int abort_words[2];
  __shared__ float part[W];
  __shared__ float squares[kFold ? W : 1][16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = p.K;
  const uint32_t pitch = (uint32_t)K * 2 + 64;
  const uint32_t sW = smem_u32(smem);
  const uint32_t sLn = sW + COLS * pitch;
  const uint32_t sX = sLn + (kNorm ? (uint32_t)K * 2 : 0u);
  float* red = reinterpret_cast<float*>(smem + COLS * pitch + (kNorm ? (uint32_t)K * 2 : 0u) + (kRows ? 16 * pitch : 0u));
  const uint32_t w_bar = smem_u32(&bar_words[0]), ln_bar = smem_u32(&bar_words[1]);
  const int n0 = (int)blockIdx.x * OUT_COLS;
  grid_launch_dependents();

  // the block's weights, before anything that depends on an earlier kernel
  if (tid == 0) {
    abort_words[0] = 0;
    mbar_init(w_bar, 1);
    mbar_init(ln_bar, 1);
    fence_barrier_init();
    fence_proxy_async();
    if (kNorm) {
      mbar_expect_tx(ln_bar, (uint32_t)K * 2);
      bulk_load(sLn, p.ln, (uint32_t)K * 2, ln_bar);
    }
  }
  if (warp == 0) {                                            // one row per lane: a copy costs its issuing thread tens of cycles
    const int r = lane;
    const int n = kEpi == E_GATED ? (r < COLS / 2 ? n0 + r : p.F + n0 + r - COLS / 2) : n0 + r;
    const bool ok = r < COLS && (kEpi == E_GATED ? n0 + r % (COLS / 2) < p.F : n < p.N);
    const int rows = __popc(__ballot_sync(0xffffffffu, ok));
    if (lane == 0) mbar_expect_tx(w_bar, (uint32_t)(rows * K * 2));
    __syncwarp();
    if (ok) bulk_load(sW + r * pitch, (const char*)p.w + (int64_t)n * K * 2, (uint32_t)K * 2, w_bar);
  }
  __syncthreads();
  volatile int* abort_flag = abort_words;
  if (kFold) mbar_wait_bounded(ln_bar, 0, abort_flag);
  grid_wait();

  const int g = lane >> 2, t = lane & 3;
  for (int m0 = 0; m0 < p.B; m0 += 16) {
    const int rows = min(16, p.B - m0);
    if constexpr (kRows) {
      norm_rows<T, 16, W>(p, m0, sLn, sX, pitch, part, ln_bar, abort_flag, 1.f);
      __syncthreads();
    }
    float acc[NT][4];
    #pragma unroll
    for (int j = 0; j < NT; ++j)
      #pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    float sq_lo = 0.f, sq_hi = 0.f;
    const char* xlo = (const char*)p.x + (int64_t)(m0 + g) * K * 2 + t * 16;
    const char* xhi = xlo + (int64_t)8 * K * 2;
    const bool lo_ok = g < rows, hi_ok = g + 8 < rows;
    bool have_w = false;
    #pragma unroll 1
    for (int kb0 = warp; kb0 < (K >> 5); kb0 += 4 * W) {
      uint4 a[4], b[4];                                       // rows g and g + 8: four pieces in flight
      #pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int kb = kb0 + u * W;
        a[u] = b[u] = make_uint4(0, 0, 0, 0);
        if (kb < (K >> 5)) {
          if (kRows) {
            a[u] = lds128(sX + g * pitch + kb * 64 + t * 16);
            b[u] = lds128(sX + (g + 8) * pitch + kb * 64 + t * 16);
          } else {
            if (lo_ok) a[u] = ld_act(xlo + kb * 64);
            if (hi_ok) b[u] = ld_act(xhi + kb * 64);
          }
        }
      }
      if (!have_w) { mbar_wait_bounded(w_bar, 0, abort_flag); have_w = true; }
      #pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int kb = kb0 + u * W;
        if (kb < (K >> 5)) {
          if (kFold) {
            const uint4 l = lds128(sLn + kb * 64 + t * 16);
            uint32_t* av = reinterpret_cast<uint32_t*>(&a[u]);
            uint32_t* bv = reinterpret_cast<uint32_t*>(&b[u]);
            const uint32_t lv[4] = {l.x, l.y, l.z, l.w};
            #pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 fa = unpack2<T>(av[i]), fb = unpack2<T>(bv[i]);
              sq_lo = fmaf(fa.x, fa.x, fmaf(fa.y, fa.y, sq_lo));
              sq_hi = fmaf(fb.x, fb.x, fmaf(fb.y, fb.y, sq_hi));
              av[i] = mul2h<T>(av[i], lv[i]);
              bv[i] = mul2h<T>(bv[i], lv[i]);
            }
          }
          #pragma unroll
          for (int j = 0; j < NT; ++j) {
            const uint4 w4 = lds128(sW + (j * 8 + g) * pitch + kb * 64 + t * 16);
            mma16816<T>(acc[j], a[u].x, b[u].x, a[u].y, b[u].y, w4.x, w4.y);
            mma16816<T>(acc[j], a[u].z, b[u].z, a[u].w, b[u].w, w4.z, w4.w);
          }
        }
      }
    }
    // ---- the warps' partial sums meet: red[warp][row][column]
    #pragma unroll
    for (int j = 0; j < NT; ++j) {
      float* r0 = red + (warp * 16 + g) * COLS + j * 8 + 2 * t;
      *reinterpret_cast<float2*>(r0) = make_float2(acc[j][0], acc[j][1]);
      *reinterpret_cast<float2*>(r0 + 8 * COLS) = make_float2(acc[j][2], acc[j][3]);
    }
    if (kFold) {
      #pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        sq_lo += __shfl_xor_sync(0xffffffffu, sq_lo, o);
        sq_hi += __shfl_xor_sync(0xffffffffu, sq_hi, o);
      }
      if (t == 0) { squares[warp][g] = sq_lo; squares[warp][g + 8] = sq_hi; }
    }
    __syncthreads();
    #pragma unroll 1
    for (int idx = tid; idx < rows * OUT_COLS; idx += W * 32) {
      const int r = idx / OUT_COLS, c = idx % OUT_COLS;
      const int row = m0 + r, n = n0 + c;
      float s = warp_sums<W, COLS>(red, r, c), rstd = 1.f;
      if (kFold) {
        float ss = 0.f;
        #pragma unroll
        for (int w = 0; w < W; ++w) ss += squares[w][r];
        rstd = rsqrtf(ss / (float)K + p.eps);
        s *= rstd;
      }
      if (n >= (kEpi == E_GATED ? p.F : p.N)) continue;
      if (kEpi == E_STORE) {
        ((T*)p.out)[(int64_t)row * p.N + n] = round_to<T>(s);
      } else if (kEpi == E_RELU) {
        ((T*)p.out)[(int64_t)row * p.N + n] = round_to<T>(fmaxf(s, 0.f));
      } else if (kEpi == E_GATED) {
        const float s2 = warp_sums<W, COLS>(red, r, COLS / 2 + c) * rstd;
        ((T*)p.out)[(int64_t)row * p.F + n] = round_to<T>(rounded<T>(gelu_tanh(rounded<T>(s))) * rounded<T>(s2));
      } else if (kEpi == E_RESIDUAL) {
        T* o = (T*)p.out + (int64_t)row * p.N + n;
        *o = round_to<T>(to_float<T>(*o) + rounded<T>(s));
      } else {
        const int HD = p.H * p.D;
        if (n < HD) ((T*)p.out)[(int64_t)row * HD + n] = round_to<T>(s);
        else {
          const int kv = n >= 2 * HD ? 1 : 0, m = n - HD - kv * HD, h = m / p.D, d = m - h * p.D;
          const int pos = p.seqlens[row] - 1;
          if (pos >= 0 && pos < p.max_len)
            ((T*)p.kv)[((((int64_t)kv * p.B + row) * p.H + h) * p.max_len + pos) * p.D + d] = round_to<T>(s);
        }
      }
    }
    if (m0 + 16 < p.B) __syncthreads();                       // `red` is written again
  }
  if (tid == 0 && abort_flag[0] != 0) close_waits(abort_flag, p.status, 4001, w_bar, kNorm ? ln_bar : w_bar, T5B_WAIT_LIMIT_CYCLES);
}

// ---------------------------------------------------------------- LM head
// Final norm, logits and each block's best token.  One block per SM; the norm is done once per SM, then every warp walks
// its share of the vocabulary by itself, eight rows of w at a time over all of K, through its own ring of bulk loads
// (pieces of `piece` columns): no barrier between warps in the loop.  Bound by HBM (66 MB at 32128 x 1024).  Measured at
// 16 rows: a block per 32 rows of w 43 us, one ring per block with a barrier per tile 21 us, this 15.8 us.
constexpr int LM_MAX_STAGES = 4;

template <typename T, int M_TILES>
__global__ void __launch_bounds__(THREADS, 1)
step_logits_kernel(const __grid_constant__ GemmParams p, int piece, int stages) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) unsigned long long bar_words[WARPS * LM_MAX_STAGES + 1];
  __shared__ int abort_words[2];
  __shared__ float part[WARPS];
  __shared__ float best_v[WARPS][16 * M_TILES];
  __shared__ int best_i[WARPS][16 * M_TILES];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, K = p.K;
  const uint32_t pitch = (uint32_t)K * 2 + 64, wpitch = (uint32_t)piece * 2 + 64, stage_bytes = 8 * wpitch;
  const uint32_t sX = smem_u32(smem), sLn = sX + M_TILES * 16 * pitch, sW = sLn + (uint32_t)K * 2 + warp * stages * stage_bytes;
  const uint32_t bar0 = smem_u32(&bar_words[warp * LM_MAX_STAGES]), ln_bar = smem_u32(&bar_words[WARPS * LM_MAX_STAGES]);
  const int tiles = (p.N + 7) / 8, pieces = K / piece;
  const int first = (int)blockIdx.x * WARPS + warp, step = (int)gridDim.x * WARPS;
  const int n_mine = first < tiles ? (tiles - first + step - 1) / step : 0;
  auto load = [&](int it) {                                  // the it-th piece of this warp (a row per lane)
    if (it >= n_mine * pieces) return;
    const int tile = first + (it / pieces) * step, k0 = (it % pieces) * piece;
    const uint32_t bar = bar0 + 8 * (it % stages), dst = sW + (it % stages) * stage_bytes;
    const int rows = min(8, p.N - tile * 8);
    if (lane == 0) mbar_expect_tx(bar, (uint32_t)(rows * piece * 2));
    __syncwarp();
    if (lane < rows)
      bulk_load(dst + lane * wpitch, (const char*)p.w + ((int64_t)(tile * 8 + lane) * K + k0) * 2, (uint32_t)piece * 2, bar);
  };
  grid_launch_dependents();
  if (lane == 0) {
    for (int i = 0; i < stages; ++i) mbar_init(bar0 + 8 * i, 1);
    if (tid == 0) { abort_words[0] = 0; mbar_init(ln_bar, 1); }
    fence_barrier_init();
    fence_proxy_async();
    if (tid == 0) {
      mbar_expect_tx(ln_bar, (uint32_t)K * 2);
      bulk_load(sLn, p.ln, (uint32_t)K * 2, ln_bar);
    }
  }
  __syncwarp();
  for (int i = 0; i < stages; ++i) load(i);
  __syncthreads();
  volatile int* abort_flag = abort_words;
  grid_wait();
  #pragma unroll 1
  for (int m = 0; m < M_TILES; ++m) {
    norm_rows<T, 16, WARPS>(p, 16 * m, sLn, sX + 16 * m * pitch, pitch, part, ln_bar, abort_flag, p.x_scale);
    __syncthreads();
  }
  const int g = lane >> 2, t = lane & 3;
  float bv[M_TILES][2];                                      // best of rows g and g + 8 among this lane's columns
  int bi[M_TILES][2];
  #pragma unroll
  for (int m = 0; m < M_TILES; ++m)
    #pragma unroll
    for (int r = 0; r < 2; ++r) { bv[m][r] = -INFINITY; bi[m][r] = 0x7fffffff; }
  int it = 0;
  bool arrived = true;
  for (int i = 0; i < n_mine && arrived; ++i) {
    const int tile = first + i * step;
    float acc[M_TILES][2][4];                                // two chains per sixteen rows
    #pragma unroll
    for (int m = 0; m < M_TILES; ++m)
      #pragma unroll
      for (int e = 0; e < 8; ++e) acc[m][e >> 2][e & 3] = 0.f;
    for (int pc = 0; pc < pieces; ++pc, ++it) {
      const uint32_t w0 = sW + (it % stages) * stage_bytes + g * wpitch + t * 16;
      const uint32_t x0 = sX + g * pitch + pc * piece * 2 + t * 16;
      arrived = mbar_wait_warp_fast(bar0 + 8 * (it % stages), (uint32_t)((it / stages) & 1), abort_flag);
      if (!arrived) break;                                   // (the warp as one: its ring is drained below)
      #pragma unroll 4
      for (int kb = 0; kb < piece / 32; ++kb) {
        const uint4 w4 = lds128(w0 + kb * 64);
        #pragma unroll
        for (int m = 0; m < M_TILES; ++m) {
          const uint4 a = lds128(x0 + 16 * m * pitch + kb * 64), b = lds128(x0 + (16 * m + 8) * pitch + kb * 64);
          mma16816<T>(acc[m][0], a.x, b.x, a.y, b.y, w4.x, w4.y);
          mma16816<T>(acc[m][1], a.z, b.z, a.w, b.w, w4.z, w4.w);
        }
      }
      __syncwarp();                                          // every lane has read the piece: its slot may be filled again
      load(it + stages);
    }
    #pragma unroll
    for (int m = 0; m < M_TILES; ++m)
      #pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = 16 * m + g + (e >> 1) * 8, n = tile * 8 + 2 * t + (e & 1);
        if (row < p.B && n < p.N) {
          const T o = round_to<T>(acc[m][0][e] + acc[m][1][e]);
          ((T*)p.out)[(int64_t)row * p.N + n] = o;
          const float v = to_float<T>(o);
          // (n increases from tile to tile: a tie stays with the first)
          if (bi[m][e >> 1] == 0x7fffffff || v > bv[m][e >> 1] || (isnan(v) && !isnan(bv[m][e >> 1]))) { bv[m][e >> 1] = v; bi[m][e >> 1] = n; }
        }
      }
  }
  if (!arrived && lane == 0) {                               // the pieces that were requested and not used
    abort_words[1] = 0;
    for (int j = it; j < it + stages && j < n_mine * pieces; ++j)
      mbar_wait_bounded(bar0 + 8 * (j % stages), (uint32_t)((j / stages) & 1), abort_words + 1);
  }
  __syncwarp();
  #pragma unroll
  for (int m = 0; m < M_TILES; ++m)
    #pragma unroll
    for (int r = 0; r < 2; ++r) {
      #pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv[m][r], o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi[m][r], o);
        if (argmax_before(ov, oi, bv[m][r], bi[m][r])) { bv[m][r] = ov; bi[m][r] = oi; }
      }
      if (t == 0) { best_v[warp][16 * m + g + 8 * r] = bv[m][r]; best_i[warp][16 * m + g + 8 * r] = bi[m][r]; }
    }
  __syncthreads();
  if (tid < p.B) {
    float v = best_v[0][tid];
    int n = best_i[0][tid];
    for (int w = 1; w < WARPS; ++w)
      if (argmax_before(best_v[w][tid], best_i[w][tid], v, n)) { v = best_v[w][tid]; n = best_i[w][tid]; }
    p.cand[(int64_t)tid * gridDim.x + blockIdx.x] = make_float2(v, __int_as_float(n));
  }
  if (tid == 0 && abort_flag[0] != 0) close_waits(abort_flag, p.status, 4002, ln_bar, ln_bar, T5B_WAIT_LIMIT_CYCLES);
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

template <typename T, int D, int AW, bool kSelf>
__global__ void __launch_bounds__(AW * 32)
step_attention_kernel(const __grid_constant__ AttnStepParams p) {
  constexpr int LPK = D / 8, KPW = 32 / LPK, UNROLL = 4, KPI = KPW * UNROLL;
  __shared__ float sm_m[AW], sm_l[AW];
  __shared__ float sm_o[AW][D];
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
    chunk = (chunk + AW * KPI - 1) / (AW * KPI) * (AW * KPI);
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
  grid_launch_dependents();
  if (!kSelf) {                      // the lengths of the memory are constant too
    len = range();
    load(n_begin + warp * KPI, kr[0], vr[0]);
  }
  grid_wait();
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
    load(it + AW * KPI, kr[1], vr[1]);
    consume(it, kr[0], vr[0]);
    it += AW * KPI;
    if (it >= n_end) break;
    load(it + AW * KPI, kr[0], vr[0]);
    consume(it, kr[1], vr[1]);
    it += AW * KPI;
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
    for (int w = 0; w < AW; ++w) mm = fmaxf(mm, sm_m[w]);
    const float m_safe = mm == -INFINITY ? 0.f : mm;
    #pragma unroll
    for (int w = 0; w < AW; ++w) {
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
  grid_launch_dependents();
  grid_wait();
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

// Self-test of close_waits: two barriers, a copy's worth of bytes announced on one and never sent.
__global__ void wait_selftest_kernel(int32_t* status, long long limit) {
  __shared__ __align__(8) unsigned long long bar_words[2];
  __shared__ int abort_words[2];
  const uint32_t bar = smem_u32(&bar_words[0]), done_bar = smem_u32(&bar_words[1]);
  if (threadIdx.x == 0) {
    abort_words[0] = 0;
    mbar_init(bar, 1);
    mbar_init(done_bar, 1);
    fence_barrier_init();
    mbar_expect_tx(bar, 64);
    mbar_arrive(done_bar);
  }
  __syncthreads();
  volatile int* flags = abort_words;
  mbar_wait_bounded(bar, 0, flags, limit);
  __syncthreads();
  if (threadIdx.x == 0 && flags[0] != 0) close_waits(flags, status, 4003, done_bar, bar, limit);
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

// Opt in to all of an SM's shared memory, once per device and kernel (`done`: a static of the call site).
template <typename F>
static bool allow_smem(F kern, std::atomic<bool>* done) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return true;
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - (int)fa.sharedSizeBytes) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
  return true;
}
constexpr size_t kMaxSmem = 223 * 1024, kLmSmem = 220 * 1024;       // dynamic; the kernels' own words take the rest

// ---- tiles of every product, for `validate` and for the launches alike
constexpr int GEMM_WARPS = 16;
static size_t gemm_smem(int K, int nt, bool norm, bool bf16) {
  const size_t pitch = (size_t)K * 2 + 64;
  return nt * 8 * pitch + (norm ? (size_t)K * 2 : 0) + (norm && !bf16 ? 16 * pitch : 0) + (size_t)GEMM_WARPS * 16 * nt * 8 * 4;
}
// `want` tiles of eight rows of w per block, or fewer where their rows do not fit in shared memory; 0: none fits
static int fitting_tiles(int want, int least, int K, bool norm, bool bf16) {
  while (want > least && gemm_smem(K, want, norm, bf16) > kMaxSmem) want /= 2;
  return gemm_smem(K, want, norm, bf16) <= kMaxSmem ? want : 0;
}
// Rows of w per block of the products that start with a norm: one tensor-core tile (8 rows) while that gives at
// most two blocks per SM, so that all SMs pull weights and the successor's blocks still find room; two or
// four tiles beyond.
static int norm_tiles(int K, int n_rows, bool gated, bool bf16) {
  const int tiles = (n_rows + 7) / 8;
  return gated ? fitting_tiles(tiles <= 592 ? 2 : 4, 2, K, true, bf16)
               : fitting_tiles(tiles <= 296 ? 1 : tiles <= 592 ? 2 : 4, 1, K, true, bf16);
}
// Output projections: at K = 4096 a block of one tile reads 128 KB of activations for 64 KB of weights, so from there
// on a block takes two (4.2 us against 5.2 us at 16 rows) while they fit.
static int residual_tiles(int K) { return fitting_tiles(K >= 4096 ? 2 : 1, 1, K, false, true); }

// LM head: sixteen-row tiles of the normed rows that a block holds (further rows take a launch of their own), and the
// ring beside them: pieces of K / 2, K / 4, ... columns until two fit, else of the largest divisor of K in whole 32s.
struct LmPlan { int m_tiles = 0, piece = 0, stages = 0; };
static LmPlan lm_plan(int K, int B) {
  LmPlan best;
  for (int m = B <= 16 ? 1 : B <= 32 ? 2 : 4; m >= 1; m /= 2) {
    const size_t fixed = (size_t)K * 2 + (size_t)m * 16 * ((size_t)K * 2 + 64);
    auto stages = [&](int piece) {
      const size_t n = fixed < kLmSmem ? (kLmSmem - fixed) / ((size_t)WARPS * 8 * ((size_t)piece * 2 + 64)) : 0;
      return n > LM_MAX_STAGES ? LM_MAX_STAGES : (int)n;
    };
    int piece = K;
    while (stages(piece) < 2 && piece % 64 == 0) piece /= 2;
    for (int p = K; stages(piece) < 2 && p >= 32; p -= 32)
      if (K % p == 0 && stages(p) >= 2) piece = p;
    if (stages(piece) > best.stages) { best.m_tiles = m; best.piece = piece; best.stages = stages(piece); }
    if (best.stages >= 2) break;
  }
  return best;
}

template <typename T, int NT, bool kNorm, int kEpi>
static void launch_gemm(Launcher& go, const GemmParams& p) {
  auto kern = step_gemm_kernel<T, GEMM_WARPS, NT, kNorm, kEpi>;
  static std::atomic<bool> attributes[64];
  if (!allow_smem(kern, attributes)) { go.status = T5B_ERR_LAUNCH; return; }
  const int cols = kEpi == E_GATED ? NT * 4 : NT * 8, n = kEpi == E_GATED ? p.F : p.N;
  go(kern, dim3((unsigned)((n + cols - 1) / cols), 1, 1), GEMM_WARPS * 32, gemm_smem(p.K, NT, kNorm, kIsBf16<T>), p);
}

template <typename T, int kEpi>
static void norm_gemm(Launcher& go, const GemmParams& p) {
  switch (norm_tiles(p.K, kEpi == E_GATED ? 2 * p.F : p.N, kEpi == E_GATED, kIsBf16<T>)) {
    case 1: if constexpr (kEpi != E_GATED) launch_gemm<T, 1, true, kEpi>(go, p); break;
    case 2: launch_gemm<T, 2, true, kEpi>(go, p); break;
    case 4: launch_gemm<T, 4, true, kEpi>(go, p); break;
    default: go.status = T5B_ERR_UNSUPPORTED;
  }
}
template <typename T>
static void residual_gemm(Launcher& go, const GemmParams& p) {
  switch (residual_tiles(p.K)) {
    case 1: launch_gemm<T, 1, false, E_RESIDUAL>(go, p); break;
    case 2: launch_gemm<T, 2, false, E_RESIDUAL>(go, p); break;
    default: go.status = T5B_ERR_UNSUPPORTED;
  }
}

static int lm_blocks(int vocab) {
  static std::atomic<int> sms[64];
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) n = sms[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) { cudaGetLastError(); n = 148; }
    if (dev >= 0 && dev < 64) sms[dev].store(n, std::memory_order_relaxed);
  }
  const int blocks = ((vocab + 7) / 8 + WARPS - 1) / WARPS;
  return blocks < n ? blocks : n;
}
template <typename T, int M_TILES>
static void launch_logits(Launcher& go, const GemmParams& p, const LmPlan& plan) {
  auto kern = step_logits_kernel<T, M_TILES>;
  static std::atomic<bool> attributes[64];
  if (!allow_smem(kern, attributes)) { go.status = T5B_ERR_LAUNCH; return; }
  const size_t fixed = (size_t)p.K * 2 + (size_t)M_TILES * 16 * ((size_t)p.K * 2 + 64);
  const size_t ring = (size_t)plan.stages * WARPS * 8 * ((size_t)plan.piece * 2 + 64);
  for (int row = 0; row < p.B; row += M_TILES * 16) {
    GemmParams q = p;
    q.B = p.B - row < M_TILES * 16 ? p.B - row : M_TILES * 16;
    q.x = (const T*)p.x + (int64_t)row * p.K;
    q.out = (T*)p.out + (int64_t)row * p.N;
    q.cand = p.cand + (int64_t)row * lm_blocks(p.N);
    go(kern, dim3((unsigned)lm_blocks(p.N), 1, 1), THREADS, fixed + ring, q, plan.piece, plan.stages);
  }
}
template <typename T>
static void logits(Launcher& go, const GemmParams& p) {
  const LmPlan plan = lm_plan(p.K, p.B);
  switch (plan.m_tiles) {
    case 1: launch_logits<T, 1>(go, p, plan); break;
    case 2: launch_logits<T, 2>(go, p, plan); break;
    case 4: launch_logits<T, 4>(go, p, plan); break;
    default: go.status = T5B_ERR_UNSUPPORTED;
  }
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
    case 128: go(step_attention_kernel<T, 128, W, kSelf>, grid, W * 32, 0, p); break;
    default: go.status = T5B_ERR_HEAD_DIM;
  }
}

// Splits of the keys: a block per SM, at least 128 keys per split.  (More blocks than that lose: at 16 x 16 heads and
// 1024 keys one split takes 12.4 us, two 17.3 us, four 20.0 us.)
static int splits_for(int B, int H, int N) {
  const long long bh = (long long)B * H;
  long long want = (148 + bh - 1) / bh, cap = (N + 127) / 128;
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
  l.n_cand = lm_blocks(a.vocab);
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
    g.B = a.B; g.eps = a.eps; g.x_scale = 1.f; g.status = a.device_status; g.H = a.H; g.D = a.D; g.max_len = a.max_len; g.F = a.d_ff;
    auto project = [&](const void* x, int K, const void* weight, const void* ln, void* out, int N) {
      g.x = x; g.K = K; g.w = weight; g.ln = ln; g.out = out; g.N = N;
    };
    project(a.hidden, a.d_model, w.wqkv, w.ln_self, ws + l.q, 3 * HD);
    g.kv = w.self_kv; g.seqlens = a.seqlens;
    norm_gemm<T, E_QKV>(go, g);
    AttnStepParams s = {};
    s.B = a.B; s.H = a.H; s.q = ws + l.q; s.out = ws + l.attn;
    s.counters = (int32_t*)(ws + l.counters); s.part_ml = (float*)(ws + l.ml); s.part_o = (float*)(ws + l.o);
    s.k = w.self_kv; s.v = (const char*)w.self_kv + (int64_t)a.B * a.H * a.max_len * a.D * 2;
    s.k_stride_b = (int64_t)a.H * a.max_len * a.D; s.k_stride_h = (int64_t)a.max_len * a.D; s.k_stride_n = a.D;
    s.lens = a.seqlens; s.bias = (const float*)(ws + l.bias); s.md = a.max_distance; s.N = a.max_len; s.splits = l.self_splits;
    attention<T, true>(go, s, a.D);
    project(ws + l.attn, HD, w.wo, nullptr, a.hidden, a.d_model);
    residual_gemm<T>(go, g);

    project(a.hidden, a.d_model, w.wcq, w.ln_cross, ws + l.q, HD);
    norm_gemm<T, E_STORE>(go, g);
    s.k = w.cross_k; s.v = w.cross_v;
    s.k_stride_b = a.cross_stride_b; s.k_stride_h = a.cross_stride_h; s.k_stride_n = a.cross_stride_n;
    s.lens = a.enc_seqlens; s.bias = nullptr; s.N = a.enc_len; s.splits = l.cross_splits;
    attention<T, false>(go, s, a.D);
    project(ws + l.attn, HD, w.wco, nullptr, a.hidden, a.d_model);
    residual_gemm<T>(go, g);

    project(a.hidden, a.d_model, w.wi, w.ln_ff, ws + l.act, a.gated ? 2 * a.d_ff : a.d_ff);
    if (a.gated) norm_gemm<T, E_GATED>(go, g);
    else norm_gemm<T, E_RELU>(go, g);
    project(ws + l.act, a.d_ff, w.wff, nullptr, a.hidden, a.d_model);
    residual_gemm<T>(go, g);
  }
  GemmParams g = {};
  g.B = a.B; g.eps = a.eps; g.x_scale = a.lm_scale; g.status = a.device_status; g.x = a.hidden; g.K = a.d_model;
  g.w = a.lm_head; g.ln = a.final_ln; g.out = a.logits; g.N = a.vocab; g.cand = (float2*)(ws + l.cand);
  logits<T>(go, g);
  go(step_choose_kernel<T>, dim3((unsigned)a.B, 1, 1), 256, 0, (const float2*)(ws + l.cand), l.n_cand, a.tokens, a.tokens_stride,
     a.seqlens, (const T*)a.embedding, (T*)a.hidden, a.d_model, a.max_len);
  return go.status;
}

// What the kernels take, the same answer for every entry point: sizes the launches would refuse show before anything runs.
static int validate_sizes(const t5b_decoder_step_args& a) {
  if (a.dtype != T5B_BF16 && a.dtype != T5B_F16) return T5B_ERR_DTYPE;
  if (a.D != 16 && a.D != 32 && a.D != 64 && a.D != 128) return T5B_ERR_HEAD_DIM;
  if (a.B <= 0 || a.H <= 0 || a.d_model <= 0 || a.d_ff <= 0 || a.vocab <= 0 || a.max_len <= 0 || a.enc_len <= 0) return T5B_ERR_SHAPE;
  // 32-wide pieces of every contraction; a norm's row in registers; the weights of a block in shared memory
  if (a.B > 64 || a.H > 4096 || a.d_model % 32 || (a.H * a.D) % 32 || a.d_ff % 32 || a.d_model > 2048 || a.H * a.D > 4096 ||
      a.d_ff > 8192 || a.max_distance > 2048)
    return T5B_ERR_UNSUPPORTED;
  const bool bf16 = a.dtype == T5B_BF16, gated = a.gated != 0;
  const int HD = a.H * a.D;
  if (!norm_tiles(a.d_model, 3 * HD, false, bf16) || !norm_tiles(a.d_model, HD, false, bf16) ||
      !norm_tiles(a.d_model, gated ? 2 * a.d_ff : a.d_ff, gated, bf16) || !residual_tiles(HD) || !residual_tiles(a.d_ff) ||
      !lm_plan(a.d_model, a.B).m_tiles)
    return T5B_ERR_UNSUPPORTED;
  return T5B_OK;
}
static int validate(const t5b_decoder_step_args* a) {
  if (!a || !a->layers || a->n_layers <= 0) return T5B_ERR_ARG;
  const int st = validate_sizes(*a);
  if (st != T5B_OK) return st;
  if (((uintptr_t)a->workspace & 255) != 0 || !a->workspace || a->workspace_bytes < layout(*a).total) return T5B_ERR_WORKSPACE;
  return T5B_OK;
}

// Everything that is fetched with 16-byte loads or bulk copies.
static int check_pointers(const t5b_decoder_step_args& a) {
  uintptr_t bits = (uintptr_t)a.hidden | (uintptr_t)a.lm_head | (uintptr_t)a.embedding | (uintptr_t)a.final_ln;
  for (int i = 0; i < a.n_layers; ++i) {
    const t5b_decoder_layer& l = a.layers[i];
    const void* all[] = {l.ln_self, l.wqkv, l.wo, l.ln_cross, l.wcq, l.wco, l.ln_ff, l.wi, l.wff, l.self_kv, l.cross_k, l.cross_v};
    for (const void* p : all) {
      if (!p) return T5B_ERR_ARG;
      bits |= (uintptr_t)p;
    }
  }
  if ((bits & 15) != 0 || ((a.cross_stride_b | a.cross_stride_h | a.cross_stride_n) % 8) != 0) return T5B_ERR_ALIGN;
  return T5B_OK;
}

}  // namespace step
}  // namespace t5b

using namespace t5b;

extern "C" int64_t t5b_decoder_step_workspace_bytes(const t5b_decoder_step_args* a) {
  if (!a || step::validate_sizes(*a) != T5B_OK) return 0;
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
  const int pst = step::check_pointers(*a);
  if (pst != T5B_OK) return pst;
  return a->dtype == T5B_BF16 ? step::run_step<__nv_bfloat16>(*a, (cudaStream_t)stream)
                              : step::run_step<__half>(*a, (cudaStream_t)stream);
}

extern "C" int t5b_selftest_decoder_wait(int32_t* device_status, int64_t limit_cycles, void* stream) {
  if (!device_status) return T5B_ERR_ARG;
  if (limit_cycles <= 0 || limit_cycles > 2000000000LL) return T5B_ERR_ARG;     // at most about a second
  step::wait_selftest_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(device_status, (long long)limit_cycles);
  return cudaGetLastError() == cudaSuccess ? T5B_OK : T5B_ERR_LAUNCH;
}
