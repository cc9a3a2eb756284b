// CUDA-core forward kernel for the cases the tcgen05 kernel does not take:
// float32 inputs (all arithmetic in float32, for the 1e-4 parity bound) at head
// dims 16/32/64/128, and rows that are not 16-byte aligned.  Same semantics, same
// bias lookup, same packed-sequence scheduling.
//
// Bound by the float32 pipe (128 FMA per clock and SM) as long as shared memory keeps up, so both products are
// register tiles: a block owns 16 * RPT query rows, its 16 x 16 threads hold RPT rows x KPT keys of the scores (rows
// of a thread adjacent, keys 16 apart) and RPT rows x D / 16 columns of the output.  A step of QK^T reads RPT + KPT
// vectors of four dims for 4 * RPT * KPT multiply-adds (packed in pairs of dims); with four threads per row and a
// key per step it was one vector per four multiply-adds, and the kernel waited for shared memory.  The next tile's
// keys and values are on their way to registers while this one's are used.  A whole float32 layer of 2 x 512 tokens,
// 8 heads x 64 (this kernel and four matrix products): 232 us before, 133 us now.
#include "t5b_common.cuh"
#include "attn_params.cuh"

#include <atomic>

namespace t5b {
namespace simt {

constexpr int THREADS = 256;

template <int D> struct Tile {
  static constexpr int TN = D == 128 ? 32 : 64;      // keys per tile (registers hold the next one)
  static constexpr int PQ = D + 4;                   // pitch of Q and K rows: 16 rows' vectors lie in different banks
  static constexpr int PP = TN + 4;                  // pitch of the probabilities
};
template <int D, int RPT>
constexpr int smem_floats() {
  return 16 * RPT * Tile<D>::PQ + Tile<D>::TN * Tile<D>::PQ + Tile<D>::TN * D + 16 * RPT * Tile<D>::PP;
}

// four consecutive elements as float32; `vec`: rows are aligned to four elements
template <typename T> __device__ __forceinline__ float4 load4(const T* p, bool vec) {
  if (vec) {
    if constexpr (sizeof(T) == 4) return __ldg(reinterpret_cast<const float4*>(p));
    else {
      const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
      const T* e = reinterpret_cast<const T*>(&r);
      return make_float4(to_float<T>(e[0]), to_float<T>(e[1]), to_float<T>(e[2]), to_float<T>(e[3]));
    }
  }
  return make_float4(to_float<T>(p[0]), to_float<T>(p[1]), to_float<T>(p[2]), to_float<T>(p[3]));
}
// two float32 multiply-adds: acc += a * b
__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum_pair(unsigned long long v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

template <typename T, int D, int RPT>
__global__ void __launch_bounds__(THREADS, D == 128 ? 1 : 2)
attn_fwd_simt_kernel(const __grid_constant__ AttnParams p, const __grid_constant__ BucketSpec spec, bool vec) {
  constexpr int TM = 16 * RPT, TN = Tile<D>::TN, KPT = TN / 16, PQ = Tile<D>::PQ, PP = Tile<D>::PP;
  constexpr int DPT = D / 16;                       // output columns of a thread
  constexpr int DV = DPT < 4 ? DPT : 4;             // ... in vectors of DV, 16 * DV columns apart
  constexpr int CHUNKS = TN * D / 4 / THREADS;      // vectors of four of a K or V tile per thread
  static_assert(CHUNKS >= 1 && CHUNKS * THREADS * 4 == TN * D, "tile shape");
  extern __shared__ __align__(16) float smem_f[];
  float* sQ = smem_f;
  float* sK = sQ + TM * PQ;
  float* sV = sK + TN * PQ;
  float* sP = sV + TN * D;
  float* lut = sP + TM * PP;
  __shared__ TileWork shared_work;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int h;
  int64_t batch = 0;
  TileWork w;
  if (p.cu_q == nullptr) {
    int tx, hb;
    dense_order(p, (int)blockIdx.x, p.tiles_x, tx, hb);
    h = hb % p.H;
    batch = hb / p.H;
    w = dense_tile<TM>(p, tx, (int)batch);
  } else {
    h = blockIdx.y;
    if (warp == 0) {
      TileWork f = find_varlen_tile<TM>(p, (int)blockIdx.x);
      if (lane == 0) shared_work = f;
    }
    __syncthreads();
    w = shared_work;
    if (w.b < 0) return;
  }
  const int md = spec.max_distance;
  const bool has_bias = p.table != nullptr;
  int kv_end = w.len_k;
  if (p.causal) kv_end = min(w.len_k, w.qpos0 + w.rows_in_tile);
  const T* qbase = (const T*)p.q + (int64_t)w.b * p.q_stride_b + (int64_t)h * p.q_stride_h + (int64_t)w.q_row0 * p.q_stride_m;
  const T* kbase = (const T*)p.k + (int64_t)w.b * p.k_stride_b + (int64_t)h * p.k_stride_h + (int64_t)w.k_row0 * p.k_stride_n;
  const T* vbase = (const T*)p.v + (int64_t)w.b * p.v_stride_b + (int64_t)h * p.v_stride_h + (int64_t)w.k_row0 * p.v_stride_n;

  float4 kn[CHUNKS], vn[CHUNKS];                    // the next tile
  auto fetch = [&](int n0) {
    #pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int c = tid + i * THREADS, n = n0 + c / (D / 4), d = c % (D / 4) * 4;
      kn[i] = vn[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (n < kv_end) {                             // (beyond: not visible to any row here, and 0 x NaN is NaN)
        kn[i] = load4<T>(kbase + (int64_t)n * p.k_stride_n + d, vec);
        vn[i] = load4<T>(vbase + (int64_t)n * p.v_stride_n + d, vec);
      }
    }
  };
  if (kv_end > 0) fetch(0);
  for (int c = tid; c < TM * (D / 4); c += THREADS) {
    const int r = c / (D / 4), d = c % (D / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < w.rows_in_tile) v = load4<T>(qbase + (int64_t)r * p.q_stride_m + d, vec);
    *reinterpret_cast<float4*>(sQ + r * PQ + d) =
        make_float4(v.x * p.scale_log2, v.y * p.scale_log2, v.z * p.scale_log2, v.w * p.scale_log2);
  }
  if (has_bias) {
    for (int i = tid; i < 2 * md + 1; i += THREADS) {
      const int bucket = bucket_of_delta_counted(spec, i - md);
      lut[i] = load_table(p.table, p.table_dtype, (int64_t)bucket * p.table_stride0 + h) * kLog2e;
    }
  }

  const int tx = tid & 15, r0 = (tid >> 4) * RPT;   // the 16 threads of a row group are one half of a warp
  float o[RPT][DPT], m_run[RPT], l_run[RPT];
  #pragma unroll
  for (int i = 0; i < RPT; ++i) {
    m_run[i] = -INFINITY; l_run[i] = 0.f;
    #pragma unroll
    for (int e = 0; e < DPT; ++e) o[i][e] = 0.f;
  }

  #pragma unroll 1
  for (int n0 = 0; n0 < kv_end; n0 += TN) {
    __syncthreads();                                // the tile before is done with (first: Q and the table are written)
    #pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int c = tid + i * THREADS, n = c / (D / 4), d = c % (D / 4) * 4;
      *reinterpret_cast<float4*>(sK + n * PQ + d) = kn[i];
      *reinterpret_cast<float4*>(sV + n * D + d) = vn[i];
    }
    __syncthreads();
    if (n0 + TN < kv_end) fetch(n0 + TN);

    // ---- scores of RPT rows x KPT keys
    float s[RPT][KPT];
    {
      unsigned long long acc[RPT][KPT];
      #pragma unroll
      for (int i = 0; i < RPT; ++i)
        #pragma unroll
        for (int j = 0; j < KPT; ++j) acc[i][j] = 0ull;
      #pragma unroll 2
      for (int d = 0; d < D; d += 4) {
        ulonglong2 qv[RPT], kv[KPT];
        #pragma unroll
        for (int i = 0; i < RPT; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(sQ + (r0 + i) * PQ + d);
        #pragma unroll
        for (int j = 0; j < KPT; ++j) kv[j] = *reinterpret_cast<const ulonglong2*>(sK + (tx + 16 * j) * PQ + d);
        #pragma unroll
        for (int i = 0; i < RPT; ++i)
          #pragma unroll
          for (int j = 0; j < KPT; ++j) { fma_pair(acc[i][j], qv[i].x, kv[j].x); fma_pair(acc[i][j], qv[i].y, kv[j].y); }
      }
      #pragma unroll
      for (int i = 0; i < RPT; ++i)
        #pragma unroll
        for (int j = 0; j < KPT; ++j) s[i][j] = sum_pair(acc[i][j]);
    }
    if (has_bias) {
      const int dmin = n0 - (w.qpos0 + TM - 1), dmax = n0 + TN - 1 - w.qpos0;
      if (dmin >= md || dmax <= -md) {              // far from the diagonal: one bias for the tile
        const float bias = lut[dmin >= md ? 2 * md : 0];
        #pragma unroll
        for (int i = 0; i < RPT; ++i)
          #pragma unroll
          for (int j = 0; j < KPT; ++j) s[i][j] += bias;
      } else {
        #pragma unroll
        for (int i = 0; i < RPT; ++i)
          #pragma unroll
          for (int j = 0; j < KPT; ++j) s[i][j] += lut[min(max(n0 + tx + 16 * j - (w.qpos0 + r0 + i) + md, 0), 2 * md)];
      }
    }
    if (n0 + TN > w.len_k || (p.causal && n0 + TN - 1 > w.qpos0)) {
      #pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int n_valid = p.causal ? min(w.len_k, w.qpos0 + r0 + i + 1) : w.len_k;
        #pragma unroll
        for (int j = 0; j < KPT; ++j)
          if (n0 + tx + 16 * j >= n_valid) s[i][j] = -INFINITY;
      }
    }

    // ---- running maximum of each row (over its 16 threads), probabilities to shared memory
    #pragma unroll
    for (int i = 0; i < RPT; ++i) {
      float mx = s[i][0];
      #pragma unroll
      for (int j = 1; j < KPT; ++j) mx = fmaxf(mx, s[i][j]);
      #pragma unroll
      for (int k = 1; k < 16; k <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, k));
      const float m_new = fmaxf(m_run[i], mx), m_safe = m_new == -INFINITY ? 0.f : m_new;   // nothing visible yet: all p = 0
      const float alpha = exp2f(m_run[i] - m_safe);
      m_run[i] = m_new;
      l_run[i] *= alpha;
      #pragma unroll
      for (int e = 0; e < DPT; ++e) o[i][e] *= alpha;
      #pragma unroll
      for (int j = 0; j < KPT; ++j) {
        const float pr = exp2f(s[i][j] - m_safe);
        l_run[i] += pr;
        sP[(r0 + i) * PP + tx + 16 * j] = pr;
      }
    }
    __syncwarp();                                   // a row's probabilities stay within its half warp

    // ---- O += P V
    #pragma unroll 2
    for (int n = 0; n < TN; n += 4) {
      float4 pv[RPT];
      #pragma unroll
      for (int i = 0; i < RPT; ++i) pv[i] = *reinterpret_cast<const float4*>(sP + (r0 + i) * PP + n);
      #pragma unroll
      for (int u = 0; u < 4; ++u) {
        #pragma unroll
        for (int g = 0; g < DPT / DV; ++g) {
          float vv[DV];
          const float* vr = sV + (n + u) * D + g * 16 * DV + tx * DV;
          if constexpr (DV == 4) { const float4 t = *reinterpret_cast<const float4*>(vr); vv[0] = t.x; vv[1] = t.y; vv[2] = t.z; vv[3] = t.w; }
          else if constexpr (DV == 2) { const float2 t = *reinterpret_cast<const float2*>(vr); vv[0] = t.x; vv[1] = t.y; }
          else vv[0] = *vr;
          #pragma unroll
          for (int i = 0; i < RPT; ++i) {
            const float pr = u == 0 ? pv[i].x : u == 1 ? pv[i].y : u == 2 ? pv[i].z : pv[i].w;
            #pragma unroll
            for (int e = 0; e < DV; ++e) o[i][g * DV + e] = fmaf(pr, vv[e], o[i][g * DV + e]);
          }
        }
      }
    }
  }

  #pragma unroll
  for (int i = 0; i < RPT; ++i) {
    float l = l_run[i];
    #pragma unroll
    for (int k = 1; k < 16; k <<= 1) l += __shfl_xor_sync(0xffffffffu, l, k);
    const int r = r0 + i;
    if (r < w.rows_in_tile) {
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      T* optr = (T*)p.out + (int64_t)w.b * p.o_stride_b + (int64_t)h * p.o_stride_h + (int64_t)(w.q_row0 + r) * p.o_stride_m;
      #pragma unroll
      for (int g = 0; g < DPT / DV; ++g)
        #pragma unroll
        for (int e = 0; e < DV; ++e) optr[g * 16 * DV + tx * DV + e] = from_float<T>(o[i][g * DV + e] * inv_l);
      if (p.lse != nullptr && tx == 0) {
        const float lse = l > 0.f ? (m_run[i] + log2f(l)) * kLn2 : -INFINITY;
        const int64_t row = (int64_t)w.q_row0 + r;
        if (p.cu_q == nullptr) p.lse[(batch * p.H + h) * p.M + row] = lse;
        else p.lse[row * p.H + h] = lse;
      }
    }
  }
}

template <typename T, int D, int RPT>
static int launch(const t5b_attn_args& a, AttnParams p, const BucketSpec& spec, cudaStream_t stream) {
  constexpr int TM = 16 * RPT;
  dim3 grid;
  if (a.cu_seqlens_q != nullptr) {
    grid = dim3((unsigned)((long long)a.total_q / TM + a.B), (unsigned)a.H, 1);
  } else {
    p.tiles_x = (a.M + TM - 1) / TM;
    const long long blocks = (long long)p.tiles_x * a.H * a.B;
    if (blocks > 0x7fffffffLL) return T5B_ERR_SHAPE;
    grid = dim3((unsigned)blocks, 1, 1);
  }
  const size_t smem = (smem_floats<D, RPT>() + (a.table ? 2 * spec.max_distance + 1 : 0)) * sizeof(float);
  // vectors of four elements where every row of q, k and v starts at a multiple of them
  auto aligned = [](const void* ptr, int64_t s0, int64_t s1, int64_t s2) {
    return (uintptr_t)ptr % (4 * sizeof(T)) == 0 && s0 % 4 == 0 && s1 % 4 == 0 && s2 % 4 == 0;
  };
  const bool vec = aligned(a.q, a.q_stride_b, a.q_stride_h, a.q_stride_m) && aligned(a.k, a.k_stride_b, a.k_stride_h, a.k_stride_n) &&
                   aligned(a.v, a.v_stride_b, a.v_stride_h, a.v_stride_n);
  auto kern = attn_fwd_simt_kernel<T, D, RPT>;
  // Room for the largest table, once per device and kernel: a limit set call by call would be lowered under another
  // thread's launch with a longer table.
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
    const size_t most = (smem_floats<D, RPT>() + 2 * 2048 + 1) * sizeof(float);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) {
      cudaGetLastError();
      return T5B_ERR_LAUNCH;
    }
    if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
  }
  kern<<<grid, THREADS, smem, stream>>>(p, spec, vec);
  return cudaGetLastError() == cudaSuccess ? T5B_OK : T5B_ERR_LAUNCH;
}

// 64 query rows per block where that fills the GPU (148 SMs); below, 32: half the reuse of a loaded key, twice the blocks.
template <typename T, int D>
static int launch_rows(const t5b_attn_args& a, const AttnParams& p, const BucketSpec& spec, cudaStream_t stream) {
  const long long rows = a.cu_seqlens_q != nullptr ? (long long)a.total_q : (long long)a.M * a.B;
  return rows * a.H >= 64LL * 148 ? launch<T, D, 4>(a, p, spec, stream) : launch<T, D, 2>(a, p, spec, stream);
}

template <typename T>
static int launch_for_type(const t5b_attn_args& a, const AttnParams& p, const BucketSpec& spec, cudaStream_t stream) {
  switch (a.D) {
    case 16: return launch_rows<T, 16>(a, p, spec, stream);
    case 32: return launch_rows<T, 32>(a, p, spec, stream);
    case 64: return launch_rows<T, 64>(a, p, spec, stream);
    case 128: return launch_rows<T, 128>(a, p, spec, stream);
  }
  return T5B_ERR_HEAD_DIM;
}

}  // namespace simt

int simt_attention_fwd(const t5b_attn_args& a, const BucketSpec& spec, cudaStream_t stream) {
  using namespace simt;
  if (a.table && spec.max_distance > 2048) return T5B_ERR_UNSUPPORTED;
  if (a.H > 65535 || (a.cu_seqlens_q == nullptr && a.B > 65535)) return T5B_ERR_SHAPE;
  const AttnParams p = make_attn_params(a);
  switch (a.dtype) {
    case T5B_F32: return launch_for_type<float>(a, p, spec, stream);
    case T5B_F16: return launch_for_type<__half>(a, p, spec, stream);
    case T5B_BF16: return launch_for_type<__nv_bfloat16>(a, p, spec, stream);
  }
  return T5B_ERR_DTYPE;
}

}  // namespace t5b
