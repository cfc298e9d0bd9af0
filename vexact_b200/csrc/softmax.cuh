// Row log-softmax and per-token log-probability: HBM-bound row kernels.
//
// Replaces vexact/batch_invariant_ops/batch_invariant_ops.py:232-331
// (_log_softmax_kernel / log_softmax: max pass, sum-exp pass, write pass) and
// vexact/batch_invariant_ops/standalone_logprobs.py:28-55, whose arithmetic is
// flash-attn's Triton cross-entropy forward (logprob = x[label] - logsumexp(x)).
//
// 1024 threads own one row.  Each thread walks 16-byte vectors at a fixed stride
// keeping a private (max, sum exp(x - max)) pair; pairs are merged with a fixed
// butterfly inside each warp and a second butterfly over the 32 warp results.
// The merge order is a function of the row length only.
//
// Where the 1024 threads sit is a question of speed alone (row_ctas): in one CTA,
// or as a cluster of eight CTAs of 128 threads, whose warp results meet in shared
// memory of the cluster.  151936 logits, one CTA to a row before / now: greedy 18 -> 8
// us for 1 to 7 rows, 18 -> 11 for 64, 256 -> 175 for 2000; log-softmax of 7 rows 28 -> 11.
#pragma once
#include "common.cuh"

namespace b200 {

struct MaxSum {
  float m, s;
};

__device__ __forceinline__ MaxSum ms_merge(MaxSum a, MaxSum b) {
  const float m = fmaxf(a.m, b.m);
  MaxSum r;
  r.m = m;
  // exp(-inf - finite) = 0; the (m == -inf) guard keeps empty partials NaN free.
  const float ea = (a.m == -INFINITY) ? 0.f : expf(a.m - m);
  const float eb = (b.m == -INFINITY) ? 0.f : expf(b.m - m);
  r.s = a.s * ea + b.s * eb;
  return r;
}

// exp of two values that are at most 0 (-inf gives 0, NaN stays): 2^h (1 + l ln 2) with h + l = t log2(e), the product
// carried in two floats (the exact remainder of h by fma, and log2(e) itself in two parts), 2^h on the special-function
// unit.  TINY: results below the normal range are subnormal, as the exact exponential's, and not 0; a term of a sum whose largest
// is 1 does not need that.  The walk over 2000 x 151936 bf16 logits is bound by issue slots, not by HBM,
// and the exact exponential took most of them: 214 us with it, 164 so.
template <bool TINY = false>
__device__ __forceinline__ Two exp_nonpos(const Two& t_in) {
  float a, b;
  t_in.get(a, b);
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(a) : "f"(a), "f"(-160.f));
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(b) : "f"(b), "f"(-160.f));
  constexpr float L = 1.4426950408889634f, L_LO = (float)(1.4426950408889634 - (double)L), LN2 = 0.6931471805599453f;
  const Two t(a, b), h = t * Two(L, L);
  const Two neg_l = fma2(t, Two(-L_LO, -L_LO), fma2(t, Two(-L, -L), h));
  h.get(a, b);
  if constexpr (TINY) {
    asm("ex2.approx.f32 %0, %1;" : "=f"(a) : "f"(a));
    asm("ex2.approx.f32 %0, %1;" : "=f"(b) : "f"(b));
  } else {
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(a));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(b));
  }
  const Two e(a, b);
  return fma2(e, neg_l * Two(-LN2, -LN2), e);
}

// A thread's running pair; the sum is kept as two chains (even and odd elements), joined at the end.
struct RowAcc {
  float m = -INFINITY;
  Two s = Two(0.f, 0.f);
  __device__ __forceinline__ MaxSum pair() const {
    float a, b;
    s.get(a, b);
    return MaxSum{m, a + b};
  }
};

// VEC values: one rescale per vector, then the exps.  True where the running maximum moved.
template <int VEC>
__device__ __forceinline__ bool ms_push_vec(RowAcc& a, const float* x) {
  float vm = x[0];
#pragma unroll
  for (int j = 1; j < VEC; ++j) vm = fmaxf(vm, x[j]);
  const bool more = vm > a.m;
  if (more) {
    const float r = a.m == -INFINITY ? 0.f : expf(a.m - vm);
    a.s = a.s * Two(r, r);
    a.m = vm;
  }
  if (a.m > -INFINITY) {
#pragma unroll
    for (int j = 0; j < VEC; j += 2) a.s = a.s + exp_nonpos(Two(x[j], x[j + 1]) + Two(-a.m, -a.m));
  }
  return more;
}
__device__ __forceinline__ bool ms_push(RowAcc& a, float x) {
  const float v[2] = {x, -INFINITY};
  return ms_push_vec<2>(a, v);
}

__device__ __forceinline__ MaxSum ms_block_reduce(MaxSum v, float* sm, float* ss) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum t;
    t.m = __shfl_xor_sync(0xffffffffu, v.m, o);
    t.s = __shfl_xor_sync(0xffffffffu, v.s, o);
    // Merge in lane order so both partners compute the same bits.
    v = (lane & o) ? ms_merge(t, v) : ms_merge(v, t);
  }
  __syncthreads();
  if (lane == 0) {
    sm[warp] = v.m;
    ss[warp] = v.s;
  }
  __syncthreads();
  MaxSum t;
  t.m = lane < nwarps ? sm[lane] : -INFINITY;
  t.s = lane < nwarps ? ss[lane] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum u;
    u.m = __shfl_xor_sync(0xffffffffu, t.m, o);
    u.s = __shfl_xor_sync(0xffffffffu, t.s, o);
    t = (lane & o) ? ms_merge(u, t) : ms_merge(t, u);
  }
  return t;
}

template <typename T>
struct RowLoader;

template <>
struct RowLoader<float> {
  static constexpr int VEC = 4;
  static __device__ __forceinline__ void unpack(const uint4& t, float* v) {
    v[0] = __uint_as_float(t.x), v[1] = __uint_as_float(t.y), v[2] = __uint_as_float(t.z), v[3] = __uint_as_float(t.w);
  }
  static __device__ __forceinline__ uint4 pack(const float* v) {
    return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  }
};
template <>
struct RowLoader<__nv_bfloat16> {
  static constexpr int VEC = 8;
  static __device__ __forceinline__ void unpack(const uint4& t, float* v) {
    unpack_bf2(t.x, v[0], v[1]), unpack_bf2(t.y, v[2], v[3]), unpack_bf2(t.z, v[4], v[5]), unpack_bf2(t.w, v[6], v[7]);
  }
  static __device__ __forceinline__ uint4 pack(const float* v) {
    return make_uint4(pack_bf2(v[0], v[1]), pack_bf2(v[2], v[3]), pack_bf2(v[4], v[5]), pack_bf2(v[6], v[7]));
  }
};

// The walk of one of a row's 1024 threads: vectors vt, vt + 1024, ... in that order, AHEAD requested at a
// time: 8 where the row is spread over a cluster and latency is all, 2 in a full CTA, where more of them cost a resident CTA
// its registers (log-probabilities of 2000 x 151936 bf16: 164 us with 2, 192 with 8).
constexpr int ROW_THREADS = 1024;
template <int AHEAD, typename T, typename F>
__device__ __forceinline__ void row_walk(const T* row, int nvec, int vt, F&& use) {
  constexpr int VEC = RowLoader<T>::VEC;
  for (int v = vt; v < nvec; v += AHEAD * ROW_THREADS) {
    uint4 raw[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (v + u * ROW_THREADS < nvec) raw[u] = *reinterpret_cast<const uint4*>(row + (size_t)(v + u * ROW_THREADS) * VEC);
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (v + u * ROW_THREADS < nvec) {
        float x[VEC];
        RowLoader<T>::unpack(raw[u], x);
        use(x, v + u * ROW_THREADS);
      }
  }
}

// Streams one row and returns its (max, sum exp) pair.  `vec_ok` is a launch-wide
// property (base pointer 16-byte aligned and row stride a multiple of the vector
// width), so every row of a launch, and the same row in any other batch, walks
// its elements in the same order.
template <int CL, typename T>
__device__ __forceinline__ MaxSum row_max_sum_part(const T* __restrict__ row, int n, bool vec_ok, int vt) {
  constexpr int VEC = RowLoader<T>::VEC;
  RowAcc acc;
  const int nvec = vec_ok ? n / VEC : 0;
  row_walk<CL == 1 ? 2 : 8>(row, nvec, vt, [&](const float* x, int) { ms_push_vec<VEC>(acc, x); });
  for (int i = nvec * VEC + vt; i < n; i += ROW_THREADS) ms_push(acc, (float)row[i]);
  return acc.pair();
}
template <typename T>
__device__ __forceinline__ MaxSum row_max_sum(const T* __restrict__ row, int n, bool vec_ok, float* sm,
                                              float* ss) {
  return ms_block_reduce(row_max_sum_part<1>(row, n, vec_ok, threadIdx.x), sm, ss);
}

// ------------------------------------------------------------------ a row's threads spread over CL CTAs
struct RowScratch {
  float m[32], s[32];
  int i[32];
};

// Thread of the row and the row itself.  Ends with the arrival of a cluster's start barrier.
template <int CL>
__device__ __forceinline__ int row_thread(long long& row) {
  row = blockIdx.x / CL;
  if (CL > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  return (int)(blockIdx.x % CL) * (ROW_THREADS / CL) + threadIdx.x;
}

// ms_block_reduce over the row's threads wherever they sit, and the lowest of the indices `idx` whose value `at` is the
// row's maximum (INDEX).  Every thread gets the result.
template <int CL, bool INDEX = false>
__device__ __forceinline__ MaxSum row_reduce(MaxSum v, int vt, RowScratch& sh, float at = 0.f, int* idx = nullptr) {
  const int lane = threadIdx.x & 31, warp = vt >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum t;
    t.m = __shfl_xor_sync(0xffffffffu, v.m, o);
    t.s = __shfl_xor_sync(0xffffffffu, v.s, o);
    v = (lane & o) ? ms_merge(t, v) : ms_merge(v, t);
  }
  int best = 0;
  if (INDEX) best = __reduce_min_sync(0xffffffffu, at == v.m ? *idx : 0x7fffffff);
  if (CL == 1) {
    if (lane == 0) {
      sh.m[warp] = v.m;
      sh.s[warp] = v.s;
      if (INDEX) sh.i[warp] = best;
    }
    __syncthreads();
  } else {
    // every CTA of the cluster has started before its shared memory is written, and all have written before it is read
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (lane < CL) {
      auto put = [&](const void* local, uint32_t bits) {
        uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
        asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(lane));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(bits) : "memory");
      };
      put(&sh.m[warp], __float_as_uint(v.m));
      put(&sh.s[warp], __float_as_uint(v.s));
      if (INDEX) put(&sh.i[warp], (uint32_t)best);
    }
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
  }
  MaxSum t;
  t.m = sh.m[lane];
  t.s = sh.s[lane];
  const float wm = t.m;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum u;
    u.m = __shfl_xor_sync(0xffffffffu, t.m, o);
    u.s = __shfl_xor_sync(0xffffffffu, t.s, o);
    t = (lane & o) ? ms_merge(u, t) : ms_merge(t, u);
  }
  if (INDEX) *idx = __reduce_min_sync(0xffffffffu, wm == t.m ? sh.i[lane] : 0x7fffffff);
  return t;
}

template <int CL>
__global__ void __launch_bounds__(ROW_THREADS / CL, CL == 1 ? 2 : 1)
log_softmax_f32_kernel(const float* __restrict__ x, float* __restrict__ out, int n, long long x_stride,
                       long long out_stride, bool vec) {
  pdl_trigger();
  __shared__ RowScratch sh;
  long long r0;
  const int vt = row_thread<CL>(r0);
  pdl_wait();
  const float* row = x + r0 * x_stride;
  float* orow = out + r0 * out_stride;
  const MaxSum r = row_reduce<CL>(row_max_sum_part<CL>(row, n, vec, vt), vt, sh);
  const float lse = logf(r.s);
  // out = x - max - log(sum), in that order, as the reference kernel's third pass.
  const int nvec = vec ? n >> 2 : 0;
  row_walk<CL == 1 ? 2 : 8>(row, nvec, vt, [&](const float* t, int v) {
    reinterpret_cast<float4*>(orow)[v] = make_float4(t[0] - r.m - lse, t[1] - r.m - lse, t[2] - r.m - lse, t[3] - r.m - lse);
  });
  for (int i = nvec * 4 + vt; i < n; i += ROW_THREADS) orow[i] = row[i] - r.m - lse;
}

// lse (may be null): the rows' log-sum-exp, for the backward.
template <typename T, int CL>
__global__ void __launch_bounds__(ROW_THREADS / CL, CL == 1 ? 2 : 1)
gather_logprob_kernel(const T* __restrict__ x, const long long* __restrict__ labels,
                      float* __restrict__ out, float* __restrict__ lse_out, int n, long long x_stride,
                      long long ignore_index, bool vec) {
  pdl_trigger();
  __shared__ RowScratch sh;
  long long r0;
  const int vt = row_thread<CL>(r0);
  pdl_wait();
  const T* row = x + r0 * x_stride;
  const MaxSum r = row_reduce<CL>(row_max_sum_part<CL>(row, n, vec, vt), vt, sh);
  if (vt == 0) {
    const long long label = labels[r0];
    const float lse = logf(r.s) + r.m;
    float lp = 0.f;  // ignored labels produce a zero loss in the reference kernel
    if (label != ignore_index && label >= 0 && label < n) lp = (float)row[label] - lse;
    out[r0] = lp;
    if (lse_out) lse_out[r0] = lse;
  }
}

// Gradient of gather_logprob_kernel with respect to the logits (flash-attn's cross-entropy backward with the sign
// of a log-probability, flash_attn/ops/triton/cross_entropy.py): dx[i] = g * ((i == label) - exp(x[i] - lse)),
// a zero row for an ignored label.  One read and one write of the row, LPB_CHUNK bytes of it per CTA, where the forward left
// its log-sum-exp; with lse == null a CTA of 1024 threads owns the row and makes the forward's walk first (the same bits).
// dx may be x itself, so x is read before dx is written and through no read-only path.
// 2000 x 151936 bf16: 702 us with the walk made again and 2-byte accesses, 230 now (5.3 TB/s).
constexpr int LPB_THREADS = 256, LPB_CHUNK = LPB_THREADS * 16 * 4;
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
gather_logprob_backward_kernel(const T* x, const long long* __restrict__ labels, const float* __restrict__ grad_out,
                               const float* __restrict__ lse_in, T* dx, int n, long long x_stride, long long dx_stride,
                               long long ignore_index, bool vec_in, bool vec) {
  constexpr int VEC = RowLoader<T>::VEC, PER = LPB_CHUNK / (int)sizeof(T);
  pdl_trigger();
  pdl_wait();
  __shared__ float sm[32], ss[32];
  const long long r0 = blockIdx.y;
  const T* row = x + r0 * x_stride;
  T* drow = dx + r0 * dx_stride;
  const long long label = labels[r0];
  const bool live = label != ignore_index && label >= 0 && label < n;
  float lse;
  int lo = 0, hi = n;
  if (lse_in) {
    lse = lse_in[r0];
    lo = (int)blockIdx.x * PER;
    hi = min(n - lo, PER) + lo;
  } else {
    const MaxSum r = row_max_sum<T>(row, n, vec_in, sm, ss);
    lse = logf(r.s) + r.m;
  }
  const float g = live ? grad_out[r0] : 0.f;
  const int lab = live ? (int)label : -1;
  const Two neg_lse(-lse, -lse);
  auto grad = [&](float& u, float& v, int i) {   // elements i and i + 1
    float a, b;
    exp_nonpos<true>(Two(u, v) + neg_lse).get(a, b);
    u = live ? g * ((i == lab ? 1.f : 0.f) - a) : 0.f;
    v = live ? g * ((i + 1 == lab ? 1.f : 0.f) - b) : 0.f;
  };
  const int vhi = vec ? lo + (hi - lo) / VEC * VEC : lo;
  const int step = blockDim.x * VEC;
  for (int at = lo + threadIdx.x * VEC; at < vhi; at += 4 * step) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (at + u * step < vhi) raw[u] = *reinterpret_cast<const uint4*>(row + at + u * step);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (at + u * step < vhi) {
        float v[VEC];
        RowLoader<T>::unpack(raw[u], v);
#pragma unroll
        for (int j = 0; j < VEC; j += 2) grad(v[j], v[j + 1], at + u * step + j);
        *reinterpret_cast<uint4*>(drow + at + u * step) = RowLoader<T>::pack(v);
      }
  }
  for (int i = vhi + threadIdx.x; i < hi; i += blockDim.x) {
    float u = (float)row[i], none = 0.f;
    grad(u, none, i);
    drow[i] = (T)u;
  }
}

// Greedy token and its log-probability in one pass over a row of logits: argmax (lowest index on
// ties, as torch.argmax) and logprob = max - logsumexp = -log(sum exp(x - max)).  Replaces the
// torch.argmax + cross-entropy pair of Inferencer._select_tokens (inferencer.py:393-449) for greedy
// decoding; the log-probability has the same bits as gather_logprob_kernel given the same label.
template <typename T, int CL>
__global__ void __launch_bounds__(ROW_THREADS / CL, CL == 1 ? 2 : 1)
greedy_logprob_kernel(const T* __restrict__ x, long long* __restrict__ tokens, float* __restrict__ logprobs,
                      int n, long long x_stride, bool vec) {
  pdl_trigger();
  __shared__ RowScratch sh;
  long long r0;
  const int vt = row_thread<CL>(r0);
  pdl_wait();
  const T* row = x + r0 * x_stride;
  // One pass: the (max, sum) walk of row_max_sum, element for element, plus this thread's first
  // index of its own maximum (a thread's indices ascend, and the maximum moves on `>` alone).
  constexpr int VEC = RowLoader<T>::VEC;
  RowAcc acc;
  int bi = 0x7fffffff;
  const int nvec = vec ? n / VEC : 0;
  row_walk<CL == 1 ? 2 : 8>(row, nvec, vt, [&](const float* xv, int v) {
    if (ms_push_vec<VEC>(acc, xv)) {
#pragma unroll
      for (int j = VEC - 1; j >= 0; --j)
        if (xv[j] == acc.m) bi = v * VEC + j;
    }
  });
  for (int i = nvec * VEC + vt; i < n; i += ROW_THREADS)
    if (ms_push(acc, (float)row[i])) bi = i;
  const MaxSum r = row_reduce<CL, true>(acc.pair(), vt, sh, acc.m, &bi);
  if (vt == 0) {
    const int b = bi == 0x7fffffff ? 0 : bi;  // a row without any value above -inf
    tokens[r0] = b;
    logprobs[r0] = (float)row[b] - (logf(r.s) + r.m);
  }
}

// CTAs per row.  A cluster spreads few rows over idle SMs; from about a row per two SMs on, whole
// CTAs do better (log-probabilities of 64 / 148 rows of 151936 bf16: 15 / 14 us in one CTA each, 10 / 24 in eight), and from a
// row per four SMs on where rows are short (64 fp32 rows of 1000 / 4096 / 16384, log-softmax: 5.2 / 5.8 / 7.7 us in one CTA, 5.7 /
// 6.8 / 7.8 in eight; 64 bf16 rows of 1000 / 4096, greedy: 5.1 / 5.5 and 6.3 / 5.2; 33 rows gain or stay at every length, 48 of bf16 too).
template <typename T>
inline int row_ctas(long long rows, int n) { return rows <= 40 || (rows <= 64 && n >= (sizeof(T) == 2 ? 4096 : 16384)) ? 8 : 1; }

// The row kernels' launch: programmatic like launch_k's, `cl` CTAs to a row and to a cluster.
template <typename... KArgs, typename... Args>
inline void launch_rows(void (*kernel)(KArgs...), long long rows, int cl, cudaStream_t st, Args&&... args) {
  launch_k_pdl(kernel, dim3((unsigned)(rows * cl)), dim3(ROW_THREADS / cl), 0, st, pdl_mode() >= 1, cl, static_cast<Args&&>(args)...);
}

}  // namespace b200

extern "C" int b200_log_softmax_f32(const void* x, void* out, long long rows, int n, long long x_row_stride,
                                    long long out_row_stride, void* stream) {
  using namespace b200;
  if (!x || !out || rows < 0 || n <= 0) return B200_ERR_ARG;
  if (rows == 0) return B200_OK;
  const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
                   x_row_stride % 4 == 0 && out_row_stride % 4 == 0;
  const int cl = row_ctas<float>(rows, n);
  launch_rows(cl == 1 ? log_softmax_f32_kernel<1> : log_softmax_f32_kernel<8>, rows, cl, (cudaStream_t)stream,
              (const float*)x, (float*)out, n, x_row_stride, out_row_stride, vec);
  return launch_status();
}

namespace b200 {
template <typename T>
inline int gather_logprob_launch(const void* logits, const void* labels, void* out, void* lse, long long rows, int n,
                                 long long row_stride, long long ignore_index, void* stream) {
  const bool vec = (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && row_stride % RowLoader<T>::VEC == 0;
  const int cl = row_ctas<T>(rows, n);
  launch_rows(cl == 1 ? gather_logprob_kernel<T, 1> : gather_logprob_kernel<T, 8>, rows, cl, (cudaStream_t)stream,
              (const T*)logits, (const long long*)labels, (float*)out, (float*)lse, n, row_stride, ignore_index, vec);
  return launch_status();
}
template <typename T>
inline int gather_logprob_backward_launch(const void* logits, const void* labels, const void* grad, const void* lse,
                                          void* dlogits, long long rows, int n, long long row_stride,
                                          long long d_row_stride, long long ignore_index, void* stream) {
  constexpr int VEC = RowLoader<T>::VEC, PER = LPB_CHUNK / (int)sizeof(T);
  const bool vec_in = (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && row_stride % VEC == 0;
  const bool vec = vec_in && (reinterpret_cast<uintptr_t>(dlogits) & 15) == 0 && d_row_stride % VEC == 0;
  // rows sit on grid y, at most 65535 of them in a launch
  for (long long r = 0; r < rows; r += 65535) {
    const long long m = rows - r < 65535 ? rows - r : 65535;
    launch_k(gather_logprob_backward_kernel<T>, dim3(lse ? (unsigned)((n + PER - 1) / PER) : 1u, (unsigned)m),
             dim3(lse ? LPB_THREADS : ROW_THREADS), 0, (cudaStream_t)stream, (const T*)logits + r * row_stride,
             (const long long*)labels + r, (const float*)grad + r, lse ? (const float*)lse + r : nullptr,
             (T*)dlogits + r * d_row_stride, n, row_stride, d_row_stride, ignore_index, vec_in, vec);
  }
  return launch_status();
}
}  // namespace b200

// lse_f32 (may be null) receives every row's log-sum-exp, which b200_gather_logprob_backward_lse takes.
extern "C" int b200_gather_logprob_lse(const void* logits, const void* labels, void* out, void* lse_f32, long long rows,
                                       int n, long long row_stride, int dtype /*0 = f32, 1 = bf16*/,
                                       long long ignore_index, void* stream) {
  using namespace b200;
  if (!logits || !labels || !out || rows < 0 || n <= 0 || (dtype != 0 && dtype != 1)) return B200_ERR_ARG;
  if (rows == 0) return B200_OK;
  return dtype == 0 ? gather_logprob_launch<float>(logits, labels, out, lse_f32, rows, n, row_stride, ignore_index, stream)
                    : gather_logprob_launch<__nv_bfloat16>(logits, labels, out, lse_f32, rows, n, row_stride, ignore_index, stream);
}

extern "C" int b200_gather_logprob(const void* logits, const void* labels, void* out, long long rows, int n,
                                   long long row_stride, int dtype /*0 = f32, 1 = bf16*/,
                                   long long ignore_index, void* stream) {
  return b200_gather_logprob_lse(logits, labels, out, nullptr, rows, n, row_stride, dtype, ignore_index, stream);
}

// d logprob / d logits for b200_gather_logprob: dlogits[r, i] = grad_out[r] * ((i == label[r]) - softmax(logits[r])[i])
// in the logits' dtype; dlogits may alias logits.  lse_f32: what b200_gather_logprob_lse left, or null.
extern "C" int b200_gather_logprob_backward_lse(const void* logits, const void* labels, const void* grad_out_f32,
                                                const void* lse_f32, void* dlogits, long long rows, int n,
                                                long long row_stride, long long d_row_stride,
                                                int dtype /*0 = f32, 1 = bf16*/, long long ignore_index, void* stream) {
  using namespace b200;
  if (!logits || !labels || !grad_out_f32 || !dlogits || rows < 0 || n <= 0 || (dtype != 0 && dtype != 1))
    return B200_ERR_ARG;
  return dtype == 0 ? gather_logprob_backward_launch<float>(logits, labels, grad_out_f32, lse_f32, dlogits, rows, n, row_stride,
                                                            d_row_stride, ignore_index, stream)
                    : gather_logprob_backward_launch<__nv_bfloat16>(logits, labels, grad_out_f32, lse_f32, dlogits, rows, n,
                                                                    row_stride, d_row_stride, ignore_index, stream);
}

extern "C" int b200_gather_logprob_backward(const void* logits, const void* labels, const void* grad_out_f32,
                                            void* dlogits, long long rows, int n, long long row_stride,
                                            long long d_row_stride, int dtype /*0 = f32, 1 = bf16*/,
                                            long long ignore_index, void* stream) {
  return b200_gather_logprob_backward_lse(logits, labels, grad_out_f32, nullptr, dlogits, rows, n, row_stride, d_row_stride,
                                          dtype, ignore_index, stream);
}

namespace b200 {
template <typename T>
inline int greedy_logprob_launch(const void* logits, void* tokens, void* logprobs, long long rows, int n, long long row_stride,
                                 void* stream) {
  const bool vec = (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && row_stride % RowLoader<T>::VEC == 0;
  const int cl = row_ctas<T>(rows, n);
  launch_rows(cl == 1 ? greedy_logprob_kernel<T, 1> : greedy_logprob_kernel<T, 8>, rows, cl, (cudaStream_t)stream,
              (const T*)logits, (long long*)tokens, (float*)logprobs, n, row_stride, vec);
  return launch_status();
}
}  // namespace b200

extern "C" int b200_greedy_logprob(const void* logits, void* tokens_i64, void* logprobs_f32, long long rows, int n,
                                   long long row_stride, int dtype /*0 = f32, 1 = bf16*/, void* stream) {
  using namespace b200;
  if (!logits || !tokens_i64 || !logprobs_f32 || rows < 0 || n <= 0 || (dtype != 0 && dtype != 1)) return B200_ERR_ARG;
  if (rows == 0) return B200_OK;
  return dtype == 0 ? greedy_logprob_launch<float>(logits, tokens_i64, logprobs_f32, rows, n, row_stride, stream)
                    : greedy_logprob_launch<__nv_bfloat16>(logits, tokens_i64, logprobs_f32, rows, n, row_stride, stream);
}
