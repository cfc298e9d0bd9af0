// Shared device/host helpers for the sm_100a rollout-forward kernels.
//
// Conventions used by every kernel in this directory:
//   * every entry point launches on the caller's stream, allocates nothing and
//     never synchronises, so it can be captured into a CUDA graph;
//   * every reduction uses one fixed tree that depends only on the row length,
//     never on the number of rows, so a row's result is bitwise independent of
//     the batch it is computed in;
//   * every spin-wait is bounded: on expiry the kernel writes a code into the
//     device status word (see b200_status_read) and returns.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>

#define B200_OK 0
#define B200_ERR_ARG (-1)
#define B200_ERR_SHAPE (-2)
#define B200_ERR_LAUNCH (-3)
#define B200_ERR_DRIVER (-4)

// Codes a kernel may leave in the device status word.
#define B200_STATUS_OK 0
#define B200_STATUS_WAIT_EXPIRED 1
#define B200_STATUS_BAD_INDEX 2

namespace b200 {

// Device status word: [0] = first non-zero code seen, [1] = detail (barrier id
// or offending index), [2] = block id, [3] = spare.
__device__ int g_status[4];  // one copy: all kernels are built as a single translation unit

__device__ __forceinline__ void report_status(int code, int detail) {
  if (atomicCAS(&g_status[0], 0, code) == 0) {
    g_status[1] = detail;
    g_status[2] = (int)blockIdx.x;
  }
}

__device__ __forceinline__ float bf2f(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ __nv_bfloat16 f2bf(float v) { return __float2bfloat16_rn(v); }
// Round an fp32 value to bf16 precision and keep it in fp32 (models a bf16
// tensor being materialised between two torch ops).
__device__ __forceinline__ float round_bf(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi) {
  __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&t);
}
__device__ __forceinline__ void unpack_bf2(uint32_t v, float& lo, float& hi) {
  __nv_bfloat162 t = *reinterpret_cast<__nv_bfloat162*>(&v);
  lo = __low2float(t);
  hi = __high2float(t);
}

// Two neighbouring values in one register pair: one instruction for both.
struct Two {
  unsigned long long v;
  __device__ __forceinline__ Two() {}
  __device__ __forceinline__ Two(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
  __device__ __forceinline__ explicit Two(float a) : Two(a, a) {}
  __device__ __forceinline__ void get(float& a, float& b) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
};
__device__ __forceinline__ Two operator+(const Two& a, const Two& b) {
  Two r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Two operator*(const Two& a, const Two& b) {
  Two r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Two fma2(const Two& a, const Two& b, const Two& c) {
  Two r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// silu(g) = g / (1 + exp(-g)) on the special-function unit.  The error grows with |g|, the rounding of g log2 e being one of
// the exponent: a relative |g| 2^-24 and 2^-22 from the unit.  For bf16 gates, which is what every use has, the result rounded to
// bf16 is that of the exact exponential and division for each of the 65536 values (tests/test_gpu_moe.py); the denominator is
// scaled by 2^-24 where it may pass 2^126, whose reciprocal the unit flushes to zero.  (The exact forms took 45 of the 60
// instructions per element of the SwiGLU kernels, which they bound.)
__device__ __forceinline__ float silu_sfu(float g) {
  const float s = g < 0.f ? 0x1p-24f : 1.f;
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaf(e, s, s)));
  return g * r * s;
}
// One element of the expert and dense SwiGLU with the rounding points of fused_moe.py:319-336: silu(g) and its product with u
// are bf16 tensors.  g holds a bf16 value.
__device__ __forceinline__ float swiglu_reference(float g, float u) { return round_bf(round_bf(silu_sfu(g)) * u); }

// Fixed butterfly reductions over a full warp.
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum with a fixed order: warp butterflies, then warp 0 folds the
// per-warp partials with another butterfly.  `scratch` holds 32 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nwarps) ? scratch[lane] : 0.f;
  t = warp_sum(t);
  return t;
}
__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nwarps) ? scratch[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Programmatic dependent launch.  Kernels of the per-layer chain are launched with the
// programmatic-stream-serialization attribute: a kernel may start (and run its prologue) while
// its predecessor drains, and touches global memory only after pdl_wait(), which returns once
// the predecessor has completed and its writes are visible.  pdl_trigger() lets the successor
// begin launching; every CTA calls it first thing, so a successor can become resident only
// when every CTA of this kernel has started.  Without the attribute both are no-ops.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Programmatic dependent launch (B200_PDL): 0 = off, 1 = every kernel, 3 = only kernels without dynamic
// shared memory, i.e. the short row / routing / permutation kernels, which can be resident beside a
// finishing GEMM or attention CTA and then start the moment it is done; 2 (default) = those plus the dense
// GEMMs, which request their first weight tiles before they wait.  Every kernel waits
// (griddepcontrol.wait) before it touches what its predecessor wrote.  Measured inside the captured
// decode step: mode 3 is worth 2.5 % on the small dense models and neutral on the 30B-A3B shape;
// mode 1 costs the latter 0.4 %.
inline int pdl_mode() {
  static const int mode = []() {
    const char* v = getenv("B200_PDL");
    return v ? atoi(v) : 2;
  }();
  return mode;
}

// What the calling thread has said about its launches (b200_settled_weights): `ordered`, that its next one waits for all work
// before it in full, and `settled`, that the weights of its dense products are written by nothing launched since.
struct LaunchScope {
  bool settled = false, ordered = false;
};
inline LaunchScope& launch_scope() {
  static thread_local LaunchScope scope;
  return scope;
}
inline bool launch_programmatic(bool pdl) {
  LaunchScope& scope = launch_scope();
  pdl = pdl && !scope.ordered;
  scope.ordered = false;
  return pdl;
}

// cluster: CTAs of a cluster along x (1: no cluster launch).
template <typename... KArgs, typename... Args>
inline void launch_k_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl, int cluster,
                         Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  if (launch_programmatic(pdl)) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  cfg.attrs = attr;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
inline void launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  const int mode = pdl_mode();
  cfg.numAttrs = launch_programmatic(mode == 1 || (mode >= 2 && smem == 0)) ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Facts and one-time settings that belong to a device, not to the process: a process that drives
// several GPUs gets each of them looked up / set once, with that device current.
constexpr int B200_MAX_DEVICES = 64;

struct PerDeviceFlags {
  std::atomic<int> v[B200_MAX_DEVICES];  // static storage: zero-initialised
};

inline int current_device_index() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= B200_MAX_DEVICES) return -1;
  return dev;
}

// Raises a kernel's dynamic shared-memory limit once per device (the attribute is per device).
template <typename KernelT>
inline int set_max_dyn_smem_once(PerDeviceFlags& done, KernelT kernel, int bytes) {
  const int dev = current_device_index();
  if (dev < 0) return B200_ERR_LAUNCH;
  if (done.v[dev].load(std::memory_order_acquire) == 0) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
      return B200_ERR_LAUNCH;
    done.v[dev].store(1, std::memory_order_release);
  }
  return B200_OK;
}

// SM count of the current device (cached per device).
inline int sm_count() {
  static PerDeviceFlags cache;
  const int dev = current_device_index();
  if (dev < 0) return 148;
  int n = cache.v[dev].load(std::memory_order_acquire);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache.v[dev].store(n, std::memory_order_release);
  }
  return n;
}

// Token tiles of the grouped GEMMs.  Height for `rows` rows over `groups` groups of products with at least `features` outputs:
// few rows per group want one low tile each (its pipeline stages are smaller and deeper); many want tall ones, on CTA pairs,
// which read a weight tile less often.  128 experts, 2048 -> 1536, the same rows for each, at 64 / 128 / 256 rows per tile: 163 /
// 133 / 142 us for 65 rows per expert, 172 / 146 / 151 for 112, 234 / 206 / 161 for 160, 298 / 223 / 185 for 256.  (Rows are not
// evenly spread: from a mean of 112 on, some experts pass 128.)
// A tall tile must not leave the chip idle: there are to be two thirds as many as there are pairs, if they are spread evenly.
// 8 experts, 1024 -> 1024: 8.7 / 10.6 / 10.7 us for 128 rows per expert (128 tiles, 32 pairs, 32 pairs), 11.8 / 10.7 / 11.2 for 160
// (192, 64, 32), 15.3 / 14.8 / 12.4 for 384 (384, 96, 64).
inline int grouped_tile_rows(long long rows, long long groups, int features, int sms) {
  const long long per = (rows + groups - 1) / groups;
  for (int h = rows <= 64 * groups ? 64 : rows <= 112 * groups ? 128 : 256; h > 64; h >>= 1)
    if (3 * groups * ((per + h - 1) / h) * ((features + 255) / 256) >= sms) return h;
  return 64;
}
// Tile j of a group's `tiles`, which is rows / tile_rows rounded up: {group, first row, rows, 0}.  The tiles of a group are equally
// high, in steps of 16, so that none is a remainder that pays for a whole weight tile, and at most tile_rows, which need not be
// such a step.  With h <= tile_rows the first tiles - 1 cover less than the rows, so that the last has some.
__device__ __forceinline__ int4 token_tile(int group, int row0, int rows, int tiles, int j, int tile_rows) {
  const int h = min(((rows + tiles - 1) / tiles + 15) & ~15, tile_rows);
  return make_int4(group, row0 + j * h, min(h, rows - j * h), 0);
}

inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? B200_OK : B200_ERR_LAUNCH;
}

}  // namespace b200
