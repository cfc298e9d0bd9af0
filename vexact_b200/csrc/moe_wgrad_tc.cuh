// Weight gradient of a grouped GEMM on tcgen05, the contraction running over each group's own rows ("ragged K"):
//   c[g, m, n] = sum over rows r of group g, ascending, of a[r, m] * b[r, n]      (fp32 accumulation, one rounding)
// (group_gemm/kernel/group_gemm.py:255-400 group_gemm_same_mn with transpose_a).
//
// Both operands lie with the contraction as their row dimension, so both are read MN-major, as TMA leaves them: boxes of
// 64 columns x 64 rows with the 128-byte swizzle.  A tile is 128 x 256 of one group's gradient: 48 KB of operands per 64 rows
// against 512 cycles of tensor pipe, two tensor-memory accumulators so that a tile's epilogue runs beside the next one's
// products, and the result through shared memory by TMA (rows of c are written in whole 128-byte lines; edges are clipped by
// the map).  Persistent CTAs walk the tiles group by group, so a group's rows come from HBM once.
//
// Bound: shared-memory fill, 768 cycles per 64 rows at 64 B a cycle, then writing c.  128 groups of 256 rows, 768 x 2048:
// 656 us on mma.sync.
//
// A group's last step holds rows of the next group (or, at the end, zeros): the MMA warp clears them up to the 16 rows of an
// instruction and issues no instruction beyond.  An empty group gets zeros.  A group whose bounds leave [0, rows] or decrease
// is clipped and reported through the status word.
//
// Warps (12): 0 TMA producer, 1 MMA issuer and TMEM owner, 2 - 3 idle, 4 - 11 epilogue, two per tensor-memory quadrant.
#pragma once
#include "attn_tc.cuh"
#include "gemm.cuh"

namespace b200 {

constexpr int WGT_THREADS = 384, WGT_M = 128, WGT_N = 256, WGT_ROWS = 64, WGT_STAGES = 3;
constexpr int WGT_BOX = WGT_ROWS * 128;                              // bytes of a 64 x 64 operand box
constexpr int WGT_BOXES = (WGT_M + WGT_N) / 64, WGT_STAGE = WGT_BOXES * WGT_BOX;
constexpr int WGT_OUT = WGT_M * WGT_N * 2;
constexpr int WGT_SMEM = 1024 + WGT_STAGES * WGT_STAGE + WGT_OUT + 256;
static_assert(WGT_SMEM <= 227 * 1024, "shared memory budget");

struct WgradMaps {
  CUtensorMap a, b, c;
};

// Rows of group g, clipped to [0, rows].
__device__ __forceinline__ int wgrad_rows(const int* cu_seqlens, int g, int rows, int& r0, bool report) {
  const int lo = cu_seqlens[g], hi = cu_seqlens[g + 1];
  if (report && (lo < 0 || hi > rows || hi < lo)) report_status(B200_STATUS_BAD_INDEX, g);
  r0 = min(max(lo, 0), rows);
  return max(min(hi, rows) - r0, 0);
}

__global__ void __launch_bounds__(WGT_THREADS, 1)
moe_wgrad_tc_kernel(const __grid_constant__ WgradMaps tm, const int* __restrict__ cu_seqlens, int rows, int groups, int m_tiles,
                    int n_tiles, int N, bool deep, int M, __nv_bfloat16* c_words) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t stage0 = (raw + 1023) & ~1023u, out0 = stage0 + WGT_STAGES * WGT_STAGE;
  uint8_t* base = smem_raw + (stage0 - raw);
  uint8_t* out_ptr = base + WGT_STAGES * WGT_STAGE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_ptr + WGT_OUT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 17);
  auto full = [&](int s) { return ptx::smem_u32(&bars[s]); };
  auto empty = [&](int s) { return ptx::smem_u32(&bars[4 + s]); };
  auto tfull = [&](int b) { return ptx::smem_u32(&bars[8 + b]); };
  auto tempty = [&](int b) { return ptx::smem_u32(&bars[10 + b]); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < WGT_STAGES; ++s) {
      ptx::mbar_init(full(s), 1);
      ptx::mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(tfull(b), 1);
      ptx::mbar_init(tempty(b), 256);
    }
    ptx::fence_barrier_init();
    ptx::prefetch_tensormap(&tm.a);
    ptx::prefetch_tensormap(&tm.b);
    ptx::prefetch_tensormap(&tm.c);
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();
  const int per_group = m_tiles * n_tiles;
  const long long total = (long long)per_group * groups;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (ptx::elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (long long lin = blockIdx.x; ok && lin < total; lin += gridDim.x) {
        const int g = (int)(lin / per_group), t = (int)(lin % per_group);
        int r0;
        const int n = wgrad_rows(cu_seqlens, g, rows, r0, t == 0);
        const int m0 = t / n_tiles * WGT_M, n0 = t % n_tiles * WGT_N;
        for (int r = 0; r < n; r += WGT_ROWS, ++it) {
          const int s = it % WGT_STAGES;
          if (!ptx::mbar_wait(empty(s), ((it / WGT_STAGES) & 1) ^ 1, abort_flag, 900 + s)) {
            ok = false;
            break;
          }
          ptx::mbar_expect_tx(full(s), WGT_STAGE);
          const uint32_t at = stage0 + s * WGT_STAGE;
          if (deep) {      // one copy an operand (make_tmap_deep): six boxes a step took longer to issue than to arrive
            ptx::tma_load_3d(at, &tm.a, full(s), 0, r0 + r, m0 / 64, ptx::kEvictLast);
            ptx::tma_load_3d(at + WGT_M / 64 * WGT_BOX, &tm.b, full(s), 0, r0 + r, n0 / 64, ptx::kEvictLast);
            continue;
          }
#pragma unroll
          for (int h = 0; h < WGT_M / 64; ++h)
            ptx::tma_load_2d(at + h * WGT_BOX, &tm.a, full(s), m0 + h * 64, r0 + r, ptx::kEvictLast);
#pragma unroll
          for (int h = 0; h < WGT_N / 64; ++h)
            ptx::tma_load_2d(at + (WGT_M / 64 + h) * WGT_BOX, &tm.b, full(s), n0 + h * 64, r0 + r, ptx::kEvictLast);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the whole warp walks; one lane issues)
    const uint32_t idesc = umma_idesc_bf16(WGT_N, true) | (1u << 16);
    uint32_t it = 0, tile_it = 0;
    bool ok = true;
    for (long long lin = blockIdx.x; ok && lin < total; lin += gridDim.x, ++tile_it) {
      int r0;
      const int n = wgrad_rows(cu_seqlens, (int)(lin / per_group), rows, r0, false), buf = tile_it & 1;
      if (!ptx::mbar_wait_warp(tempty(buf), ((tile_it >> 1) & 1) ^ 1, abort_flag, 910 + buf)) break;
      ptx::tc_fence_after();
      for (int r = 0; r < n; r += WGT_ROWS, ++it) {
        const int s = it % WGT_STAGES, live = min(WGT_ROWS, n - r), k_steps = (live + 15) >> 4;
        if (!ptx::mbar_wait_warp(full(s), (it / WGT_STAGES) & 1, abort_flag, 920 + s)) {
          ok = false;
          break;
        }
        if (live & 15) {
          // rows live .. 16 k_steps of every box: 128 bytes each, whatever the swizzle
          const int per = (16 * k_steps - live) * 8;
          for (int e = lane; e < per * WGT_BOXES; e += 32) {
            const int box = e / per, w = e % per;
            *reinterpret_cast<uint4*>(base + s * WGT_STAGE + box * WGT_BOX + live * 128 + w * 16) = make_uint4(0, 0, 0, 0);
          }
          ptx::fence_proxy_async_smem();
          __syncwarp();
        }
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          const uint32_t at = stage0 + s * WGT_STAGE;
          for (int kk = 0; kk < k_steps; ++kk)
            ptx::umma_bf16(tmem + buf * WGT_N, umma_desc_mn_sw128(at + kk * 2048, WGT_BOX),
                           umma_desc_mn_sw128(at + WGT_M / 64 * WGT_BOX + kk * 2048, WGT_BOX), idesc, (r | kk) != 0 ? 1u : 0u);
          ptx::umma_commit(empty(s));
          if (r + WGT_ROWS >= n) ptx::umma_commit(tfull(buf));
        }
        __syncwarp();
      }
      if (ok && n == 0 && ptx::elect_one()) ptx::umma_commit(tfull(buf));
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3, row = q * 32 + lane, half = (warp - 4) >> 2;
    uint32_t tile_it = 0;
    for (long long lin = blockIdx.x; lin < total; lin += gridDim.x, ++tile_it) {
      const int g = (int)(lin / per_group), t = (int)(lin % per_group), buf = tile_it & 1;
      const int m0 = t / n_tiles * WGT_M, n0 = t % n_tiles * WGT_N;
      int r0;
      const int n = wgrad_rows(cu_seqlens, g, rows, r0, false);
      const bool ready = ptx::mbar_wait(tfull(buf), (tile_it >> 1) & 1, abort_flag, 930 + buf);
      if (threadIdx.x == 128) ptx::bulk_wait_read0();      // the previous tile's copy out has read the staging tile
      if (ptx::named_barrier_any(1, 256, !ready)) break;   // all eight warps leave together
      ptx::tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + buf * WGT_N;
#pragma unroll
      for (int i = 0; i < WGT_N / 2; i += 16) {
        const int c = half * (WGT_N / 2) + i;
        uint32_t r[16];
        ptx::tmem_ld16(taddr + c, r);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (n) {
            const float* f = reinterpret_cast<const float*>(r) + 8 * h;
            v = make_uint4(pack_bf2(f[0], f[1]), pack_bf2(f[2], f[3]), pack_bf2(f[4], f[5]), pack_bf2(f[6], f[7]));
          }
          const int chunk = (c & 63) / 8 + h;              // 16-byte chunk of the row's 128 bytes, swizzled by the row
          *reinterpret_cast<uint4*>(out_ptr + c / 64 * (WGT_M * 128) + row * 128 + ((chunk ^ (row & 7)) << 4)) = v;
        }
      }
      ptx::tc_fence_before();
      ptx::mbar_arrive(tempty(buf));
      ptx::fence_proxy_async_smem();
      ptx::named_barrier_sync(1, 256);
      if (c_words) {
        // c on a 4-byte boundary: the staged tile leaves as words, a warp's 128 bytes of a row together
        for (int i = warp - 4; i < WGT_M * (WGT_N / 64); i += 8) {
          const int h = i / WGT_M, r = i % WGT_M, col = n0 + h * 64 + lane * 2;
          if (m0 + r < M && col < N)
            *reinterpret_cast<uint32_t*>(c_words + ((long long)g * M + m0 + r) * N + col) =
                *reinterpret_cast<const uint32_t*>(out_ptr + h * (WGT_M * 128) + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
        }
      } else if (threadIdx.x == 128) {
        for (int h = 0; h < WGT_N / 64; ++h)
          if (n0 + h * 64 < N) ptx::tma_store_3d(&tm.c, out0 + h * (WGT_M * 128), n0 + h * 64, m0, g);
        ptx::bulk_commit();
      }
    }
    if (threadIdx.x == 128) ptx::bulk_wait0();
  }

  // Teardown.  On an aborted run give in-flight TMA copies time to land before the CTA exits.
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
  }
  ptx::tc_fence_after();
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_dealloc(tmem, 512);
  }
}

// a and b are 16-byte aligned with rows of a multiple of 8 elements, c is 4-byte aligned; M, N multiples of 8.  A c that no tensor
// map takes (16 bytes) is written by the epilogue warps: 32 groups of 256 rows, 768 x 2048, 60 us
// against 55 by TMA (the CUDA-core kernel: 794).
inline int moe_wgrad_tc_launch(const void* a, long long a_stride, const void* b, long long b_stride, void* c, const int* cu_seqlens,
                               long long rows, int groups, int M, int N, cudaStream_t st) {
  static PerDeviceFlags attr_set;
  if (int rc = set_max_dyn_smem_once(attr_set, moe_wgrad_tc_kernel, WGT_SMEM)) return rc;
  WgradMaps tm;
  // a map has at least one row; without rows nothing is read
  const uint64_t map_rows = rows > 0 ? (uint64_t)rows : 1;
  const bool deep = M % 64 == 0 && N % 64 == 0;
  int rc = deep ? make_tmap_deep(&tm.a, a, map_rows, (uint64_t)M, (uint64_t)a_stride, WGT_ROWS, WGT_M / 64)
                : make_tmap_2d(&tm.a, a, map_rows, (uint64_t)M, (uint64_t)a_stride, WGT_ROWS);
  if (!rc)
    rc = deep ? make_tmap_deep(&tm.b, b, map_rows, (uint64_t)N, (uint64_t)b_stride, WGT_ROWS, WGT_N / 64)
              : make_tmap_2d(&tm.b, b, map_rows, (uint64_t)N, (uint64_t)b_stride, WGT_ROWS);
  const bool words = (reinterpret_cast<uintptr_t>(c) & 15) != 0;
  if (words) tm.c = tm.a;
  else if (!rc) rc = make_tmap_3d(&tm.c, c, (uint64_t)groups, (uint64_t)M, (uint64_t)N, (uint64_t)M * N, (uint64_t)N, WGT_M);
  if (rc) return rc;
  const int m_tiles = (M + WGT_M - 1) / WGT_M, n_tiles = (N + WGT_N - 1) / WGT_N;
  const long long total = (long long)m_tiles * n_tiles * groups;
  launch_k(moe_wgrad_tc_kernel, dim3((unsigned)(total < sm_count() ? total : sm_count())), dim3(WGT_THREADS), WGT_SMEM, st, tm,
           cu_seqlens, (int)rows, groups, m_tiles, n_tiles, N, deep, M, words ? (__nv_bfloat16*)c : nullptr);
  return launch_status();
}

}  // namespace b200
