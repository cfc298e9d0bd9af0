// The backward of attn_bwd.cuh on tcgen05: the same two kernels with the same rounding points (p and ds become bf16 before
// their products, fp32 accumulation, fixed order, no atomics), 128-row tiles owned by a CTA, the other side streamed past it
// 64 rows at a time.
//
//   dq kernel:  a CTA owns 128 queries of one head (A operands Q and dO) and walks the keys:
//               S = Q K^T, dP = dO V^T, dQ += bf16(dS) K.  A first walk over the keys (S alone) gives the log-sum-exp, where the
//               forward did not leave it (4 x 2048 tokens, 32 / 4 heads of 128: 534 us
//               with that walk, 388 without; the forward's second row sum costs it 334 -> 367).
//   dkv kernel: a CTA owns 128 keys of one KV head (A operands K and V) and walks its query heads and their queries:
//               S^T = K Q^T, dP^T = V dO^T, dV += bf16(P^T) dO, dK += bf16(dS^T) Q.
//
// Owned rows sit on the 128 TMEM lanes in both, so the kernels are one template: two owned tiles X1, X2, a ring of streamed
// tile pairs Y1, Y2 (TMA boxes of 64 rows x 64 columns, 128-byte swizzle), scores = X1 Y1^T and dP = X2 Y2^T double buffered
// in TMEM.  A streamed tile is read K-major for the scores and MN-major, as it lies, for the gradients; P and dS go through
// shared memory as K-major A tiles.  The issuer puts the scores of step i + 1 ahead of the gradients of step i, so the tensor
// core works while the eight compute warps exponentiate.
//
// Bound: per 128 x 64 step 1280 cycles of shared-memory operand reads for the four products of the dkv kernel (1024 of tensor
// pipe) against about 900 issue slots of the compute warps per scheduler; HBM traffic is negligible beside either.
// 4 x 2048 tokens, 32 / 4 heads of 128: dk / dv 356 us, dq 388 us.
//
// Warps (12): 0 TMA producer, 1 UMMA issuer + TMEM owner, 2 keeper (clears streamed rows past the sequence's end, fetches
// their log-sum-exp and delta), 3 idle, 4 - 11 compute: two threads per owned row, 32 streamed rows each.
#pragma once
#include "attn_bwd_mma.cuh"
#include "attn_rows.cuh"

namespace b200 {

constexpr int ABT_THREADS = 384, ABT_M = 128, ABT_N = 64;

// Shared memory of one form, from a 1024-byte boundary.
template <int DK, int DV, bool DKV>
struct AbtLayout {
  static constexpr int X1H = DK / 64, X2H = DV / 64;                     // 64-column halves of an owned tile
  static constexpr int X1 = ABT_M * DK * 2, X2 = ABT_M * DV * 2;
  static constexpr int Y1 = ABT_N * DK * 2, Y2 = ABT_N * DV * 2;         // one streamed tile
  static constexpr int PT = ABT_M * ABT_N * 2;                           // one P or dS tile
  static constexpr int NP = DKV ? 4 : 2;                                 // double-buffered dS, and P
  // barriers; then lse and delta of every stage (dkv) or the halves' row sums (dq)
  static constexpr int small(int stages) { return 256 + (DKV ? stages * 2 * ABT_N : 2 * ABT_M) * 4; }
  static constexpr int total(int stages) { return X1 + X2 + stages * (Y1 + Y2) + NP * PT + small(stages) + 1023; }
  static constexpr int STAGES = total(4) <= 227 * 1024 ? 4 : total(3) <= 227 * 1024 ? 3 : 2;
  static constexpr int BYTES = total(STAGES);
  static constexpr int NBUF = 2 * 2 * ABT_N + DK + (DKV ? DV : 0) <= 512 ? 2 : 1;   // score buffers in TMEM
  static_assert(BYTES <= 227 * 1024, "shared memory budget");
  static_assert(NBUF * 2 * ABT_N + DK + (DKV ? DV : 0) <= 512, "tensor memory budget");
};

struct AbtMaps {
  CUtensorMap x1, x2, y1, y2;
};

template <int DK, int DV, bool DKV>
__global__ void __launch_bounds__(ABT_THREADS, 1)
attn_bwd_tc_kernel(const __grid_constant__ AbtMaps tm, const AttnBwdParams p, int tiles, int num_seqs) {
  using L = AbtLayout<DK, DV, DKV>;
  constexpr int ST = L::STAGES, NBUF = L::NBUF;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t x1 = (raw + 1023) & ~1023u;
  uint8_t* base = smem_raw + (x1 - raw);
  const uint32_t x2 = x1 + L::X1, y1 = x2 + L::X2, y2 = y1 + ST * L::Y1, ps = y2 + ST * L::Y2;   // ps: dS tiles, then P tiles
  uint8_t* p_ptr = base + (ps - x1);
  uint8_t* small = p_ptr + L::NP * L::PT;
  uint64_t* bars = reinterpret_cast<uint64_t*>(small);
  float (*s_lse)[ABT_N] = reinterpret_cast<float (*)[ABT_N]>(small + 256);
  float (*s_delta)[ABT_N] = s_lse + ST;
  float* s_row = reinterpret_cast<float*>(small + 256);   // [2][128]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(small + 240);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(small + 248);
  auto bar = [&](int i) { return ptx::smem_u32(&bars[i]); };
  const uint32_t xfull = bar(0);
  auto yfull = [&](int s) { return bar(1 + s); };
  auto yready = [&](int s) { return bar(5 + s); };
  auto yempty = [&](int s) { return bar(9 + s); };
  auto sfull = [&](int b) { return bar(13 + b); };
  auto sfree = [&](int b) { return bar(15 + b); };
  auto pready = [&](int b) { return bar(17 + b); };
  auto pfree = [&](int b) { return bar(19 + b); };
  const uint32_t done = bar(21);

  // ---- which tile: the longest walks come first (dkv: first keys; dq: last queries)
  const int per_tile = (DKV ? p.hkv : p.hq) * num_seqs;
  const int order = (int)(blockIdx.x / per_tile), who = (int)(blockIdx.x % per_tile);
  const int seq = who / (DKV ? p.hkv : p.hq), head = who % (DKV ? p.hkv : p.hq);
  const int tile = DKV ? order : tiles - 1 - order;
  pdl_trigger();
  pdl_wait();
  int q0, q_len, k0, kv_len;
  if (!ab_bounds(p, seq, q0, q_len, k0, kv_len)) return;
  const int own_len = DKV ? kv_len : q_len;
  if (tile == tiles - 1 && own_len > tiles * ABT_M && threadIdx.x == 0 && head == 0) report_status(B200_STATUS_BAD_INDEX, seq);
  const int m0 = tile * ABT_M;                       // first owned row in the sequence
  if (m0 >= own_len) return;
  const int rows = min(ABT_M, own_len - m0);
  const int group = p.hq / p.hkv, shift = kv_len - q_len;
  const int kvh = DKV ? head : head / group;
  // streamed tiles: dq: keys 0 .. last visible; dkv: for every query head, queries from the first that sees m0
  const int first = DKV ? max(0, m0 - shift) / ABT_N : 0;
  const int end = DKV ? q_len : min(kv_len, m0 + rows + shift);
  const int nt = max(0, (end + ABT_N - 1) / ABT_N - first);
  const int walk1 = DKV || p.have_lse ? 0 : nt;      // dq: steps of the first walk
  const int steps = walk1 + (DKV ? group * nt : nt);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    ptx::mbar_init(xfull, 1);
    for (int s = 0; s < 4; ++s) {
      ptx::mbar_init(yfull(s), 1);
      ptx::mbar_init(yready(s), 1);
      ptx::mbar_init(yempty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(sfull(b), 1);
      ptx::mbar_init(sfree(b), 8);
      ptx::mbar_init(pready(b), 8);
      ptx::mbar_init(pfree(b), 1);
    }
    ptx::mbar_init(done, 1);
    ptx::fence_barrier_init();
    ptx::prefetch_tensormap(&tm.x1);
    ptx::prefetch_tensormap(&tm.x2);
    ptx::prefetch_tensormap(&tm.y1);
    ptx::prefetch_tensormap(&tm.y2);
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tm_s = tmem, tm_dp = tmem + NBUF * ABT_N, tm_a2 = tmem + 2 * NBUF * ABT_N, tm_a1 = tm_a2 + DK;
  // tm_a2: the gradient through dS (dK / dQ, DK columns), tm_a1: dV

  // step -> streamed head, first streamed row in the sequence
  auto step_row = [&](int i) { return (first + (i < walk1 ? i : (i - walk1) % max(nt, 1))) * ABT_N; };
  auto step_head = [&](int i) { return DKV ? kvh * group + i / max(nt, 1) : kvh; };
  const int own_tok = (DKV ? k0 : q0) + m0, other0 = DKV ? q0 : k0, other_len = DKV ? q_len : kv_len;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (keys that no query sees: nothing to load)
    if (steps > 0 && ptx::elect_one()) {
      ptx::mbar_expect_tx(xfull, L::X1 + L::X2);
      for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int h = 0; h < L::X1H; ++h)
          ptx::tma_load_3d(x1 + h * (ABT_M * 128) + r * (64 * 128), &tm.x1, xfull, h * 64, head, own_tok + r * 64, ptx::kEvictNormal);
#pragma unroll
        for (int h = 0; h < L::X2H; ++h)
          ptx::tma_load_3d(x2 + h * (ABT_M * 128) + r * (64 * 128), &tm.x2, xfull, h * 64, head, own_tok + r * 64, ptx::kEvictNormal);
      }
      for (int i = 0; i < steps; ++i) {
        const int s = i % ST;
        if (!ptx::mbar_wait(yempty(s), ((i / ST) & 1) ^ 1, abort_flag, 800 + s)) break;
        const bool both = i >= walk1;
        ptx::mbar_expect_tx(yfull(s), L::Y1 + (both ? L::Y2 : 0));
        const int tok = other0 + step_row(i), h0 = step_head(i);
#pragma unroll
        for (int h = 0; h < L::X1H; ++h)
          ptx::tma_load_3d(y1 + s * L::Y1 + h * (ABT_N * 128), &tm.y1, yfull(s), h * 64, h0, tok, ptx::kEvictLast);
        if (both) {
#pragma unroll
          for (int h = 0; h < L::X2H; ++h)
            ptx::tma_load_3d(y2 + s * L::Y2 + h * (ABT_N * 128), &tm.y2, yfull(s), h * 64, h0, tok, ptx::kEvictLast);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ UMMA issuer
    if (ptx::elect_one()) {
      const uint32_t idesc_s = umma_idesc_bf16_b(ABT_N, false);
      const uint32_t idesc_k = umma_idesc_bf16_b(DK, true), idesc_v = umma_idesc_bf16_b(DV, true);
      const uint64_t hi = ptx::umma_desc_k_sw128(0) & 0xFFFFFFFF00000000ull;
      auto kdesc = [&](uint32_t a) { return hi | (uint64_t)(((a & 0x3FFFFu) >> 4) | (1u << 16)); };
      auto scores = [&](int i) {
        const int s = i % ST, b = i % NBUF;
        if (!ptx::mbar_wait(yready(s), (i / ST) & 1, abort_flag, 810 + s)) return false;
        if (!ptx::mbar_wait(sfree(b), ((i / NBUF) & 1) ^ 1, abort_flag, 820 + b)) return false;
        ptx::tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < DK / 16; ++kk)
          ptx::umma_bf16(tm_s + b * ABT_N, kdesc(x1 + (kk >> 2) * (ABT_M * 128) + (kk & 3) * 32),
                         kdesc(y1 + s * L::Y1 + (kk >> 2) * (ABT_N * 128) + (kk & 3) * 32), idesc_s, kk != 0 ? 1u : 0u);
        if (i >= walk1) {
#pragma unroll
          for (int kk = 0; kk < DV / 16; ++kk)
            ptx::umma_bf16(tm_dp + b * ABT_N, kdesc(x2 + (kk >> 2) * (ABT_M * 128) + (kk & 3) * 32),
                           kdesc(y2 + s * L::Y2 + (kk >> 2) * (ABT_N * 128) + (kk & 3) * 32), idesc_s, kk != 0 ? 1u : 0u);
        } else {
          ptx::umma_commit(yempty(s));             // the first walk needs the tile for nothing else
        }
        ptx::umma_commit(sfull(b));
        return true;
      };
      bool ok = steps > 0 && ptx::mbar_wait(xfull, 0, abort_flag, 830);
      int issued = 0;
      for (; ok && issued < walk1; ++issued) ok = scores(issued);
      const int u0 = walk1;
      if (ok && issued < steps) {
        ok = scores(issued);
        ++issued;
      }
      for (int i = u0; ok && i < steps; ++i) {
        if (issued < steps) {
          if (!scores(issued)) break;
          ++issued;
        }
        const int s = i % ST, u = i - u0, b = u & 1;
        if (!ptx::mbar_wait(pready(b), (u >> 1) & 1, abort_flag, 840 + b)) break;
        ptx::tc_fence_after();
        if constexpr (DKV) {
#pragma unroll
          for (int kk = 0; kk < ABT_N / 16; ++kk)
            ptx::umma_bf16(tm_a1, kdesc(ps + (2 + b) * L::PT + kk * 32), umma_desc_mn_sw128(y2 + s * L::Y2 + kk * 16 * 128, ABT_N * 128),
                           idesc_v, (u | kk) != 0 ? 1u : 0u);
        }
#pragma unroll
        for (int kk = 0; kk < ABT_N / 16; ++kk)
          ptx::umma_bf16(tm_a2, kdesc(ps + b * L::PT + kk * 32), umma_desc_mn_sw128(y1 + s * L::Y1 + kk * 16 * 128, ABT_N * 128),
                         idesc_k, (u | kk) != 0 ? 1u : 0u);
        ptx::umma_commit(yempty(s));
        ptx::umma_commit(pfree(b));
        if (i == steps - 1) ptx::umma_commit(done);
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ keeper: streamed tiles become usable here
    for (int i = 0; i < steps; ++i) {
      const int s = i % ST, row = step_row(i), n = min(ABT_N, other_len - row);
      float l[2] = {INFINITY, INFINITY}, dl[2] = {0.f, 0.f};
      if constexpr (DKV) {
        const long long at = (long long)step_head(i) * p.total_q + q0 + row;
#pragma unroll
        for (int k = 0; k < 2; ++k)
          if (lane + 32 * k < n) {
            l[k] = p.lse[at + lane + 32 * k];
            dl[k] = p.delta[at + lane + 32 * k];
          }
      }
      if (!ptx::mbar_wait_warp(yfull(s), (i / ST) & 1, abort_flag, 850 + s)) break;
      if constexpr (DKV) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          s_lse[s][lane + 32 * k] = l[k];
          s_delta[s][lane + 32 * k] = dl[k];
        }
      }
      if (n < ABT_N) {
        // rows past the sequence's end are a neighbour's: their weights are zeros, and 0 times anything must stay 0
        for (int r = n; r < ABT_N; ++r) {
#pragma unroll
          for (int h = 0; h < L::X1H; ++h)
            reinterpret_cast<uint32_t*>(base + (y1 - x1) + s * L::Y1 + h * (ABT_N * 128) + r * 128)[lane] = 0u;
          if (i >= walk1) {
#pragma unroll
            for (int h = 0; h < L::X2H; ++h)
              reinterpret_cast<uint32_t*>(base + (y2 - x1) + s * L::Y2 + h * (ABT_N * 128) + r * 128)[lane] = 0u;
          }
        }
        ptx::fence_proxy_async_smem();
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(yready(s));
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ compute: thread = (owned row, half of the streamed rows)
    const int q4 = warp & 3, half = (warp - 4) >> 2, row = q4 * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(q4 * 32) << 16;
    const float scale2 = p.scale * kLog2e;
    const int own = m0 + row;                                    // in the sequence
    bool alive = true;
    float lse = 0.f, delta = 0.f;                                // of this row (dq)
    if constexpr (!DKV) {
      // delta = sum_d out * dout: 64 columns per thread
      const bool live = row < rows;
      float acc = 0.f;
      const long long at = ((long long)(q0 + min(own, q_len - 1)) * p.hq + head) * DV + half * 64;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint4 a = *reinterpret_cast<const uint4*>(p.out + at + c * 8), b = *reinterpret_cast<const uint4*>(p.dout + at + c * 8);
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float a0, a1, b0, b1;
          unpack_bf2(av[k], a0, a1);
          unpack_bf2(bv[k], b0, b1);
          acc = fmaf(a0, b0, acc);
          acc = fmaf(a1, b1, acc);
        }
      }
      s_row[half * ABT_M + row] = acc;
      ptx::named_barrier_sync(1, 256);
      delta = s_row[row] + s_row[ABT_M + row];
      if (p.have_lse) lse = live ? p.lse[(long long)head * p.total_q + q0 + own] : INFINITY;
      // first walk: running maximum and sum over this thread's half of every key tile, in units of log2
      float m = -INFINITY, l = 0.f;
      const int pos = own + shift;
      for (int i = 0; i < walk1; ++i) {
        const int b = i % NBUF;
        if (!ptx::mbar_wait_warp(sfull(b), (i / NBUF) & 1, abort_flag, 860 + b)) {
          alive = false;
          break;
        }
        ptx::tc_fence_after();
        uint32_t r[32];
        tmem_ld32(tm_s + b * ABT_N + lane_addr + half * 32, r);
        ptx::tmem_ld_wait();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(sfree(b));
        const int key0 = step_row(i) + half * 32;
        float v[32], mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]) * scale2;
        if (key0 + 31 > pos) {
#pragma unroll
          for (int k = 0; k < 32; ++k)
            if (key0 + k > pos) v[k] = -INFINITY;
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) mx[k & 3] = fmaxf(mx[k & 3], v[k]);
        const float mn = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), m);
        if (mn > -INFINITY) {
          float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int k = 0; k < 32; ++k) s4[k & 3] += fast_exp2(v[k] - mn);
          l = l * fast_exp2(m - mn) + ((s4[0] + s4[1]) + (s4[2] + s4[3]));
          m = mn;
        }
      }
      ptx::named_barrier_sync(1, 256);
      if (*abort_flag) alive = false;
      // join the halves: (m, l) of the partner through shared memory, the sums in the order half 0, half 1
      if (!p.have_lse) {
        s_row[half * ABT_M + row] = m;
        ptx::named_barrier_sync(1, 256);
        const float mj = fmaxf(s_row[row], s_row[ABT_M + row]);
        ptx::named_barrier_sync(1, 256);
        s_row[half * ABT_M + row] = m > -INFINITY ? l * fast_exp2(m - mj) : 0.f;
        ptx::named_barrier_sync(1, 256);
        const float sum = s_row[row] + s_row[ABT_M + row];
        lse = sum > 0.f ? mj + log2f(sum) : INFINITY;              // no key: every weight is zero
      }
      if (live && half == 0 && alive) {
        if (!p.have_lse) p.lse[(long long)head * p.total_q + q0 + own] = lse;
        p.delta[(long long)head * p.total_q + q0 + own] = delta;
      }
    }
    for (int i = walk1; i < steps && alive; ++i) {
      const int b = i % NBUF, s = i % ST, u = i - walk1, pb = u & 1;
      if (!ptx::mbar_wait_warp(sfull(b), (i / NBUF) & 1, abort_flag, 860 + b)) break;
      if (DKV && !ptx::mbar_wait_warp(yready(s), (i / ST) & 1, abort_flag, 865 + s)) break;   // lse and delta are there
      ptx::tc_fence_after();
      uint32_t rs[32], rd[32];
      tmem_ld32(tm_s + b * ABT_N + lane_addr + half * 32, rs);
      tmem_ld32(tm_dp + b * ABT_N + lane_addr + half * 32, rd);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(sfree(b));
      const int c0 = step_row(i) + half * 32;                    // first streamed row of this thread
      // dq: key c0 + k is seen up to own + shift; dkv: queries from own - shift on see this key, up to q_len
      const bool masked = DKV ? c0 < own - shift || c0 + 32 > q_len : c0 + 31 > own + shift;
      uint32_t pk[16], dk[16];
#pragma unroll
      for (int k = 0; k < 32; k += 4) {
        float l4[4], d4[4], pr[4], ds[4];
        if constexpr (DKV) {
          const float4 lv = *reinterpret_cast<const float4*>(&s_lse[s][half * 32 + k]);
          const float4 dv = *reinterpret_cast<const float4*>(&s_delta[s][half * 32 + k]);
          l4[0] = lv.x, l4[1] = lv.y, l4[2] = lv.z, l4[3] = lv.w;
          d4[0] = dv.x, d4[1] = dv.y, d4[2] = dv.z, d4[3] = dv.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) l4[e] = lse, d4[e] = delta;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) pr[e] = fast_exp2(fmaf(__uint_as_float(rs[k + e]), scale2, -l4[e]));
        if (masked) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = c0 + k + e;
            if (DKV ? (c < own - shift || c >= q_len) : c > own + shift) pr[e] = 0.f;
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) ds[e] = pr[e] * (__uint_as_float(rd[k + e]) - d4[e]) * p.scale;
        dk[k / 2] = pack_bf2(ds[0], ds[1]);
        dk[k / 2 + 1] = pack_bf2(ds[2], ds[3]);
        if constexpr (DKV) {
          pk[k / 2] = pack_bf2(pr[0], pr[1]);
          pk[k / 2 + 1] = pack_bf2(pr[2], pr[3]);
        }
      }
      if (!ptx::mbar_wait_warp(pfree(pb), ((u >> 1) & 1) ^ 1, abort_flag, 870 + pb)) break;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(p_ptr + pb * L::PT + sw128(row, half * 4 + c)) = make_uint4(dk[c * 4], dk[c * 4 + 1], dk[c * 4 + 2], dk[c * 4 + 3]);
      if constexpr (DKV) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(p_ptr + (2 + pb) * L::PT + sw128(row, half * 4 + c)) = make_uint4(pk[c * 4], pk[c * 4 + 1], pk[c * 4 + 2], pk[c * 4 + 3]);
      }
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(pready(pb));
    }
    // ---- the gradients of this row
    const bool some = steps > walk1;
    if (alive && some) alive = ptx::mbar_wait_warp(done, 0, abort_flag, 880);
    if (alive && !*abort_flag) {
      ptx::tc_fence_after();
      auto store = [&](uint32_t acc, __nv_bfloat16* dst, int cols) {   // 32 columns at a time, the halves taking turns
        for (int c = half * 32; c < cols; c += 64) {
          uint32_t r[32];
          if (some) {
            tmem_ld32(acc + lane_addr + c, r);
            ptx::tmem_ld_wait();
          } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) r[k] = 0u;      // keys that no query sees
          }
          if (row < rows) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              auto pair = [&](int e) { return pack_bf2(__uint_as_float(r[k * 8 + e]), __uint_as_float(r[k * 8 + e + 1])); };
              *reinterpret_cast<uint4*>(dst + c + k * 8) = make_uint4(pair(0), pair(2), pair(4), pair(6));
            }
          }
        }
      };
      const long long at = (long long)((DKV ? k0 : q0) + own) * (DKV ? p.hkv : p.hq) + head;
      store(tm_a2, (DKV ? p.dk : p.dq) + at * DK, DK);
      if constexpr (DKV) store(tm_a1, p.dv + at * DV, DV);
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (*abort_flag) {      // in-flight copies land before the CTA leaves
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

// bf16 [tokens, heads, d] contiguous; box = 64 columns of one head of 64 tokens, 128-byte swizzle.
inline int abt_map(CUtensorMap* m, const void* base, long long tokens, int heads, int d) {
  EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return B200_ERR_DRIVER;
  cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)tokens};
  cuuint64_t strides[2] = {(cuuint64_t)d * 2, (cuuint64_t)heads * d * 2};
  cuuint32_t box[3] = {64, 1, 64}, estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200_OK : B200_ERR_DRIVER;
}

template <int DK, int DV, bool DKV>
inline int attn_bwd_tc_one(const AbtMaps& tm, const AttnBwdParams& p, int num_seqs, int max_len, cudaStream_t st) {
  using L = AbtLayout<DK, DV, DKV>;
  static PerDeviceFlags attr;
  if (int rc = set_max_dyn_smem_once(attr, attn_bwd_tc_kernel<DK, DV, DKV>, L::BYTES)) return rc;
  const int tiles = (max_len + ABT_M - 1) / ABT_M;
  const long long grid = (long long)tiles * num_seqs * (DKV ? p.hkv : p.hq);
  if (grid > 0x7fffffffLL) return B200_ERR_SHAPE;
  launch_k(attn_bwd_tc_kernel<DK, DV, DKV>, dim3((unsigned)grid), dim3(ABT_THREADS), (size_t)L::BYTES, st, tm, p, tiles, num_seqs);
  return launch_status();
}

template <int DK, int DV>
inline int attn_bwd_tc_launch(const AttnBwdParams& p, int num_seqs, int max_seqlen_q, int max_seqlen_k, cudaStream_t st) {
  CUtensorMap q, k, v, dout;
  int rc = abt_map(&q, p.q, p.total_q, p.hq, DK);
  if (!rc) rc = abt_map(&k, p.k, p.total_k, p.hkv, DK);
  if (!rc) rc = abt_map(&v, p.v, p.total_k, p.hkv, DV);
  if (!rc) rc = abt_map(&dout, p.dout, p.total_q, p.hq, DV);
  if (!rc) rc = attn_bwd_tc_one<DK, DV, false>(AbtMaps{q, dout, k, v}, p, num_seqs, max_seqlen_q, st);
  if (!rc) rc = attn_bwd_tc_one<DK, DV, true>(AbtMaps{k, v, q, dout}, p, num_seqs, max_seqlen_k, st);
  return rc;
}

}  // namespace b200

namespace b200 {
inline int varlen_attn_backward_impl(const void* q, const void* k, const void* v, const void* out, const void* dout,
                                         const void* cu_seqlens_q, const void* cu_seqlens_k, void* dq, void* dk,
                                         void* dv, void* lse_scratch_f32, void* delta_scratch_f32, int num_seqs,
                                         int max_seqlen_q, int max_seqlen_k, long long total_q, long long total_k,
                                         int num_q_heads, int num_kv_heads, int dk_dim, int dv_dim,
                                         float softmax_scale, int have_lse, void* stream) {
  if (!q || !k || !v || !out || !dout || !cu_seqlens_q || !cu_seqlens_k || !dq || !dk || !dv || !lse_scratch_f32 ||
      !delta_scratch_f32 || num_seqs < 0 || max_seqlen_q < 0 || max_seqlen_k < 0 || total_q < 0 || total_k < 0 ||
      num_q_heads <= 0 || num_kv_heads <= 0)
    return B200_ERR_ARG;
  if (num_q_heads % num_kv_heads != 0 || num_seqs > 65535 || num_q_heads > 65535) return B200_ERR_SHAPE;
  if (total_q > 0x7fffffffLL || total_k > 0x7fffffffLL) return B200_ERR_SHAPE;
  if (num_seqs == 0 || max_seqlen_q == 0 || max_seqlen_k == 0) return B200_OK;
  AttnBwdParams p{(const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v,
                  (const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dq, (__nv_bfloat16*)dk,
                  (__nv_bfloat16*)dv, (float*)lse_scratch_f32, (float*)delta_scratch_f32, (const int*)cu_seqlens_q,
                  (const int*)cu_seqlens_k, num_q_heads, num_kv_heads, total_q, total_k, softmax_scale};
  cudaStream_t st = (cudaStream_t)stream;
  static const int simt = env_int("B200_ATTN_BWD_SIMT", 0);     // development knob: the CUDA-core kernels
  if (simt) {     // (these make their own log-sum-exp, over the forward's)
    if (dk_dim == 64 && dv_dim == 64) return attn_bwd_launch<64, 64>(p, num_seqs, max_seqlen_q, max_seqlen_k, st);
    if (dk_dim == 128 && dv_dim == 128) return attn_bwd_launch<128, 128>(p, num_seqs, max_seqlen_q, max_seqlen_k, st);
    if (dk_dim == 192 && dv_dim == 128) return attn_bwd_launch<192, 128>(p, num_seqs, max_seqlen_q, max_seqlen_k, st);
    return B200_ERR_SHAPE;
  }
  p.have_lse = have_lse;
  if (dk_dim == 64 && dv_dim == 64) return have_lse ? B200_ERR_SHAPE : attn_bwd_mma_launch<64, 64>(p, num_seqs, max_seqlen_q, max_seqlen_k, st);
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dq) |
       reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 15)
    return B200_ERR_ARG;
  if (dk_dim == 128 && dv_dim == 128) return attn_bwd_tc_launch<128, 128>(p, num_seqs, max_seqlen_q, max_seqlen_k, st);
  if (dk_dim == 192 && dv_dim == 128) return attn_bwd_tc_launch<192, 128>(p, num_seqs, max_seqlen_q, max_seqlen_k, st);
  return B200_ERR_SHAPE;
}
}  // namespace b200

// dq, dk, dv of packed causal varlen attention (triton_invariant_attention.py:194-431).  All tensors bf16 and
// contiguous: q / dq [total_q, hq, dk_dim], k / dk [total_k, hkv, dk_dim], v / dv [total_k, hkv, dv_dim], out /
// dout [total_q, hq, dv_dim]; cu_seqlens_q / _k [num_seqs + 1] int32; lse / delta: fp32 scratch of total_q * hq values.
// (dk_dim, dv_dim) one of (64, 64), (128, 128), (192, 128).  Keys or queries of no sequence keep what dq / dk / dv
// held (pass zero-filled tensors).  Sequences longer than max_seqlen_q / max_seqlen_k are reported (status code 2).
extern "C" int b200_varlen_attn_backward(const void* q, const void* k, const void* v, const void* out, const void* dout,
                                         const void* cu_seqlens_q, const void* cu_seqlens_k, void* dq, void* dk,
                                         void* dv, void* lse_scratch_f32, void* delta_scratch_f32, int num_seqs,
                                         int max_seqlen_q, int max_seqlen_k, long long total_q, long long total_k,
                                         int num_q_heads, int num_kv_heads, int dk_dim, int dv_dim,
                                         float softmax_scale, void* stream) {
  return b200::varlen_attn_backward_impl(q, k, v, out, dout, cu_seqlens_q, cu_seqlens_k, dq, dk, dv, lse_scratch_f32, delta_scratch_f32,
                                         num_seqs, max_seqlen_q, max_seqlen_k, total_q, total_k, num_q_heads, num_kv_heads, dk_dim,
                                         dv_dim, softmax_scale, 0, stream);
}

// The same with lse_scratch_f32 as b200_paged_attn_fwd_lse left it ([num_q_heads, total_q]); it is overwritten where the
// development knob selects the CUDA-core kernels.  Head dims (128, 128) and (192, 128).
extern "C" int b200_varlen_attn_backward_lse(const void* q, const void* k, const void* v, const void* out, const void* dout,
                                         const void* cu_seqlens_q, const void* cu_seqlens_k, void* dq, void* dk,
                                         void* dv, void* lse_scratch_f32, void* delta_scratch_f32, int num_seqs,
                                         int max_seqlen_q, int max_seqlen_k, long long total_q, long long total_k,
                                         int num_q_heads, int num_kv_heads, int dk_dim, int dv_dim,
                                         float softmax_scale, void* stream) {
  return b200::varlen_attn_backward_impl(q, k, v, out, dout, cu_seqlens_q, cu_seqlens_k, dq, dk, dv, lse_scratch_f32, delta_scratch_f32,
                                         num_seqs, max_seqlen_q, max_seqlen_k, total_q, total_k, num_q_heads, num_kv_heads, dk_dim,
                                         dv_dim, softmax_scale, 1, stream);
}
