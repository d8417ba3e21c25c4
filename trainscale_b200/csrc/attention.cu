// Flash attention for sm_100a on tcgen05 / TMEM / TMA: causal or full, GQA, packed documents (cu_seqlens).
//
// Forward, per CTA (one 256-row query block of one head = two 128-row tiles that ping-pong):
//   warp 0        TMA loader: Q tiles once, then a 2-deep ring of 128-row K and V tiles (128-byte swizzle)
//   warp 1        MMA issuer (one thread): S_t = Q_t K^T into TMEM, later O_t += P_t V with P_t read from TMEM
//   warps 2..5    softmax for tile 0, warps 6..9 for tile 1: one thread per query row (its own TMEM lane), so row
//                 max / sum need no shuffles; P is written back over S as packed bf16, O is rescaled in TMEM
//                 only when the running max moved by more than 2^8 (exact: O and the row sum share the stale max).
//                 `SPLIT` (portions of prompts against a cache): P = high + low bf16 parts, both multiplied with V, which
//                 leaves 16 bits of every weight; the low part takes the other 64 columns of S, and with heads of 128 the
//                 tensor memory is full.  Against 64 bits, relative to the same in fp32 throughout (rows x keys, heads of 64 and
//                 128): error larger by 1e-6 of itself at 2 x 700, 2e-6 at 300 x 1300, 9e-6 at 512 x 3000; most of it is the order
//                 in which the tensor core adds up long rows, the rest the weights.  The result's rounding to bf16 is the error.
//                 An infinite value gives NaN (the low part may be zero or negative), as it does in every row that masks its key
// While one tile's rows are in softmax the tensor core works on the other tile.
// Backward is two kernels that recompute S and dP: one owns a K/V tile and accumulates dK, dV over the query
// tiles of its head group; one owns a Q tile and accumulates dQ over the K/V tiles.  No atomics, deterministic.
//
// Replaces data_pipeline/trainer/kernels/flash_attention.py:147-560 (Triton forward, dq and dk/dv kernels).
#include <type_traits>
#include "common.cuh"
#include "host_common.h"

namespace ts {

struct AttnParams {
  // strides are in elements; q/k/v/o/do/dq/dk/dv rows are tokens, heads are laid out along the row
  int q_col0, k_col0, v_col0;   // column of head 0 inside the q / k / v tensor maps
  int Hq, Hkv, group;           // group = Hq / Hkv
  int B, S;                     // uniform batch (ignored when cu_seqlens != nullptr)
  const int* cu_seqlens;        // [B + 1] or nullptr
  const int* k_starts;          // keys apart from the queries: first key row of every sequence (nullptr: the queries' rows)
  const int* k_lens;            // and its keys; the queries are its last ones
  int causal;
  float scale_log2;             // softmax scale * log2(e)
  __nv_bfloat16* o;             // [rows][o_stride], head h at column h*D
  int o_stride;
  float* lse;                   // [Hq][total_rows]
  long long total_rows;
  // backward
  const __nv_bfloat16* dout;    // [rows][o_stride]
  const float* delta;           // [Hq][total_rows] rowsum(dO * O)
  __nv_bfloat16* dq;            // written at column q_col0 + h*D of rows with stride dqkv_stride
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  int dqkv_stride;
  float scale;                  // softmax scale (natural units)
  int window;                   // > 0: key j is visible to query i only if j > i - window (sliding window)
  float cap_inv, cap_log2;      // logit soft-cap c: s' = c * tanh(s * scale / c); cap_inv = scale / c, cap_log2 = c * log2(e)
};

__device__ __forceinline__ float fast_tanh(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void seq_bounds(const AttnParams& p, int b, int& start, int& len) {
  if (p.cu_seqlens) {
    start = p.cu_seqlens[b];
    len = p.cu_seqlens[b + 1] - start;
  } else {
    start = b * p.S;
    len = p.S;
  }
}

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
template <int D>
struct FwdSmem {
  static constexpr int TILE = 128 * D * 2;
  static constexpr int KV_STAGES = 2;
  static constexpr int Q_OFF = 0;
  static constexpr int K_OFF = 2 * TILE;
  static constexpr int V_OFF = K_OFF + KV_STAGES * TILE;
  static constexpr int BAR_OFF = V_OFF + KV_STAGES * TILE;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

constexpr int FWD_THREADS = 320;

template <int D, bool EXT, bool SPLIT>   // EXT: sliding window / logit soft-cap code paths compiled in
__global__ void __launch_bounds__(FWD_THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, AttnParams p) {
  using SM = FwdSmem<D>;
  constexpr int DCH = D / 64;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t O_COL0 = 256;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::BAR_OFF);
  uint64_t* q_full = bars;          // [2]
  uint64_t* k_full = bars + 2;      // [2]
  uint64_t* k_empty = bars + 4;     // [2]
  uint64_t* v_full = bars + 6;      // [2]
  uint64_t* v_empty = bars + 8;     // [2]
  uint64_t* s_full = bars + 10;     // [2]
  uint64_t* p_full = bars + 12;     // [2]
  uint64_t* o_full = bars + 14;     // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // grid: x = head + heads * batch (fastest), y = tile: the whole grid is dispatched longest-tile-first
  const int h = blockIdx.x % p.Hq, b = blockIdx.x / p.Hq;
  const int hk = h / p.group;
  int q_start, Lq, k_start, Lk;
  seq_bounds(p, b, q_start, Lq);
  k_start = SPLIT ? p.k_starts[b] : q_start;
  Lk = SPLIT ? p.k_lens[b] : Lq;
  const int n_qblocks = (Lq + 255) / 256;
  if ((int)blockIdx.y >= n_qblocks) return;
  const int qb = n_qblocks - 1 - blockIdx.y;   // heaviest (latest) causal blocks first
  const int off = Lk - Lq;
  int r0[2], nkv[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    r0[t] = qb * 256 + t * 128;
    if (r0[t] >= Lq) {
      nkv[t] = 0;
    } else {
      const int kv_end = p.causal ? min(Lk, r0[t] + 128 + off) : Lk;
      nkv[t] = (kv_end + 127) / 128;
    }
  }
  // sliding window: key blocks entirely left of the first row's window are never loaded
  const int kb_lo = (EXT && p.window > 0) ? max(0, qb * 256 + off - p.window + 1) / 128 : 0;
#pragma unroll
  for (int t = 0; t < 2; ++t) nkv[t] = max(0, nkv[t] - kb_lo);
  const int n = max(nkv[0], nkv[1]);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    for (int i = 0; i < 16; ++i) mbar_init(&bars[i], (i == 12 || i == 13) ? 4 : 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  bool alive = true;

  if (warp == 0) {
    if (elect_one_sync()) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (nkv[t] == 0) continue;
        mbar_expect_tx(&q_full[t], SM::TILE);
#pragma unroll
        for (int j = 0; j < DCH; ++j)
          tma_load_2d(smem + SM::Q_OFF + t * SM::TILE + j * 16384, &tmQ, &q_full[t], p.q_col0 + h * D + j * 64,
                      q_start + r0[t]);
      }
      for (int i = 0; i < n && alive; ++i) {
        const int s = i & 1;
        const uint32_t ph = (i >> 1) & 1u;
        if (!mbar_wait(&k_empty[s], ph ^ 1u, alive, 400)) break;
        mbar_expect_tx(&k_full[s], SM::TILE);
#pragma unroll
        for (int j = 0; j < DCH; ++j)
          tma_load_2d(smem + SM::K_OFF + s * SM::TILE + j * 16384, &tmK, &k_full[s], p.k_col0 + hk * D + j * 64,
                      k_start + (kb_lo + i) * 128);
        if (!mbar_wait(&v_empty[s], ph ^ 1u, alive, 401)) break;
        mbar_expect_tx(&v_full[s], SM::TILE);
#pragma unroll
        for (int j = 0; j < DCH; ++j)
          tma_load_2d(smem + SM::V_OFF + s * SM::TILE + j * 16384, &tmV, &v_full[s], p.v_col0 + hk * D + j * 64,
                      k_start + (kb_lo + i) * 128);
      }
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      const uint32_t idesc_s = make_idesc(128, 128, 1, 1, 0, 0);
      const uint32_t idesc_o = make_idesc(128, D, 1, 1, 0, 1);
      auto issue_s = [&](int t, int stage) {
        const uint32_t qa = smem_u32(smem + SM::Q_OFF + t * SM::TILE);
        const uint32_t ka = smem_u32(smem + SM::K_OFF + stage * SM::TILE);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t o = (k >> 2) * 16384 + (k & 3) * 32;
          umma_f16_ss(tmem_base + t * 128, make_smem_desc_sw128(qa + o, 16, 1024),
                      make_smem_desc_sw128(ka + o, 16, 1024), idesc_s, k != 0);
        }
        umma_commit(&s_full[t]);
      };
      for (int t = 0; t < 2; ++t)
        if (nkv[t] > 0) mbar_wait(&q_full[t], 0, alive, 500);
      if (n > 0 && mbar_wait(&k_full[0], 0, alive, 501)) {
        tc_fence_after_sync();
        for (int t = 0; t < 2; ++t)
          if (nkv[t] > 0) issue_s(t, 0);
        umma_commit(&k_empty[0]);
      }
      for (int i = 0; i < n && alive; ++i) {
        const int s = i & 1;
        if (!mbar_wait(&v_full[s], (i >> 1) & 1u, alive, 502)) break;
        bool k_waited = false;
        for (int t = 0; t < 2 && alive; ++t) {
          if (i < nkv[t]) {
            if (!mbar_wait(&p_full[t], i & 1u, alive, 503)) break;
            tc_fence_after_sync();
            const uint32_t va = smem_u32(smem + SM::V_OFF + s * SM::TILE);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_f16_ts(tmem_base + O_COL0 + t * D, tmem_base + t * 128 + kk * 8,
                          make_smem_desc_sw128(va + kk * 2048, 16384, 1024), idesc_o, (i | kk) != 0);
            if (SPLIT) {
#pragma unroll
              for (int kk = 0; kk < 8; ++kk)
                umma_f16_ts(tmem_base + O_COL0 + t * D, tmem_base + t * 128 + 64 + kk * 8,
                            make_smem_desc_sw128(va + kk * 2048, 16384, 1024), idesc_o, 1u);
            }
            if (i == nkv[t] - 1) umma_commit(&o_full[t]);
          }
          if (i + 1 < nkv[t]) {
            if (!k_waited) {
              if (!mbar_wait(&k_full[(i + 1) & 1], ((i + 1) >> 1) & 1u, alive, 504)) break;
              tc_fence_after_sync();
              k_waited = true;
            }
            issue_s(t, (i + 1) & 1);
          }
        }
        if (!alive) break;
        if (i + 1 < n) umma_commit(&k_empty[(i + 1) & 1]);
        umma_commit(&v_empty[s]);
      }
    }
  } else {
    // ------------------------------ softmax / correction / epilogue ------------------------------
    const int t = (warp - 2) >> 2;
    const int q4 = warp & 3;
    const int r = q4 * 32 + lane;
    const int row = r0[t] + r;                  // row inside the sequence
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q4 * 32) << 16);
    const uint32_t t_s = t_lane + t * 128;
    const uint32_t t_o = t_lane + O_COL0 + t * D;
    float m_used = -INFINITY, l = 0.f;
    const int nt = nkv[t];
    for (int i = 0; i < nt && alive; ++i) {
      if (!mbar_wait(&s_full[t], i & 1u, alive, 600)) break;
      tc_fence_after_sync();
      const int c0 = (kb_lo + i) * 128;
      const bool need_mask = (p.causal && (c0 + 127 > r0[t] + off)) || (c0 + 128 > Lk) ||
                             (EXT && p.window > 0 && c0 <= r0[t] + 127 + off - p.window);
      const int limit = p.causal ? min(Lk - 1, row + off) : Lk - 1;   // last visible column
      const int lo = (EXT && p.window > 0) ? row + off - p.window + 1 : 0;  // first visible column
      // the thread's whole row of S (128 columns) comes into registers once
      uint32_t v[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_s + c * 32, v + c * 32);
      tc_wait_ld();
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
      float sc = p.scale_log2;
      if (EXT && p.cap_log2 > 0.f) {   // soft-capped logits, already in log2 units
#pragma unroll
        for (int j = 0; j < 128; ++j) v[j] = __float_as_uint(p.cap_log2 * fast_tanh(__uint_as_float(v[j]) * p.cap_inv));
        sc = 1.f;
      }
      if (need_mask) {
#pragma unroll
        for (int j = 0; j < 128; ++j)
          if (c0 + j > limit || c0 + j < lo) v[j] = 0xff800000u;   // -inf: drops out of the max, exp2 gives 0
      }
#pragma unroll
      for (int j = 0; j < 128; j += 4) {
        mx0 = fmaxf(mx0, __uint_as_float(v[j]));
        mx1 = fmaxf(mx1, __uint_as_float(v[j + 1]));
        mx2 = fmaxf(mx2, __uint_as_float(v[j + 2]));
        mx3 = fmaxf(mx3, __uint_as_float(v[j + 3]));
      }
      const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
      const float m_new = fmaxf(m_used, mx * sc);
      const bool grow = (m_new - m_used > 8.0f);   // also true on the first block (m_used = -inf)
      if (__any_sync(0xffffffffu, grow)) {
        const float alpha = (m_used == -INFINITY) ? 0.f : fast_ex2(m_used - m_new);
        m_used = m_new;
        l *= alpha;
        if (i > 0) {
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(t_o + c * 16, o);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
            tmem_st_32x32b_x16(t_o + c * 16, o);
          }
        }
      }
      const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;
      // P = exp2(S*scale - m), packed bf16 written over the first 64 columns of S
      float l0 = 0.f, l1 = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16], low[16];
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float p0 = fast_ex2(fmaf(__uint_as_float(v[c * 32 + j]), sc, -m_sub));
          const float p1 = fast_ex2(fmaf(__uint_as_float(v[c * 32 + j + 1]), sc, -m_sub));
          l0 += p0;
          l1 += p1;
          pk[j >> 1] = pack_bf16x2(p0, p1);
          if (SPLIT) {
            const float2 high = unpack_bf16x2(pk[j >> 1]);
            low[j >> 1] = pack_bf16x2(p0 - high.x, p1 - high.y);
          }
        }
        tmem_st_32x32b_x16(t_s + c * 16, pk);
        if (SPLIT) tmem_st_32x32b_x16(t_s + 64 + c * 16, low);
      }
      l += l0 + l1;
      tc_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[t]);
    }
    if (nt > 0 && alive && mbar_wait(&o_full[t], 0, alive, 601)) {
      tc_fence_after_sync();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const bool valid = row < Lq;
      __nv_bfloat16* dst = p.o + static_cast<size_t>(q_start + row) * p.o_stride + h * D;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(t_o + c * 32, v);
        tc_wait_ld();
        if (valid) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 o4;
            o4.x = pack_bf16x2(__uint_as_float(v[8 * j]) * inv, __uint_as_float(v[8 * j + 1]) * inv);
            o4.y = pack_bf16x2(__uint_as_float(v[8 * j + 2]) * inv, __uint_as_float(v[8 * j + 3]) * inv);
            o4.z = pack_bf16x2(__uint_as_float(v[8 * j + 4]) * inv, __uint_as_float(v[8 * j + 5]) * inv);
            o4.w = pack_bf16x2(__uint_as_float(v[8 * j + 6]) * inv, __uint_as_float(v[8 * j + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + j * 8) = o4;
          }
        }
      }
      if (valid && p.lse)
        p.lse[static_cast<size_t>(h) * p.total_rows + q_start + row] =
            l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// delta[h][row] = sum_d dO[row][h*D + d] * O[row][h*D + d]
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                  float* __restrict__ delta, long long total_rows, int Hq, int D, int o_stride) {
  const long long gw = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= total_rows * Hq) return;
  const long long row = gw / Hq;
  const int h = static_cast<int>(gw - row * Hq);
  const __nv_bfloat16* a = o + row * o_stride + h * D;
  const __nv_bfloat16* g = dout + row * o_stride + h * D;
  float s = 0.f;
  for (int d = lane * 2; d < D; d += 64) {
    const float2 x = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(a + d));
    const float2 y = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(g + d));
    s += x.x * y.x + x.y * y.y;
  }
  s = warp_sum(s);
  if (lane == 0) delta[static_cast<size_t>(h) * total_rows + row] = s;
}


// 32 accumulator columns of the thread's row, scaled, as bf16
__device__ __forceinline__ void store_rows_32(uint32_t taddr, float scale, __nv_bfloat16* dst, bool valid) {
  uint32_t v[32];
  tmem_ld_32x32b_x32(taddr, v);
  tc_wait_ld();
  if (!valid) return;
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    uint32_t o[4];
#pragma unroll
    for (int y = 0; y < 4; ++y)
      o[y] = pack_bf16x2(__uint_as_float(v[8 * x + 2 * y]) * scale, __uint_as_float(v[8 * x + 2 * y + 1]) * scale);
    *reinterpret_cast<uint4*>(dst + x * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// ------------------------------------------------------------------------------------------------
// backward.  Both kernels work on 128 x 128 blocks of S: an SS product of 128 x 128 takes from shared memory what the tensor core
// takes in the same time, one of 128 x 64 half as much again.  Bounds per block (D = 128): tensor core 2048 (dK, dV) and 1536 (dQ)
// cycles, exponentials 1024 cycles of the special-function units, so the products of one block run while the other half of its
// neighbour is in the compute warps:
//   dK, dV   dV += P dO and the next block's S   beside   dS = P (dP - delta)
//            dK += dS Q and the next block's dP  beside   the next block's P = exp2(S - lse)
//   dQ       dQ += dS K, the next dP, S after it beside   the next block's P and dS (two S buffers)
// P stays in fp32 registers between its two uses.  Two warpgroups share a row: each has 64 columns of S and dP and writes its
// bf16 P and dS over the first 32 columns of ITS half, so neither touches columns the other has still to read.
// 64-wide sub-tiles with P and dS in one phase / this, both kernels, ms (tensor rate over the seven products): S = 8192, 32 / 8
// heads of 128 1.86 / 1.41 (1360 TFLOP/s), S = 32768 30.5 / 24.9 (1236, power-capped), S = 8192 with heads of 64 2.01 / 1.54 (bound
// by the exponentials).
// ------------------------------------------------------------------------------------------------
constexpr int BWD_THREADS = 320;   // warp 0 TMA, warp 1 MMA, warps 2..5 and 6..9: two compute warpgroups (64 columns each)

// TMEM column of reduction step kk (16 values) of a bf16 operand that the two warpgroups wrote over their halves
__device__ __forceinline__ uint32_t half_col(int kk) { return (kk >> 2) * 64 + (kk & 3) * 8; }

// ------------------------------------------------------------------------------------------------
// kernel 1: dK / dV.  One CTA owns a 128-row K/V tile of one kv head and walks the 128-row query tiles of every query head in its
// group.  TMEM: S^T, dP^T, dV, dK of 128 columns each.  P^T and dS^T are fed to the MMA from TMEM.
// ------------------------------------------------------------------------------------------------
template <int D>
struct DkvSmem {
  static constexpr int TILE = 128 * D * 2;
  static constexpr int Q_STAGES = 3, DO_STAGES = 2;                   // Q(i + 1) is wanted while Q(i) waits for dK's product
  static constexpr int K_OFF = 0, V_OFF = TILE;                       // resident
  static constexpr int Q_OFF = 2 * TILE, DO_OFF = Q_OFF + Q_STAGES * TILE;   // streamed
  static constexpr int VEC_OFF = DO_OFF + DO_STAGES * TILE;           // two of: 128 x lse * log2e, 128 x delta
  static constexpr int BAR_OFF = VEC_OFF + 2 * 1024;
  static constexpr int TOTAL = BAR_OFF + 256;                         // (no room for slack: the block itself is aligned)
};

template <int D, bool EXT>   // EXT: sliding window / logit soft-cap code paths compiled in
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, AttnParams p) {
  using SM = DkvSmem<D>;
  constexpr int DCH = D / 64;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t DP_COL = 128, DV_COL = 256, DK_COL = 384;

  extern __shared__ __align__(1024) uint8_t smem_aligned[];
  uint8_t* smem = smem_aligned;
  if (smem_u32(smem) & 1023u) {            // the swizzled tiles need it
    if (threadIdx.x == 0) ts_report_error(ERR_BAD_ARGUMENT, 730);
    return;
  }
  float* vec = reinterpret_cast<float*>(smem + SM::VEC_OFF);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::BAR_OFF);
  uint64_t* kv_full = bars;
  uint64_t* s_full = bars + 1;
  uint64_t* p_full = bars + 2;
  uint64_t* dp_full = bars + 3;
  uint64_t* ds_full = bars + 4;
  uint64_t* acc_full = bars + 5;
  uint64_t* q_full = bars + 6;      // [3]
  uint64_t* q_empty = bars + 9;     // [3]
  uint64_t* do_full = bars + 12;    // [2]
  uint64_t* do_empty = bars + 14;   // [2]
  uint64_t* vec_full = bars + 16;   // [2]
  uint64_t* vec_empty = bars + 18;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // grid: x = kv head + kv heads * batch (fastest), y = kv tile; low tiles see the most queries and go first
  const int j = blockIdx.y, hk = blockIdx.x % p.Hkv, b = blockIdx.x / p.Hkv;
  int q_start, Lq;
  seq_bounds(p, b, q_start, Lq);
  const int k_start = q_start, Lk = Lq;
  if (j * 128 >= Lk) return;
  const int off = Lk - Lq;
  const int n_u = (Lq + 127) / 128;
  const int u_start = p.causal ? max(0, (j * 128 - off) / 128) : 0;
  // sliding window: the last query row that sees any key of this tile is (j*128 + 127) - off + window - 1
  const int u_end = (EXT && p.window > 0) ? min(n_u, (j * 128 + 127 - off + p.window - 1) / 128 + 1) : n_u;
  const int per_head = u_end - u_start;
  const int total = per_head * p.group;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
    for (int i = 0; i < 20; ++i) mbar_init(&bars[i], (i == 2 || i == 4 || i >= 18) ? 8 : 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  bool alive = true;

  if (warp == 0) {
    // the whole warp runs the producer loop: lane 0 issues the tiled loads, every lane brings four columns' lse * log2e and
    // delta into the stage's vector buffer (fetched one stage ahead)
    if (lane == 0) {
      mbar_expect_tx(kv_full, 2 * SM::TILE);
#pragma unroll
      for (int c = 0; c < DCH; ++c) {
        tma_load_2d(smem + SM::K_OFF + c * 16384, &tmK, kv_full, p.k_col0 + hk * D + c * 64, k_start + j * 128);
        tma_load_2d(smem + SM::V_OFF + c * 16384, &tmV, kv_full, p.v_col0 + hk * D + c * 64, k_start + j * 128);
      }
    }
    float nl[4], nd[4];
    auto fetch_vec = [&](int it) {
      const int g = it / per_head, u = u_start + it % per_head;
      const size_t row0 = static_cast<size_t>(hk * p.group + g) * p.total_rows + q_start;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int qrow = u * 128 + lane + c * 32;
        const bool in = it < total && qrow < Lq;
        nl[c] = in ? p.lse[row0 + qrow] * 1.4426950408889634f : 0.f;
        nd[c] = in ? p.delta[row0 + qrow] : 0.f;
      }
    };
    fetch_vec(0);
    for (int it = 0; it < total && alive; ++it) {
      const int s = it & 1, qs = it % SM::Q_STAGES;
      const uint32_t ph = ((it >> 1) & 1u) ^ 1u;
      const int u = u_start + it % per_head, h = hk * p.group + it / per_head;
      if (!mbar_wait(&q_empty[qs], ((it / SM::Q_STAGES) & 1u) ^ 1u, alive, 700)) break;
      if (lane == 0) {
        mbar_expect_tx(&q_full[qs], SM::TILE);
#pragma unroll
        for (int c = 0; c < DCH; ++c)
          tma_load_2d(smem + SM::Q_OFF + qs * SM::TILE + c * 16384, &tmQ, &q_full[qs], p.q_col0 + h * D + c * 64, q_start + u * 128);
      }
      if (!mbar_wait(&vec_empty[s], ph, alive, 702)) break;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        vec[s * 256 + lane + c * 32] = nl[c];
        vec[s * 256 + 128 + lane + c * 32] = nd[c];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&vec_full[s]);
      fetch_vec(it + 1);
      if (!mbar_wait(&do_empty[s], ph, alive, 701)) break;
      if (lane == 0) {
        mbar_expect_tx(&do_full[s], SM::TILE);
#pragma unroll
        for (int c = 0; c < DCH; ++c)
          tma_load_2d(smem + SM::DO_OFF + s * SM::TILE + c * 16384, &tmdO, &do_full[s], h * D + c * 64, q_start + u * 128);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      const uint32_t idesc_s = make_idesc(128, 128, 1, 1, 0, 0);
      const uint32_t idesc_acc = make_idesc(128, D, 1, 1, 0, 1);
      // a (resident) times b (streamed), both K-major
      auto issue_ss = [&](uint32_t d_col, uint32_t a, uint32_t bb) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t o = (k >> 2) * 16384 + (k & 3) * 32;
          umma_f16_ss(tmem_base + d_col, make_smem_desc_sw128(a + o, 16, 1024), make_smem_desc_sw128(bb + o, 16, 1024), idesc_s,
                      k != 0);
        }
      };
      auto issue_ts = [&](uint32_t d_col, uint32_t a_col, uint32_t bb, bool add) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_f16_ts(tmem_base + d_col, tmem_base + a_col + half_col(kk), make_smem_desc_sw128(bb + kk * 2048, 16384, 1024),
                      idesc_acc, add || kk != 0);
      };
      const uint32_t ka = smem_u32(smem + SM::K_OFF), va = smem_u32(smem + SM::V_OFF);
      const uint32_t qa = smem_u32(smem + SM::Q_OFF), da = smem_u32(smem + SM::DO_OFF);
      if (mbar_wait(kv_full, 0, alive, 710) && mbar_wait(&q_full[0], 0, alive, 711)) {
        tc_fence_after_sync();
        issue_ss(0, ka, qa);
        umma_commit(s_full);
        if (mbar_wait(&do_full[0], 0, alive, 712)) {
          tc_fence_after_sync();
          issue_ss(DP_COL, va, da);
          umma_commit(dp_full);
        }
      }
      for (int it = 0; it < total && alive; ++it) {
        const int s = it & 1, sn = s ^ 1, qs = it % SM::Q_STAGES, qn = (it + 1) % SM::Q_STAGES;
        if (!mbar_wait(p_full, it & 1u, alive, 713)) break;
        tc_fence_after_sync();
        issue_ts(DV_COL, 0, da + s * SM::TILE, it != 0);
        umma_commit(&do_empty[s]);
        if (it + 1 < total) {
          if (!mbar_wait(&q_full[qn], ((it + 1) / SM::Q_STAGES) & 1u, alive, 714)) break;
          tc_fence_after_sync();
          issue_ss(0, ka, qa + qn * SM::TILE);       // over P^T, which dV has read by then (products run in order)
          umma_commit(s_full);
        }
        if (!mbar_wait(ds_full, it & 1u, alive, 715)) break;
        tc_fence_after_sync();
        issue_ts(DK_COL, DP_COL, qa + qs * SM::TILE, it != 0);
        umma_commit(&q_empty[qs]);
        if (it + 1 < total) {
          if (!mbar_wait(&do_full[sn], ((it + 1) >> 1) & 1u, alive, 716)) break;
          tc_fence_after_sync();
          issue_ss(DP_COL, va, da + sn * SM::TILE);
          umma_commit(dp_full);
        }
      }
      if (alive) umma_commit(acc_full);
    }
  } else {
    const int q4 = warp & 3;
    const int wg = (warp - 2) >> 2;          // compute warpgroup: owns query columns [wg*64, wg*64+64) of the tile
    const int r = q4 * 32 + lane;            // kv row inside the tile
    const int kv_row = j * 128 + r;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q4 * 32) << 16);
    const uint32_t t_s = t_lane + wg * 64, t_dp = t_lane + DP_COL + wg * 64;
    for (int it = 0; it < total && alive; ++it) {
      const int u = u_start + it % per_head;
      const float* lse2 = vec + (it & 1) * 256 + wg * 64;
      const float* delta = lse2 + 128;
      const int q0 = u * 128 + wg * 64;
      const bool need_mask = (p.causal && (j * 128 + 127 > q0 + off)) || (q0 + 64 > Lq) || (j * 128 + 128 > Lk) ||
                             (EXT && p.window > 0 && j * 128 <= q0 + 63 + off - p.window);
      // visible columns of this row: [lo, hi)
      int lo = 0, hi = 64;
      if (need_mask) {
        lo = p.causal ? max(0, kv_row - off - q0) : 0;
        hi = kv_row < Lk ? min(64, Lq - q0) : 0;
        if (EXT && p.window > 0) hi = min(hi, kv_row - off + p.window - q0);
      }
      if (!mbar_wait(&vec_full[it & 1], (it >> 1) & 1u, alive, 723)) break;
      if (!mbar_wait(s_full, it & 1u, alive, 720)) break;
      tc_fence_after_sync();
      uint32_t pv[64];                       // S, then P (times the soft cap's derivative), fp32
#pragma unroll
      for (int c = 0; c < 2; ++c) tmem_ld_32x32b_x32(t_s + c * 32, pv + c * 32);
      tc_wait_ld();
      const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const int x = c * 32 + e;
          const float4 l4 = *reinterpret_cast<const float4*>(lse2 + x);   // warp-wide broadcast
          float v[4];
          if (EXT && p.cap_log2 > 0.f) {
            const float lv[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int y = 0; y < 4; ++y) {
              const float t = fast_tanh(__uint_as_float(pv[x + y]) * p.cap_inv);
              v[y] = fast_ex2(fmaf(t, p.cap_log2, -lv[y]));
              if (x + y < lo || x + y >= hi) v[y] = 0.f;
              pv[x + y] = __float_as_uint(v[y] * (1.f - t * t));   // d(capped logit) / d(scaled logit)
            }
          } else {
            const float2 a = unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(pv[x]), __uint_as_float(pv[x + 1])), sc2,
                                                    pack_f32x2(-l4.x, -l4.y)));
            const float2 bq = unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(pv[x + 2]), __uint_as_float(pv[x + 3])), sc2,
                                                     pack_f32x2(-l4.z, -l4.w)));
            v[0] = fast_ex2(a.x);
            v[1] = fast_ex2(a.y);
            v[2] = fast_ex2(bq.x);
            v[3] = fast_ex2(bq.y);
#pragma unroll
            for (int y = 0; y < 4; ++y) pv[x + y] = __float_as_uint(v[y]);
          }
          pk[e >> 1] = pack_bf16x2(v[0], v[1]);
          pk[(e >> 1) + 1] = pack_bf16x2(v[2], v[3]);
        }
        if (need_mask && !(EXT && p.cap_log2 > 0.f)) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (c * 32 + e < lo || c * 32 + e >= hi) pv[c * 32 + e] = 0u;
#pragma unroll
          for (int e = 0; e < 32; e += 2)
            pk[e >> 1] = pack_bf16x2(__uint_as_float(pv[c * 32 + e]), __uint_as_float(pv[c * 32 + e + 1]));
        }
        tmem_st_32x32b_x16(t_s + c * 16, pk);
      }
      tc_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);

      if (!mbar_wait(dp_full, it & 1u, alive, 721)) break;
      tc_fence_after_sync();
      uint32_t ds[32];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t dv[32];
        tmem_ld_32x32b_x32(t_dp + c * 32, dv);
        tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const int x = c * 32 + e;
          const float4 d4 = *reinterpret_cast<const float4*>(delta + x);
          const float2 a = unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(pv[x]), __uint_as_float(pv[x + 1])),
                                                  add_f32x2(pack_f32x2(__uint_as_float(dv[e]), __uint_as_float(dv[e + 1])),
                                                            pack_f32x2(-d4.x, -d4.y))));
          const float2 bq = unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(pv[x + 2]), __uint_as_float(pv[x + 3])),
                                                   add_f32x2(pack_f32x2(__uint_as_float(dv[e + 2]), __uint_as_float(dv[e + 3])),
                                                             pack_f32x2(-d4.z, -d4.w))));
          ds[x >> 1] = pack_bf16x2(a.x, a.y);
          ds[(x >> 1) + 1] = pack_bf16x2(bq.x, bq.y);
        }
      }
      tmem_st_32x32b_x32(t_dp, ds);
      tc_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&vec_empty[it & 1]);
        mbar_arrive(ds_full);
      }
    }
    if (alive && mbar_wait(acc_full, 0, alive, 722)) {
      tc_fence_after_sync();
      const bool valid = kv_row < Lk;
      __nv_bfloat16* dvp = p.dv + static_cast<size_t>(k_start + kv_row) * p.dqkv_stride + p.v_col0 + hk * D;
      __nv_bfloat16* dkp = p.dk + static_cast<size_t>(k_start + kv_row) * p.dqkv_stride + p.k_col0 + hk * D;
#pragma unroll 1
      for (int c = wg; c < D / 32; c += 2) {
        store_rows_32(t_lane + DV_COL + c * 32, 1.f, dvp + c * 32, valid);
        store_rows_32(t_lane + DK_COL + c * 32, p.scale, dkp + c * 32, valid);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------
// kernel 2: dQ.  One CTA owns a 128-row query tile of one head (Q and dO resident) and walks the 128-row K/V tiles it can see.
// TMEM: two S buffers, dP, dQ of 128 columns each.  Three K stages: K(i + 2) is wanted for S while K(i) is in dQ's product.
// ------------------------------------------------------------------------------------------------
template <int D>
struct DqSmem {
  static constexpr int TILE = 128 * D * 2;
  static constexpr int K_STAGES = 3, V_STAGES = 2;
  static constexpr int Q_OFF = 0, DO_OFF = TILE;
  static constexpr int K_OFF = 2 * TILE, V_OFF = K_OFF + K_STAGES * TILE;
  static constexpr int BAR_OFF = V_OFF + V_STAGES * TILE;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

template <int D, bool EXT>   // EXT: sliding window / logit soft-cap code paths compiled in
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, AttnParams p) {
  using SM = DqSmem<D>;
  constexpr int DCH = D / 64;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t DP_COL = 256, DQ_COL = 384;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::BAR_OFF);
  uint64_t* qd_full = bars;         // [1]
  uint64_t* s_full = bars + 1;      // [2]
  uint64_t* dp_full = bars + 3;     // [1]
  uint64_t* ds_full = bars + 4;     // [1]
  uint64_t* acc_full = bars + 5;    // [1]
  uint64_t* k_full = bars + 6;      // [3]
  uint64_t* k_empty = bars + 9;     // [3]
  uint64_t* v_full = bars + 12;     // [2]
  uint64_t* v_empty = bars + 14;    // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // grid: x = head + heads * batch (fastest), y = tile: the whole grid is dispatched longest-tile-first
  const int h = blockIdx.x % p.Hq, b = blockIdx.x / p.Hq;
  const int hk = h / p.group;
  int q_start, Lq;
  seq_bounds(p, b, q_start, Lq);
  const int k_start = q_start, Lk = Lq;
  const int n_qt = (Lq + 127) / 128;
  if ((int)blockIdx.y >= n_qt) return;
  const int i = n_qt - 1 - blockIdx.y;
  const int off = Lk - Lq;
  const int kv_end = p.causal ? min(Lk, i * 128 + 128 + off) : Lk;
  // sliding window: key tiles entirely left of the first row's window are skipped
  const int tile0 = (EXT && p.window > 0) ? max(0, i * 128 + off - p.window + 1) / 128 : 0;
  const int total = (kv_end + 127) / 128 - tile0;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
    for (int x = 0; x < 16; ++x) mbar_init(&bars[x], x == 4 ? 8 : 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  bool alive = true;

  if (warp == 0) {
    if (elect_one_sync()) {
      mbar_expect_tx(qd_full, 2 * SM::TILE);
#pragma unroll
      for (int c = 0; c < DCH; ++c) {
        tma_load_2d(smem + SM::Q_OFF + c * 16384, &tmQ, qd_full, p.q_col0 + h * D + c * 64, q_start + i * 128);
        tma_load_2d(smem + SM::DO_OFF + c * 16384, &tmdO, qd_full, h * D + c * 64, q_start + i * 128);
      }
      // in the order the products want them: K(0) V(0) K(1), then V(i), K(i + 1)
      auto load_k = [&](int it) {
        const int s = it % SM::K_STAGES;
        if (!mbar_wait(&k_empty[s], ((it / SM::K_STAGES) & 1u) ^ 1u, alive, 800)) return;
        mbar_expect_tx(&k_full[s], SM::TILE);
#pragma unroll
        for (int c = 0; c < DCH; ++c)
          tma_load_2d(smem + SM::K_OFF + s * SM::TILE + c * 16384, &tmK, &k_full[s], p.k_col0 + hk * D + c * 64,
                      k_start + (tile0 + it) * 128);
      };
      auto load_v = [&](int it) {
        const int s = it % SM::V_STAGES;
        if (!mbar_wait(&v_empty[s], ((it / SM::V_STAGES) & 1u) ^ 1u, alive, 801)) return;
        mbar_expect_tx(&v_full[s], SM::TILE);
#pragma unroll
        for (int c = 0; c < DCH; ++c)
          tma_load_2d(smem + SM::V_OFF + s * SM::TILE + c * 16384, &tmV, &v_full[s], p.v_col0 + hk * D + c * 64,
                      k_start + (tile0 + it) * 128);
      };
      if (total > 0) load_k(0);
      for (int it = 0; it < total && alive; ++it) {
        load_v(it);
        if (it + 1 < total && alive) load_k(it + 1);
      }
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      const uint32_t idesc_s = make_idesc(128, 128, 1, 1, 0, 0);
      const uint32_t idesc_acc = make_idesc(128, D, 1, 1, 0, 1);
      const uint32_t qa = smem_u32(smem + SM::Q_OFF), da = smem_u32(smem + SM::DO_OFF);
      const uint32_t ka = smem_u32(smem + SM::K_OFF), va = smem_u32(smem + SM::V_OFF);
      auto issue_ss = [&](uint32_t d_col, uint32_t a, uint32_t bb) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t o = (k >> 2) * 16384 + (k & 3) * 32;
          umma_f16_ss(tmem_base + d_col, make_smem_desc_sw128(a + o, 16, 1024), make_smem_desc_sw128(bb + o, 16, 1024), idesc_s,
                      k != 0);
        }
      };
      auto issue_s = [&](int it) {
        const int s = it % SM::K_STAGES;
        if (!mbar_wait(&k_full[s], (it / SM::K_STAGES) & 1u, alive, 810)) return;
        tc_fence_after_sync();
        issue_ss((it & 1) * 128, qa, ka + s * SM::TILE);
        umma_commit(&s_full[it & 1]);
      };
      auto issue_dp = [&](int it) {
        const int s = it % SM::V_STAGES;
        if (!mbar_wait(&v_full[s], (it / SM::V_STAGES) & 1u, alive, 811)) return;
        tc_fence_after_sync();
        issue_ss(DP_COL, da, va + s * SM::TILE);
        umma_commit(dp_full);
        umma_commit(&v_empty[s]);
      };
      if (total > 0 && mbar_wait(qd_full, 0, alive, 812)) {
        issue_s(0);
        if (alive) issue_dp(0);
        if (total > 1 && alive) issue_s(1);
        for (int it = 0; it < total && alive; ++it) {
          const int s = it % SM::K_STAGES;
          if (!mbar_wait(ds_full, it & 1u, alive, 813)) break;
          tc_fence_after_sync();
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_ts(tmem_base + DQ_COL, tmem_base + DP_COL + half_col(kk),
                        make_smem_desc_sw128(ka + s * SM::TILE + kk * 2048, 16384, 1024), idesc_acc, (it | kk) != 0);
          umma_commit(&k_empty[s]);
          if (it + 1 < total) issue_dp(it + 1);                // over dS, which dQ has read by then
          if (it + 2 < total && alive) issue_s(it + 2);        // S(it) was read before dS(it) was written
        }
        if (alive) umma_commit(acc_full);
      }
    }
  } else {
    const int q4 = warp & 3;
    const int wg = (warp - 2) >> 2;
    const int r = q4 * 32 + lane;
    const int qrow = i * 128 + r;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q4 * 32) << 16);
    const uint32_t t_dp = t_lane + DP_COL + wg * 64;
    float lse2 = 0.f, delta = 0.f;
    if (qrow < Lq) {
      const size_t idx = static_cast<size_t>(h) * p.total_rows + q_start + qrow;
      lse2 = p.lse[idx] * 1.4426950408889634f;
      delta = p.delta[idx];
    }
    const int limit = (qrow < Lq) ? (p.causal ? min(Lk - 1, qrow + off) : Lk - 1) : -1;
    const int first = (EXT && p.window > 0) ? qrow + off - p.window + 1 : 0;
    const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2), ml2 = pack_f32x2(-lse2, -lse2), md2 = pack_f32x2(-delta, -delta);
    for (int it = 0; it < total && alive; ++it) {
      const int col0 = (tile0 + it) * 128 + wg * 64;
      const bool need_mask = (p.causal && col0 + 63 > i * 128 + off) || (col0 + 64 > Lk) || (i * 128 + 128 > Lq) ||
                             (EXT && p.window > 0 && col0 <= i * 128 + 127 + off - p.window);
      if (!mbar_wait(&s_full[it & 1], (it >> 1) & 1u, alive, 820)) break;
      tc_fence_after_sync();
      uint32_t pv[64];
#pragma unroll
      for (int c = 0; c < 2; ++c) tmem_ld_32x32b_x32(t_lane + (it & 1) * 128 + wg * 64 + c * 32, pv + c * 32);
      tc_wait_ld();
      if (EXT && p.cap_log2 > 0.f) {
#pragma unroll
        for (int e = 0; e < 64; ++e) {
          const float t = fast_tanh(__uint_as_float(pv[e]) * p.cap_inv);
          pv[e] = __float_as_uint(fast_ex2(fmaf(t, p.cap_log2, -lse2)) * (1.f - t * t));
        }
      } else {
#pragma unroll
        for (int e = 0; e < 64; e += 2) {
          const float2 a = unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(pv[e]), __uint_as_float(pv[e + 1])), sc2, ml2));
          pv[e] = __float_as_uint(fast_ex2(a.x));
          pv[e + 1] = __float_as_uint(fast_ex2(a.y));
        }
      }
      if (need_mask) {
#pragma unroll
        for (int e = 0; e < 64; ++e)
          if (col0 + e > limit || (EXT && col0 + e < first)) pv[e] = 0u;
      }
      if (!mbar_wait(dp_full, it & 1u, alive, 821)) break;
      tc_fence_after_sync();
      uint32_t ds[32];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t dv[32];
        tmem_ld_32x32b_x32(t_dp + c * 32, dv);
        tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const int x = c * 32 + e;
          const float2 a = unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(pv[x]), __uint_as_float(pv[x + 1])),
                                                  add_f32x2(pack_f32x2(__uint_as_float(dv[e]), __uint_as_float(dv[e + 1])), md2)));
          ds[x >> 1] = pack_bf16x2(a.x, a.y);
        }
      }
      tmem_st_32x32b_x32(t_dp, ds);
      tc_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    if (total > 0 && alive && mbar_wait(acc_full, 0, alive, 822)) {
      tc_fence_after_sync();
      __nv_bfloat16* dqp = p.dq + static_cast<size_t>(q_start + qrow) * p.dqkv_stride + p.q_col0 + h * D;
#pragma unroll 1
      for (int c = wg; c < D / 32; c += 2) store_rows_32(t_lane + DQ_COL + c * 32, p.scale, dqp + c * 32, qrow < Lq);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int D, bool EXT>
static int launch_bwd(const CUtensorMap* m, const AttnParams& p, int max_len, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(flash_bwd_dkdv_kernel<D, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         DkvSmem<D>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(flash_bwd_dq_kernel<D, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize, DqSmem<D>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  // m: q, k, v, dO
  dim3 g1(p.Hkv * p.B, (max_len + 127) / 128, 1);
  flash_bwd_dkdv_kernel<D, EXT><<<g1, BWD_THREADS, DkvSmem<D>::TOTAL, st>>>(m[0], m[1], m[2], m[3], p);
  dim3 g2(p.Hq * p.B, (max_len + 127) / 128, 1);
  flash_bwd_dq_kernel<D, EXT><<<g2, BWD_THREADS, DqSmem<D>::TOTAL, st>>>(m[0], m[1], m[2], m[3], p);
  return (int)cudaGetLastError();
}

template <int D, bool EXT, bool SPLIT = false>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& p,
                      int max_len, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(flash_fwd_kernel<D, EXT, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         FwdSmem<D>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  dim3 grid(p.Hq * p.B, (max_len + 255) / 256, 1);
  flash_fwd_kernel<D, EXT, SPLIT><<<grid, FWD_THREADS, FwdSmem<D>::TOTAL, st>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

}  // namespace ts

TS_DEFINE_ERROR_API(ts_attention)

using namespace ts;

// q, k, v: bf16 row-major token matrices [total_rows][*_stride]; head h of q starts at column h*D (+ col0).
// They may alias one fused qkv buffer (pass the same base with different col0).
// cu_seqlens: device int32 [B+1] for packed documents or nullptr for B sequences of S tokens.
// max_len: longest sequence (host knowledge; S for the uniform case).
// window > 0 restricts every query to the last `window` keys; softcap > 0 applies c * tanh(s / c) to the scaled logits.
extern "C" int ts_flash_fwd_ex(const void* q, const void* k, const void* v, void* o, float* lse, long long total_rows,
                               int q_stride, int k_stride, int v_stride, int o_stride, int q_col0, int k_col0,
                               int v_col0, int Hq, int Hkv, int D, int B, int S, const int* cu_seqlens, int max_len,
                               int causal, float scale, int window, float softcap, void* stream) {
  if ((D != 64 && D != 128) || Hq % Hkv != 0 || total_rows <= 0) return -10;
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_2d(&tq, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)total_rows, (uint64_t)q_stride,
                        (uint64_t)q_stride, 128, 64);
  if (rc) return rc * 100 - 1;
  rc = make_tmap_2d(&tk, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)total_rows, (uint64_t)k_stride,
                    (uint64_t)k_stride, 128, 64);
  if (rc) return rc * 100 - 2;
  rc = make_tmap_2d(&tv, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)total_rows, (uint64_t)v_stride,
                    (uint64_t)v_stride, 128, 64);
  if (rc) return rc * 100 - 3;
  AttnParams p{};
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.Hq = Hq; p.Hkv = Hkv; p.group = Hq / Hkv; p.B = B; p.S = S; p.cu_seqlens = cu_seqlens; p.causal = causal;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.window = window > 0 ? window : 0;
  p.cap_inv = softcap > 0.f ? scale / softcap : 0.f;
  p.cap_log2 = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
  p.o = (__nv_bfloat16*)o; p.o_stride = o_stride; p.lse = lse; p.total_rows = total_rows;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool ext = p.window > 0 || p.cap_log2 > 0.f;
  if (D == 128) return ext ? launch_fwd<128, true>(tq, tk, tv, p, max_len, st) : launch_fwd<128, false>(tq, tk, tv, p, max_len, st);
  return ext ? launch_fwd<64, true>(tq, tk, tv, p, max_len, st) : launch_fwd<64, false>(tq, tk, tv, p, max_len, st);
}

extern "C" int ts_flash_fwd(const void* q, const void* k, const void* v, void* o, float* lse, long long total_rows,
                            int q_stride, int k_stride, int v_stride, int o_stride, int q_col0, int k_col0,
                            int v_col0, int Hq, int Hkv, int D, int B, int S, const int* cu_seqlens, int max_len,
                            int causal, float scale, void* stream) {
  return ts_flash_fwd_ex(q, k, v, o, lse, total_rows, q_stride, k_stride, v_stride, o_stride, q_col0, k_col0, v_col0, Hq,
                         Hkv, D, B, S, cu_seqlens, max_len, causal, scale, 0, 0.f, stream);
}

// Portions of prompts against keys of a cache: sequence b's queries are rows [cu_q[b], cu_q[b + 1]) of q and the LAST of its
// k_lens[b] keys, which lie at rows k_starts[b] on of k / v (head g of k at column g * D, of v too); rows up to the next
// multiple of 128 are read, so they hold finite values.  Causal; window and softcap as above.  Weights keep 16 bits (SPLIT).
// Tensor-bound (the split is half as much again as plain bf16 weights): 0.65 ms for 8192 query rows of up to 10000 keys, 32 / 8 heads of
// 128; three such prompts with 24 decoding steps took 438 ms with fp32 scores in memory, 101 ms with this.
extern "C" int ts_flash_portions(const void* q, const void* k, const void* v, void* o, long long q_rows, long long k_rows,
                                 int q_stride, int kv_stride, int o_stride, int Hq, int Hkv, int D, int B, const int* cu_q,
                                 const int* k_starts, const int* k_lens, int max_q, float scale, int window, float softcap,
                                 void* stream) {
  if ((D != 64 && D != 128) || Hkv <= 0 || Hq % Hkv != 0 || q_rows <= 0 || k_rows <= 0 || B <= 0 || max_q <= 0) return -10;
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_2d(&tq, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)q_rows, (uint64_t)Hq * D, (uint64_t)q_stride, 128, 64);
  if (rc) return rc * 100 - 1;
  rc = make_tmap_2d(&tk, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)k_rows, (uint64_t)Hkv * D, (uint64_t)kv_stride, 128, 64);
  if (rc) return rc * 100 - 2;
  rc = make_tmap_2d(&tv, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)k_rows, (uint64_t)Hkv * D, (uint64_t)kv_stride, 128, 64);
  if (rc) return rc * 100 - 3;
  AttnParams p{};
  p.Hq = Hq; p.Hkv = Hkv; p.group = Hq / Hkv; p.B = B; p.cu_seqlens = cu_q; p.k_starts = k_starts; p.k_lens = k_lens;
  p.causal = 1; p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.window = window > 0 ? window : 0;
  p.cap_inv = softcap > 0.f ? scale / softcap : 0.f;
  p.cap_log2 = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
  p.o = (__nv_bfloat16*)o; p.o_stride = o_stride; p.total_rows = q_rows;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (p.window > 0 || p.cap_log2 > 0.f)
    return D == 128 ? launch_fwd<128, true, true>(tq, tk, tv, p, max_q, st) : launch_fwd<64, true, true>(tq, tk, tv, p, max_q, st);
  return D == 128 ? launch_fwd<128, false, true>(tq, tk, tv, p, max_q, st) : launch_fwd<64, false, true>(tq, tk, tv, p, max_q, st);
}

extern "C" int ts_attn_delta(const void* o, const void* dout, float* delta, long long total_rows, int Hq, int D,
                             int o_stride, void* stream) {
  const long long warps = total_rows * Hq;
  const int threads = 256;
  const long long blocks = (warps * 32 + threads - 1) / threads;
  attn_delta_kernel<<<(unsigned)blocks, threads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, total_rows, Hq, D, o_stride);
  return (int)cudaGetLastError();
}

// Gradient of ts_flash_fwd. dq/dk/dv are written into `dqkv` (same row layout and column offsets as q/k/v inside
// a fused buffer of row stride `qkv_stride`); every element of the q|k|v column range is written.
extern "C" int ts_flash_bwd_ex(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                               const float* delta, void* dqkv, long long total_rows, int qkv_stride, int o_stride,
                               int q_col0, int k_col0, int v_col0, int Hq, int Hkv, int D, int B, int S,
                               const int* cu_seqlens, int max_len, int causal, float scale, int window, float softcap,
                               void* stream) {
  if ((D != 64 && D != 128) || Hq % Hkv != 0 || total_rows <= 0) return -10;
  CUtensorMap m[4];
  const void* bases[4] = {q, k, v, dout};
  const int strides[4] = {qkv_stride, qkv_stride, qkv_stride, o_stride};
  for (int t = 0; t < 4; ++t) {
    int rc = make_tmap_2d(&m[t], bases[t], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)total_rows,
                          (uint64_t)strides[t], (uint64_t)strides[t], 128, 64);
    if (rc) return rc * 100 - 10 - t;
  }
  AttnParams p{};
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.Hq = Hq; p.Hkv = Hkv; p.group = Hq / Hkv; p.B = B; p.S = S; p.cu_seqlens = cu_seqlens; p.causal = causal;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.window = window > 0 ? window : 0;
  p.cap_inv = softcap > 0.f ? scale / softcap : 0.f;
  p.cap_log2 = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
  p.o_stride = o_stride; p.lse = const_cast<float*>(lse); p.delta = delta; p.total_rows = total_rows;
  p.dout = (const __nv_bfloat16*)dout;
  p.dq = p.dk = p.dv = (__nv_bfloat16*)dqkv;
  p.dqkv_stride = qkv_stride;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool ext = p.window > 0 || p.cap_log2 > 0.f;
  if (D == 128) return ext ? launch_bwd<128, true>(m, p, max_len, st) : launch_bwd<128, false>(m, p, max_len, st);
  return ext ? launch_bwd<64, true>(m, p, max_len, st) : launch_bwd<64, false>(m, p, max_len, st);
}

extern "C" int ts_flash_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                            const float* delta, void* dqkv, long long total_rows, int qkv_stride, int o_stride,
                            int q_col0, int k_col0, int v_col0, int Hq, int Hkv, int D, int B, int S,
                            const int* cu_seqlens, int max_len, int causal, float scale, void* stream) {
  return ts_flash_bwd_ex(q, k, v, dout, lse, delta, dqkv, total_rows, qkv_stride, o_stride, q_col0, k_col0, v_col0, Hq,
                         Hkv, D, B, S, cu_seqlens, max_len, causal, scale, 0, 0.f, stream);
}
