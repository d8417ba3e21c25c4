// Inference kernels: paged KV-cache writes and single-token (decode) attention over a paged cache with split-KV.
//
// Decode attention reads every K/V byte of a sequence once per step; the q heads of a GQA group share each K/V row.
// Serves the role of the vLLM paged-attention kernels configured in the reference
// (data_pipeline/trainer/inference.py:786-921) and of data_pipeline/trainer/kernels/flex_attention.py:1032.
#include "common.cuh"
#include "host_common.h"

namespace ts {

// Rotary embedding (partners i and i + D / 2) of the q and k heads of projection rows, in place, and the cache write of the rotated
// keys and the values: one launch and one pass instead of a copy of the rows, a rotation and a write.  One CTA per row: a thread
// owns eight pairs of a head or eight values.
constexpr int RC_THREADS = 256;
__global__ void __launch_bounds__(RC_THREADS)
rope_cache_kernel(__nv_bfloat16* __restrict__ qkv, long long row_stride, const float* __restrict__ cos_t,
                  const float* __restrict__ sin_t, const int* __restrict__ pos, const long long* __restrict__ slot_mapping,
                  __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache, int Hq, int Hkv, int D) {
  grid_trigger();
  grid_wait();
  const long long row = blockIdx.x, slot = slot_mapping[row];
  const int half = D >> 1, vecs = half >> 3, rot = (Hq + Hkv) * vecs, kv_width = Hkv * D;
  const size_t table = static_cast<size_t>(pos[row]) * half;
  __nv_bfloat16* r = qkv + row * row_stride;
  for (int idx = threadIdx.x; idx < rot + (kv_width >> 3); idx += RC_THREADS) {
    if (idx >= rot) {
      const int v = idx - rot;
      if (slot >= 0)
        reinterpret_cast<uint4*>(v_cache + slot * kv_width)[v] = reinterpret_cast<const uint4*>(r + (Hq + Hkv) * D)[v];
      continue;
    }
    const int head = idx / vecs, c = (idx - head * vecs) * 8;
    __nv_bfloat16* base = r + head * D + c;
    const uint4 a4 = *reinterpret_cast<const uint4*>(base), b4 = *reinterpret_cast<const uint4*>(base + half);
    const uint32_t aw[4] = {a4.x, a4.y, a4.z, a4.w}, bw[4] = {b4.x, b4.y, b4.z, b4.w};
    uint32_t oa[4], ob[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 cs = *reinterpret_cast<const float2*>(cos_t + table + c + 2 * e);
      const float2 sn = *reinterpret_cast<const float2*>(sin_t + table + c + 2 * e);
      const float2 a = unpack_bf16x2(aw[e]), b = unpack_bf16x2(bw[e]);
      oa[e] = pack_bf16x2(a.x * cs.x - b.x * sn.x, a.y * cs.y - b.y * sn.y);
      ob[e] = pack_bf16x2(b.x * cs.x + a.x * sn.x, b.y * cs.y + a.y * sn.y);
    }
    const uint4 ra = make_uint4(oa[0], oa[1], oa[2], oa[3]), rb = make_uint4(ob[0], ob[1], ob[2], ob[3]);
    *reinterpret_cast<uint4*>(base) = ra;
    *reinterpret_cast<uint4*>(base + half) = rb;
    if (head >= Hq && slot >= 0) {
      __nv_bfloat16* dst = k_cache + slot * kv_width + (head - Hq) * D + c;
      *reinterpret_cast<uint4*>(dst) = ra;
      *reinterpret_cast<uint4*>(dst + half) = rb;
    }
  }
}

// k_cache / v_cache: [num_blocks][block_size][Hkv][D] bf16.  slot = block * block_size + offset.
__global__ void kv_cache_write_kernel(const __nv_bfloat16* __restrict__ qkv, int row_stride, int k_col0, int v_col0,
                                      __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache,
                                      const long long* __restrict__ slot_mapping, long long rows, int kv_width) {
  const int vec_per_row = kv_width >> 3;
  const long long total = rows * vec_per_row;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long row = idx / vec_per_row;
    const int v = static_cast<int>(idx - row * vec_per_row);
    const long long slot = slot_mapping[row];
    if (slot < 0) continue;
    const uint4 kk = *reinterpret_cast<const uint4*>(qkv + row * row_stride + k_col0 + v * 8);
    const uint4 vv = *reinterpret_cast<const uint4*>(qkv + row * row_stride + v_col0 + v * 8);
    *reinterpret_cast<uint4*>(k_cache + slot * kv_width + v * 8) = kk;
    *reinterpret_cast<uint4*>(v_cache + slot * kv_width + v * 8) = vv;
  }
}

// Cached keys and values of sequences side by side, in key order: rows [starts[s], starts[s] + lens[s]) of out
// [rows][2 * kv_width], the rows up to the next multiple of 128 zero (attention reads whole tiles of 128 keys).
// grid (rows of the longest / KV_GATHER_ROWS, sequences); one warp per row.
constexpr int KV_GATHER_ROWS = 8;
__global__ void __launch_bounds__(KV_GATHER_ROWS * 32)
kv_gather_kernel(const __nv_bfloat16* __restrict__ k_cache, const __nv_bfloat16* __restrict__ v_cache,
                 const int* __restrict__ block_table, int max_blocks, const int* __restrict__ starts,
                 const int* __restrict__ lens, int block_size, int kv_width, __nv_bfloat16* __restrict__ out) {
  const int s = blockIdx.y, j = blockIdx.x * KV_GATHER_ROWS + (threadIdx.x >> 5), lane = threadIdx.x & 31, len = lens[s];
  if (j >= (len + 127) / 128 * 128) return;
  uint4* dst = reinterpret_cast<uint4*>(out + (static_cast<size_t>(starts[s]) + j) * 2 * kv_width);
  const int vecs = kv_width >> 3;
  if (j >= len) {
    for (int v = lane; v < 2 * vecs; v += 32) dst[v] = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const size_t slot = static_cast<size_t>(block_table[static_cast<size_t>(s) * max_blocks + j / block_size]) * block_size + j % block_size;
  const uint4* ks = reinterpret_cast<const uint4*>(k_cache + slot * kv_width);
  const uint4* vs = reinterpret_cast<const uint4*>(v_cache + slot * kv_width);
  for (int v = lane; v < vecs; v += 32) {
    dst[v] = ks[v];
    dst[vecs + v] = vs[v];
  }
}

constexpr int DEC_WARPS = 4;
constexpr int DEC_MAX_GROUP = 8;
constexpr int DEC_MAX_CLUSTER = 8;
constexpr int DEC_MOST_KEYS = 12288;

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the leading eight bits of a value, and those of two as an operand word
__device__ __forceinline__ float high_part(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
// and what they leave, at least `least`
__device__ __forceinline__ float rest_part(float x, float least) { return fmaxf(x - high_part(x), least); }
__device__ __forceinline__ uint32_t pack_high(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }
// eight values of a row of any alignment (query rows may be anybody's; caches are whole 16-byte vectors)
__device__ __forceinline__ uint4 load_row8(const __nv_bfloat16* p) {
  if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) return *reinterpret_cast<const uint4*>(p);
  const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
  return make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
}
__device__ __forceinline__ void put_float4(float* dst, const float* v) { *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]); }

// grid (splits, Hkv, sequences).  A CTA takes an even share of one sequence's keys for one kv head and all query heads that share
// it.  Memory should bound this; scalar code for four heads of 128 spends 5 - 10 times as many issue slots per key as the loads
// leave (shuffles of the dot products, conversions), so both products are warp MMAs whose operands come straight from global
// memory as 16-byte vectors:
//   S = Q K^T  rows are heads; a lane's eight consecutive dimensions feed two reduction steps (Q in the same order)
//   O += P V   a lane has the same dimensions of four keys, two keys of one dimension are one operand word; P comes from S in
//              registers, cut into three bf16 parts of eight bits each, which hold all of an fp32 weight.  No part of a weight is
//              zero (2^-24 of it at least): an infinite value stays infinite in every product.  The heads use eight
//              of the sixteen rows, so rows 8 - 15 take the second part; up to four heads are given twice (rows 4 - 7 repeat
//              rows 0 - 3) and rows 4 - 7 take the third at no cost, more (WIDE) need a second product for it, 3 - 10 % of the
//              time (8 heads per key head, 64 sequences: 2000 keys of 128 117.6 -> 120.8 us, 300 of 64 26.6 -> 28.7)
// Every warp walks its own 16-key tiles with a softmax state of its own; states meet in shared memory, then over the splits: up
// to DEC_MAX_CLUSTER in distributed shared memory, more through partial results [seq][Hq][split][D] fp32 and lse
// [seq][Hq][split] for decode_merge_kernel.
// One warp per key with shuffled dot products / this (32 query heads of 8 kv heads, us between events with nothing cached; at the
// copy bandwidth): 64 sequences of 300 keys of 64 110 / 25.5 (6.1), of 2000 keys of 128 580 / 113 (81), 4 of 10000 keys of 128
// 261 / 50 (25), 17 of 10000 779 / 132 (108), 1 of 97 of 64 27.7 / 10.2.
// EXT: a window (the last `window` keys, 0: all) or a soft cap of the scores (cap_log2 * tanh(s * cap_inv), cap_log2 0: none).
template <int D, bool CLUSTER, bool EXT, bool WIDE>
__global__ void __launch_bounds__(DEC_WARPS * 32)
decode_attention_kernel(const __nv_bfloat16* __restrict__ q, int q_stride, const __nv_bfloat16* __restrict__ k_cache,
                        const __nv_bfloat16* __restrict__ v_cache, const int* __restrict__ block_table,
                        int max_blocks, const int* __restrict__ seq_lens, __nv_bfloat16* __restrict__ out, int out_stride,
                        float* __restrict__ part_out, float* __restrict__ part_lse, int Hq, int Hkv, int block_size,
                        int chunk, int splits, float scale_log2, int window, float cap_inv, float cap_log2) {
  constexpr int KT = D == 64 ? 2 : 1;      // 16-key tiles in flight: 8 KB of keys and values per warp
  constexpr int NK = D / 32, NV = D / 64;
  const int split = blockIdx.x, hk = blockIdx.y, seq = blockIdx.z;
  const int group = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int head = WIDE ? gid : gid & 3;           // of this lane's row
  const bool third = !WIDE && gid >= 4;            // whose weights are the third parts
  grid_trigger();
  grid_wait();
  const int len = seq_lens[seq];
  const int seen = EXT && window > 0 ? max(0, len - window) : 0, base0 = seen & ~15;      // first visible key, and its tile
  const int share = (max(chunk, (len - base0 + splits - 1) / splits) + 15) & ~15;
  const int t0 = base0 + split * share, t1 = min(len, t0 + share);
  __shared__ __align__(16) float s_acc[DEC_WARPS][DEC_MAX_GROUP][D];
  __shared__ float s_m[DEC_WARPS][DEC_MAX_GROUP], s_l[DEC_WARPS][DEC_MAX_GROUP];
  __shared__ __align__(16) float c_acc[DEC_MAX_GROUP][D];      // the CTA's result, not normalised
  __shared__ float c_m[DEC_MAX_GROUP], c_l[DEC_MAX_GROUP];

  uint4 qv[NK];
#pragma unroll
  for (int i = 0; i < NK; ++i)
    qv[i] = head < group ? load_row8(q + static_cast<size_t>(seq) * q_stride + (hk * group + head) * D + i * 32 + tig * 8)
                         : make_uint4(0u, 0u, 0u, 0u);
  float m = -INFINITY, l = 0.f;            // of the lane's head; l of this lane's keys
  float acc[NV * 8][4];                    // [n]: columns 2 tig, 2 tig + 1 <-> dimensions 64 (n / 8) + 8 column + n % 8
#pragma unroll
  for (int n = 0; n < NV * 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
  const int kv_width = Hkv * D;
  const int* table = block_table + static_cast<size_t>(seq) * max_blocks;
  // first cache row of a 16-key tile whose keys lie in one block; one past the end repeats the last one, masked below.  A step's
  // keys are loaded as soon as the products with the keys before have read their registers, its values likewise; the lines come
  // from L2, into which they are asked a step earlier, and the block table is read three steps ahead
  const bool whole = (block_size & 15) == 0;
  constexpr int STRIDE = DEC_WARPS * 16 * KT;
  auto tile_base = [&](int t) { return min(t, (t1 - 1) & ~15); };
  auto tile_first = [&](int t) {
    const int base = tile_base(t);
    return whole ? table[base / block_size] * block_size + base % block_size : 0;
  };
  auto row_at = [&](int base, int first, int j) {
    const int key = min(base + j, t1 - 1);
    const int slot = whole ? first + (key - base) : table[key / block_size] * block_size + key % block_size;
    return static_cast<size_t>(slot) * kv_width + hk * D;
  };
  uint4 kr[KT][2][NK], vr[KT][4][NV];
  auto load_k = [&](int t, const int (&first)[KT]) {
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const __nv_bfloat16* p = k_cache + row_at(tile_base(t + x * 16), first[x], n * 8 + gid) + tig * 8;
#pragma unroll
        for (int i = 0; i < NK; ++i) kr[x][n][i] = *reinterpret_cast<const uint4*>(p + i * 32);
      }
  };
  auto load_v = [&](int t, const int (&first)[KT]) {
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat16* p = v_cache + row_at(tile_base(t + x * 16), first[x], (j >> 1) * 8 + tig * 2 + (j & 1)) + gid * 8;
#pragma unroll
        for (int i = 0; i < NV; ++i) vr[x][j][i] = *reinterpret_cast<const uint4*>(p + i * 64);
      }
    if (t + KT * 16 > t1 || (EXT && t < seen)) {
      // keys that do not count: their weights are zero, their values must be too (an infinite one would give NaN)
#pragma unroll
      for (int x = 0; x < KT; ++x)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = t + x * 16 + (j >> 1) * 8 + tig * 2 + (j & 1);
          if (key >= t1 || (EXT && key < seen))
#pragma unroll
            for (int i = 0; i < NV; ++i) vr[x][j][i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
  };
  const int begin = t0 + warp * 16 * KT;
  int next[KT], later[KT];
  if (begin < t1) {
    int first[KT];
#pragma unroll
    for (int x = 0; x < KT; ++x) {
      first[x] = tile_first(begin + x * 16);
      next[x] = tile_first(begin + STRIDE + x * 16);
      later[x] = tile_first(begin + 2 * STRIDE + x * 16);
    }
    load_k(begin, first);
    load_v(begin, first);
  }
  for (int t = begin; t < t1; t += STRIDE) {
    int far[KT];
#pragma unroll
    for (int x = 0; x < KT; ++x) far[x] = tile_first(t + 3 * STRIDE + x * 16);
    if (whole) {
      // 32 lines of keys and of values: rows of one 128-byte line each (D = 64, two tiles) or of two (D = 128)
      const int x = KT == 2 ? lane >> 4 : 0, j = KT == 2 ? lane & 15 : lane >> 1;
      const size_t at = row_at(tile_base(t + 2 * STRIDE + x * 16), KT == 2 && x ? later[KT - 1] : later[0], j) + (KT == 2 ? 0 : (lane & 1) * 64);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(k_cache + at));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(v_cache + at));
    }
    float sc[KT][2][4];
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[x][n][e] = 0.f;
#pragma unroll
        for (int i = 0; i < NK; ++i) {
          mma_bf16_16816(sc[x][n], qv[i].x, 0u, qv[i].y, 0u, kr[x][n][i].x, kr[x][n][i].y);
          mma_bf16_16816(sc[x][n], qv[i].z, 0u, qv[i].w, 0u, kr[x][n][i].z, kr[x][n][i].w);
        }
      }
    if (t + STRIDE < t1) load_k(t + STRIDE, next);
#pragma unroll
    for (int x = 0; x < KT; ++x) {
      float (&s)[2][4] = sc[x];
      const int k0 = t + x * 16 + tig * 2;
      float mn = m;
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          s[n][e] = EXT && cap_log2 > 0.f ? cap_log2 * tanhf(s[n][e] * cap_inv) : s[n][e] * scale_log2;
          if (k0 + n * 8 + e >= t1 || (EXT && k0 + n * 8 + e < seen)) s[n][e] = -INFINITY;
          mn = fmaxf(mn, s[n][e]);
        }
      mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
      mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
      const float sub = mn == -INFINITY ? 0.f : mn;
      if (__any_sync(0xffffffffu, mn > m)) {
        const float a = fast_ex2(m - sub);
        l *= a;
#pragma unroll
        for (int n = 0; n < NV * 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[n][e] *= a;
        m = mn;
      }
      uint32_t a0[2], a8[2], last[2];        // operand words of rows gid and gid + 8; the third parts
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float p0 = fast_ex2(s[n][0] - sub), p1 = fast_ex2(s[n][1] - sub);
        l += p0 + p1;
        const float r0 = rest_part(p0, p0 * 0x1p-24f), r1 = rest_part(p1, p1 * 0x1p-24f);
        a0[n] = pack_high(p0, p1);
        a8[n] = pack_high(r0, r1);
        const float x0 = rest_part(r0, p0 * 0x1p-40f), x1 = rest_part(r1, p1 * 0x1p-40f);
        last[n] = WIDE ? pack_bf16x2(0.5f * x0, 0.5f * x1) : pack_bf16x2(x0, x1);     // (WIDE: in two rows, so that none is zero)
        if (third) {
          a0[n] = last[n];
          a8[n] = 0u;
        }
      }
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const uint32_t v[4][4] = {{vr[x][0][i].x, vr[x][0][i].y, vr[x][0][i].z, vr[x][0][i].w},
                                  {vr[x][1][i].x, vr[x][1][i].y, vr[x][1][i].z, vr[x][1][i].w},
                                  {vr[x][2][i].x, vr[x][2][i].y, vr[x][2][i].z, vr[x][2][i].w},
                                  {vr[x][3][i].x, vr[x][3][i].y, vr[x][3][i].z, vr[x][3][i].w}};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t b0[2] = {__byte_perm(v[0][e], v[1][e], 0x5410), __byte_perm(v[2][e], v[3][e], 0x5410)};
          const uint32_t b1[2] = {__byte_perm(v[0][e], v[1][e], 0x7632), __byte_perm(v[2][e], v[3][e], 0x7632)};
          mma_bf16_16816(acc[i * 8 + 2 * e], a0[0], a8[0], a0[1], a8[1], b0[0], b0[1]);
          mma_bf16_16816(acc[i * 8 + 2 * e + 1], a0[0], a8[0], a0[1], a8[1], b1[0], b1[1]);
          if (WIDE) {
            mma_bf16_16816(acc[i * 8 + 2 * e], last[0], last[0], last[1], last[1], b0[0], b0[1]);
            mma_bf16_16816(acc[i * 8 + 2 * e + 1], last[0], last[0], last[1], last[1], b1[0], b1[1]);
          }
        }
      }
    }
    if (t + STRIDE < t1) load_v(t + STRIDE, next);
#pragma unroll
    for (int x = 0; x < KT; ++x) {
      next[x] = later[x];
      later[x] = far[x];
    }
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (tig == 0 && !third) {
    s_m[warp][head] = m;
    s_l[warp][head] = l;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float sum[8];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const float x = acc[i * 8 + n][c];
        sum[n] = (WIDE ? 0.f : __shfl_down_sync(0xffffffffu, x, 16)) + acc[i * 8 + n][c + 2] + x;     // smallest parts first
      }
      if (third) continue;
      float* dst = &s_acc[warp][head][i * 64 + (2 * tig + c) * 8];
      put_float4(dst, sum);
      put_float4(dst + 4, sum + 4);
    }
  __syncthreads();
  for (int idx = threadIdx.x; idx < group * D; idx += blockDim.x) {
    const int g = idx / D, d = idx % D;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) mm = fmaxf(mm, s_m[w][g]);
    const float sub = mm == -INFINITY ? 0.f : mm;
    float ll = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) {
      const float a = fast_ex2(s_m[w][g] - sub);
      ll += s_l[w][g] * a;
      o += s_acc[w][g][d] * a;
    }
    if (CLUSTER) {
      c_acc[g][d] = o;
      if (d == 0) {
        c_m[g] = mm;
        c_l[g] = ll;
      }
    } else {
      const size_t base = (static_cast<size_t>(seq) * Hq + hk * group + g) * splits + split;
      part_out[base * D + d] = ll > 0.f ? o / ll : 0.f;
      if (d == 0) part_lse[base] = ll > 0.f ? mm + log2f(ll) : -INFINITY;
    }
  }
  if (CLUSTER) {
    if (splits > 1) cluster_sync_all();
    else __syncthreads();
    for (int idx = split * (DEC_WARPS * 32) + threadIdx.x; idx < group * D; idx += splits * (DEC_WARPS * 32)) {
      const int g = idx / D, d = idx % D;
      float mm = -INFINITY, ll = 0.f, o = 0.f;
      for (int r = 0; r < splits; ++r) mm = fmaxf(mm, splits > 1 ? ld_shared_cluster(&c_m[g], r) : c_m[g]);
      const float sub = mm == -INFINITY ? 0.f : mm;
      for (int r = 0; r < splits; ++r) {
        const float a = fast_ex2((splits > 1 ? ld_shared_cluster(&c_m[g], r) : c_m[g]) - sub);
        ll += a * (splits > 1 ? ld_shared_cluster(&c_l[g], r) : c_l[g]);
        o += a * (splits > 1 ? ld_shared_cluster(&c_acc[g][d], r) : c_acc[g][d]);
      }
      out[static_cast<size_t>(seq) * out_stride + (hk * group + g) * D + d] = __float2bfloat16(ll > 0.f ? o / ll : 0.f);
    }
    if (splits > 1) cluster_sync_all();            // nobody leaves while a peer may still read its result
  }
}

template <int D>
__global__ void decode_merge_kernel(const float* __restrict__ part_out, const float* __restrict__ part_lse,
                                    __nv_bfloat16* __restrict__ out, int out_stride, int Hq, int splits) {
  const int seq = blockIdx.x, h = blockIdx.y, d = threadIdx.x;
  const size_t base = (static_cast<size_t>(seq) * Hq + h) * splits;
  float mm = -INFINITY;
  for (int s = 0; s < splits; ++s) mm = fmaxf(mm, part_lse[base + s]);
  float den = 0.f, o = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float w = (part_lse[base + s] == -INFINITY) ? 0.f : fast_ex2(part_lse[base + s] - mm);
    den += w;
    o += w * part_out[(base + s) * D + d];
  }
  out[static_cast<size_t>(seq) * out_stride + h * D + d] = __float2bfloat16(den > 0.f ? o / den : 0.f);
}

}  // namespace ts

TS_DEFINE_ERROR_API(ts_decode)
using namespace ts;

extern "C" int ts_kv_cache_write(const void* qkv, int row_stride, int k_col0, int v_col0, void* k_cache, void* v_cache,
                                 const long long* slot_mapping, long long rows, int kv_width, void* stream) {
  if (rows <= 0) return 0;
  if (kv_width % 8 != 0) return -10;
  long long blocks = (rows * (kv_width / 8) + 255) / 256;
  if (blocks > (long long)sm_count() * 16) blocks = (long long)sm_count() * 16;
  kv_cache_write_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      (const __nv_bfloat16*)qkv, row_stride, k_col0, v_col0, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache,
      slot_mapping, rows, kv_width);
  return (int)cudaGetLastError();
}

// D a multiple of 16; rows of qkv (q | k | v heads) 16-byte aligned; cos / sin: fp32 [positions][D / 2], read at pos[row] without
// a check: the caller refuses sequences longer than the tables (inference/engine.py check_length); slot < 0: not cached.
extern "C" int ts_rope_cache(void* qkv, long long row_stride, const float* cos_t, const float* sin_t, const int* pos,
                             const long long* slot_mapping, void* k_cache, void* v_cache, long long rows, int Hq, int Hkv, int D,
                             void* stream) {
  if (rows <= 0) return 0;
  if (D <= 0 || D % 16 || row_stride % 8 || (reinterpret_cast<uintptr_t>(qkv) & 15u) || rows > 0x7fffffffll) return -10;
  return launch_chained(rope_cache_kernel, dim3((unsigned)rows), dim3(RC_THREADS), 0, reinterpret_cast<cudaStream_t>(stream), 1,
                        true, (__nv_bfloat16*)qkv, row_stride, cos_t, sin_t, pos, slot_mapping, (__nv_bfloat16*)k_cache,
                        (__nv_bfloat16*)v_cache, Hq, Hkv, D);
}

extern "C" int ts_kv_gather(const void* k_cache, const void* v_cache, const int* block_table, int max_blocks,
                            const int* starts, const int* lens, int sequences, int max_len, int block_size, int kv_width,
                            void* out, void* stream) {
  if (sequences <= 0 || max_len <= 0) return 0;
  if (kv_width % 8 != 0 || block_size <= 0 || sequences > 65535) return -10;
  const int rows = (max_len + 127) / 128 * 128;
  kv_gather_kernel<<<dim3(rows / KV_GATHER_ROWS, sequences), KV_GATHER_ROWS * 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache, block_table, max_blocks, starts, lens, block_size, kv_width,
      (__nv_bfloat16*)out);
  return (int)cudaGetLastError();
}

namespace ts {

template <int D, bool CLUSTER, bool EXT, bool WIDE>
static int launch_decode(const void* q, int q_stride, const void* k_cache, const void* v_cache, const int* block_table,
                         int max_blocks, const int* seq_lens, void* out, int out_stride, float* part_out, float* part_lse,
                         int num_seqs, int Hq, int Hkv, int block_size, int chunk, int splits, float scale_log2, int window,
                         float cap_inv, float cap_log2, cudaStream_t st) {
  return launch_chained(decode_attention_kernel<D, CLUSTER, EXT, WIDE>, dim3(splits, Hkv, num_seqs), dim3(DEC_WARPS * 32), 0, st,
                        CLUSTER ? splits : 1, true, (const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k_cache,
                        (const __nv_bfloat16*)v_cache, block_table, max_blocks, seq_lens, (__nv_bfloat16*)out, out_stride, part_out,
                        part_lse, Hq, Hkv, block_size, chunk, splits, scale_log2, window, cap_inv, cap_log2);
}

template <int D, bool CLUSTER>
static auto pick_decode(bool ext, bool wide) {
  return ext ? (wide ? launch_decode<D, CLUSTER, true, true> : launch_decode<D, CLUSTER, true, false>)
             : (wide ? launch_decode<D, CLUSTER, false, true> : launch_decode<D, CLUSTER, false, false>);
}

}  // namespace ts

// Shares of a sequence's keys: 256 CTAs in all, at least 128 keys each.  Up to eight are merged inside the kernel; more (long sequences, few heads) cost a second
// launch and are taken where the eight would have more than 512 keys each.  Measured (us by splits, 8 kv heads, nothing cached):
// 1 x 10000 keys of 128 34 (8) / 28 (32), 4 x 10000 56 (4) / 50 (8) / 56 (16), 64 x 300 keys of 64 25.5 (1) / 31.7 (2), 16 x 300 of
// 128 17.4 (1, 2) / 24.6 (3).
// The rule knows the number of sequences and the longest, not the others: one long sequence among many short ones would be left to
// one CTA per head, 18 us for every 1000 keys of 128.  So no share is longer than DEC_MOST_KEYS: 63 of 100 keys and one of 60000
// 1018 -> 293 us (5 splits).  Shorter shares cost even batches: 32 x 9000 204 us whole, 218 in two, 222 in three.
extern "C" int ts_decode_splits(int num_seqs, int Hkv, int max_len) {
  const long long ctas = static_cast<long long>(num_seqs) * Hkv;
  int want = ctas > 0 ? static_cast<int>((256 + ctas - 1) / ctas) : 1;
  const int most = max_len / 128;
  if (want > most) want = most;
  if (want > DEC_MAX_CLUSTER && max_len <= DEC_MAX_CLUSTER * 512) want = DEC_MAX_CLUSTER;
  const int least = static_cast<int>((max_len + static_cast<long long>(DEC_MOST_KEYS) - 1) / DEC_MOST_KEYS);
  return want > least ? want : least < 1 ? 1 : least;
}

// chunk: least number of keys of a split (multiples of 16 keep whole cache blocks together); splits * chunk may exceed the keys.
// splits > 8 (DEC_MAX_CLUSTER): part_out fp32 [num_seqs][Hq][splits][D], part_lse fp32 [num_seqs][Hq][splits] (caller-provided
// workspace); else they are not used.  window > 0: the last `window` keys of a sequence only; softcap > 0: scaled scores become
// softcap * tanh(score / softcap).
extern "C" int ts_decode_attention_ex(const void* q, int q_stride, const void* k_cache, const void* v_cache,
                                      const int* block_table, int max_blocks, const int* seq_lens, void* out,
                                      int out_stride, float* part_out, float* part_lse, int num_seqs, int Hq, int Hkv,
                                      int D, int block_size, int chunk, int splits, float scale, int window, float softcap,
                                      void* stream) {
  if (num_seqs <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv != 0 || Hq / Hkv > DEC_MAX_GROUP || (D != 64 && D != 128) || splits <= 0 || Hkv > 65535)
    return -10;
  if ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15u) return -11;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const float log2e = 1.4426950408889634f;
  const bool cluster = splits <= DEC_MAX_CLUSTER;
  const bool ext = window > 0 || softcap > 0.f, wide = Hq / Hkv > 4;
  auto launch = D == 128 ? (cluster ? pick_decode<128, true>(ext, wide) : pick_decode<128, false>(ext, wide))
                         : (cluster ? pick_decode<64, true>(ext, wide) : pick_decode<64, false>(ext, wide));
  int rc = 0;
  for (int s0 = 0; s0 < num_seqs && !rc; s0 += 65535) {          // the grid's third dimension ends there
    const size_t part = static_cast<size_t>(s0) * Hq * splits;
    rc = launch((const __nv_bfloat16*)q + static_cast<size_t>(s0) * q_stride, q_stride, k_cache, v_cache,
                block_table + static_cast<size_t>(s0) * max_blocks, max_blocks, seq_lens + s0,
                (__nv_bfloat16*)out + static_cast<size_t>(s0) * out_stride, out_stride, cluster ? nullptr : part_out + part * D,
                cluster ? nullptr : part_lse + part, num_seqs - s0 < 65535 ? num_seqs - s0 : 65535, Hq, Hkv, block_size, chunk, splits,
                scale * log2e, window, softcap > 0.f ? scale / softcap : 0.f, softcap > 0.f ? softcap * log2e : 0.f, st);
  }
  if (rc || cluster) return rc;
  if (D == 128)
    decode_merge_kernel<128><<<dim3(num_seqs, Hq), 128, 0, st>>>(part_out, part_lse, (__nv_bfloat16*)out, out_stride, Hq, splits);
  else
    decode_merge_kernel<64><<<dim3(num_seqs, Hq), 64, 0, st>>>(part_out, part_lse, (__nv_bfloat16*)out, out_stride, Hq, splits);
  return (int)cudaGetLastError();
}

extern "C" int ts_decode_attention(const void* q, int q_stride, const void* k_cache, const void* v_cache,
                                   const int* block_table, int max_blocks, const int* seq_lens, void* out,
                                   int out_stride, float* part_out, float* part_lse, int num_seqs, int Hq, int Hkv,
                                   int D, int block_size, int chunk, int splits, float scale, void* stream) {
  return ts_decode_attention_ex(q, q_stride, k_cache, v_cache, block_table, max_blocks, seq_lens, out, out_stride, part_out, part_lse,
                                num_seqs, Hq, Hkv, D, block_size, chunk, splits, scale, 0, 0.f, stream);
}
