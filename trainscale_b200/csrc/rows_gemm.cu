// Products of a few hundred token rows with a weight matrix: out[r, n] = sum_k X[r, k] W[n, k] (tcgen05 / TMEM / TMA).
//
// Serving multiplies a few rows with every weight of the model, so the cost is one pass over the weights.  Tiles of 128 TOKEN
// rows leave most of a tensor-core tile empty and give a projection of N columns N / 128 (or N / 64) CTAs, each of which has to
// pull its whole share of the weights through one shared-memory ring: 16 to 48 CTAs for the projections of a small model.  Here the WEIGHTS are the 128 rows of the MMA, tokens its N columns (a multiple of 16), and the reduction of one
// 128-row weight tile is split over a cluster of up to eight CTAs, so that (almost) every SM streams weights.  Per CTA:
//   warp 0      TMA producer: 128x64 weight and (tokens)x64 activation blocks into a ring sized for two CTAs per SM
//   warp 1      MMA issuer: D[128 weight rows][tokens] in TMEM
//   warps 2..5  TMEM -> shared memory, fp32 [token][128] (over the ring, which is drained by then)
//   all warps   sum of the cluster's partial results through distributed shared memory, in rank order (the same bits every
//               time); every rank finishes its own share of the tokens
// Gated products: a tile is 64 gate rows and the 64 up rows of the same outputs (the two halves of a gate|up matrix), which meet
// in the last step: act(gate) * up is rounded once.
#include "common.cuh"
#include "host_common.h"

namespace ts {

constexpr int RG_THREADS = 192;
constexpr int RG_W_BYTES = 128 * 64 * 2;     // a weight block of the ring
constexpr int RG_TOKENS = 128;               // token rows of a CTA; grid.y walks further ones, whose weights then come from L2
constexpr int RG_MAX_STAGES = 8;
constexpr int RG_RING = 108 * 1024;

struct RowsGemmParams {
  int M, N, K;              // token rows, outputs (gated: half of the weight rows), reduction
  int mt;                   // token rows of a CTA: M rounded up to 16, at most RG_TOKENS
  int stages, k_blocks, splits;
  void* out;
  size_t out_bytes;         // extent of the result (debug build)
  long long ldo;
  int out_fp32;
};

// ACT of a gated product: 0 silu, 1 gelu, 2 gelu (tanh form); -1: not gated
template <int ACT>
__device__ __forceinline__ float rows_glu(float g, float u) {
  if (ACT == 0) return g / (1.f + expf(-g)) * u;
  if (ACT == 1) return 0.5f * g * (1.f + erff(g * 0.70710678118654752f)) * u;
  return 0.5f * g * (1.f + tanhf(0.7978845608f * (g + 0.044715f * g * g * g))) * u;
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t cta) {
  float4 v;
  asm volatile(
      "{\n\t"
      ".reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t"
      "}\n"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(addr), "r"(cta)
      : "memory");
  return v;
}

template <int ACT>
__global__ void __launch_bounds__(RG_THREADS)
rows_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, RowsGemmParams p) {
  constexpr bool GLU = ACT >= 0;
  constexpr int COLS = GLU ? 64 : 128;         // outputs of a tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int x_bytes = p.mt * 128, stage_bytes = RG_W_BYTES + x_bytes;
  __shared__ uint64_t bars[2 * RG_MAX_STAGES + 1];
  __shared__ uint32_t tmem_slot;
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + RG_MAX_STAGES;
  uint64_t* acc_bar = bars + 2 * RG_MAX_STAGES;
  float* part = reinterpret_cast<float*>(smem);          // [mt][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = p.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int n0 = static_cast<int>(blockIdx.x) / p.splits * COLS;
  const int m0 = static_cast<int>(blockIdx.y) * RG_TOKENS, m = min(p.M - m0, RG_TOKENS);
  const int kb0 = static_cast<int>(static_cast<long long>(p.k_blocks) * rank / p.splits);
  const int kb1 = static_cast<int>(static_cast<long long>(p.k_blocks) * (rank + 1) / p.splits);
  uint32_t tmem_cols = 32;
  while (tmem_cols < static_cast<uint32_t>(p.mt)) tmem_cols *= 2;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_bar, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, tmem_cols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  bool alive = true;

  auto load_w = [&](int s, int kb) {
    uint8_t* dst = smem + s * stage_bytes;
    mbar_expect_tx(&full_bar[s], stage_bytes);
    tma_load_2d(dst, &tmW, &full_bar[s], kb * 64, n0);
    if (GLU) tma_load_2d(dst + RG_W_BYTES / 2, &tmW, &full_bar[s], kb * 64, p.N + n0);
  };
  auto load_x = [&](int s, int kb) {
    tma_load_2d(smem + s * stage_bytes + RG_W_BYTES, &tmX, &full_bar[s], kb * 64, m0);
  };
  grid_trigger();                    // (this block has its TMEM)
  // the first weights come while the kernels before may still be running
  const int ahead = min(p.stages, kb1 - kb0);
  const bool producer = warp == 0 && elect_one_sync();
  if (producer)
    for (int it = 0; it < ahead; ++it) load_w(it, kb0 + it);
  __syncwarp();
  grid_wait();

  if (warp == 0) {
    if (producer) {
      int it = 0;
      for (; it < ahead; ++it) load_x(it, kb0 + it);
      for (int kb = kb0 + ahead; kb < kb1; ++kb, ++it) {
        const int s = it % p.stages;
        if (!mbar_wait(&empty_bar[s], ((it / p.stages) & 1u) ^ 1u, alive, 100)) break;
        load_w(s, kb);
        load_x(s, kb);
      }
      if (!alive) {
        // tear-down after a failed wait: give the loads that are still in flight a bounded time to land
        for (int i = it > p.stages ? it - p.stages : 0; i < it; ++i) {
          const long long t0 = clock64();
          while (!mbar_try_wait(&full_bar[i % p.stages], (i / p.stages) & 1u) && clock64() - t0 < 2000000ll) {
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      const uint32_t idesc = make_idesc(128, p.mt, 1, 1, 0, 0);
      int it = 0;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % p.stages;
        if (!mbar_wait(&full_bar[s], (it / p.stages) & 1u, alive, 200)) break;
        tc_fence_after_sync();
        const uint32_t w = smem_u32(smem + s * stage_bytes), x = w + RG_W_BYTES;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16_ss(tmem_base, make_smem_desc_sw128(w + k * 32, 16, 1024), make_smem_desc_sw128(x + k * 32, 16, 1024), idesc,
                      (it | k) != 0);
        umma_commit(&empty_bar[s]);
      }
      if (alive) umma_commit(acc_bar);
    }
  } else {
    // every load has been consumed when the accumulator is complete, so its ring can hold the partial results
    const int q = warp & 3;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    if (mbar_wait(acc_bar, 0, alive, 300)) {
      tc_fence_after_sync();
#pragma unroll 1
      for (int c = 0; c < p.mt; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_row + c, r);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) part[(c + j) * 128 + q * 32 + lane] = __uint_as_float(r[j]);
      }
      tc_fence_before_sync();
    }
  }
  __syncwarp();
  __syncthreads();
  if (p.splits > 1) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, tmem_cols);
  }

  // tokens rank, rank + splits, ...: four outputs per thread
  constexpr int VECS = COLS / 4;
  const int mine = m > rank ? (m - rank + p.splits - 1) / p.splits : 0;
  const uint32_t base = smem_u32(part);
  for (int i = threadIdx.x; i < mine * VECS; i += RG_THREADS) {
    const int t = rank + i / VECS * p.splits, c = i % VECS * 4;
    const uint32_t at = base + (t * 128 + c) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f), u = v;
    if (p.splits == 1) {
      v = *reinterpret_cast<const float4*>(part + t * 128 + c);
      if (GLU) u = *reinterpret_cast<const float4*>(part + t * 128 + 64 + c);
    } else {
      float4 a[8], b[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        if (s < p.splits) {
          a[s] = ld_cluster_f4(at, s);
          if (GLU) b[s] = ld_cluster_f4(at + 256, s);
        }
      }
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        if (s < p.splits) {
          v.x += a[s].x; v.y += a[s].y; v.z += a[s].z; v.w += a[s].w;
          if (GLU) {
            u.x += b[s].x; u.y += b[s].y; u.z += b[s].z; u.w += b[s].w;
          }
        }
      }
    }
    if (GLU) v = make_float4(rows_glu<ACT>(v.x, u.x), rows_glu<ACT>(v.y, u.y), rows_glu<ACT>(v.z, u.z), rows_glu<ACT>(v.w, u.w));
    const int n = n0 + c;
    if (n >= p.N) continue;
    const float f[4] = {v.x, v.y, v.z, v.w};
    if (p.out_fp32) {
      float* dst = reinterpret_cast<float*>(p.out) + (m0 + t) * p.ldo + n;
      if (!TS_IN_BOUNDS(dst, min(4, p.N - n) * 4, p.out, p.out_bytes, 7200)) continue;
      if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        *reinterpret_cast<float4*>(dst) = v;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) dst[j] = f[j];
      }
    } else {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + (m0 + t) * p.ldo + n;
      if (!TS_IN_BOUNDS(dst, min(4, p.N - n) * 2, p.out, p.out_bytes, 7200)) continue;
      if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) dst[j] = __float2bfloat16(f[j]);
      }
    }
  }
  if (p.splits > 1) cluster_sync_all();      // nobody leaves while a peer may still read its partial results
}

// CTAs of a weight tile: as many (1, 2, 4, 8) as keep all CTAs resident at once, with at least four 64-wide blocks of the
// reduction for each.  Measured against every other split (1 - 8) and rings of 54 and 200 KB: within 7 % of the best.
static int rows_splits(int tiles, int k_blocks, int resident) {
  int s = 1;
  while (s < 8 && tiles * s * 2 <= resident && k_blocks >= s * 2 * 4) s *= 2;
  return s;
}

template <int ACT>
static int launch_rows(const CUtensorMap& tW, const CUtensorMap& tX, const RowsGemmParams& p, int tiles, size_t smem, bool chained, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(rows_gemm_kernel<ACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, RG_RING + 1024);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const dim3 grid((unsigned)(tiles * p.splits), (unsigned)((p.M + RG_TOKENS - 1) / RG_TOKENS));
  return launch_chained(rows_gemm_kernel<ACT>, grid, dim3(RG_THREADS), smem, st, p.splits, chained, tW, tX, p);
}

}  // namespace ts

TS_DEFINE_ERROR_API(ts_rows_gemm)
using namespace ts;

// X [M][ldx], W [rows][ldw], out [M][ldo] (bf16, or fp32 with out_fp32).  glu < 0: W has N rows.  glu 0 silu, 1 gelu, 2 gelu in its
// tanh form: W has 2 N rows, gates first, out = act(gate) * up.  Rows of X and W are 16-byte aligned.  chained: see launch_chained;
// no chained kernel and not the last ordinary one before them may write W.
extern "C" int ts_rows_gemm(const void* X, const void* W, void* out, int M, int N, int K, long long ldx, long long ldw,
                            long long ldo, int out_fp32, int glu, int chained, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || glu > 2) return -10;
  RowsGemmParams p;
  p.M = M; p.N = N; p.K = K; p.out = out; p.ldo = ldo; p.out_fp32 = out_fp32;
  p.out_bytes = (static_cast<size_t>(M - 1) * ldo + N) * (out_fp32 ? 4 : 2);
  p.mt = M > RG_TOKENS ? RG_TOKENS : (M + 15) / 16 * 16;
  p.k_blocks = (K + 63) / 64;
  const int cols = glu >= 0 ? 64 : 128, tiles = (N + cols - 1) / cols, blocks = (M + RG_TOKENS - 1) / RG_TOKENS;
  // two CTAs share an SM: one fills its ring while the other finishes
  const int stage = RG_W_BYTES + p.mt * 128;
  p.splits = rows_splits(tiles * blocks, p.k_blocks, 2 * sm_count());
  p.stages = RG_RING / stage;
  if (p.stages > RG_MAX_STAGES) p.stages = RG_MAX_STAGES;
  const int longest = (p.k_blocks + p.splits - 1) / p.splits;
  if (p.stages > longest) p.stages = longest;
  size_t ring = static_cast<size_t>(p.stages) * stage;
  const size_t part = static_cast<size_t>(p.mt) * 512;
  if (ring < part) ring = part;
  const size_t smem = ring + 1024;
  CUtensorMap tW, tX;
  int rc = make_tmap_2d(&tW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)N * (glu >= 0 ? 2 : 1), (uint64_t)K, (uint64_t)ldw,
                        (uint32_t)cols, 64);
  if (rc) return rc * 100 - 1;
  rc = make_tmap_2d(&tX, X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, (uint32_t)p.mt, 64);
  if (rc) return rc * 100 - 2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (glu < 0) return launch_rows<-1>(tW, tX, p, tiles, smem, chained != 0, st);
  if (glu == 0) return launch_rows<0>(tW, tX, p, tiles, smem, chained != 0, st);
  if (glu == 1) return launch_rows<1>(tW, tX, p, tiles, smem, chained != 0, st);
  return launch_rows<2>(tW, tX, p, tiles, smem, chained != 0, st);
}
