// Linear layers of few rows (decoded tokens, short text streams): C[M, N] = epilogue(A[M, K] W[N, K]^T) for M <= 128.  The time
// is that of streaming W from HBM plus a launch's fixed chain of latencies, and a tile per 128..256 columns leaves most SMs
// idle (16 tiles of 128 columns for a 2048-wide layer).
//
// gemm_rows_kernel     M <= 24: 16 columns of C per block, the contraction dealt out to its warps.  W goes from HBM straight into
//                      MMA fragments: no shared-memory ring, no barriers and no tensor memory to set up, which is what a
//                      launch of a few microseconds is made of.
// gemm_skinny_kernel   M <= 128: the operands change places, 128 rows of W are the M side of a tcgen05 MMA and MT = 32 / 64 /
//                      128 rows of A its N side; the contraction is split over the S = 1, 2, 4 or 8 CTAs of a cluster, each
//                      streaming its own K range through a TMA ring.  Partial sums (fp32) meet over distributed shared
//                      memory in rank order: the result does not depend on timing.
#pragma once
#include "host_util.h"
#include "ptx_sm100.cuh"

namespace omni {

template <int MT, bool ALONE>
struct SkinnyCfg {
  static constexpr int A_BYTES = 128 * 128;                 // 128 rows of W x 64 bf16
  static constexpr int STAGE_BYTES = A_BYTES + MT * 128;
  static constexpr int STAGES = (ALONE ? 200 * 1024 : 108 * 1024) / STAGE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
  static constexpr int TMEM_COLS = MT < 32 ? 32 : MT;
  static_assert(MT * 128 * 4 <= STAGES * STAGE_BYTES, "partial sums reuse the ring");
};
constexpr int SKINNY_THREADS = 192;   // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue (TMEM quadrant = warp & 3)

__device__ __forceinline__ float ld_shared_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// bias, activation, gate, residual and the store of B rows m, m + step, ... of column n.  All operands are read before the
// first store, because the residual may be the output.
template <int B>
__device__ __forceinline__ void skinny_finish(float (&x)[B], int m, int step, int M, int n, __nv_bfloat16* __restrict__ C, int ldc,
                                              const GemmEpilogue& epi, float bias) {
  float add[B];
#pragma unroll
  for (int j = 0; j < B; ++j) {
    x[j] += bias;
    const int r = m + j * step;
    add[j] = epi.residual && r < M ? __bfloat162float(epi.residual[(size_t)r * epi.ldr + n]) : 0.f;
  }
  if (epi.act == ACT_GELU_TANH) {
#pragma unroll
    for (int j = 0; j < B; ++j) x[j] = gelu_tanh(x[j]);
  } else if (epi.act == ACT_SILU) {
#pragma unroll
    for (int j = 0; j < B; ++j) x[j] = silu(x[j]);
  } else if (epi.act == ACT_RELU2) {
#pragma unroll
    for (int j = 0; j < B; ++j) x[j] = fmaxf(x[j], 0.f) * fmaxf(x[j], 0.f);
  } else if (epi.act == ACT_XIELU) {
#pragma unroll
    for (int j = 0; j < B; ++j) x[j] = xielu(x[j], epi.act_c0, epi.act_c1);
  }
  if (epi.gate) {
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int r = m + j * step;
      if (r < M) x[j] *= __bfloat162float(epi.gate[(size_t)(r / epi.rows_per_batch) * epi.gate_stride + n]);
    }
  }
#pragma unroll
  for (int j = 0; j < B; ++j) {
    const int r = m + j * step;
    if (r < M) {
      __nv_bfloat16* out = C + (size_t)r * ldc;
      if (epi.c_rows_per_batch > 0) {
        const int cb = r / epi.c_rows_per_batch;
        out = C + (size_t)cb * epi.c_batch_stride + (size_t)(r - cb * epi.c_rows_per_batch) * ldc;
      }
      out[n] = __float2bfloat16(x[j] + add[j]);
    }
  }
}

// ---------------------------------------------------------------------------------------------------- at most 24 rows
// NT * 8 rows of A; 16 resident warps x U chunks x 1 KB = up to 128 KB of W in flight per SM.
// GATED: W holds N / 2 gate rows and then their lift rows; a block makes 8 columns of C, silu(gate) * lift, from 8 rows of each.
template <int NT, int NW, int U, int BLOCKS, bool GATED>
__global__ void __launch_bounds__(32 * NW, BLOCKS)
gemm_rows_kernel(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, __nv_bfloat16* C, int ldc,
                 int M, int N, int K, const __grid_constant__ GemmEpilogue epi, int resident) {
  __shared__ float part[NW][NT * 8][16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  const int n0 = blockIdx.x * 16;
  auto w_row = [&](int i) { return GATED ? min(n0 / 2 + (i & 7), N / 2 - 1) + (i >> 3) * (N / 2) : min(n0 + i, N - 1); };
  if ((int)blockIdx.x < resident) {             // W does not come from the kernel before: the first blocks' share is on its way to L2 meanwhile
    const __nv_bfloat16* w = W + (size_t)w_row(threadIdx.x & 15) * ldw;
    for (int c = (threadIdx.x >> 4) * 64; c < K; c += 2 * NW * 64) prefetch_l2(w + c);
  }
  pdl_begin();
  const __nv_bfloat16* x[NT];
  float acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    x[t] = t * 8 + g < M ? A + (size_t)(t * 8 + g) * lda : nullptr;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
  }
  // columns past N repeat the last one and are not stored
  few_rows_products<NT, NW, U>(acc, W + (size_t)w_row(g) * ldw, W + (size_t)w_row(8 + g) * ldw, x, K, warp, j);
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) part[warp][t * 8 + j * 2 + (i & 1)][g + 8 * (i >> 1)] = acc[t][i];
  __syncthreads();
  if constexpr (GATED) {
    for (int e = threadIdx.x; e < NT * 64; e += 32 * NW) {
      const int n = n0 / 2 + (e & 7), m = e >> 3;
      if (n < N / 2 && m < M) {
        float gate = 0.f, lift = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          gate += part[w][m][e & 7];
          lift += part[w][m][8 + (e & 7)];
        }
        C[(size_t)m * ldc + n] = __float2bfloat16(silu(gate) * lift);
      }
    }
    return;
  }
#pragma unroll
  for (int e = threadIdx.x; e < NT * 128; e += 32 * NW) {
    const int n = n0 + (e & 15), m = e >> 4;
    if (n < N && m < M) {
      const float bias = epi.bias ? __bfloat162float(epi.bias[n]) : 0.f;
      float y[1] = {0.f};
#pragma unroll
      for (int w = 0; w < NW; ++w) y[0] += part[w][m][e & 15];
      skinny_finish<1>(y, m, 1, M, n, C, ldc, epi, bias);
    }
  }
}

// How a tile's contraction is split over warps (NW), loads in flight per warp (U) and blocks on an SM, by the number of 16-column
// tiles per SM.  Measured with 8 and 16 rows in us, streaming the weights from memory:
//   up to one    a block of 16 warps, so that a long contraction still is one or two rounds of loads: 2048 x 9216 12.7 / 15.2 with
//                8 warps, 9.8 / 11.0 with 16; a contraction of at most 1024 is one round with 8 warps, 2.6 / 2.6 against 2.9 / 2.9
//   two to three three blocks of 8 with half the loads, since two blocks would leave a second round that is nearly empty:
//                6144 x 4096 14.0 / 17.4 with two blocks, 11.4 / 14.3 with three; 5120 x 2048 7.0 / 9.7 and 6.2 / 7.4
//   more, 9 rows and up: four blocks of 4 warps where their last round is at least half full (24576 x 4096 46.1 with two blocks
//                of 8, 42.1 with four of 4; 9216 x 2048 10.2 and 9.2), not where it is emptier (12288 x 4096 25.3 and 27.8)
//   else         two blocks of 8 (8 rows, 32768 x 4096: 46.2; four of 4 48.0, three of 8 47.9; the copy rate would be 40.4)
// 17 to 24 rows, whose products leave registers for fewer loads (17 and 24 rows; gemm_skinny_kernel in brackets): up to one tile per SM 16 warps
// (2048 x 6144 8.1 / 8.7 (10.0)), up to two two blocks of 8 with twice the loads (4096 x 4096 9.1 / 9.8 (10.6)), up to three those with half
// (6144 x 4096 12.2 / 13.3 (14.3)), more four of 4 (9216 x 2048 9.4 / 10.2 (11.6)), with half the loads past a round of them (12288 x 2048 12.0 / 12.8 (14.9)).
template <int NT, bool GATED>
static void launch_rows(int tiles, const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, __nv_bfloat16* C, int ldc, int M,
                        int N, int K, const GemmEpilogue& epi, cudaStream_t stream) {
  constexpr int U = NT == 1 ? 8 : 4;
  const int sms = sm_count(), last = tiles % (4 * sms);
  const auto go = [&](auto kernel, int warps, int blocks) {
    launch_overlapped(kernel, tiles, 32 * warps, 0, stream, A, lda, W, ldw, C, ldc, M, N, K, epi, blocks * sms);
  };
  if constexpr (NT == 3) {
    if (tiles <= sms) go(gemm_rows_kernel<3, 16, 2, 1, GATED>, 16, 1);
    else if (tiles <= 2 * sms) go(gemm_rows_kernel<3, 8, 4, 2, GATED>, 8, 2);
    else if (tiles <= 3 * sms) go(gemm_rows_kernel<3, 8, 2, 2, GATED>, 8, 2);
    else if (tiles <= 4 * sms) go(gemm_rows_kernel<3, 4, 4, 4, GATED>, 4, 4);
    else go(gemm_rows_kernel<3, 4, 2, 4, GATED>, 4, 4);
  } else if (tiles <= sms && K > 1024) go(gemm_rows_kernel<NT, 16, U, 1, GATED>, 16, 1);
  else if (tiles > 2 * sms && tiles <= 3 * sms) go(gemm_rows_kernel<NT, 8, U / 2, 3, GATED>, 8, 3);
  else if (NT == 2 && tiles > 3 * sms && (last == 0 || last >= 2 * sms)) go(gemm_rows_kernel<NT, 4, U, 4, GATED>, 4, 4);
  else go(gemm_rows_kernel<NT, 8, U, 2, GATED>, 8, 2);
}

static int launch_rows(const void* A, int lda, const void* W, int ldw, __nv_bfloat16* C, int ldc, int M, int N, int K,
                       const GemmEpilogue& epi, cudaStream_t stream) {
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) return RC_BAD_ARG;
  const auto a = static_cast<const __nv_bfloat16*>(A), w = static_cast<const __nv_bfloat16*>(W);
  const int tiles = (N + 15) / 16;
  const bool gated = epi.act == EPI_SWIGLU;
  const auto go = M <= 8 ? (gated ? launch_rows<1, true> : launch_rows<1, false>)
                : M <= 16 ? (gated ? launch_rows<2, true> : launch_rows<2, false>) : (gated ? launch_rows<3, true> : launch_rows<3, false>);
  go(tiles, a, lda, w, ldw, C, ldc, M, N, K, epi, stream);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------- 17 to 128 rows
template <int MT, int S, bool ALONE>
__global__ void __launch_bounds__(SKINNY_THREADS)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, __nv_bfloat16* __restrict__ C,
                   int ldc, int M, int N, int K, const __grid_constant__ GemmEpilogue epi, int* status) {
  using Cfg = SkinnyCfg<MT, ALONE>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t done_bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = S > 1 ? (int)cluster_ctarank() : 0;
  const int n0 = (blockIdx.x / S) * 128;
  const int num_kb = (K + 63) / 64;
  const int kb0 = rank * num_kb / S, kb1 = (rank + 1) * num_kb / S;      // never empty: the launcher keeps num_kb >= S
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    mbar_init(smem_u32(&done_bar), 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  if (threadIdx.x == 0)
    for (int kb = kb0; kb < kb1 && kb < kb0 + 16; ++kb) tma_prefetch_2d(&tmW, kb * 64, n0);
  pdl_begin();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
        const uint32_t fb = smem_u32(&full_bar[stage]);
        const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
        mbar_expect_tx(fb, Cfg::STAGE_BYTES);
        tma_load_2d(sa, &tmW, fb, kb * 64, n0);
        tma_load_2d(sa + Cfg::A_BYTES, &tmX, fb, kb * 64, 0);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc(128, MT, 1, 1, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(smem_u32(&full_bar[stage]), phase, &s_abort, status, ERR_WAIT_FULL);
        tc_fence_after_sync();
        const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
        const uint64_t w_desc = umma_desc_kmajor_sw128(sa), x_desc = umma_desc_kmajor_sw128(sa + Cfg::A_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_ss(tmem_base, w_desc + 2 * k, x_desc + 2 * k, idesc, kb != kb0 || k != 0);
        tc_commit(smem_u32(&empty_bar[stage]));
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      tc_commit(smem_u32(&done_bar));
    }
  } else {
    const int q = warp & 3;
    const int n = n0 + q * 32 + lane;
    const float bias = epi.bias && n < N ? __bfloat162float(epi.bias[n]) : 0.f;
    mbar_wait(smem_u32(&done_bar), 0, &s_abort, status, ERR_WAIT_TMEM_FULL);
    tc_fence_after_sync();
    // a lane holds one column of C, the registers 16 of its rows
#pragma unroll 1
    for (int c = 0; c < MT && (S > 1 || c < M); c += 16) {
      uint32_t v[16];
      tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + c, v);
      tmem_wait_ld();
      if (S > 1) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(smem_base + ((c + j) * 128 + q * 32 + lane) * 4), "r"(v[j]) : "memory");
      } else if (n < N) {
        float x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = __uint_as_float(v[j]);
        skinny_finish<16>(x, c, 1, M, n, C, ldc, epi, bias);
      }
    }
    tc_fence_before_sync();
  }
  __syncthreads();
  if (S > 1) {
    cluster_sync_all();                                     // every rank's partial sums lie in its shared memory
    if (warp >= 2) {
      const int col = (warp & 3) * 32 + lane, n = n0 + col;
      const float bias = epi.bias && n < N ? __bfloat162float(epi.bias[n]) : 0.f;
      uint32_t src[S];
#pragma unroll
      for (int s = 0; s < S; ++s) src[s] = mapa_shared(smem_base + col * 4, s);
      if (n < N) {
        constexpr int B = MT / S < 8 ? MT / S : 8;
#pragma unroll 1
        for (int m = rank; m < M; m += B * S) {             // rows of C are dealt out to the ranks, B at a time
          float x[B];
#pragma unroll
          for (int j = 0; j < B; ++j) {
            float p[S];                                     // rows past M are zero products: there to be read, never stored
#pragma unroll
            for (int s = 0; s < S; ++s) p[s] = ld_shared_cluster_f32(src[s] + (m + j * S) * 512);
            x[j] = p[0];
#pragma unroll
            for (int s = 1; s < S; ++s) x[j] += p[s];
          }
          skinny_finish<B>(x, m, S, M, n, C, ldc, epi, bias);
        }
      }
    }
    __syncthreads();
    cluster_sync_all();                                     // no rank leaves while another reads its shared memory
  }
  if (s_abort) {                                            // copies and MMAs in flight land before the memory is handed back
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

template <int MT, int S, bool ALONE>
static int launch_skinny_s(const CUtensorMap& tmX, const CUtensorMap& tmW, __nv_bfloat16* C, int ldc, int M, int N, int K,
                           const GemmEpilogue& epi, int* status, cudaStream_t stream) {
  static unsigned long long prepared = 0;
  if (int e = ensure_dynamic_smem((const void*)gemm_skinny_kernel<MT, S, ALONE>, SkinnyCfg<MT, ALONE>::SMEM_BYTES, prepared)) return e;
  launch_with(true, S, gemm_skinny_kernel<MT, S, ALONE>, (unsigned)((N + 127) / 128 * S), SKINNY_THREADS, SkinnyCfg<MT, ALONE>::SMEM_BYTES, stream,
              tmX, tmW, C, ldc, M, N, K, epi, status);
  return (int)cudaGetLastError();
}

// CTAs that one SM holds one of (ALONE) all run at once up to as many clusters as the device places; whole clusters do not use every SM of
// a group of SMs, so that is less than the SMs divided by S: 37 tiles of 4 CTAs would be one cluster short of a round (48 rows 4736 x 2048
// took 15.5 us, the general kernel 12.1).
template <int MT, int S>
static int clusters_alone() {
  static int cached = 0;
  if (cached) return cached;
  int n = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sm_count() / S * S);
  cfg.blockDim = dim3(SKINNY_THREADS);
  cfg.dynamicSmemBytes = SkinnyCfg<MT, true>::SMEM_BYTES;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = S; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  static unsigned long long prepared = 0;
  if (ensure_dynamic_smem((const void*)gemm_skinny_kernel<MT, S, true>, SkinnyCfg<MT, true>::SMEM_BYTES, prepared) ||
      cudaOccupancyMaxActiveClusters(&n, gemm_skinny_kernel<MT, S, true>, &cfg) != cudaSuccess)
    n = 0;
  (void)cudaGetLastError();
  return cached = n > 0 ? n : 1;
}

// CTAs per tile: up to about 200 in all (two share an SM), each with at least two K blocks.
// us with a limit of 148, 200, 296: 64 rows 3072 x 4096 9.9, 9.5, 9.4; 6144 x 4096 15.5, 16.9, 16.9; 9216 x 2048 12.7, 12.7, 18.7.
static int skinny_split(int N, int K) {
  const int tiles = (N + 127) / 128, num_kb = (K + 63) / 64;
  for (int s = 8; s > 1; s >>= 1)
    if (tiles * s <= 200 && num_kb >= 2 * s) return s;
  return 1;
}

template <int MT>
static int launch_skinny_mt(const CUtensorMap& tmW, const void* A, int lda, __nv_bfloat16* C, int ldc, int M, int N, int K,
                            const GemmEpilogue& epi, int split, int* status, cudaStream_t stream) {
  CUtensorMap tmX;
  if (int rc = make_tmap_2d(&tmX, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, MT, 64)) return rc;
  const int tiles = (N + 127) / 128;
#define OMNI_SKINNY(S)                                                                                                           \
  return tiles <= clusters_alone<MT, S>() ? launch_skinny_s<MT, S, true>(tmX, tmW, C, ldc, M, N, K, epi, status, stream)         \
                                          : launch_skinny_s<MT, S, false>(tmX, tmW, C, ldc, M, N, K, epi, status, stream)
  // clusters of 8 CTAs do not fit every GPC's SMs one by one
  if (split == 8) return launch_skinny_s<MT, 8, false>(tmX, tmW, C, ldc, M, N, K, epi, status, stream);
  if constexpr (MT < 128) {                // few_rows() leaves 128 rows 49 tiles at most, of 16 K blocks at least
    if (split == 2) OMNI_SKINNY(2);
    if (split == 1) OMNI_SKINNY(1);
  }
  OMNI_SKINNY(4);
#undef OMNI_SKINNY
}

// Which problems leave the general kernels (tiles of 128 or 256 rows).
//   up to 16 rows    all but those whose rows of A do not stay in L1 (120 KB) between the blocks of an SM: every block reads them all, and past six
//                    blocks per SM, or four of very long rows, that costs more than it saves.  us, general kernel in brackets: 13 rows 16384 x 4096 30.0
//                    (37.3), 16 rows 16384 x 3584 28.3 (33.9), 16384 x 4096 31.5 (28.7), 13824 x 4096 24.4 (25.7), 12288 x 12288 1.05 times
//                    as long, 8192 x 4096 18.1 (20.5).  Up to 8 rows the products are half as many and it pays at any length.
//   17 to 24         gemm_rows_kernel up to 5 blocks per SM and contractions of 2048; of 9216, 4096, 4096 and 2560 with one to four where those fill four fifths of
//                    a round, and of 3072 and 2560 with three and four that do not.  17 and 24 rows on weights from memory, gemm_skinny_kernel in brackets: 10240 x 2048 12.8
//                    and 13.4 (13.2, 13.5), 2048 x 9216 11.6, 12.3 (12.3, 12.4), 4096 x 4096 9.5, 10.2 (10.7), 8192 x 2560 10.9, 11.7 (11.8); beyond: 1024 x 8192
//                    9.6, 10.0 (8.6), 2560 x 4096 9.2, 9.4 (8.5), 7168 x 4096 16.2, 17.3 (15.0), 10240 x 4096 23.8, 25.6 (21.0), 12288 x 4096 24.3, 25.4 (23.4).  A
//                    gated layer, for which the alternative is two launches: up to 9216, 4096 with two to four blocks per SM, 2560 with five (17 and 24 rows, two
//                    launches in brackets: 2560 x 4096 8.5, 9.0 (10.0), 8192 x 4096 16.0, 17.4 (17.4), 10240 x 3072 18.0, 19.0 (17.6), 12288 x 2048 12.3, 13.1 (16.5)).
//                    Which rows these are: steps that are not replayed from a captured batch (mixed ones, contexts past the captured tables),
//                    since captured batches have 16 or 32 rows and a vocabulary is wider than that
//   17 to 32         else up to as many tiles as SMs: 17 rows 10240 x 2048 12.5 (17.1), 12288 x 1024 8.0 (11.6), 32 rows 18432 x 2048 15.4 (16.7)
//   33 to 64         up to half as many; above, the general kernels stream W as fast and read A less often: 64 rows 9216 x 2048 12.7 (13.8),
//                    10240 x 2048 14.4 (13.2)
//   65 to 128        up to a third, and contractions long enough for the split: exchange and epilogue of 128 rows take 4 us, which a split
//                    wins back from 16 K blocks on and, with less to split by, from three quarters of the number of tiles: 128 rows 1536 x 768
//                    9.8 (9.2), 1536 x 1024 8.1 (10.0), 4096 x 1024 11.2 (10.0), 4096 x 2048 12.9 (13.0); 65 rows 4096 x 1536 10.3 (10.7)
enum class FewRows { no, rows, skinny };
static FewRows few_rows(int M, int N, int K, bool gated = false) {
  const int tiles = (N + 127) / 128, num_kb = (K + 63) / 64;
  if (M <= 16) {
    const long a_kb = (long)M * K * 2 / 1024, blocks = (N + 15) / 16;
    return M > 8 && ((a_kb > 120 && blocks > 6L * sm_count()) || (a_kb >= 384 && blocks > 4L * sm_count())) ? FewRows::no : FewRows::rows;
  }
  const long blocks = (N + 15) / 16;
  if (M <= 24 && blocks <= 5.25 * sm_count()) {
    const long rounds = (blocks + sm_count() - 1) / sm_count();
    const bool full = 5 * blocks >= 4 * rounds * sm_count();
    const int most = gated ? (rounds == 1 ? 9216 : rounds > 4 ? 2560 : 4096) : rounds > 4 ? 2048 : rounds == 4 ? 2560 : full ? (rounds == 1 ? 9216 : 4096) : rounds == 3 ? 3072 : 2048;
    if (K <= most) return FewRows::rows;
  }
  if (M <= 64) return tiles * (M <= 32 ? 1 : 2) <= sm_count() ? FewRows::skinny : FewRows::no;
  return M <= 128 && tiles * 3 <= sm_count() && num_kb >= 16 && num_kb * 4 >= tiles * 3 ? FewRows::skinny : FewRows::no;
}

static int launch_skinny(const void* A, int lda, const void* W, int ldw, __nv_bfloat16* C, int ldc, int M, int N, int K,
                         const GemmEpilogue& epi, int* status, cudaStream_t stream) {
  CUtensorMap tmW;
  if (int rc = make_tmap_2d(&tmW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)N, (uint64_t)K, (uint64_t)ldw * 2, 128, 64)) return rc;
  const int s = skinny_split(N, K);
  if (M <= 32) return launch_skinny_mt<32>(tmW, A, lda, C, ldc, M, N, K, epi, s, status, stream);
  if (M <= 64) return launch_skinny_mt<64>(tmW, A, lda, C, ldc, M, N, K, epi, s, status, stream);
  return launch_skinny_mt<128>(tmW, A, lda, C, ldc, M, N, K, epi, s, status, stream);
}

}  // namespace omni
