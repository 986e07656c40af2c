// Expert GEMMs over rows that sit back to back (mixture of experts, more than a few tokens):  C[r, n] = act(sum_k A[r, k] W[e(r), n, k]).
//
// The weights are the M side of the MMA (128 rows of W) and a tile's rows of A its N side, because experts get any number of rows: the N of an
// MMA goes in steps of 16, or of 32 on CTA pairs (154 rows cost 160, not the 256 of two 128-row tiles), every weight is fetched once per tile of up to
// 256 rows, and a tile of few rows leaves the shared memory to the weights' ring.  XR is the most rows a tile may have: 64 or 128 on single CTAs
// (expert_gemm_kernel), 256 on pairs (expert_pair_kernel).
// GATED: W [E, 2 N, K] holds gate and lift rows; one 5-D box brings 8 gate rows, their 8 lift rows, the next 8 gate rows and so on, so that both
// values of an output lie 8 lanes apart in a warp and silu(gate) * lift leaves the accumulators without passing through memory.
// 128 experts, 2048 -> 2 x 768 -> 2048, top 8, whole layer on cold caches: 64 tokens 200 us (two grouped launches of 128-row tiles around a SwiGLU
// kernel: 239), 256 tokens 211 us (241), 2463 tokens 290 us (about 440); the weights alone take 182 us.
#pragma once

namespace omni {

template <int XR>
struct ExpertCfg {
  static constexpr int W_BYTES = 128 * 128, STAGE_BYTES = W_BYTES + XR * 128;
  static constexpr int STAGES = 200 * 1024 / STAGE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
  static constexpr int ACC_STRIDE = XR, TMEM_COLS = 2 * XR;
};

struct ExpertArgs {
  CUtensorMap tmX, tmW;
  __nv_bfloat16* c;
  long ldc;
  int N, K;                                   // outputs per row, contraction
  const int *tile_expert, *tile_row0, *tile_rows;
  int max_tiles, act;
  int by16;                                   // rows of C begin on 16 bytes
};

// A warp's share of a finished tile: its 32 lanes of the accumulator, every other chunk of 16 rows; `out` and `cols` from the warp's first column on.  A lane
// holds a column of the result.  GATED: lanes of a gate row take the even rows of C, lanes of its lift row the odd ones, and store where they stand.  Else the
// chunk is turned in `turned` (1 KB of this warp) and leaves in pieces of 16 bytes where C lies on such: 16000 tokens of 128 x (768 -> 2048) on pairs 480 -> 349 us (427 -> 396 on
// single CTAs); the gated half as many stores are no faster that way (560 us, 611 turned).
template <bool GATED>
__device__ __forceinline__ void expert_drain(uint32_t acc, __nv_bfloat16* turned, __nv_bfloat16* out, int rows, int half, int lane, int cols, const ExpertArgs& a) {
  const bool lift = lane & 8;
  const int col = (lane >> 4) * 8 + (lane & 7);
#pragma unroll 1
  for (int c = half * 16; c < rows; c += 32) {
    uint32_t v[16];
    tmem_ld_32x16(acc + c, v);
    tmem_wait_ld();
    if (GATED) {
#pragma unroll
      for (int i = 0; i < 16; i += 2) {
        const float even = __uint_as_float(v[i]), odd = __uint_as_float(v[i + 1]);
        const float mine = lift ? odd : even, theirs = __shfl_xor_sync(0xffffffffu, lift ? even : odd, 8);
        const int r = c + i + (lift ? 1 : 0);
        if (r < rows && col < cols) out[(long)r * a.ldc + col] = __float2bfloat16(lift ? silu(theirs) * mine : silu(mine) * theirs);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float x = __uint_as_float(v[i]);
        if (a.act == ACT_RELU2) x = fmaxf(x, 0.f) * fmaxf(x, 0.f);
        turned[i * 32 + lane] = __float2bfloat16(x);
      }
      if (!a.by16) {                          // a lane's own column
        for (int i = 0; i < 16; ++i)
          if (c + i < rows && lane < cols) out[(long)(c + i) * a.ldc + lane] = turned[i * 32 + lane];
        continue;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = i * 8 + (lane >> 2), n = (lane & 3) * 8;
        if (c + r < rows && n < cols) *reinterpret_cast<uint4*>(out + (long)(c + r) * a.ldc + n) = *reinterpret_cast<const uint4*>(turned + r * 32 + n);
      }
      __syncwarp();
    }
  }
}

template <int XR, bool GATED>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
expert_gemm_kernel(const __grid_constant__ ExpertArgs a, int* status) {
  using Cfg = ExpertCfg<XR>;
  constexpr int STAGES = Cfg::STAGES, COLS = GATED ? 64 : 128;        // outputs per tile
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t tfull_bar[2];
  __shared__ __align__(8) uint64_t tempty_bar[2];
  __shared__ __align__(16) __nv_bfloat16 turned[8][GATED ? 8 : 512];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int num_n = (a.N + COLS - 1) / COLS, num_items = a.max_tiles * num_n, num_kb = (a.K + 63) / 64;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 8);
    }
    fence_mbar_init();
    tma_prefetch_desc(&a.tmX);
    tma_prefetch_desc(&a.tmW);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  pdl_begin();

  // item -> (tile of rows, block of outputs): neighbours share rows; the tiles of an expert follow one another and share its weights in L2.
  // Used tiles come first, so the walk ends at the first unused one.
  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int it = blockIdx.x; it < num_items; it += gridDim.x) {
        const int t = it / num_n, nb = it - t * num_n, e = a.tile_expert[t];
        if (e < 0) break;
        const int row0 = a.tile_row0[t], boxes = (a.tile_rows[t] + 63) / 64;
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
          const uint32_t fb = smem_u32(&full_bar[stage]), sa = smem_base + stage * Cfg::STAGE_BYTES;
          mbar_expect_tx(fb, Cfg::W_BYTES + boxes * 64 * 128);
          if (GATED) tma_load_5d(sa, &a.tmW, fb, kb * 64, 0, 0, nb * 8, e);
          else tma_load_3d(sa, &a.tmW, fb, kb * 64, nb * 128, e);
          for (int b = 0; b < boxes; ++b) tma_load_2d(sa + Cfg::W_BYTES + b * 64 * 128, &a.tmX, fb, kb * 64, row0 + b * 64);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int it = blockIdx.x; it < num_items; it += gridDim.x) {
        const int t = it / num_n;
        if (a.tile_expert[t] < 0) break;
        const uint32_t idesc = umma_idesc(128, 0, 1, 1, 0, 0) | ((uint32_t)((a.tile_rows[t] + 15) / 16 * 2) << 17);
        mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1, &s_abort, status, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * Cfg::ACC_STRIDE;
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(smem_u32(&full_bar[stage]), phase, &s_abort, status, ERR_WAIT_FULL);
          tc_fence_after_sync();
          const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
          const uint64_t w_desc = umma_desc_kmajor_sw128(sa), x_desc = umma_desc_kmajor_sw128(sa + Cfg::W_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_ss(d_tmem, w_desc + 2 * k, x_desc + 2 * k, idesc, (kb | k) != 0);
          tc_commit(smem_u32(&empty_bar[stage]));
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        tc_commit(smem_u32(&tfull_bar[acc]));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;           // TMEM quadrant; every other chunk of 16 rows
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int it = blockIdx.x; it < num_items; it += gridDim.x) {
      const int t = it / num_n, nb = it - t * num_n;
      if (a.tile_expert[t] < 0) break;
      const int row0 = a.tile_row0[t], rows = a.tile_rows[t];
      const int n = nb * COLS + q * (COLS / 4);
      __nv_bfloat16* out = a.c + (long)row0 * a.ldc + n;
      mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase, &s_abort, status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      expert_drain<GATED>(tmem_base + ((uint32_t)(q * 32) << 16) + acc * Cfg::ACC_STRIDE, turned[warp - 2], out, rows, half, lane, a.N - n, a);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (s_abort) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// Tiles of up to 256 rows, on CTA pairs: each CTA brings 128 rows of W and half of the tile's rows, and one MMA of 256 outputs reads both.  On single CTAs these
// tiles are bound by what L2 delivers (154 rows: 1.1 MB per 128 x 2048 weights, 10.5 TB/s in all); a pair fetches 0.8, and what bounds it is HBM
// (2463 tokens: weights and rows at 0.94 and 0.96 of the copy rate).  128 experts, 2048 -> 2 x 768 and
// 768 -> 2048, top 8, both with the drain of this file: 1400 tokens 152 -> 144 and 79 -> 77 us, 2463 162 -> 155 and 89 -> 86, 4000 204 -> 192 and 124 -> 111,
// 8000 340 -> 322 and 210 -> 191.  Tiles of up to 128 rows gain nothing (600 tokens 132.6 -> 132 and 70.7 -> 72.7, 1000 135 -> 135 and 72.7 -> 75.3).
struct ExpertPairCfg {
  static constexpr int XR = 256;
  static constexpr int W_BYTES = 128 * 128, BOX = 32, STAGE_BYTES = W_BYTES + XR / 2 * 128;
  static constexpr int STAGES = 200 * 1024 / STAGE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
};

template <bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
expert_pair_kernel(const __grid_constant__ ExpertArgs a, int* status) {
  using Cfg = ExpertPairCfg;
  constexpr int XR = Cfg::XR, STAGES = Cfg::STAGES, COLS = GATED ? 64 : 128;        // outputs per CTA and tile
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES];                  // even CTA: the bytes of both
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t tfull_bar[2];
  __shared__ __align__(8) uint64_t tempty_bar[2];                     // even CTA: the warps of both
  __shared__ __align__(16) __nv_bfloat16 turned[8][GATED ? 8 : 512];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_ctarank();
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int num_n = (a.N + 2 * COLS - 1) / (2 * COLS), num_items = a.max_tiles * num_n, num_kb = (a.K + 63) / 64;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 16);
    }
    fence_mbar_init();
    tma_prefetch_desc(&a.tmX);
    tma_prefetch_desc(&a.tmW);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&tmem_base_s), 2 * XR);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  pdl_begin();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int it = first; it < num_items; it += step) {
        const int t = it / num_n, nb = (it - t * num_n) * 2 + rank, e = a.tile_expert[t];
        if (e < 0) break;
        // N of an MMA on pairs goes in steps of 32, half of it per CTA
        const int mine = (a.tile_rows[t] + 31) / 32 * 16, row0 = a.tile_row0[t] + rank * mine, boxes = (mine + Cfg::BOX - 1) / Cfg::BOX;
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
          if (rank == 0) mbar_expect_tx(smem_u32(&full_bar[stage]), 2 * (Cfg::W_BYTES + boxes * Cfg::BOX * 128));
          const uint32_t fb = mapa_shared(smem_u32(&full_bar[stage]), 0), sa = smem_base + stage * Cfg::STAGE_BYTES;
          if (GATED) tma_load_5d_pair(sa, &a.tmW, fb, kb * 64, 0, 0, nb * 8, e);
          else tma_load_3d_pair(sa, &a.tmW, fb, kb * 64, nb * 128, e);
          for (int b = 0; b < boxes; ++b) tma_load_2d_pair(sa + Cfg::W_BYTES + b * Cfg::BOX * 128, &a.tmX, fb, kb * 64, row0 + b * Cfg::BOX);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int it = first; it < num_items; it += step) {
        const int t = it / num_n;
        if (a.tile_expert[t] < 0) break;
        const uint32_t idesc = umma_idesc(256, 0, 1, 1, 0, 0) | ((uint32_t)((a.tile_rows[t] + 31) / 32 * 4) << 17);
        mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1, &s_abort, status, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * XR;
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(smem_u32(&full_bar[stage]), phase, &s_abort, status, ERR_WAIT_FULL);
          tc_fence_after_sync();
          const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
          const uint64_t w_desc = umma_desc_kmajor_sw128(sa), x_desc = umma_desc_kmajor_sw128(sa + Cfg::W_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_ss_pair(d_tmem, w_desc + 2 * k, x_desc + 2 * k, idesc, (kb | k) != 0);
          tc_commit_pair(mapa_shared(smem_u32(&empty_bar[stage]), 0));
          tc_commit_pair(mapa_shared(smem_u32(&empty_bar[stage]), 1));
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        tc_commit_pair(mapa_shared(smem_u32(&tfull_bar[acc]), 0));
        tc_commit_pair(mapa_shared(smem_u32(&tfull_bar[acc]), 1));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int it = first; it < num_items; it += step) {
      const int t = it / num_n, nb = (it - t * num_n) * 2 + rank;
      if (a.tile_expert[t] < 0) break;
      const int rows = a.tile_rows[t], n = nb * COLS + q * (COLS / 4);
      __nv_bfloat16* out = a.c + (long)a.tile_row0[t] * a.ldc + n;
      mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase, &s_abort, status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      expert_drain<GATED>(tmem_base + ((uint32_t)(q * 32) << 16) + acc * XR, turned[warp - 2], out, rows, half, lane, a.N - n, a);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[acc]), 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (s_abort) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  cluster_sync_all();   // neither CTA frees TMEM or exits while its partner may still signal it
  if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * XR);
}

template <int XR, bool GATED>
static int launch_expert_as(const ExpertArgs& a, int* status, cudaStream_t stream) {
  static unsigned long long prepared = 0;
  if (int e = ensure_dynamic_smem((const void*)expert_gemm_kernel<XR, GATED>, ExpertCfg<XR>::SMEM_BYTES, prepared)) return e;
  const long items = (long)a.max_tiles * ((a.N + (GATED ? 63 : 127)) / (GATED ? 64 : 128));
  const int grid = items < sm_count() ? (int)items : sm_count();
  launch_overlapped(expert_gemm_kernel<XR, GATED>, grid, GEMM_THREADS, ExpertCfg<XR>::SMEM_BYTES, stream, a, status);
  return (int)cudaGetLastError();
}

template <bool GATED>
static int launch_expert_pair(const ExpertArgs& a, int* status, cudaStream_t stream) {
  static unsigned long long prepared = 0;
  if (int e = ensure_dynamic_smem((const void*)expert_pair_kernel<GATED>, ExpertPairCfg::SMEM_BYTES, prepared)) return e;
  const long items = (long)a.max_tiles * ((a.N + (GATED ? 127 : 255)) / (GATED ? 128 : 256));
  const int pairs = items < max_resident_pairs() ? (int)items : max_resident_pairs();
  launch_overlapped(expert_pair_kernel<GATED>, 2 * pairs, GEMM_THREADS, ExpertPairCfg::SMEM_BYTES, stream, a, status);
  return (int)cudaGetLastError();
}

template <bool GATED>
static int launch_expert(const ExpertArgs& a, int tile, int* status, cudaStream_t stream) {
  switch (tile) {
    case 64: return launch_expert_as<64, GATED>(a, status, stream);
    case 128: return launch_expert_as<128, GATED>(a, status, stream);
    case 256: return launch_expert_pair<GATED>(a, status, stream);
    default: return RC_BAD_ARG;
  }
}

}  // namespace omni
