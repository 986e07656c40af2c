// 3 x 3 convolution, stride 1, zero padding, channels-last, as an implicit GEMM on CTA pairs (cta_group::2).
//
// What bounds the one-CTA kernel (gemm_bf16_kernel) here is the way from L2 to shared memory: it fetches the pixels of a tile once per tap
// and the weights once per 128 pixels, 32 to 40 KB per 64 channels and tap, 1.6 to 2 times what an SM takes in while its MMAs run.  This
// kernel fetches both less often:
//   pixels   a tile is 16 x 8 pixels per CTA; one TMA box of 18 x 8 pixels (one column offset dx, 64 channels) serves the three taps (dy, dx):
//            a group of 8 rows of the MMA operand is the 8 pixels of one image row, so tap dy is the box from its (dy + 1)-th group on
//   weights  each CTA of a pair holds half of the TN output channels' weights and the pair's MMA reads both
// A channel block of which only some channels exist (96 = 64 + 32) issues the K steps that hold any.  Per 64 channels and three taps
// a CTA takes in 18 KB + 3 * 64 * TN bytes, 36 KB at TN = 96; the one-CTA kernel, whose narrowest tile has 128 columns, 3 * (16 KB + 16 KB).
// With residual, one-CTA kernel before: 1024 x 1024 pixels, 96 -> 96 channels 211 us (461), 192 -> 96 257 us (662), 96 -> 8 127 us (743);
// 512 x 512, 192 -> 192 160 us (193), 384 -> 192 221 us (350); 256 x 256, 384 -> 384 119 us (180).
// Up to 96 output channels the epilogue was what a tile waited for (16 -> 96 took as long as 96 -> 96): a lane's 16 bytes at the pitch of a
// pixel fill half a sector.  Results and residuals therefore move as boxes by TMA: 268 -> 211 us, 317 -> 257 us, 145 -> 127 us in the order
// above.  Wider outputs have MMAs enough to hide it behind and no shared memory to spare.
#pragma once

namespace omni {

constexpr int C3_W = 8, C3_H = 16;                       // pixels of a CTA's tile
constexpr int C3_A_BYTES = (C3_H + 2) * C3_W * 128;      // 18 groups of 8 pixels x 64 channels

template <int TN>
struct Conv3Cfg {
  static constexpr int B_BYTES = (TN / 2) * 128;         // one tap's weights of this CTA's half
  static constexpr int STAGE_BYTES = C3_A_BYTES + 3 * B_BYTES;
  static constexpr bool STAGED = TN <= 96;               // results leave, and the residual arrives, by TMA through shared memory
  static constexpr int OUT_BYTES = STAGED ? TN * 2 * C3_W * C3_H : 0;        // a tile's outputs, two of them
  static constexpr int FIT = (220 * 1024 - 2 * OUT_BYTES) / STAGE_BYTES, STAGES = FIT < 6 ? FIT : 6;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 2 * OUT_BYTES + 1024;
  static constexpr int ACC_STRIDE = TN <= 32 ? 32 : (TN <= 128 ? 128 : 256);
  static constexpr int TMEM_COLS = 2 * ACC_STRIDE;
};

struct Conv3Args {
  CUtensorMap tmX, tmW, tmY, tmR;         // Y, residual: 32 channels of a tile
  __nv_bfloat16* y;
  int ldy;
  // The image as the tiles see it: rows of W pixels, H of them, in tiles of 16 x 8.  An image that is flat (see conv3_flat) is seen with
  // its columns as rows: the maps swap the two, tap (dy, dx) is weight dy * tap_y + dx and pixel (y, x) is y * px_y + x * px_x.
  int H, W, n_img, tiles_x, tiles_y;
  int tap_y, tap_x, px_y, px_x;
  int Cout, cin, cin_blocks;
  GemmEpilogue epi;
};

__device__ __forceinline__ void add8(float (&f)[8], const uint4& u) {
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  f[0] += a.x; f[1] += a.y; f[2] += b.x; f[3] += b.y;
  f[4] += c.x; f[5] += c.y; f[6] += d.x; f[7] += d.y;
}

__device__ __forceinline__ void conv3_finish(float (&f)[8], const GemmEpilogue& epi, int col) {
  if (epi.bias) add8(f, *reinterpret_cast<const uint4*>(epi.bias + col));
  if (epi.act == ACT_GELU_TANH) {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = gelu_tanh(f[e]);
  } else if (epi.act == ACT_SILU) {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = silu(f[e]);
  } else if (epi.act == ACT_RELU2) {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = fmaxf(f[e], 0.f) * fmaxf(f[e], 0.f);
  }
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* tmap, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(tmap)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

template <int TN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
conv3x3_pair_kernel(const __grid_constant__ Conv3Args a, int* status) {
  using Cfg = Conv3Cfg<TN>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t tfull_bar[2];
  __shared__ __align__(8) uint64_t tempty_bar[2];
  __shared__ __align__(8) uint64_t res_bar[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int per_img = a.tiles_x * a.tiles_y, m_tiles = a.n_img * per_img;
  const int num_m = (m_tiles + 1) / 2, num_n = (a.Cout + TN - 1) / TN, num_tiles = num_m * num_n;
  const int num_st = 3 * a.cin_blocks;                    // stages per tile: (channel block, dx)

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), Cfg::STAGED ? 8 : 16);
      mbar_init(smem_u32(&res_bar[i]), 1);
    }
    fence_mbar_init();
    tma_prefetch_desc(&a.tmX);
    tma_prefetch_desc(&a.tmW);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&tmem_base_s), Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  pdl_begin();

  // the pair's two pixel tiles are neighbours in the tile list; a tile past the end (odd counts) lies below the last image's rows
  auto place = [&](int t, int& nb, int& img, int& y0, int& x0) {
    const int mb = (t / num_n) * 2 + (int)rank;
    nb = t % num_n;
    img = min(mb / per_img, a.n_img - 1);
    const int rem = mb - img * per_img;
    y0 = rem / a.tiles_x * C3_H;
    x0 = rem % a.tiles_x * C3_W;
  };

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int t = pair; t < num_tiles; t += num_pairs) {
        int nb, img, y0, x0;
        place(t, nb, img, y0, x0);
        for (int s = 0; s < num_st; ++s) {
          const int cb = s / 3, dx = s - cb * 3;
          mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
          if (rank == 0) mbar_expect_tx(smem_u32(&full_bar[stage]), 2 * Cfg::STAGE_BYTES);
          const uint32_t fb = mapa_shared(smem_u32(&full_bar[stage]), 0);
          const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
          tma_load_4d_pair(sa, &a.tmX, fb, cb * 64, x0 + dx - 1, y0 - 1, img);
#pragma unroll
          for (int dy = 0; dy < 3; ++dy)
            tma_load_2d_pair(sa + C3_A_BYTES + dy * Cfg::B_BYTES, &a.tmW, fb, ((dy * a.tap_y + dx * a.tap_x) * a.cin_blocks + cb) * 64,
                             nb * TN + (int)rank * (TN / 2));
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc(256, TN, 1, 1, 0, 0);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int t = pair; t < num_tiles; t += num_pairs) {
        mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1, &s_abort, status, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * Cfg::ACC_STRIDE;
        for (int s = 0; s < num_st; ++s) {
          const int steps = min(4, (a.cin - s / 3 * 64 + 15) / 16);          // 16 channels each
          mbar_wait(smem_u32(&full_bar[stage]), phase, &s_abort, status, ERR_WAIT_FULL);
          tc_fence_after_sync();
          const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
          const uint64_t a_desc = umma_desc_kmajor_sw128(sa), b_desc = umma_desc_kmajor_sw128(sa + C3_A_BYTES);
#pragma unroll
          for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (k < steps)
                mma_f16_ss_pair(d_tmem, a_desc + dy * (C3_W * 128 / 16) + 2 * k, b_desc + dy * (Cfg::B_BYTES / 16) + 2 * k, idesc,
                                (s | dy | k) != 0);
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
  } else if constexpr (Cfg::STAGED) {
    // A tile of few channels is over in 1 to 3 us, less than one epilogue takes from the accumulator to memory: four warps have the even
    // tiles and four the odd ones.  A pixel's channels are a row of their own in memory, so each group of 32 channels goes out, and its
    // residual comes in a tile ahead, as one box through shared memory (64 bytes per pixel, swizzled: no bank conflicts).
    constexpr int GROUPS = TN / 32;
    const int q = warp & 3, mine = (warp - 2) >> 2, r = q * 32 + lane;
    const uint32_t buf = smem_base + STAGES * Cfg::STAGE_BYTES + mine * Cfg::OUT_BYTES;
    const bool leader = q == 2 && lane == 0;                // warps 2 and 6
    const uint32_t swizzle = (r >> 1) & 3;
    auto fetch_residual = [&](int t) {
      int nb, img, y0, x0;
      place(t, nb, img, y0, x0);
      const int groups = min(GROUPS, (a.Cout - nb * TN + 31) / 32);
      mbar_expect_tx(smem_u32(&res_bar[mine]), groups * (Cfg::OUT_BYTES / GROUPS));
      for (int g = 0; g < groups; ++g)
        tma_load_4d(buf + g * (Cfg::OUT_BYTES / GROUPS), &a.tmR, smem_u32(&res_bar[mine]), nb * TN + g * 32, x0, y0, img);
    };
    uint32_t phase = 0;
    int t = pair + mine * num_pairs;
    if (leader && a.epi.residual && t < num_tiles) fetch_residual(t);
    for (; t < num_tiles; t += 2 * num_pairs, phase ^= 1) {
      int nb, img, y0, x0;
      place(t, nb, img, y0, x0);
      if (a.epi.residual) mbar_wait(smem_u32(&res_bar[mine]), phase, &s_abort, status, ERR_WAIT_FULL);
      mbar_wait(smem_u32(&tfull_bar[mine]), phase, &s_abort, status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        uint32_t v[32];
        tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + mine * Cfg::ACC_STRIDE + g * 32, v);
        tmem_wait_ld();
        if (g == GROUPS - 1) {                              // the accumulator is read: the next but one tile may have it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[mine]), 0));
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int col = nb * TN + g * 32 + c * 8;
          if (col >= a.Cout) break;
          const uint32_t at = buf + g * (Cfg::OUT_BYTES / GROUPS) + r * 64 + ((c ^ swizzle) << 4);
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[c * 8 + e]);
          conv3_finish(f, a.epi, col);
          if (a.epi.residual) add8(f, lds128(at));
          sts128(at, make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7])));
        }
      }
      fence_proxy_async_smem();
      asm volatile("bar.sync %0, 128;" ::"r"(1 + mine) : "memory");
      if (leader) {
        if ((t / num_n) * 2 + (int)rank < m_tiles)
          for (int g = 0; g < GROUPS && nb * TN + g * 32 < a.Cout; ++g)
            tma_store_4d(&a.tmY, buf + g * (Cfg::OUT_BYTES / GROUPS), nb * TN + g * 32, x0, y0, img);
        bulk_commit();
        bulk_wait_read();
        if (a.epi.residual && t + 2 * num_pairs < num_tiles) fetch_residual(t + 2 * num_pairs);
      }
      __syncwarp();
      asm volatile("bar.sync %0, 128;" ::"r"(1 + mine) : "memory");          // the buffer is free
    }
    if (leader) bulk_wait_all();
  } else {
    // the residual is requested while the MMAs of the tile run
    constexpr int CH = TN / 32;                             // 16-column chunks per warp: half of the tile's columns
    const int q = warp & 3, first = ((warp - 2) >> 2) * (TN / 2);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = pair; t < num_tiles; t += num_pairs) {
      int nb, img, y0, x0;
      place(t, nb, img, y0, x0);
      const int r = q * 32 + lane, y = y0 + r / C3_W, x = x0 + r % C3_W;
      const bool row_ok = y < a.H && x < a.W;
      const long row = (long)img * a.H * a.W + (long)y * a.px_y + (long)x * a.px_x;
      const int col = nb * TN + first;
      uint4 res[CH][2];
      if (a.epi.residual) {
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
          for (int g = 0; g < 2; ++g)
            res[c][g] = row_ok && col + c * 16 + g * 8 < a.Cout
                            ? *reinterpret_cast<const uint4*>(a.epi.residual + row * a.epi.ldr + col + c * 16 + g * 8)
                            : make_uint4(0u, 0u, 0u, 0u);
      }
      mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase, &s_abort, status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        uint32_t v[16];
        tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + acc * Cfg::ACC_STRIDE + first + c * 16, v);
        tmem_wait_ld();
        if (c == CH - 1) {                                  // the accumulator is read: the next but one tile may have it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[acc]), 0));
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int cc = col + c * 16 + g * 8;
          if (!row_ok || cc >= a.Cout) continue;
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[g * 8 + e]);
          conv3_finish(f, a.epi, cc);
          if (a.epi.residual) add8(f, res[c][g]);
          *reinterpret_cast<uint4*>(a.y + row * a.ldy + cc) =
              make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
        }
      }
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
  cluster_sync_all();
  if (warp == 1) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
}

// Boxes of `chans` channels x 8 pixels x `rows` rows of an image of C channels, `ld` elements per pixel.
static int conv3_map(CUtensorMap* map, const Conv3Args& a, const void* p, long ld, int C, int chans, int rows, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return RC_NO_DRIVER;
  if (reinterpret_cast<uintptr_t>(p) & 15) return RC_BAD_ARG;
  const cuuint64_t px = (cuuint64_t)ld * 2;
  cuuint64_t gdim[4] = {(cuuint64_t)C, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.n_img};
  cuuint64_t gstr[3] = {px * a.px_x, px * a.px_y, px * a.W * a.H};
  cuuint32_t box[4] = {(cuuint32_t)chans, C3_W, (cuuint32_t)rows, 1}, estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? RC_OK : RC_TMAP;
}

static long conv3_tiles(long n_img, int H, int W) { return n_img * ((W + C3_W - 1) / C3_W) * ((H + C3_H - 1) / C3_H); }


template <int TN>
static int launch_conv3(Conv3Args& a, const void* w, int pairs, int* status, cudaStream_t stream) {
  using Cfg = Conv3Cfg<TN>;
  const uint64_t K = 9ull * a.cin_blocks * 64;
  if (int rc = make_tmap_2d(&a.tmW, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)a.Cout, K, K * 2, TN / 2, 64)) return rc;
  if (Cfg::STAGED) {
    if (int rc = conv3_map(&a.tmY, a, a.y, a.ldy, a.Cout, 32, C3_H, CU_TENSOR_MAP_SWIZZLE_64B)) return rc;
    if (a.epi.residual)
      if (int rc = conv3_map(&a.tmR, a, a.epi.residual, a.epi.ldr, a.Cout, 32, C3_H, CU_TENSOR_MAP_SWIZZLE_64B)) return rc;
  }
  static unsigned long long prepared = 0;
  if (int e = ensure_dynamic_smem((const void*)conv3x3_pair_kernel<TN>, Cfg::SMEM_BYTES, prepared)) return e;
  const long tiles = (long)((a.n_img * a.tiles_x * a.tiles_y + 1) / 2) * ((a.Cout + TN - 1) / TN);
  const int grid = tiles < pairs ? (int)tiles : pairs;
  launch_overlapped(conv3x3_pair_kernel<TN>, 2 * grid, GEMM_THREADS, Cfg::SMEM_BYTES, stream, a, status);
  return (int)cudaGetLastError();
}

// Widths that leave the fewest columns empty, then the fewest waves; the narrowest for outputs of a few channels (an image).
static int pick_conv3_tn(long m_pairs, int Cout, int pairs) {
  const int cand[5] = {256, 192, 128, 96, 32};
  int best = 256;
  long best_cost = -1;
  for (int i = 0; i < 5; ++i) {
    const int tn = cand[i];
    const long waves = (m_pairs * ((Cout + tn - 1) / tn) + pairs - 1) / pairs;
    const long cost = waves * (tn + 24);                  // a tile's pixels are fetched whatever its width
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = tn; }
  }
  return best;
}

// Whether an image is seen with its columns as rows: where that takes at least a quarter fewer tiles (images of up to 8 rows: half as many), still
// a quarter of a wave of them, and fewer waves.  us, seen as it is in brackets: 4 images of 8 x 512, 256 -> 256 channels 24.2 (31.9; the
// one-CTA kernel 27.3), 512 -> 256 35.1 (52.1; 43.1), one of 3 x 1000, 512 -> 512 30.7 (50.0; 39.6).
static bool conv3_flat(long n_img, int H, int W, int Cout, int pairs) {
  const long seen = (conv3_tiles(n_img, H, W) + 1) / 2, turned = (conv3_tiles(n_img, W, H) + 1) / 2;
  if (turned * 4 > seen * 3 || turned * 4 < pairs) return false;
  const int tn = pick_conv3_tn(seen, Cout, pairs), num_n = (Cout + tn - 1) / tn;
  return (turned * num_n + pairs - 1) / pairs < (seen * num_n + pairs - 1) / pairs;
}

}  // namespace omni
