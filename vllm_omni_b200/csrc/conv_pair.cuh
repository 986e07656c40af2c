// 3 x 3 convolution, stride 1, zero padding, channels-last, as an implicit GEMM on CTA pairs (cta_group::2).
//
// What bounds the one-CTA kernel (gemm_bf16_kernel) here is the way from L2 to shared memory: it fetches the pixels of a tile once per tap
// and the weights once per 128 pixels.  This kernel fetches both less often:
//   pixels   a tile is 16 x 8 pixels per CTA; ONE TMA box of 18 x 10 pixels (64 channels) serves all nine taps: a group of 8 rows of the MMA
//            operand is 8 neighbouring pixels of an image row, 128 bytes each, groups lie one box row (1280 bytes) apart, and a tap is the
//            operand that begins some rows and pixels further into the box (the swizzle goes by address, not by operand row)
//   weights  each CTA of a pair holds half of the TN output channels' weights and the pair's MMA reads both; where all of a layer's weights fit
//            beside the tiles they are fetched once per CTA, otherwise tap by tap through a ring
// A last channel block of at most 32 channels (96 = 64 + 32) is 32 wide: 64-byte rows, swizzled as such, in half the space.
// Results leave, and residuals arrive, as boxes by TMA through shared memory: a lane's 16 bytes at the pitch of a pixel fill half a sector.
// Where a tile holds all channels of its pixels, the RMS norm (+ SiLU) that follows is made there as well, beside or instead of the result.
// An image that is to be doubled first (nearest neighbour) is read as it is: output pixels of one parity of (y, x) see, tap by tap, the same
// shifted box of the small image, so a tile takes 16 x 8 pixels of one parity.
//
// us with residual where it says +, in brackets the form before, with a box per dx, weights by the ring and results of wide tiles by plain stores:
// 1024 x 1024 pixels, 96 -> 96 channels 133 (179), + 166 (206), 192 -> 96 247 (261), 96 -> 8 87 (116); 512 x 512, 192 -> 192 110 (128), + 119 (153),
// 384 -> 192 205 (220); 256 x 256, 384 -> 384 + 105 (117).  With the norm: 96 -> 96 163 (179 + 72 as its own launch), + beside the result 210 (206 + 72);
// 192 -> 192 117 (128 + 42), + 143 (153 + 42).  Without epilogue and loads the MMAs of 96 -> 96 take 109.  Four warps per team instead of eight: 198 and 265
// for 96 -> 96 with the norm, even without.
#pragma once
#include <type_traits>

namespace omni {

constexpr int C3_W = 8, C3_H = 16;                       // pixels of a CTA's tile
constexpr int C3_BOX_ROW = (C3_W + 2) * 128;             // a box row: 10 pixels x 64 channels
constexpr int C3_PX_BYTES = (C3_H + 2) * C3_BOX_ROW, C3_PX_STAGE = (C3_PX_BYTES + 1023) / 1024 * 1024;
constexpr int C3_MAX_PX = 8, C3_MAX_W = 16;              // stages of the pixel and the weight ring
constexpr int C3_THREADS = 64 + 512;                     // TMA, MMA, 16 epilogue warps

template <int TN>
struct Conv3Cfg {
  static constexpr int W_BYTES = (TN / 2) * 128;         // one tap's weights of this CTA's half, 64 channels
  static constexpr int TAPS = TN <= 128 ? 3 : 1;         // per stage of the weight ring: narrow MMAs are over before the next wait is through
  static constexpr int TEAMS = TN <= 96 ? 2 : 1;         // narrow: eight warps have the even tiles and eight the odd ones; wide: sixteen share a tile
  static constexpr int SHARE = 4 / TEAMS, COLS = TN / SHARE;                           // threads per pixel, columns of each
  static constexpr int OUT_BYTES = TN * 2 * C3_W * C3_H; // a tile's outputs
  static constexpr int FIXED = TEAMS * OUT_BYTES + 4 * 128 * 4 + 1024;               // + sums of squares of a thread's columns, alignment
  static constexpr int DYN_MAX = 231424;
  static constexpr int ACC_STRIDE = TN <= 32 ? 32 : (TN <= 128 ? 128 : 256);
  static constexpr int TMEM_COLS = 2 * ACC_STRIDE;
};

struct Conv3Args {
  CUtensorMap tmX, tmW, tmX32, tmW32, tmY, tmR, tmZ;      // X32, W32: of a last block of 32 channels; Y, Z (norm), residual: 32 channels of a tile
  // The image as the tiles see it: rows of W pixels, H of them, in tiles of 16 x 8.  An image that is flat (see conv3_flat) is seen with
  // its columns as rows: the maps swap the two, tap (dy, dx) is weight dy * tap_y + dx * tap_x and pixel (y, x) is y * px_y + x * px_x.
  // up: H and W are those of the small image, and every tile exists for the four parities of output pixels.
  int H, W, n_img, tiles_x, tiles_y, up;
  int tap_y, tap_x, px_y, px_x;
  int Cout, cin, cin_blocks, tail32;      // tail32: the last block is 32 channels wide
  int px_stages, w_stages;
  int has_y, norm_silu, z_apart;          // z_apart: the norm has buffers of its own
  const __nv_bfloat16* gamma;             // of the norm; null: none
  GemmEpilogue epi;
};

template <bool ACT>
__device__ __forceinline__ void conv3_finish(float (&f)[8], const GemmEpilogue& epi, int col) {
  if (epi.bias) add_bf16x8(f, *reinterpret_cast<const uint4*>(epi.bias + col));
  if (!ACT) return;
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
__device__ __forceinline__ void tma_store_5d(const CUtensorMap* tmap, uint32_t src, int c0, int c1, int c2, int c3, int c4) {
  asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(tmap)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// RESIDENT: all weights stay in shared memory.  ACT: an activation follows; few convolutions have one, and its code would crowd the instruction cache of the
// others (128 x 128 pixels with SiLU, 96 -> 96 8.8 us, 11.8 with a function that is called for each value; inlined for all, 16 -> 384 without took 2 % more).
template <int TN, bool RESIDENT, bool ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(C3_THREADS, 1)
conv3x3_pair_kernel(const __grid_constant__ Conv3Args a, int* status) {
  using Cfg = Conv3Cfg<TN>;
  constexpr int TEAMS = Cfg::TEAMS, SHARE = Cfg::SHARE, COLS = Cfg::COLS, GROUP_BYTES = C3_W * C3_H * 64;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t px_full[C3_MAX_PX], px_empty[C3_MAX_PX], w_full[C3_MAX_W], w_empty[C3_MAX_W];
  __shared__ __align__(8) uint64_t tfull_bar[2], tempty_bar[2], res_bar[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const uint32_t s_px = (smem_u32(smem_raw) + 1023u) & ~1023u, s_w = s_px + a.px_stages * C3_PX_STAGE;
  const uint32_t s_out = s_w + (RESIDENT ? 18 * a.cin_blocks - 9 * a.tail32 : 2 * a.w_stages * Cfg::TAPS) * (Cfg::W_BYTES / 2);
  float* part_ss = reinterpret_cast<float*>(smem_raw + (s_out - smem_u32(smem_raw)) + (1 + a.z_apart) * TEAMS * Cfg::OUT_BYTES);      // [team][share][128]
  const int per_img = a.tiles_x * a.tiles_y, m_tiles = a.n_img * per_img, phases = a.up ? 4 : 1;
  const int num_m = (m_tiles + 1) / 2 * phases, num_n = (a.Cout + TN - 1) / TN, num_tiles = num_m * num_n;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < C3_MAX_PX; ++i) {
      mbar_init(smem_u32(&px_full[i]), 1);
      mbar_init(smem_u32(&px_empty[i]), 1);
    }
    for (int i = 0; i < C3_MAX_W; ++i) {
      mbar_init(smem_u32(&w_full[i]), 1);
      mbar_init(smem_u32(&w_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 2 * 4 * SHARE);
      mbar_init(smem_u32(&res_bar[i]), 1);
    }
    fence_mbar_init();
    tma_prefetch_desc(&a.tmX);
    tma_prefetch_desc(&a.tmW);
  }
  const int full_blocks = a.cin_blocks - a.tail32;
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
  auto place = [&](int t, int& mb, int& nb, int& phase, int& img, int& y0, int& x0) {
    const int p = t / num_n;
    nb = t - p * num_n;
    phase = a.up ? p & 3 : 0;
    mb = (a.up ? p >> 2 : p) * 2 + (int)rank;
    img = min(mb / per_img, a.n_img - 1);
    const int rem = mb - img * per_img;
    y0 = rem / a.tiles_x * C3_H;
    x0 = rem % a.tiles_x * C3_W;
  };

  if (warp == 0) {
    if (elect_one()) {
      int ps = 0, ws = 0;
      uint32_t pphase = 0, wphase = 0;
      auto load_w = [&](uint32_t dst, uint32_t fb, int cb, int tap, int nb) {
        const int dx = tap / 3, dy = tap - dx * 3;
        tma_load_2d_pair(dst, cb < full_blocks ? &a.tmW : &a.tmW32, fb, ((dy * a.tap_y + dx * a.tap_x) * a.cin_blocks + cb) * 64, nb * TN + (int)rank * (TN / 2));
      };
      if (RESIDENT && pair < num_tiles) {
        if (rank == 0) mbar_expect_tx(smem_u32(&w_full[0]), (18 * a.cin_blocks - 9 * a.tail32) * Cfg::W_BYTES);
        const uint32_t fb = mapa_shared(smem_u32(&w_full[0]), 0);
        for (int cb = 0; cb < a.cin_blocks; ++cb)
          for (int tap = 0; tap < 9; ++tap) load_w(s_w + (cb * 18 + (cb < full_blocks ? 2 * tap : tap)) * (Cfg::W_BYTES / 2), fb, cb, tap, 0);
      }
      for (int t = pair; t < num_tiles; t += num_pairs) {
        int mb, nb, phase, img, y0, x0;
        place(t, mb, nb, phase, img, y0, x0);
        for (int cb = 0; cb < a.cin_blocks; ++cb) {
          mbar_wait(smem_u32(&px_empty[ps]), pphase ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
          const bool wide = cb < full_blocks;
          if (rank == 0) mbar_expect_tx(smem_u32(&px_full[ps]), wide ? 2 * C3_PX_BYTES : C3_PX_BYTES);
          tma_load_4d_pair(s_px + ps * C3_PX_STAGE, wide ? &a.tmX : &a.tmX32, mapa_shared(smem_u32(&px_full[ps]), 0), cb * 64, x0 - 1, y0 - 1, img);
          if (++ps == a.px_stages) { ps = 0; pphase ^= 1; }
          if (RESIDENT) continue;
          for (int tap = 0; tap < 9; tap += Cfg::TAPS) {
            mbar_wait(smem_u32(&w_empty[ws]), wphase ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
            if (rank == 0) mbar_expect_tx(smem_u32(&w_full[ws]), (wide ? 2 : 1) * Cfg::TAPS * Cfg::W_BYTES);
            const uint32_t fb = mapa_shared(smem_u32(&w_full[ws]), 0);
            for (int i = 0; i < Cfg::TAPS; ++i) load_w(s_w + (ws * Cfg::TAPS * 2 + (wide ? 2 * i : i)) * (Cfg::W_BYTES / 2), fb, cb, tap + i, nb);
            if (++ws == a.w_stages) { ws = 0; wphase ^= 1; }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc(256, TN, 1, 1, 0, 0);
      // One thread issues everything and the tensor cores wait for it where MMAs are narrow: no test between the MMAs of a block of channels (with one
      // per K step 96 -> 96 took 40 us more), and the loop over dx stays a loop for the instruction cache.
      int ps = 0, ws = 0, acc = 0;
      uint32_t pphase = 0, wphase = 0, acc_phase = 0;
      const uint32_t w_free0 = mapa_shared(smem_u32(w_empty), 0), w_free1 = mapa_shared(smem_u32(w_empty), 1);
      const uint32_t px_free0 = mapa_shared(smem_u32(px_empty), 0), px_free1 = mapa_shared(smem_u32(px_empty), 1);
      if (RESIDENT && pair < num_tiles) mbar_wait(smem_u32(&w_full[0]), 0, &s_abort, status, ERR_WAIT_FULL);
      for (int t = pair; t < num_tiles; t += num_pairs) {
        const int phase = a.up ? (t / num_n) & 3 : 0;
        uint32_t y_at[3];                                    // where the pixels of a tap's row begin in the box
#pragma unroll
        for (int d = 0; d < 3; ++d) y_at[d] = (a.up ? (((phase >> 1) + d - 1) >> 1) + 1 : d) * (C3_BOX_ROW / 16);
        mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1, &s_abort, status, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * Cfg::ACC_STRIDE;
        for (int cb = 0; cb < a.cin_blocks; ++cb) {
          mbar_wait(smem_u32(&px_full[ps]), pphase, &s_abort, status, ERR_WAIT_FULL);
          tc_fence_after_sync();
          // N K steps of 16 channels from rows of ROW bytes
          auto products = [&](auto n, auto row) {
            constexpr int N = decltype(n)::value, ROW = decltype(row)::value;
            constexpr uint64_t swizzle = ROW == 128 ? 0 : 6ull << 61;          // umma_desc_sw128's 2 becomes 4: 64 bytes
            const uint64_t a_desc = umma_desc_sw128(s_px + ps * C3_PX_STAGE, 0, C3_BOX_ROW * ROW / 128) ^ swizzle;
            uint64_t b_desc = umma_desc_sw128(s_w + cb * 9 * Cfg::W_BYTES, 0, 8 * ROW) ^ swizzle;
#pragma unroll 1
            for (int dx = 0; dx < 3; ++dx) {
              const uint64_t col = a_desc + (uint32_t)((a.up ? (((phase & 1) + dx - 1) >> 1) + 1 : dx) * (ROW / 16));
#pragma unroll
              for (int dy = 0; dy < 3; ++dy) {
                if (!RESIDENT && (Cfg::TAPS == 1 || dy == 0)) {
                  mbar_wait(smem_u32(&w_full[ws]), wphase, &s_abort, status, ERR_WAIT_FULL);
                  tc_fence_after_sync();
                  b_desc = umma_desc_sw128(s_w + ws * Cfg::TAPS * Cfg::W_BYTES, 0, 8 * ROW) ^ swizzle;
                }
                const uint64_t at = col + y_at[dy] * ROW / 128;
#pragma unroll
                for (int k = 0; k < N; ++k) mma_f16_ss_pair(d_tmem, at + 2 * k, b_desc + 2 * k, idesc, (cb | dx | dy | k) != 0);
                b_desc += Cfg::W_BYTES * ROW / 128 / 16;
                if (!RESIDENT && (Cfg::TAPS == 1 || dy == 2)) {
                  tc_commit_pair(w_free0 + ws * 8);
                  tc_commit_pair(w_free1 + ws * 8);
                  if (++ws == a.w_stages) { ws = 0; wphase ^= 1; }
                }
              }
            }
          };
          const int steps = (a.cin - cb * 64 + 15) / 16;
          if (steps >= 4) products(std::integral_constant<int, 4>(), std::integral_constant<int, 128>());
          else if (steps == 3) products(std::integral_constant<int, 3>(), std::integral_constant<int, 128>());
          else if (steps == 2) products(std::integral_constant<int, 2>(), std::integral_constant<int, 64>());
          else products(std::integral_constant<int, 1>(), std::integral_constant<int, 64>());
          tc_commit_pair(px_free0 + ps * 8);
          tc_commit_pair(px_free1 + ps * 8);
          if (++ps == a.px_stages) { ps = 0; pphase ^= 1; }
        }
        tc_commit_pair(mapa_shared(smem_u32(&tfull_bar[acc]), 0));
        tc_commit_pair(mapa_shared(smem_u32(&tfull_bar[acc]), 1));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    // SHARE threads per pixel, COLS channels each; a team shares a buffer of 32-channel boxes (64 bytes per pixel, swizzled: no bank conflicts)
    const int q = warp & 3, team = (warp - 2) / (4 * SHARE), share = ((warp - 2) >> 2) % SHARE, r = q * 32 + lane;
    const uint32_t buf = s_out + team * Cfg::OUT_BYTES, zbuf = buf + a.z_apart * TEAMS * Cfg::OUT_BYTES, swizzle = (r >> 1) & 3;
    const bool leader = (warp - 2) % (4 * SHARE) == 0 && lane == 0, norm = a.gamma != nullptr;
    auto team_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(128 * SHARE) : "memory"); };
    auto fetch_residual = [&](int t) {
      int mb, nb, phase, img, y0, x0;
      place(t, mb, nb, phase, img, y0, x0);
      const int groups = min(TN / 32, (a.Cout - nb * TN + 31) / 32);
      mbar_expect_tx(smem_u32(&res_bar[team]), groups * GROUP_BYTES);
      for (int g = 0; g < groups; ++g) tma_load_4d(buf + g * GROUP_BYTES, &a.tmR, smem_u32(&res_bar[team]), nb * TN + g * 32, x0, y0, img);
    };
    int t = pair + team * num_pairs;
    if (leader && a.epi.residual && t < num_tiles) fetch_residual(t);
#pragma unroll 1
    for (int i = 0; t < num_tiles; t += TEAMS * num_pairs, ++i) {
      int mb, nb, phase, img, y0, x0;
      place(t, mb, nb, phase, img, y0, x0);
      const int acc = TEAMS == 2 ? team : i & 1, acc_phase = TEAMS == 2 ? i & 1 : (i >> 1) & 1;
      auto at = [&](uint32_t b, int c) { return b + (c >> 5) * GROUP_BYTES + r * 64 + ((((c >> 3) & 3) ^ swizzle) << 4); };       // 8 channels from c on
      auto store = [&](const CUtensorMap* tm, uint32_t from) {
        if (mb < m_tiles)
          for (int g = 0; g < TN / 32 && nb * TN + g * 32 < a.Cout; ++g)
            tma_store_5d(tm, from + g * GROUP_BYTES, nb * TN + g * 32, x0, y0, a.up ? phase & 1 : img, phase >> 1);
        bulk_commit();
      };
      if (a.epi.residual) mbar_wait(smem_u32(&res_bar[team]), i & 1, &s_abort, status, ERR_WAIT_FULL);
      mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase, &s_abort, status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      // Both passes are rolled and a pixel's channels wait in the buffer for the second: unrolled, with the channels in registers, the code outgrew the
      // instruction cache (96 -> 96: 306 us)
      float ss = 0.f;
#pragma unroll 1
      for (int g = 0; g < COLS; g += 16) {
        uint32_t v[16];
        tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + acc * Cfg::ACC_STRIDE + share * COLS + g, v);
        tmem_wait_ld();
        if (g == COLS - 16) {                               // the accumulator is read: the next but one tile may have it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[acc]), 0));
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int in_tile = share * COLS + g + c * 8, col = nb * TN + in_tile;
          if (col >= a.Cout) break;
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[c * 8 + e]);
          conv3_finish<ACT>(f, a.epi, col);
          if (a.epi.residual) add_bf16x8(f, lds128(at(buf, in_tile)));
          const uint4 w = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
          sts128(at(buf, in_tile), w);
          if (norm) {                                       // of the rounded values
            const float2 p0 = unpack_bf16(w.x), p1 = unpack_bf16(w.y), p2 = unpack_bf16(w.z), p3 = unpack_bf16(w.w);
            ss += (p0.x * p0.x + p0.y * p0.y + p1.x * p1.x + p1.y * p1.y) + (p2.x * p2.x + p2.y * p2.y + p3.x * p3.x + p3.y * p3.y);
          }
        }
      }
      if (norm) part_ss[(team * SHARE + share) * 128 + r] = ss;
      if (a.has_y) {
        fence_proxy_async_smem();
        team_sync();
        if (leader) {
          store(&a.tmY, buf);
          if (norm && !a.z_apart) bulk_wait_read();
        }
        if (norm && !a.z_apart) {
          __syncwarp();
          team_sync();
        }
      } else {
        team_sync();
      }
      if (norm) {
        ss = 0.f;
#pragma unroll
        for (int h = 0; h < SHARE; ++h) ss += part_ss[(team * SHARE + h) * 128 + r];
        const float inv = rsqrtf(fmaxf(ss / (float)a.Cout, 1e-24f));
#pragma unroll 2
        for (int col = share * COLS; col < (share + 1) * COLS; col += 8) {
          if (col >= a.Cout) break;
          const uint4 u = lds128(at(buf, col)), gm = *reinterpret_cast<const uint4*>(a.gamma + col);
          const uint32_t uw[4] = {u.x, u.y, u.z, u.w}, gw[4] = {gm.x, gm.y, gm.z, gm.w};
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 p = unpack_bf16(uw[e]), g2 = unpack_bf16(gw[e]);
            const float x = p.x * inv * g2.x, y = p.y * inv * g2.y;
            o[e] = a.norm_silu ? pack_bf16(silu(x), silu(y)) : pack_bf16(x, y);
          }
          sts128(at(zbuf, col), make_uint4(o[0], o[1], o[2], o[3]));
        }
        fence_proxy_async_smem();
        team_sync();
        if (leader) store(&a.tmZ, zbuf);
      }
      if (leader) {
        bulk_wait_read();
        if (a.epi.residual && t + TEAMS * num_pairs < num_tiles) fetch_residual(t + TEAMS * num_pairs);
      }
      __syncwarp();
      team_sync();                                          // the buffer is free
    }
    if (leader) bulk_wait_all();
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

// Boxes of `chans` channels x `cols` x `rows` pixels of an image of C channels, `ld` elements per pixel, that is read.
static int conv3_map(CUtensorMap* map, const Conv3Args& a, const void* p, long ld, int C, int chans, int cols, int rows, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return RC_NO_DRIVER;
  if (reinterpret_cast<uintptr_t>(p) & 15) return RC_BAD_ARG;
  const cuuint64_t px = (cuuint64_t)ld * 2;
  cuuint64_t gdim[4] = {(cuuint64_t)C, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.n_img};
  cuuint64_t gstr[3] = {px * a.px_x, px * a.px_y, px * a.W * a.H};
  cuuint32_t box[4] = {(cuuint32_t)chans, (cuuint32_t)cols, (cuuint32_t)rows, 1}, estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? RC_OK : RC_TMAP;
}
// The same of an image that is written: 32 channels of a tile; the fourth and fifth coordinates are the image and 0, or the parities of x and y.
static int conv3_out_map(CUtensorMap* map, const Conv3Args& a, const void* p, long ld) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return RC_NO_DRIVER;
  if (reinterpret_cast<uintptr_t>(p) & 15) return RC_BAD_ARG;
  const cuuint64_t px = (cuuint64_t)ld * 2, image = px * a.W * a.H;
  cuuint64_t gdim[5] = {(cuuint64_t)a.Cout, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)(a.up ? 2 : a.n_img), (cuuint64_t)(a.up ? 2 : 1)};
  cuuint64_t gstr[4] = {px * a.px_x, px * a.px_y, image, image * a.n_img};
  if (a.up) { gstr[0] = px * 2; gstr[1] = px * 4 * a.W; gstr[2] = px; gstr[3] = px * 2 * a.W; }
  cuuint32_t box[5] = {32, C3_W, C3_H, 1, 1}, estr[5] = {1, 1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(p), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? RC_OK : RC_TMAP;
}

static long conv3_tiles(long n_img, int H, int W) { return n_img * ((W + C3_W - 1) / C3_W) * ((H + C3_H - 1) / C3_H); }


template <int TN>
static int launch_conv3(Conv3Args& a, const void* w, const void* y, long ldy, const void* z, long ldz, int pairs, int* status, cudaStream_t stream) {
  using Cfg = Conv3Cfg<TN>;
  const uint64_t K = 9ull * a.cin_blocks * 64;
  if (int rc = make_tmap_2d(&a.tmW, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)a.Cout, K, K * 2, TN / 2, 64)) return rc;
  if (int rc = make_tmap_2d(&a.tmW32, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)a.Cout, K, K * 2, TN / 2, 32, CU_TENSOR_MAP_SWIZZLE_64B)) return rc;
  if (y)
    if (int rc = conv3_out_map(&a.tmY, a, y, ldy)) return rc;
  if (z)
    if (int rc = conv3_out_map(&a.tmZ, a, z, ldz)) return rc;
  if (a.epi.residual)
    if (int rc = conv3_map(&a.tmR, a, a.epi.residual, a.epi.ldr, a.Cout, 32, C3_W, C3_H, CU_TENSOR_MAP_SWIZZLE_64B)) return rc;
  // weights stay where they leave room for two channel blocks of pixels; otherwise two or more blocks of pixels and the rest for the weights' ring
  constexpr int RING = Cfg::TAPS * Cfg::W_BYTES, Z = Cfg::TEAMS * Cfg::OUT_BYTES;
  constexpr bool MAY_STAY = Cfg::TEAMS == 2;
  const int all_w = (18 * a.cin_blocks - 9 * a.tail32) * (Cfg::W_BYTES / 2);
  int room = Cfg::DYN_MAX - Cfg::FIXED;
  const bool stay = MAY_STAY && a.Cout <= TN && all_w + 2 * C3_PX_STAGE <= room;
  // Result and norm from one buffer wait for each other; apart they cost pixel stages or the weights' ring (not below six stages).  Both of 96 -> 96 at
  // 1024 x 1024 with residual 210 us (233 from one buffer), 192 -> 192 at 512 x 512 143 (147).
  a.z_apart = y && z && (stay ? all_w : 6 * RING) + 2 * C3_PX_STAGE + Z <= room;
  room -= a.z_apart * Z;
  const int fit = (room - 2 * C3_PX_STAGE) / RING;
  a.w_stages = stay ? 0 : (fit < C3_MAX_W ? fit : C3_MAX_W);
  const int w_bytes = stay ? all_w : a.w_stages * RING;
  a.px_stages = (room - w_bytes) / C3_PX_STAGE < C3_MAX_PX ? (room - w_bytes) / C3_PX_STAGE : C3_MAX_PX;
  const int bytes = w_bytes + a.px_stages * C3_PX_STAGE + Cfg::FIXED + a.z_apart * Z;
  const long tiles = (long)((a.n_img * a.tiles_x * a.tiles_y + 1) / 2) * (a.up ? 4 : 1) * ((a.Cout + TN - 1) / TN);
  const int grid = tiles < pairs ? (int)tiles : pairs;
  static unsigned long long prepared[4] = {};
  const bool act = a.epi.act != ACT_NONE;
  const auto kernel = act ? (stay ? conv3x3_pair_kernel<TN, MAY_STAY, true> : conv3x3_pair_kernel<TN, false, true>)
                          : (stay ? conv3x3_pair_kernel<TN, MAY_STAY, false> : conv3x3_pair_kernel<TN, false, false>);
  if (int e = ensure_dynamic_smem((const void*)kernel, Cfg::DYN_MAX, prepared[2 * act + stay])) return e;
  launch_overlapped(kernel, 2 * grid, C3_THREADS, bytes, stream, a, status);
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

static bool conv3_fits(long n_img, int H, int W) { return conv3_tiles(n_img, H, W) < (1L << 22); }

static int conv3_run(const void* x, long ldx, const void* w, void* y, long ldy, void* z, long ldz, int n_img, int H, int W, int Cin, int Cout, bool up,
                     const void* bias, const void* residual, int ldr, int act, const void* gamma, int norm_silu, int* status, cudaStream_t stream) {
  const int pairs = max_resident_pairs();
  const bool flat = conv3_flat(n_img, H, W, Cout, pairs);
  Conv3Args a = {};
  a.n_img = n_img;
  a.H = flat ? W : H; a.W = flat ? H : W;
  a.tap_y = flat ? 1 : 3; a.tap_x = flat ? 3 : 1;
  a.px_y = flat ? 1 : W; a.px_x = flat ? W : 1;
  a.tiles_x = (a.W + C3_W - 1) / C3_W; a.tiles_y = (a.H + C3_H - 1) / C3_H;
  a.up = up;
  a.Cout = Cout; a.cin = Cin; a.cin_blocks = (Cin + 63) / 64;
  a.tail32 = (Cin - 1) % 64 < 32;
  if (int rc = conv3_map(&a.tmX, a, x, ldx, Cin, 64, C3_W + 2, C3_H + 2, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
  if (int rc = conv3_map(&a.tmX32, a, x, ldx, Cin, 32, C3_W + 2, C3_H + 2, CU_TENSOR_MAP_SWIZZLE_64B)) return rc;
  a.epi.bias = static_cast<const __nv_bfloat16*>(bias);
  a.epi.residual = static_cast<const __nv_bfloat16*>(residual);
  a.epi.ldr = ldr;
  a.epi.rows_per_batch = 1;
  a.epi.act = act;
  a.has_y = y != nullptr;
  a.gamma = static_cast<const __nv_bfloat16*>(gamma);
  a.norm_silu = norm_silu;
  const long m_pairs = (conv3_tiles(n_img, a.H, a.W) + 1) / 2 * (up ? 4 : 1);
  const int tn = pick_conv3_tn(m_pairs, Cout, pairs);
  if ((gamma && tn < Cout) || (up && (flat || n_img != 1 || residual))) return RC_BAD_ARG;
  switch (tn) {
    case 256: return launch_conv3<256>(a, w, y, ldy, z, ldz, pairs, status, stream);
    case 192: return launch_conv3<192>(a, w, y, ldy, z, ldz, pairs, status, stream);
    case 128: return launch_conv3<128>(a, w, y, ldy, z, ldz, pairs, status, stream);
    case 96: return launch_conv3<96>(a, w, y, ldy, z, ldz, pairs, status, stream);
    default: return launch_conv3<32>(a, w, y, ldy, z, ldz, pairs, status, stream);
  }
}

}  // namespace omni
