// Attention of one head as wide as 384 channels (the mid block of the image and video decoders), outside the head sizes of attention_sm100.cu.
//
// A CTA pair (cta_group::2) owns 256 query rows.  TMEM holds the 128 x 384 fp32 result of a CTA's rows and one block of scores against 128 keys, all
// 512 columns.  The softmax warps take a row's 128 scores into registers at once, so the scores of step j + 1 are computed while those of step j become
// probabilities, which pass to the product with V as bf16 through shared memory.  K and V come through one ring of 24 KB stages: half of the channels
// of the K rows of a CTA's 64 keys, or half of the channels of V for 64 keys.  Shared memory: queries 96 KB, probabilities 32 KB, four stages 96 KB.
//   warp 0      TMA producer          warp 1   MMA issuer (even CTA)
//   warps 4-7   softmax, one thread per query row; result
// Scores and row sums are fp32 throughout.  O is rescaled only when a row maximum grows by more than 2^8 (as in attention_sm100.cu).
//
// Bound by the tensor cores: 128 keys cost a CTA 3072 clocks of MMAs.  (Scores against 64 keys in two alternating TMEM blocks: 350 us where this takes
// 321; an MMA 64 wide waits for its query operand in shared memory.)  us, and two GEMMs around a row softmax in chunks of 4096 rows before: 256 rows
// 17 (23), 1024 23 (28), 4096 46 (86), 8192 103 (249), 16384 321 (872) = 1284 TFLOP/s; the error against 64 bits is half of theirs, whose
// scores pass through bf16.  Work is dealt out as runs of (tile, 128 keys) units, equally long for every pair; a tile that
// two or more pairs share leaves fp32 sums behind that a second kernel merges.
#include "host_util.h"
#include "ptx_sm100.cuh"
#include "f32x2.cuh"

namespace omni {

constexpr int AW_C = 384, AW_KEYS = 128, AW_CHUNKS = AW_C / 64, AW_THREADS = 256;
constexpr int AW_Q_BYTES = 128 * AW_C * 2, AW_P_BYTES = 128 * AW_KEYS * 2, AW_STAGE_BYTES = 64 * AW_C, AW_STAGES = 4;
constexpr int AW_SMEM = AW_Q_BYTES + AW_P_BYTES + AW_STAGES * AW_STAGE_BYTES + 1024;
constexpr int AW_S_COL = AW_C;                               // first column of the scores

struct WideAttn {
  CUtensorMap tmQ, tmK, tmV;
  __nv_bfloat16* o;
  long o_rs, o_bs;
  int N, tiles_per, tiles, steps, workers;                   // rows (= keys) per batch entry; tiles of 256 rows; steps of 128 keys; pairs
  float scale_log2;
  float4* part_o;                                            // [slot][CTA][96 column quads][128 rows]
  float2* part_ml;                                           // [slot][CTA][128 rows]: reference exponent, row sum
};

// worker w has the units [wide_start(w), wide_start(w + 1)) of tiles * steps
__device__ __forceinline__ int wide_start(const WideAttn& a, int w) { return (int)((long)w * a.tiles * a.steps / a.workers); }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(AW_THREADS, 1)
wide_attn_kernel(const __grid_constant__ WideAttn a, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t q_full, q_empty, kv_full[AW_STAGES], kv_empty[AW_STAGES], s_full, s_empty, p_full, pv_done, o_full, o_empty;
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int worker = blockIdx.x >> 1;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u, sP = smem_base + AW_Q_BYTES, sKV = sP + AW_P_BYTES;
  const int u0 = wide_start(a, worker), u1 = wide_start(a, worker + 1);

  if (threadIdx.x == 0) {
    s_abort = 0;
    mbar_init(smem_u32(&q_full), 1);
    mbar_init(smem_u32(&q_empty), 1);
    for (int i = 0; i < AW_STAGES; ++i) {
      mbar_init(smem_u32(&kv_full[i]), 1);
      mbar_init(smem_u32(&kv_empty[i]), 1);
    }
    mbar_init(smem_u32(&s_full), 1);
    mbar_init(smem_u32(&s_empty), 8);                        // one arrival per softmax warp of both CTAs
    mbar_init(smem_u32(&p_full), 8);
    mbar_init(smem_u32(&pv_done), 1);
    mbar_init(smem_u32(&o_full), 1);
    mbar_init(smem_u32(&o_empty), 8);
    fence_mbar_init();
    tma_prefetch_desc(&a.tmQ);
    tma_prefetch_desc(&a.tmK);
    tma_prefetch_desc(&a.tmV);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&tmem_base_s), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  pdl_begin();

  // Both roles walk the same order: S(first), then per step S(next) before P V(this) inside a tile, after it where the tile ends.
  if (warp == 0) {
    if (elect_one()) {
      int stage = 0, seg = -1;
      uint32_t phase = 0;
      auto acquire = [&]() {
        mbar_wait(smem_u32(&kv_empty[stage]), phase ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
        if (rank == 0) mbar_expect_tx(smem_u32(&kv_full[stage]), 2 * AW_STAGE_BYTES);
        return mapa_shared(smem_u32(&kv_full[stage]), 0);
      };
      auto advance = [&]() {
        if (++stage == AW_STAGES) { stage = 0; phase ^= 1; }
      };
      auto load_k = [&](int u) {
        const int tile = u / a.steps, j = u - tile * a.steps, b = tile / a.tiles_per;
        if (u == u0 || j == 0) {                             // a tile begins: its queries
          ++seg;
          mbar_wait(smem_u32(&q_empty), (seg & 1) ^ 1, &s_abort, status, ERR_WAIT_EMPTY);
          if (rank == 0) mbar_expect_tx(smem_u32(&q_full), 2 * AW_Q_BYTES);
          const uint32_t qb = mapa_shared(smem_u32(&q_full), 0);
          for (int x = 0; x < AW_CHUNKS; ++x)
            tma_load_3d_pair(smem_base + x * 128 * 128, &a.tmQ, qb, 64 * x, (tile - b * a.tiles_per) * 256 + (int)rank * 128, b);
        }
        for (int h = 0; h < 2; ++h) {
          const uint32_t fb = acquire();
          for (int x = 0; x < AW_CHUNKS / 2; ++x)
            tma_load_3d_pair(sKV + stage * AW_STAGE_BYTES + x * 64 * 128, &a.tmK, fb, 64 * (h * (AW_CHUNKS / 2) + x), j * AW_KEYS + (int)rank * 64, b);
          advance();
        }
      };
      auto load_v = [&](int u) {                             // this CTA's half of channels 0..255 and of 256..383
        const int tile = u / a.steps, j = u - tile * a.steps, b = tile / a.tiles_per;
        for (int h = 0; h < 2; ++h) {
          const uint32_t fb = acquire(), at = sKV + stage * AW_STAGE_BYTES;
          tma_load_3d_pair(at, &a.tmV, fb, (int)rank * 128, j * AW_KEYS + h * 64, b);
          tma_load_3d_pair(at + 64 * 128, &a.tmV, fb, (int)rank * 128 + 64, j * AW_KEYS + h * 64, b);
          tma_load_3d_pair(at + 2 * 64 * 128, &a.tmV, fb, 256 + (int)rank * 64, j * AW_KEYS + h * 64, b);
          advance();
        }
      };
      if (u0 < u1) load_k(u0);
      for (int u = u0; u < u1; ++u) {
        const bool more = u + 1 < u1, same = more && (u + 1) % a.steps != 0;
        if (same) load_k(u + 1);
        load_v(u);
        if (more && !same) load_k(u + 1);
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc(256, AW_KEYS, 1, 1, 0, 0), idesc_wide = umma_idesc(256, 256, 1, 1, 0, 1), idesc_rest = umma_idesc(256, 128, 1, 1, 0, 1);
      int stage = 0, seg = -1;
      uint32_t phase = 0;
      const uint64_t dQ = umma_desc_kmajor_sw128(smem_base), dP = umma_desc_kmajor_sw128(sP);
      auto take = [&]() {
        mbar_wait(smem_u32(&kv_full[stage]), phase, &s_abort, status, ERR_WAIT_FULL);
        tc_fence_after_sync();
        return sKV + stage * AW_STAGE_BYTES;
      };
      auto release = [&]() {
        tc_commit_pair(mapa_shared(smem_u32(&kv_empty[stage]), 0));
        tc_commit_pair(mapa_shared(smem_u32(&kv_empty[stage]), 1));
        if (++stage == AW_STAGES) { stage = 0; phase ^= 1; }
      };
      auto scores = [&](int u) {
        const int g = u - u0, j = u % a.steps;
        if (g == 0 || j == 0) {
          ++seg;
          mbar_wait(smem_u32(&q_full), seg & 1, &s_abort, status, ERR_WAIT_FULL);
        }
        mbar_wait(smem_u32(&s_empty), (g & 1) ^ 1, &s_abort, status, ERR_WAIT_TMEM_EMPTY);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const uint64_t dK = umma_desc_kmajor_sw128(take()), dA = dQ + h * (AW_Q_BYTES / 2 / 16);
#pragma unroll
          for (int k = 0; k < AW_C / 32; ++k)
            mma_f16_ss_pair(tmem_base + AW_S_COL, dA + (k >> 2) * (128 * 128 / 16) + (k & 3) * 2, dK + (k >> 2) * (64 * 128 / 16) + (k & 3) * 2, idesc_s,
                            (h | k) != 0);
          release();
        }
        tc_commit_pair(mapa_shared(smem_u32(&s_full), 0));
        tc_commit_pair(mapa_shared(smem_u32(&s_full), 1));
        if (u + 1 == u1 || j + 1 == a.steps) {               // the tile's last scores here: its queries may go
          tc_commit_pair(mapa_shared(smem_u32(&q_empty), 0));
          tc_commit_pair(mapa_shared(smem_u32(&q_empty), 1));
        }
      };
      if (u0 < u1) scores(u0);
      int pv_seg = -1;
      for (int u = u0; u < u1; ++u) {
        const int g = u - u0, j = u % a.steps;
        const bool more = u + 1 < u1, same = more && j + 1 != a.steps, first = g == 0 || j == 0;
        if (same) scores(u + 1);
        if (first) {
          ++pv_seg;
          mbar_wait(smem_u32(&o_empty), (pv_seg & 1) ^ 1, &s_abort, status, ERR_WAIT_TMEM_EMPTY);   // the tile before has left TMEM
        }
        mbar_wait(smem_u32(&p_full), g & 1, &s_abort, status, ERR_WAIT_SOFTMAX);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const uint64_t dV = umma_desc_sw128(take(), 64 * 128, 1024), dA = dP + h * (AW_P_BYTES / 2 / 16);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            mma_f16_ss_pair(tmem_base, dA + k * 2, dV + k * (16 * 128 / 16), idesc_wide, !(first && (h | k) == 0));
            mma_f16_ss_pair(tmem_base + 256, dA + k * 2, dV + 2 * (64 * 128 / 16) + k * (16 * 128 / 16), idesc_rest, !(first && (h | k) == 0));
          }
          release();
        }
        tc_commit_pair(mapa_shared(smem_u32(&pv_done), 0));
        tc_commit_pair(mapa_shared(smem_u32(&pv_done), 1));
        if (!same) {
          tc_commit_pair(mapa_shared(smem_u32(&o_full), 0));
          tc_commit_pair(mapa_shared(smem_u32(&o_full), 1));
        }
        if (more && !same) scores(u + 1);
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t tO = tmem_base + ((uint32_t)(q * 32) << 16);
    const uint64_t scale2 = pack2(a.scale_log2, a.scale_log2);
    float m = -INFINITY;
    uint64_t la = 0ull, lb = 0ull;
    int seg = 0;
    for (int u = u0; u < u1; ++u) {
      const int g = u - u0, tile = u / a.steps, j = u - tile * a.steps;
      const bool first = g == 0 || j == 0, last = u + 1 == u1 || j + 1 == a.steps;
      const int valid = a.N - j * AW_KEYS;
      mbar_wait(smem_u32(&s_full), g & 1, &s_abort, status, ERR_WAIT_FULL);
      tc_fence_after_sync();
      uint32_t v0[32], v1[32], v2[32], v3[32];
      tmem_ld_32x32(tO + AW_S_COL, v0);
      tmem_ld_32x32(tO + AW_S_COL + 32, v1);
      tmem_ld_32x32(tO + AW_S_COL + 64, v2);
      tmem_ld_32x32(tO + AW_S_COL + 96, v3);
      tmem_wait_ld(v0);
      tmem_wait_ld(v1);
      tmem_wait_ld(v2);
      tmem_wait_ld(v3);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&s_empty), 0));
      if (valid < AW_KEYS) {
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          if (e >= valid) v0[e] = 0xff800000u;
          if (e + 32 >= valid) v1[e] = 0xff800000u;
          if (e + 64 >= valid) v2[e] = 0xff800000u;
          if (e + 96 >= valid) v3[e] = 0xff800000u;
        }
      }
      float x0 = __uint_as_float(v0[0]), x1 = __uint_as_float(v1[0]), x2 = __uint_as_float(v2[0]), x3 = __uint_as_float(v3[0]);
#pragma unroll
      for (int e = 1; e < 31; e += 2) {
        x0 = max3(x0, __uint_as_float(v0[e]), __uint_as_float(v0[e + 1]));
        x1 = max3(x1, __uint_as_float(v1[e]), __uint_as_float(v1[e + 1]));
        x2 = max3(x2, __uint_as_float(v2[e]), __uint_as_float(v2[e + 1]));
        x3 = max3(x3, __uint_as_float(v3[e]), __uint_as_float(v3[e + 1]));
      }
      x0 = fmaxf(fmaxf(x0, __uint_as_float(v0[31])), fmaxf(x1, __uint_as_float(v1[31])));
      x2 = fmaxf(fmaxf(x2, __uint_as_float(v2[31])), fmaxf(x3, __uint_as_float(v3[31])));
      if (first) {
        m = -INFINITY;
        la = lb = 0ull;
      }
      const float m_new = fmaxf(m, fmaxf(x0, x2) * a.scale_log2);
      const bool grow = __any_sync(0xffffffffu, m_new > m + 8.0f) && !first;
      float alpha = 1.f;
      if (grow) {
        alpha = m_new == -INFINITY ? 1.f : ex2_approx(m - m_new);      // a row of -inf scores so far beside one that grows
        la = mul2(la, pack2(alpha, alpha));
        lb = mul2(lb, pack2(alpha, alpha));
      }
      if (grow || first) m = m_new;
      const float m_use = m == -INFINITY ? 0.f : m;
      const uint64_t negm2 = pack2(-m_use, -m_use);
      auto probabilities = [&](uint32_t (&v)[32]) {          // the packed pairs stay in the first half of v
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float p0, p1;
          unpack2(fma2(pack2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), scale2, negm2), p0, p1);
          p0 = ex2_approx(p0);
          p1 = ex2_approx(p1);
          if (e & 2) lb = add2(lb, pack2(p0, p1)); else la = add2(la, pack2(p0, p1));
          v[e >> 1] = pack_bf16(p0, p1);
        }
      };
      probabilities(v0);
      probabilities(v1);
      probabilities(v2);
      probabilities(v3);
      // the product of the step before has read its probabilities, and O may be rescaled
      if (g > 0) mbar_wait(smem_u32(&pv_done), (g - 1) & 1, &s_abort, status, ERR_WAIT_PV);
      if (grow) {
        tc_fence_after_sync();
#pragma unroll 1
        for (int c = 0; c < AW_C / 16; ++c) {
          uint32_t o[16];
          tmem_ld_32x16(tO + c * 16, o);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
          tmem_st_32x16(tO + c * 16, o);
        }
        tmem_wait_st();
        tc_fence_before_sync();
      }
      auto put = [&](const uint32_t (&v)[32], int i) {       // 32 keys: four 16-byte groups of the row, swizzled as the MMA reads them
#pragma unroll
        for (int c = 0; c < 4; ++c)
          st_shared_v4(sP + (i >> 1) * 128 * 128 + row * 128 + ((((i & 1) * 4 + c) ^ (row & 7)) << 4),
                       make_uint4(v[c * 4], v[c * 4 + 1], v[c * 4 + 2], v[c * 4 + 3]));
      };
      put(v0, 0);
      put(v1, 1);
      put(v2, 2);
      put(v3, 3);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&p_full), 0));
      if (!last) continue;

      float l;
      {
        float s0, s1, s2, s3;
        unpack2(la, s0, s1);
        unpack2(lb, s2, s3);
        l = (s0 + s1) + (s2 + s3);
      }
      const int b = tile / a.tiles_per, srow = (tile - b * a.tiles_per) * 256 + (int)rank * 128 + row;
      const bool begins = u - j >= u0;                        // this pair has the tile's first keys
      const bool whole = begins && j + 1 == a.steps;
      const long slot = ((long)worker * 2 + (begins ? 1 : 0)) * 2 + rank;
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      mbar_wait(smem_u32(&o_full), seg & 1, &s_abort, status, ERR_WAIT_PV);
      ++seg;
      tc_fence_after_sync();
      __nv_bfloat16* orow = a.o + (long)b * a.o_bs + (long)srow * a.o_rs;
      if (!whole) a.part_ml[slot * 128 + row] = make_float2(m, l);
#pragma unroll 1
      for (int c = 0; c < AW_C / 32; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(tO + c * 32, v);
        tmem_wait_ld();
        if (whole) {
          if (srow < a.N) {
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
              uint4 w;
              w.x = pack_bf16(__uint_as_float(v[e]) * inv, __uint_as_float(v[e + 1]) * inv);
              w.y = pack_bf16(__uint_as_float(v[e + 2]) * inv, __uint_as_float(v[e + 3]) * inv);
              w.z = pack_bf16(__uint_as_float(v[e + 4]) * inv, __uint_as_float(v[e + 5]) * inv);
              w.w = pack_bf16(__uint_as_float(v[e + 6]) * inv, __uint_as_float(v[e + 7]) * inv);
              *reinterpret_cast<uint4*>(orow + c * 32 + e) = w;
            }
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; e += 4)
            a.part_o[(slot * (AW_C / 4) + c * 8 + e / 4) * 128 + row] =
                make_float4(__uint_as_float(v[e]), __uint_as_float(v[e + 1]), __uint_as_float(v[e + 2]), __uint_as_float(v[e + 3]));
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&o_empty), 0));
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
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// One thread per row and 32 channels of a tile that several pairs share.
__global__ void __launch_bounds__(128)
wide_attn_merge_kernel(const __grid_constant__ WideAttn a) {
  pdl_begin();
  const int tile = blockIdx.x, rank = blockIdx.y, c0 = blockIdx.z * 8, row = threadIdx.x;
  const int first = tile * a.steps, end = first + a.steps;
  int w = (int)((long)first * a.workers / ((long)a.tiles * a.steps));
  while (wide_start(a, w + 1) <= first) ++w;
  if (wide_start(a, w + 1) >= end) return;                   // one pair had all keys and wrote the rows
  const int b = tile / a.tiles_per, srow = (tile - b * a.tiles_per) * 256 + rank * 128 + row;
  if (srow >= a.N) return;
  auto slot_of = [&](int p) { return ((long)p * 2 + (wide_start(a, p) <= first ? 1 : 0)) * 2 + rank; };
  float M = -INFINITY, l = 0.f;
  for (int p = w; wide_start(a, p) < end && p < a.workers; ++p) M = fmaxf(M, a.part_ml[slot_of(p) * 128 + row].x);
  float acc[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) acc[e] = 0.f;
  for (int p = w; wide_start(a, p) < end && p < a.workers; ++p) {
    const long slot = slot_of(p);
    const float2 ml = a.part_ml[slot * 128 + row];
    const float s = ml.x == -INFINITY ? 0.f : ex2_approx(ml.x - M);
    l = fmaf(ml.y, s, l);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 v = a.part_o[(slot * (AW_C / 4) + c0 + i) * 128 + row];
      acc[i * 4] = fmaf(v.x, s, acc[i * 4]);
      acc[i * 4 + 1] = fmaf(v.y, s, acc[i * 4 + 1]);
      acc[i * 4 + 2] = fmaf(v.z, s, acc[i * 4 + 2]);
      acc[i * 4 + 3] = fmaf(v.w, s, acc[i * 4 + 3]);
    }
  }
  const float inv = l > 0.f ? 1.0f / l : 0.f;
  __nv_bfloat16* out = a.o + (long)b * a.o_bs + (long)srow * a.o_rs + c0 * 4;
#pragma unroll
  for (int e = 0; e < 32; e += 8)
    *reinterpret_cast<uint4*>(out + e) = make_uint4(pack_bf16(acc[e] * inv, acc[e + 1] * inv), pack_bf16(acc[e + 2] * inv, acc[e + 3] * inv),
                                                    pack_bf16(acc[e + 4] * inv, acc[e + 5] * inv), pack_bf16(acc[e + 6] * inv, acc[e + 7] * inv));
}

// Pairs that share the work: a tile each, in waves; or each tile cut into equally many shares; or every pair of the chip in runs that begin and end
// inside tiles.  Estimated in steps of 128 keys (about 2.6 us): the longest run, 0.08 per pair for sums that are written and merged, and as much per
// tile and 3 for the second tile of a run (its queries come in while nothing else can run) where runs cross tiles.  us, a tile each / shares / runs:
// 2048 rows 52 / 29 (4 shares) / 45; 8192 174 / 104 (2) / 104; 10000 211 / - / 140; 16384 340 / - / 321.
static int wide_workers(long tiles, long steps, int pairs) {
  const long units = tiles * steps;
  double best = (double)((tiles + pairs - 1) / pairs * steps);
  long workers = tiles;
  auto consider = [&](long w, double extra) {
    const double cost = (double)((units + w - 1) / w) + extra;
    if (cost < best) { best = cost; workers = w; }
  };
  for (long n = 2; n <= steps && n * tiles <= pairs; ++n) consider(n * tiles, 0.08 * (n * tiles));
  if (units >= pairs && pairs % tiles != 0) consider(pairs, 0.08 * (pairs + tiles) + 3);
  return (int)workers;
}

static int wide_map(CUtensorMap* m, const void* p, long N, long B, long rs, long bs, int rows) {
  if ((rs & 7) || (bs & 7)) return RC_BAD_ARG;
  return make_tmap_3d(m, p, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, AW_C, (uint64_t)N, (uint64_t)B, (uint64_t)rs * 2, (uint64_t)bs * 2, 64, rows);
}

}  // namespace omni

// Pairs of CTAs that omni_attn_wide uses for B entries of N rows; scratch_floats (may be null) takes the fp32 scratch it needs, 0 where no tile is shared.
extern "C" int omni_attn_wide_workers(int B, int N, long* scratch_floats) {
  using namespace omni;
  if (scratch_floats) *scratch_floats = 0;
  if (B <= 0 || N <= 0) return 0;
  const long tiles = (long)B * ((N + 255) / 256), steps = (N + AW_KEYS - 1) / AW_KEYS;
  const int w = wide_workers(tiles, steps, sm_count() / 2);
  if (scratch_floats) *scratch_floats = w == tiles ? 0 : (long)w * 4 * 128 * (AW_C + 2);
  return w;
}

// out[b, r, :] = softmax(scale q[b, r] k[b]^T) v[b] for one head of 384 channels; q, k, v, out bf16 [B, N, 384] with row and batch strides in elements
// (multiples of 8) and contiguous channels, bases on 16 bytes.  workers: what omni_attn_wide_workers says, or any other number of pairs; scratch (may be null where
// no tile is shared): 4 * 128 * (384 + 2) floats for each.
extern "C" int omni_attn_wide(const void* q, long q_rs, long q_bs, const void* k, long k_rs, long k_bs, const void* v, long v_rs, long v_bs, void* out,
                              long o_rs, long o_bs, int B, int N, int C, float scale, int workers, float* scratch, int* status, void* stream) {
  using namespace omni;
  if (C != AW_C || B < 0 || N < 0 || (reinterpret_cast<uintptr_t>(out) & 15) || (o_rs & 7) || (o_bs & 7)) return RC_BAD_ARG;
  if (B == 0 || N == 0) return RC_OK;
  WideAttn a;
  if (int rc = wide_map(&a.tmQ, q, N, B, q_rs, q_bs, 128)) return rc;
  if (int rc = wide_map(&a.tmK, k, N, B, k_rs, k_bs, 64)) return rc;
  if (int rc = wide_map(&a.tmV, v, N, B, v_rs, v_bs, 64)) return rc;
  a.o = static_cast<__nv_bfloat16*>(out);
  a.o_rs = o_rs; a.o_bs = o_bs;
  a.N = N;
  a.tiles_per = (N + 255) / 256;
  a.steps = (N + AW_KEYS - 1) / AW_KEYS;
  const long tiles = (long)B * a.tiles_per;
  if (tiles * a.steps > 0x3fffffffL) return RC_TOO_LARGE;
  a.tiles = (int)tiles;
  if (workers < 1 || workers > tiles * a.steps) return RC_BAD_ARG;
  a.workers = workers;
  a.scale_log2 = scale * 1.4426950408889634f;
  const bool shared = a.workers != a.tiles;
  if (shared && (scratch == nullptr || (reinterpret_cast<uintptr_t>(scratch) & 15))) return RC_BAD_ARG;
  a.part_o = reinterpret_cast<float4*>(scratch);
  a.part_ml = reinterpret_cast<float2*>(scratch + (shared ? (long)a.workers * 4 * 128 * AW_C : 0));
  static unsigned long long prepared = 0;
  if (int e = ensure_dynamic_smem((const void*)wide_attn_kernel, AW_SMEM, prepared)) return e;
  cudaStream_t st = (cudaStream_t)stream;
  launch_overlapped(wide_attn_kernel, 2 * a.workers, AW_THREADS, AW_SMEM, st, a, status);
  if (shared) launch_overlapped(wide_attn_merge_kernel, dim3(a.tiles, 2, AW_C / 32), 128, 0, st, a);
  return (int)cudaGetLastError();
}
