// Paged attention of decoded tokens (one query token per sequence), bf16, head size 128.
//
// A decode step reads every cached K and V byte once, so the kernel is a stream from HBM with a little arithmetic on the way.
// Nothing is staged: K and V go from their pages straight into the registers of the warp that uses them, as operands of
// 16 x 8 x 16 products.
//   S[head, key]   = q K^T      the heads of a group are the rows, keys the columns; lane group j of a quad owns channels 8 j .. 8 j + 7 of every
//                               32-channel chunk for both operands (one 16-byte load per key and chunk; the contraction is
//                               permuted alike on both sides)
//   O^T[ch, head] += V^T P^T    channels are the rows: lane (g, j) loads channels 8 g .. 8 g + 7 (and 64 more) of keys 2 j, 2 j + 1, 2 j + 8, 2 j + 9
//                               and pairs neighbouring keys with byte permutes; P^T needs no exchange, because the accumulator of S is laid
//                               out as this operand
// A warp owns one KV head of one share of the keys, the warps of a block neighbouring heads of the same keys, so that a block
// reads whole page rows.  The next 16 keys are requested as soon as their registers are free: 12 warps x 8 KB are in flight per SM.
// Caches cold, launches included:
// 64 sequences of about 1800 keys, 32 / 4 heads (236 MB) 58 us (tcgen05 kernel: 95), 64 of 4000 with 32 / 8 heads 183 us (212), one of 1414 keys
// 18 us (20).  The tcgen05 kernel (attention_sm100.cu) stays for groups of more than 16 heads.
#include "host_util.h"
#include "ptx_sm100.cuh"

namespace omni {

constexpr int DA_D = 128, DA_WARPS = 4, DA_KEYS = 16;

struct DecodeAttn {
  const __nv_bfloat16 *q, *k, *v;
  long q_rs;
  const int* block_tables;
  int bt_stride, block_size;
  const int* lens;
  int max_keys;                      // no sequence has more
  int H, Hkv, splits, subs;          // shares of the keys: blocks, and warps of a block
  float scale_log2;
  float *part_o, *part_ml;
  __nv_bfloat16* out;
  long o_rs;
  const long long* rows;             // sequence -> row of q and out (below zero: from the end); null: the sequence's number
  int n_rows;
  int* status;
};

// Row of q and out; -1 where there is none, which the status word tells the host.
template <bool ROWS>
__device__ __forceinline__ long da_row(const DecodeAttn& p, int seq) {
  if (!ROWS) return seq;
  long long r = p.rows[seq];
  if (r < 0) r += p.n_rows;
  if (r >= 0 && r < p.n_rows) return (long)r;
  atomicCAS(p.status, 0, ERR_BOUNDS);
  return -1;
}

// UP: 9 .. 16 heads per group, the second half of the MMA's 16 rows is live.
template <bool UP, bool ROWS>
__global__ void __launch_bounds__(32 * DA_WARPS, UP ? 2 : 3)
paged_decode_kernel(const __grid_constant__ DecodeAttn p) {
  pdl_begin();
  constexpr int NH = UP ? 2 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  const int seq = blockIdx.y, split = blockIdx.x;
  const int per_block = min(DA_WARPS, p.Hkv), sub = warp / per_block;
  const int hk = blockIdx.z * DA_WARPS + warp % per_block;
  if (sub >= p.subs || hk >= p.Hkv) return;
  const int G = p.H / p.Hkv, h0 = hk * G, parts = p.splits * p.subs;
  const long q_row = da_row<ROWS>(p, seq);
  if (q_row < 0) return;
  const int len = min(p.lens[seq], p.max_keys);
  const int tiles = (len + DA_KEYS - 1) / DA_KEYS, per = (tiles + p.splits - 1) / p.splits;
  const int t1 = min(tiles, (split + 1) * per);
  if (split * per + sub >= t1) {      // no keys (a table wider than the sequence): weight zero, and no sum for the merge to read
    if (parts > 1 && lane < G) {
      float* ml = p.part_ml + (((long)seq * p.H + h0 + lane) * parts + split * p.subs + sub) * 2;
      ml[0] = -INFINITY;
      ml[1] = 0.f;
    }
    if (parts > 1) return;
  }
  const int* bt = p.block_tables + (long)seq * p.bt_stride;
  const long row = (long)p.Hkv * DA_D;

  uint4 q[NH][4];
#pragma unroll
  for (int u = 0; u < NH; ++u)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      q[u][c] = u * 8 + g < G ? *reinterpret_cast<const uint4*>(p.q + q_row * p.q_rs + (long)(h0 + u * 8 + g) * DA_D + c * 32 + j * 8)
                              : make_uint4(0u, 0u, 0u, 0u);
  float m[NH], l[NH], acc[NH][8][4];
#pragma unroll
  for (int u = 0; u < NH; ++u) {
    m[u] = -INFINITY;
    l[u] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[u][i][e] = 0.f;
  }

  // first rows of the two 8-key halves of tile t (a half past the end repeats the first one)
  auto pages = [&](int t, int& a, int& b) {
    const int k0 = t * DA_KEYS, k1 = k0 + 8 < len ? k0 + 8 : k0;
    a = bt[k0 / p.block_size] * p.block_size + k0 % p.block_size;
    b = bt[k1 / p.block_size] * p.block_size + k1 % p.block_size;
  };
  // rows past the end repeat the last key: valid memory, its weight is zero
  auto row_in_half = [&](int t, int half, int r) {
    const int k0 = t * DA_KEYS + (t * DA_KEYS + 8 * half < len ? 8 * half : 0);
    return min(r, len - 1 - k0);
  };
  uint4 kr[2][4], vr[4][2];
  auto load_k = [&](int t, int a, int b) {
    const __nv_bfloat16* k0 = p.k + (long)(a + row_in_half(t, 0, g)) * row + (long)hk * DA_D + j * 8;
    const __nv_bfloat16* k1 = p.k + (long)(b + row_in_half(t, 1, g)) * row + (long)hk * DA_D + j * 8;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      kr[0][c] = ld_stream(k0 + c * 32);
      kr[1][c] = ld_stream(k1 + c * 32);
    }
  };
  auto load_v = [&](int t, int a, int b) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat16* v = p.v + (long)((i < 2 ? a : b) + row_in_half(t, i >> 1, 2 * j + (i & 1))) * row + (long)hk * DA_D + g * 8;
      vr[i][0] = ld_stream(v);
      vr[i][1] = ld_stream(v + 64);
    }
  };
  int t = split * per + sub, pa = 0, pb = 0, na = 0, nb = 0;
  if (t < t1) {
    pages(t, pa, pb);
    load_k(t, pa, pb);
    load_v(t, pa, pb);
    if (t + p.subs < t1) pages(t + p.subs, na, nb);
  }
#pragma unroll 1
  for (; t < t1; t += p.subs) {
    const int next = t + p.subs;
    float s[2][4] = {};
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const uint4 hi = UP ? q[NH - 1][c] : make_uint4(0u, 0u, 0u, 0u);
        mma_bf16_16x8(s[n], q[0][c].x, hi.x, q[0][c].y, hi.y, kr[n][c].x, kr[n][c].y);
        mma_bf16_16x8(s[n], q[0][c].z, hi.z, q[0][c].w, hi.w, kr[n][c].z, kr[n][c].w);
      }
    if (next < t1) load_k(next, na, nb);
    uint32_t pw[NH][2];
#pragma unroll
    for (int u = 0; u < NH; ++u) {
      const float before = m[u];
      float mx = -INFINITY;
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float y = t * DA_KEYS + n * 8 + 2 * j + e < len ? s[n][2 * u + e] * p.scale_log2 : -INFINITY;
          s[n][2 * u + e] = y;
          mx = fmaxf(mx, y);
        }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      m[u] = fmaxf(m[u], mx);
      const float top = m[u] == -INFINITY ? 0.f : m[u];        // only scores of -inf so far: all weights are zero
      const float alpha = ex2_approx(before - top);
      l[u] *= alpha;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float e0 = ex2_approx(s[n][2 * u] - top), e1 = ex2_approx(s[n][2 * u + 1] - top);
        l[u] += e0 + e1;
        pw[u][n] = pack_bf16(e0, e1);
      }
      const float a0 = __shfl_sync(0xffffffffu, alpha, 8 * j), a1 = __shfl_sync(0xffffffffu, alpha, 8 * j + 4);   // heads 2 j, 2 j + 1
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[u][i][0] *= a0; acc[u][i][1] *= a1;
        acc[u][i][2] *= a0; acc[u][i][3] *= a1;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int w = i >> 1, sel = i & 1 ? 0x7632 : 0x5410;
      auto word = [&](const uint4& x) { return w == 0 ? x.x : (w == 1 ? x.y : (w == 2 ? x.z : x.w)); };
      const uint32_t v0 = __byte_perm(word(vr[0][0]), word(vr[1][0]), sel), v1 = __byte_perm(word(vr[0][1]), word(vr[1][1]), sel);
      const uint32_t v2 = __byte_perm(word(vr[2][0]), word(vr[3][0]), sel), v3 = __byte_perm(word(vr[2][1]), word(vr[3][1]), sel);
#pragma unroll
      for (int u = 0; u < NH; ++u) mma_bf16_16x8(acc[u][i], v0, v1, v2, v3, pw[u][0], pw[u][1]);
    }
    if (next < t1) {
      load_v(next, na, nb);
      if (next + p.subs < t1) pages(next + p.subs, na, nb);
    }
  }
#pragma unroll
  for (int u = 0; u < NH; ++u) {
    l[u] += __shfl_xor_sync(0xffffffffu, l[u], 1);
    l[u] += __shfl_xor_sync(0xffffffffu, l[u], 2);
    const float inv = l[u] > 0.f ? 1.0f / l[u] : 0.f;
    const float i0 = __shfl_sync(0xffffffffu, inv, 8 * j), i1 = __shfl_sync(0xffffffffu, inv, 8 * j + 4);
    const long base = (long)seq * p.H + h0 + u * 8;
    if (parts > 1 && j == 0 && u * 8 + g < G) {
      float* ml = p.part_ml + ((base + g) * parts + split * p.subs + sub) * 2;
      ml[0] = m[u];
      ml[1] = l[u];
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int h = 2 * j + hh;
      if (u * 8 + h >= G) continue;
#pragma unroll
      for (int b = 0; b < 2; ++b) {                            // channels b * 64 + 8 g .. + 7
        if (parts > 1) {
          float* o = p.part_o + ((base + h) * parts + split * p.subs + sub) * DA_D + b * 64 + g * 8;
          *reinterpret_cast<float4*>(o) = make_float4(acc[u][0][2 * b + hh], acc[u][1][2 * b + hh], acc[u][2][2 * b + hh], acc[u][3][2 * b + hh]);
          *reinterpret_cast<float4*>(o + 4) = make_float4(acc[u][4][2 * b + hh], acc[u][5][2 * b + hh], acc[u][6][2 * b + hh], acc[u][7][2 * b + hh]);
        } else {
          const float f = hh ? i1 : i0;
          uint4 w;
          w.x = pack_bf16(acc[u][0][2 * b + hh] * f, acc[u][1][2 * b + hh] * f);
          w.y = pack_bf16(acc[u][2][2 * b + hh] * f, acc[u][3][2 * b + hh] * f);
          w.z = pack_bf16(acc[u][4][2 * b + hh] * f, acc[u][5][2 * b + hh] * f);
          w.w = pack_bf16(acc[u][6][2 * b + hh] * f, acc[u][7][2 * b + hh] * f);
          *reinterpret_cast<uint4*>(p.out + q_row * p.o_rs + (long)(h0 + u * 8 + h) * DA_D + b * 64 + g * 8) = w;
        }
      }
    }
  }
}

// out[seq, h] = sum_s 2^(m_s - m*) O_s / sum_s 2^(m_s - m*) l_s over a row's shares (at most 64): one block per row, its warps take
// every fourth share, four channels per lane.
template <bool ROWS>
__global__ void __launch_bounds__(128)
paged_decode_merge_kernel(const float* part_o, const float* part_ml, int parts, int H, __nv_bfloat16* __restrict__ out, long o_rs, const long long* rows, int n_rows) {
  pdl_begin();
  __shared__ float4 part[4][32];
  const long r = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + r * parts;
  const float4* po = reinterpret_cast<const float4*>(part_o) + r * parts * (DA_D / 4) + lane;
  const float2 a = lane < parts ? ml[lane] : make_float2(-INFINITY, 0.f);
  const float2 b = lane + 32 < parts ? ml[lane + 32] : make_float2(-INFINITY, 0.f);
  float top = fmaxf(a.x, b.x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  const float wa = a.x == -INFINITY ? 0.f : ex2_approx(a.x - top), wb = b.x == -INFINITY ? 0.f : ex2_approx(b.x - top);
  float den = a.y * wa + b.y * wb;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (int s0 = warp; s0 < parts; s0 += 32) {
    float w[8];
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int s = s0 + 4 * i;                                // below 64 + 32: a lane of a or b, or past the end
      w[i] = __shfl_sync(0xffffffffu, s < 32 ? wa : wb, s & 31);
      // a share without keys has written no sum
      x[i] = s < parts && w[i] != 0.f ? po[(long)s * (DA_D / 4)] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      acc.x = fmaf(x[i].x, w[i], acc.x); acc.y = fmaf(x[i].y, w[i], acc.y);
      acc.z = fmaf(x[i].z, w[i], acc.z); acc.w = fmaf(x[i].w, w[i], acc.w);
    }
  }
  part[warp][lane] = acc;
  __syncthreads();
  if (warp) return;
#pragma unroll
  for (int i = 1; i < 4; ++i) {
    const float4 x = part[i][lane];
    acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
  }
  const float f = den > 0.f ? 1.0f / den : 0.f;
  const int seq = (int)blockIdx.x / H;
  long row = seq;
  if (ROWS) {
    row = rows[seq];
    if (row < 0) row += n_rows;
    if (row < 0 || row >= n_rows) return;
  }
  uint2 w;
  w.x = pack_bf16(acc.x * f, acc.y * f);
  w.y = pack_bf16(acc.z * f, acc.w * f);
  *reinterpret_cast<uint2*>(out + row * o_rs + ((int)blockIdx.x - seq * H) * DA_D + lane * 4) = w;
}

constexpr int DA_MAX_PARTS = 64;

// Shares of a sequence's keys: about `target` warps in all, at least two tiles of 16 keys each.  Twelve warps fit an SM; two rounds of them
// even out lengths (8 sequences of 4096 keys, 8 KV heads: 20 warps per SM 1.05 and 18 1.12 times as long as 24).  The number depends on how many sequences
// there are and on the table's width, never on the lengths: a sequence's result is the same whatever its neighbours hold, and probabilities are rounded
// against the maximum of short shares.  (As many shares as make one round of warps, from the sum of the lengths: 48 sequences of about 2600 keys, 32 heads,
// 8 KV heads 93 us instead of 103, but 2 to 5 % further from 64-bit results: 64 sequences of 900 to 2700 keys, 4 KV heads 0.00214 instead of 0.00208.)  Blocks of fewer KV
// heads hold shares of one sequence, whose sums are many and small: 20, since 24 took 1.11 times the tensor-core kernel's time for 72
// sequences of 1024 keys in tables of 4096 and 1 KV head, and 20 never more than 1.01 of it.  A single sequence has at most
// 64 shares: 131072 keys of 4 KV heads take 148 us, the tensor-core kernel 246 (the copy rate would be 41; more shares would reach more SMs).
static void plan_shares(int n, int Hkv, int max_keys, int& splits, int& subs) {
  subs = Hkv < DA_WARPS ? DA_WARPS / Hkv : 1;
  const long warps = (long)n * Hkv, target = (Hkv < DA_WARPS ? 20L : 24L) * sm_count();
  const int tiles = (max_keys + DA_KEYS - 1) / DA_KEYS;
  long parts = (target + warps - 1) / warps;
  if (parts > tiles / 2) parts = tiles / 2;
  if (parts > DA_MAX_PARTS) parts = DA_MAX_PARTS;
  if (parts < 1) parts = 1;
  if (subs > parts) subs = (int)parts;
  splits = (int)(parts + subs - 1) / subs;
  if (splits * subs > DA_MAX_PARTS) splits = DA_MAX_PARTS / subs;
}

}  // namespace omni

using namespace omni;

// Shares per (sequence, head) that omni_paged_decode_attn will write: sizes its scratch (fp32, shares x 128 and shares x 2 each).
extern "C" int omni_paged_decode_shares(int n, int Hkv, int max_keys) {
  int splits, subs;
  plan_shares(n < 1 ? 1 : n, Hkv < 1 ? 1 : Hkv, max_keys, splits, subs);
  return splits * subs;
}

// q [n, H, 128] (row pitch q_rs elements, heads side by side), pages [blocks, block_size, Hkv, 128] with block_size a multiple of 8,
// block_tables int32 [n, bt_stride], lens int32 [n] (counted up to max_keys), out [n, H, 128] (pitch o_rs).  rows (may be null): int64 [n], sequence i
// is row rows[i] of q and out, which then have n_rows rows.
extern "C" int omni_paged_decode_attn(const void* q, long q_rs, const void* k, const void* v, const int* block_tables, int bt_stride,
                                      int block_size, const int* lens, int n, int H, int Hkv, int max_keys, float scale, float* part_o,
                                      float* part_ml, void* out, long o_rs, const long long* rows, int n_rows, int* status, void* stream) {
  if (n <= 0) return RC_OK;
  if (Hkv <= 0 || H % Hkv || H / Hkv > 16 || block_size < 8 || (block_size & 7) || max_keys < 1 || n > 65535 || (q_rs & 7) || (o_rs & 7))
    return RC_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out)) & 15)
    return RC_BAD_ARG;
  DecodeAttn p;
  plan_shares(n, Hkv, max_keys, p.splits, p.subs);
  const int parts = p.splits * p.subs;
  if (parts > 1 && (!part_o || !part_ml)) return RC_BAD_ARG;
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
  p.q_rs = q_rs; p.block_tables = block_tables; p.bt_stride = bt_stride; p.block_size = block_size; p.lens = lens; p.max_keys = max_keys;
  p.H = H; p.Hkv = Hkv; p.scale_log2 = scale * 1.4426950408889634f;
  p.part_o = part_o; p.part_ml = part_ml; p.out = (__nv_bfloat16*)out; p.o_rs = o_rs;
  p.rows = rows; p.n_rows = n_rows; p.status = status;
  const dim3 grid((unsigned)p.splits, (unsigned)n, (unsigned)((Hkv + DA_WARPS - 1) / DA_WARPS));
  cudaStream_t st = (cudaStream_t)stream;
  const bool up = H / Hkv > 8;
  // The blocks of many sequences are dealt out unevenly around the last blocks of the kernel before, few ones gain from the early start.  Decode steps of four
  // layers in us, ordinary launch (overlapped): 4096 wide, 8 KV heads, 50 sequences of 4000 keys 957 (1123), 24 of 1000 521 (527), 14 of 300 494.8 (493.5), 8 of 800
  // 431 (430); 2048 wide, 4 KV heads, 20 of 500 263 (270), 14 of 300 217.8 (217.3); experts, 4 KV heads, 64 of 2048 1128 (1205), 32 of 90 856 (858).
  launch_with(n <= 16, 1, rows ? (up ? paged_decode_kernel<true, true> : paged_decode_kernel<false, true>)
                         : (up ? paged_decode_kernel<true, false> : paged_decode_kernel<false, false>), grid, 32 * DA_WARPS, 0, st, p);
  if (parts == 1) return (int)cudaGetLastError();
  if (cudaError_t e = cudaGetLastError()) return (int)e;
  launch_overlapped(rows ? paged_decode_merge_kernel<true> : paged_decode_merge_kernel<false>, (unsigned)n * H, 128, 0, st, part_o, part_ml, parts, H, (__nv_bfloat16*)out, o_rs, rows, n_rows);
  return (int)cudaGetLastError();
}
