// Bandwidth-bound fused kernels of the DiT / AR blocks (K6, K7, K8, K9, K14).
// Each of them reads its inputs once with 16-byte vector loads, does all arithmetic in
// fp32 registers and writes bf16 once, so the roofline is bytes / HBM bandwidth.
//
//  omni_norm_modulate   LayerNorm / RMSNorm (+weight, +bias) fused with the AdaLN
//                       modulation y = norm(x) * (1 + scale[b]) + shift[b]
//                       (reference: vllm_omni/diffusion/layers/adalayernorm.py)
//  omni_qk_norm_rope    per-head RMSNorm of q and k fused with rotary embedding, in place on
//                       a packed [B, S, 3, H, D] qkv buffer; interleaved (complex-pair) or
//                       half-rotation layout; separate norm weights for rows >= s_alt (the text
//                       rows that follow the image rows in the joint sequence)
//                       (reference: qwen_image_transformer.py:561-661, layers/rope.py:94-154)
//  omni_cfg_euler_step  guidance mix neg + s (pos - neg), optional norm rescale, flow-match
//                       Euler update x += dt * v, bf16 copy of the new latents
//                       (reference: vllm_omni/diffusion/distributed/cfg_parallel.py:99-137)
//  omni_silu_mul        SwiGLU gate: silu(x[:, :N]) * x[:, N:] (_f32: the same in fp32)
//  omni_rel_l1_partial / omni_rel_l1_finish
//                       TeaCache residual metric sum|a-b| / sum|b| with the polynomial
//                       rescale, accumulation and skip decision kept on the device
//                       (reference: vllm_omni/diffusion/cache/teacache/hook.py:185-232)
#include "host_util.h"
#include "ptx_sm100.cuh"
#include "peer_signal.cuh"

namespace omni {

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&x)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y; x[4] = c.x; x[5] = c.y; x[6] = d.x; x[7] = d.y;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&x)[8]) {
  uint4 u;
  u.x = pack_bf16(x[0], x[1]); u.y = pack_bf16(x[2], x[3]);
  u.z = pack_bf16(x[4], x[5]); u.w = pack_bf16(x[6], x[7]);
  *reinterpret_cast<uint4*>(p) = u;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------- norm + modulate
// Up to a row per SM of more than 1024 channels: one block per row, CPT 16-byte chunks per thread.  Gains and modulation are fetched
// together with the row, so a launch is one round trip to memory and one reduction; short code matters as much, because a
// launch of a few rows spends its time fetching instructions.  Caches cold, launch included: 8 rows of 4096 8 us (one
// warp per row with all chunks unrolled: 18).
template <int CPT>
__global__ void __launch_bounds__(512)
norm_modulate_kernel(const __nv_bfloat16* x, __nv_bfloat16* __restrict__ y, int D, int ldx, int ldy,
                     const __nv_bfloat16* weight, const __nv_bfloat16* bias,
                     const __nv_bfloat16* shift, const __nv_bfloat16* scale, int mod_stride,
                     int rows_per_batch, int rms, float eps) {
  pdl_begin();
  __shared__ float2 red[16];
  const int row = blockIdx.x, nchunk = D >> 3, warps = blockDim.x >> 5;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * ldx);
  const size_t mod = (size_t)(row / rows_per_batch) * mod_stride;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 v[CPT], wv[CPT], bv[CPT], sh[CPT], sc[CPT];
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    const bool in = c < nchunk;
    v[i] = in ? xr[c] : zero;
    if (weight) wv[i] = in ? *reinterpret_cast<const uint4*>(weight + c * 8) : zero;
    if (bias) bv[i] = in ? *reinterpret_cast<const uint4*>(bias + c * 8) : zero;
    if (scale) sc[i] = in ? *reinterpret_cast<const uint4*>(scale + mod + c * 8) : zero;
    if (shift) sh[i] = in ? *reinterpret_cast<const uint4*>(shift + mod + c * 8) : zero;
  }
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16(w[j]);
      s += f.x + f.y;
      ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
    }
  }
  s = warp_sum(s);
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(s, ss);
  __syncthreads();
  s = 0.f; ss = 0.f;
  for (int w = 0; w < warps; ++w) { s += red[w].x; ss += red[w].y; }
  const float inv_d = 1.0f / (float)D;
  const float mean = rms ? 0.f : s * inv_d;
  const float var = rms ? ss * inv_d : fmaxf(ss * inv_d - mean * mean, 0.f);
  const float rstd = rsqrtf(var + eps);
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * ldy);
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c >= nchunk) break;
    uint32_t o[4];
    const uint32_t vv[4] = {v[i].x, v[i].y, v[i].z, v[i].w}, ww[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
    const uint32_t bb[4] = {bv[i].x, bv[i].y, bv[i].z, bv[i].w}, cc[4] = {sc[i].x, sc[i].y, sc[i].z, sc[i].w};
    const uint32_t hh[4] = {sh[i].x, sh[i].y, sh[i].z, sh[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = unpack_bf16(vv[j]);
      f.x = (f.x - mean) * rstd;
      f.y = (f.y - mean) * rstd;
      if (weight) { const float2 t = unpack_bf16(ww[j]); f.x *= t.x; f.y *= t.y; }
      if (bias) { const float2 t = unpack_bf16(bb[j]); f.x += t.x; f.y += t.y; }
      if (scale) { const float2 t = unpack_bf16(cc[j]); f.x = fmaf(f.x, t.x, f.x); f.y = fmaf(f.y, t.y, f.y); }
      if (shift) { const float2 t = unpack_bf16(hh[j]); f.x += t.x; f.y += t.y; }
      o[j] = pack_bf16(f.x, f.y);
    }
    yr[c] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// More rows, or rows of up to 1024 channels: WPR warps per row, the row packed (bf16) in VPL 16-byte registers per lane.  All loads of a
// row are in flight at once and 40 to 60 registers leave room for 32 warps and more per SM.  8192 rows of 4096 (134 MB): 34 us, with one
// warp per row and 16 chunks per lane 48 us; keeping rows in flight through shared memory instead (bulk copies,
// 200 KB per SM) did not help: 16 warps issue too little.
template <int VPL, int WPR>
__global__ void __launch_bounds__(256)
norm_modulate_warp_kernel(const __nv_bfloat16* x, __nv_bfloat16* __restrict__ y, int rows,
                          int D, int ldx, int ldy, const __nv_bfloat16* weight,
                          const __nv_bfloat16* bias, const __nv_bfloat16* shift,
                          const __nv_bfloat16* scale, int mod_stride, int rows_per_batch,
                          int rms, float eps) {
  pdl_begin();
  __shared__ float2 red[8];
  const int warp = threadIdx.x >> 5, row = blockIdx.x * (8 / WPR) + warp / WPR;
  const int lane = (threadIdx.x & 31) + (warp % WPR) * 32;
  if (WPR == 1 && row >= rows) return;
  const bool live = row < rows;
  const int nchunk = live ? D >> 3 : 0;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * ldx);
  uint4 v[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = lane + i * 32 * WPR;
    v[i] = c < nchunk ? xr[c] : make_uint4(0u, 0u, 0u, 0u);
  }
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16(w[j]);
      s += f.x + f.y;
      ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
    }
  }
  s = warp_sum(s);
  ss = warp_sum(ss);
  if (WPR > 1) {
    if ((threadIdx.x & 31) == 0) red[warp] = make_float2(s, ss);
    __syncthreads();
    s = 0.f; ss = 0.f;
#pragma unroll
    for (int w = 0; w < WPR; ++w) {
      const float2 p = red[warp / WPR * WPR + w];
      s += p.x; ss += p.y;
    }
  }
  const float inv_d = 1.0f / (float)D;
  const float mean = rms ? 0.f : s * inv_d;
  const float var = rms ? ss * inv_d : fmaxf(ss * inv_d - mean * mean, 0.f);
  const float rstd = rsqrtf(var + eps);
  const int b = row / rows_per_batch;
  const __nv_bfloat16* sh = shift ? shift + (size_t)b * mod_stride : nullptr;
  const __nv_bfloat16* sc = scale ? scale + (size_t)b * mod_stride : nullptr;
  __nv_bfloat16* yr = y + (size_t)row * ldy;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = lane + i * 32 * WPR;
    if (c < nchunk) {
      const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
      float o[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16(w[j]);
        o[2 * j] = (f.x - mean) * rstd;
        o[2 * j + 1] = (f.y - mean) * rstd;
      }
      if (weight) { float t[8]; load8(weight + c * 8, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] *= t[e]; }
      if (bias) { float t[8]; load8(bias + c * 8, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] += t[e]; }
      if (sc) { float t[8]; load8(sc + c * 8, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = fmaf(o[e], t[e], o[e]); }
      if (sh) { float t[8]; load8(sh + c * 8, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] += t[e]; }
      store8(yr + c * 8, o);
    }
  }
}

// Where the heads of a row also go: key and value pages (null: nowhere), at slots[r], < 0 = none.
struct HeadPages {
  __nv_bfloat16 *k, *v;
  const int* slots;
};

// Norm and rotation of one head held by half a warp, 8 consecutive elements per lane (D = 128).  c, s: this lane's rotation
// coefficients, 4 pairs of neighbours (interleaved) or the 8 frequencies of its elements (halves, the sign already on s).
__device__ __forceinline__ uint4 head_norm_rope(const uint4& v, bool norm, const float (&gain)[8], bool rope, int interleaved, const float (&c)[8],
                                                const float (&s)[8], float eps) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  float x[8];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16(w[j]);
    x[2 * j] = f.x; x[2 * j + 1] = f.y;
    ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
  }
  if (norm) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float r = rsqrtf(ss * (1.0f / 128) + eps);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = x[e] * r * gain[e];
  }
  if (rope) {
    if (interleaved) {
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const float a = x[e], b = x[e + 1];
        x[e] = fmaf(a, c[e >> 1], -b * s[e >> 1]);
        x[e + 1] = fmaf(b, c[e >> 1], a * s[e >> 1]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float partner = __shfl_xor_sync(0xffffffffu, x[e], 8);
        x[e] = fmaf(x[e], c[e], partner * s[e]);
      }
    }
  }
  return make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
}

struct HeadRows {
  __nv_bfloat16* qkv;
  long rows;
  int S, H, Hkv, ld;
  const __nv_bfloat16 *wq, *wk, *wq_alt, *wk_alt;
  int s_alt;
  const float *cosb, *sinb;
  int interleaved;
  float eps;
  const int* positions;
  HeadPages pages;
};

__device__ __forceinline__ void rope_coefficients(const HeadRows& a, long row, int s, int l16, float (&cs)[8], float (&sn)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) cs[e] = sn[e] = 0.f;
  if (!a.cosb) return;
  const int pos = a.positions ? a.positions[row] : s;
  const int f0 = a.interleaved ? 4 * l16 : (l16 & 7) * 8, n = a.interleaved ? 4 : 8;
  const float* cr = a.cosb + (size_t)pos * 64 + f0;
  const float* sr = a.sinb + (size_t)pos * 64 + f0;
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (e < n) {
      cs[e] = cr[e];
      sn[e] = a.interleaved || l16 >= 8 ? sr[e] : -sr[e];
    }
}

// A result to its places: back to the row, and key and value heads to their page.
__device__ __forceinline__ void store_head(const HeadRows& a, long row, int h, int l16, int slot, const uint4& raw, const uint4& done) {
  const int heads = a.H + a.Hkv;
  if (h < heads) *reinterpret_cast<uint4*>(a.qkv + (size_t)row * a.ld + (size_t)h * 128 + l16 * 8) = done;
  if (slot >= 0 && h >= a.H) {
    __nv_bfloat16* page = h < heads ? a.pages.k + (size_t)(h - a.H) * 128 : a.pages.v + (size_t)(h - heads) * 128;
    *reinterpret_cast<uint4*>(page + (size_t)slot * a.Hkv * 128 + l16 * 8) = h < heads ? done : raw;
  }
}

// Head norms and rotation for D = 128, a few rows: two heads to a warp, half a warp each.  With pages the key heads go there as
// well and the value heads that follow them are copied.  8 rows of 40 heads, caches cold, launch included: 8 us, 14 us
// with one warp per row; 560 rows of 48 heads 12 us (16).
__global__ void __launch_bounds__(256)
qk_norm_rope128_kernel(const __grid_constant__ HeadRows a, PeerWait wt, int* status) {
  pdl_begin();
  if (wt.counter) {
    // fused exchange: the rows come from the peers' QKV GEMM epilogues; wait for their arrivals
    // here instead of in a barrier kernel of its own
    if (threadIdx.x == 0) {
      peer_wait_arrivals(wt, nullptr, status);
      peer_wait_cta_exit(wt, gridDim.x);      // only this thread reads the epoch word
    }
    __syncthreads();
  }
  const int all = a.H + (a.pages.k ? 2 : 1) * a.Hkv, pairs = (all + 1) / 2;
  const long unit = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const long row = unit / pairs;
  if (row >= a.rows) return;
  const int lane = threadIdx.x & 31, l16 = lane & 15;
  const int h = (int)(unit - row * pairs) * 2 + (lane >> 4);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  float gain[8];
  if (h < all) v = *reinterpret_cast<const uint4*>(a.qkv + (size_t)row * a.ld + (size_t)h * 128 + l16 * 8);
  const int s = (int)(row % a.S);
  const bool alt = s >= a.s_alt;
  if (a.wq) {
    const __nv_bfloat16* g = h < a.H ? ((alt && a.wq_alt) ? a.wq_alt : a.wq) : ((alt && a.wk_alt) ? a.wk_alt : a.wk);
    load8(g + l16 * 8, gain);
  }
  float cs[8], sn[8];
  rope_coefficients(a, row, s, l16, cs, sn);
  const uint4 o = head_norm_rope(v, a.wq != nullptr, gain, a.cosb != nullptr, a.interleaved, cs, sn, a.eps);
  if (h < all) store_head(a, row, h, l16, a.pages.k ? a.pages.slots[row] : -1, v, o);
}

// The same for many rows: a warp walks all heads of its row, 8 at a time, and fetches gains and rotation coefficients once; steps of
// query heads alone neither choose a gain nor look for a page.
__global__ void __launch_bounds__(256)
qk_norm_rope128_rows_kernel(const __grid_constant__ HeadRows a, PeerWait wt, int* status) {
  pdl_begin();
  if (wt.counter) {
    if (threadIdx.x == 0) {
      peer_wait_arrivals(wt, nullptr, status);
      peer_wait_cta_exit(wt, gridDim.x);
    }
    __syncthreads();
  }
  const long row = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= a.rows) return;
  const int all = a.H + (a.pages.k ? 2 : 1) * a.Hkv;
  const int lane = threadIdx.x & 31, l16 = lane & 15, hsel = lane >> 4;
  const int s = (int)(row % a.S);
  const bool alt = s >= a.s_alt;
  float gq[8], gk[8];
  if (a.wq) {
    load8(((alt && a.wq_alt) ? a.wq_alt : a.wq) + l16 * 8, gq);
    load8(((alt && a.wk_alt) ? a.wk_alt : a.wk) + l16 * 8, gk);
  }
  float cs[8], sn[8];
  rope_coefficients(a, row, s, l16, cs, sn);
  const int page = a.pages.k ? a.pages.slots[row] : -1;
  constexpr int U = 4;
  // Both halves of the warp take every step, whether or not their last heads exist: head_norm_rope exchanges values over the whole warp.
  uint4 v[U];
  int h0 = 0;
#pragma unroll 1
  for (; h0 + 2 * U <= a.H; h0 += 2 * U) {                 // query heads alone
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = *reinterpret_cast<const uint4*>(a.qkv + (size_t)row * a.ld + (size_t)(h0 + 2 * u + hsel) * 128 + l16 * 8);
#pragma unroll
    for (int u = 0; u < U; ++u)
      *reinterpret_cast<uint4*>(a.qkv + (size_t)row * a.ld + (size_t)(h0 + 2 * u + hsel) * 128 + l16 * 8) =
          head_norm_rope(v[u], a.wq != nullptr, gq, a.cosb != nullptr, a.interleaved, cs, sn, a.eps);
  }
#pragma unroll 1
  for (; h0 < all; h0 += 2 * U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int h = h0 + 2 * u + hsel;
      v[u] = h < all ? *reinterpret_cast<const uint4*>(a.qkv + (size_t)row * a.ld + (size_t)h * 128 + l16 * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int h = h0 + 2 * u + hsel;
      float gain[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) gain[e] = h < a.H ? gq[e] : gk[e];
      const uint4 o = head_norm_rope(v[u], a.wq != nullptr, gain, a.cosb != nullptr, a.interleaved, cs, sn, a.eps);
      if (h < all) store_head(a, row, h, l16, page, v[u], o);
    }
  }
}

// ------------------------------------------------------------------ qk norm + rope
// qkv: [B, S, 3, H, D] (row pitch ld elements between consecutive s), D in {64, 128}.
// One warp per (row, head); lane owns D/32 consecutive elements (2 or 4), i.e. whole
// (even, odd) pairs for the interleaved layout.  For the half-rotation layout lane l
// owns elements {l*D/64 .. } of both halves.  cos/sin: [S, D/2] fp32.
template <int D>
__global__ void __launch_bounds__(256)
qk_norm_rope_kernel(__nv_bfloat16* __restrict__ qkv, int B, int S, int H, int Hkv, int ld,
                    const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk,
                    const __nv_bfloat16* __restrict__ wq_alt, const __nv_bfloat16* __restrict__ wk_alt,
                    int s_alt, const float* __restrict__ cosb, const float* __restrict__ sinb,
                    int interleaved, float eps, const int* __restrict__ positions) {
  constexpr int E = D / 32;  // elements per lane
  const int warps_per_block = blockDim.x >> 5;
  const long gw = (long)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int heads = H + Hkv;
  const long total = (long)B * S * heads;
  if (gw >= total) return;
  const int hh = (int)(gw % heads);
  const long rs = gw / heads;
  const int s = (int)(rs % S);
  const int b = (int)(rs / S);
  const bool is_k = hh >= H;
  const int h = is_k ? hh - H : hh;
  __nv_bfloat16* p = qkv + ((size_t)b * S + s) * ld + (is_k ? (size_t)H * D : 0) + (size_t)h * D;
  const __nv_bfloat16* w = is_k ? (s >= s_alt && wk_alt ? wk_alt : wk) : (s >= s_alt && wq_alt ? wq_alt : wq);
  const int pos = positions ? positions[(size_t)b * S + s] : s;

  float x[E];
  int idx[E];
  if (interleaved) {
#pragma unroll
    for (int e = 0; e < E; ++e) idx[e] = lane * E + e;
  } else {
    // lane owns E/2 elements in each half so that rotation partners sit in one lane
#pragma unroll
    for (int e = 0; e < E / 2; ++e) { idx[e] = lane * (E / 2) + e; idx[e + E / 2] = D / 2 + lane * (E / 2) + e; }
  }
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) { x[e] = __bfloat162float(p[idx[e]]); ss += x[e] * x[e]; }
  if (w) {
    ss = warp_sum(ss);
    const float r = rsqrtf(ss / (float)D + eps);
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = x[e] * r * __bfloat162float(w[idx[e]]);
  }
  if (cosb) {
    const float* cr = cosb + (size_t)pos * (D / 2);
    const float* sr = sinb + (size_t)pos * (D / 2);
    if (interleaved) {
#pragma unroll
      for (int e = 0; e < E; e += 2) {
        const int pi = idx[e] >> 1;
        const float c = cr[pi], sn = sr[pi];
        const float a = x[e], bb = x[e + 1];
        x[e] = a * c - bb * sn;
        x[e + 1] = a * sn + bb * c;
      }
    } else {
#pragma unroll
      for (int e = 0; e < E / 2; ++e) {
        const int pi = idx[e];
        const float c = cr[pi], sn = sr[pi];
        const float a = x[e], bb = x[e + E / 2];
        x[e] = a * c - bb * sn;
        x[e + E / 2] = bb * c + a * sn;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) p[idx[e]] = __float2bfloat16(x[e]);
}

// ------------------------------------------------------------ CFG mix + Euler step
// pos/neg: [rows, C] bf16 velocity predictions; lat: [rows, C] fp32 latents (in place);
// lat_bf16: bf16 copy of the updated latents for the next transformer call.
// One warp per row.  neg == nullptr means no guidance (v = pos).
__global__ void __launch_bounds__(256)
cfg_euler_kernel(const __nv_bfloat16* pos, const __nv_bfloat16* neg,
                 float* __restrict__ lat, __nv_bfloat16* __restrict__ lat_bf16, long rows, int C,
                 float guidance, float dt, int renorm) {
  pdl_begin();
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const size_t base = (size_t)row * C;
  float pn = 0.f, cn = 0.f;
  for (int c = lane; c < C; c += 32) {
    const float p = __bfloat162float(pos[base + c]);
    float v = p;
    if (neg) {
      const float n = __bfloat162float(neg[base + c]);
      v = n + guidance * (p - n);
    }
    pn += p * p;
    cn += v * v;
  }
  float resc = 1.0f;
  if (renorm && neg) {
    pn = warp_sum(pn);
    cn = warp_sum(cn);
    resc = sqrtf(pn) / fmaxf(sqrtf(cn), 1e-12f);
  }
  for (int c = lane; c < C; c += 32) {
    const float p = __bfloat162float(pos[base + c]);
    float v = p;
    if (neg) {
      const float n = __bfloat162float(neg[base + c]);
      v = (n + guidance * (p - n)) * resc;
    }
    const float x = lat[base + c] + dt * v;
    lat[base + c] = x;
    if (lat_bf16) lat_bf16[base + c] = __float2bfloat16(x);
  }
}

// ------------------------------------------------------------------------ SwiGLU
__global__ void __launch_bounds__(256)
silu_mul_kernel(const __nv_bfloat16* x, __nv_bfloat16* __restrict__ y, long rows, int N,
                int ldx, int ldy) {
  pdl_begin();
  const long nchunk = (long)rows * (N >> 3);
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nchunk; i += (long)gridDim.x * blockDim.x) {
    const long r = i / (N >> 3);
    const int c = (int)(i % (N >> 3)) * 8;
    float g[8], u[8], o[8];
    load8(x + r * ldx + c, g);
    load8(x + r * ldx + N + c, u);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = silu(g[e]) * u[e];
    store8(y + r * ldy + c, o);
  }
}

// the same in fp32 (exact mode)
__global__ void __launch_bounds__(256)
silu_mul_f32_kernel(const float* __restrict__ x, float* __restrict__ y, long rows, int N, long ldx, long ldy) {
  const long total = rows * N;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long r = i / N;
    const int c = (int)(i - r * N);
    const float g = x[r * ldx + c];
    y[r * ldy + c] = g / (1.0f + expf(-g)) * x[r * ldx + N + c];
  }
}

// --------------------------------------------------------- TeaCache rel-L1 metric
// Stage 1: every CTA writes its partial (sum|a-b|, sum|b|) into scratch[2*blockIdx.x].
// Stage 2 (one CTA): reduces the partials, applies the polynomial rescale, accumulates
// and decides; state = {accumulated, last_rel_l1, skip_flag(as float), steps_skipped}.
constexpr int RL_THREADS = 256;

__global__ void __launch_bounds__(RL_THREADS)
rel_l1_partial_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b, long n8,
                      float* __restrict__ scratch) {
  __shared__ float red[2][RL_THREADS / 32];
  float d = 0.f, m = 0.f;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long)gridDim.x * blockDim.x) {
    float x[8], y[8];
    load8(a + i * 8, x);
    load8(b + i * 8, y);
#pragma unroll
    for (int e = 0; e < 8; ++e) { d += fabsf(x[e] - y[e]); m += fabsf(y[e]); }
  }
  d = warp_sum(d);
  m = warp_sum(m);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = d; red[1][threadIdx.x >> 5] = m; }
  __syncthreads();
  if (threadIdx.x == 0) {
    d = 0.f; m = 0.f;
    for (int w = 0; w < RL_THREADS / 32; ++w) { d += red[0][w]; m += red[1][w]; }
    scratch[2 * blockIdx.x] = d;
    scratch[2 * blockIdx.x + 1] = m;
  }
}

__global__ void __launch_bounds__(RL_THREADS)
rel_l1_finish_kernel(const float* __restrict__ scratch, int nparts, float* __restrict__ state,
                     const float* __restrict__ coef, int ncoef, float thresh, int force_compute,
                     float* __restrict__ sums_out) {
  __shared__ float red[2][RL_THREADS / 32];
  float d = 0.f, m = 0.f;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) { d += scratch[2 * i]; m += scratch[2 * i + 1]; }
  d = warp_sum(d);
  m = warp_sum(m);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = d; red[1][threadIdx.x >> 5] = m; }
  __syncthreads();
  if (threadIdx.x == 0) {
    d = 0.f; m = 0.f;
    for (int w = 0; w < RL_THREADS / 32; ++w) { d += red[0][w]; m += red[1][w]; }
    if (sums_out) { sums_out[0] = d; sums_out[1] = m; }
    if (state) {
      // mean|a-b| / (mean|b| + 1e-8) with equal element counts reduces to the ratio of sums
      const float rel = d / (m + 1e-8f);
      float r = rel;
      if (ncoef > 0) {  // numpy.poly1d order: highest power first
        r = coef[0];
        for (int i = 1; i < ncoef; ++i) r = r * rel + coef[i];
      }
      // the reference accumulates |rescale(rel)| (teacache/hook.py:225): a polynomial that dips below
      // zero at small rel must not pull the accumulator down
      float acc = state[0] + fabsf(r);
      float skip = 0.f;
      if (!force_compute && acc < thresh) skip = 1.f; else acc = 0.f;
      state[0] = acc;
      state[1] = rel;
      state[2] = skip;
      state[3] += skip;
    }
  }
}

}  // namespace omni

using namespace omni;

extern "C" int omni_norm_modulate(const void* x, void* y, int rows, int D, int ldx, int ldy,
                                  const void* weight, const void* bias, const void* shift,
                                  const void* scale, int mod_stride, int rows_per_batch, int rms,
                                  float eps, void* stream) {
  if (rows <= 0) return RC_OK;
  if ((D & 7) || D > 8192 || (ldx & 7) || (ldy & 7) || (mod_stride & 7)) return RC_BAD_ARG;
  if (rows_per_batch <= 0) rows_per_batch = rows;
  auto xx = (const __nv_bfloat16*)x; auto yy = (__nv_bfloat16*)y;
  auto w = (const __nv_bfloat16*)weight; auto bb = (const __nv_bfloat16*)bias;
  auto sh = (const __nv_bfloat16*)shift; auto sc = (const __nv_bfloat16*)scale;
  cudaStream_t st = (cudaStream_t)stream;
  const int nchunk = D >> 3;
#define OMNI_NM_WARP(V, W) launch_overlapped(norm_modulate_warp_kernel<V, W>, (unsigned)((rows + 8 / W - 1) / (8 / W)), 256, 0, st, xx, yy, rows, D, ldx, ldy, w, bb, sh, sc, mod_stride, rows_per_batch, rms, eps)
  // Rows of more than 1024 channels, by the rows per SM, RMS norm in us on cold operands:
  //   up to 2, or 5 of up   a block per row, two chunks per thread: one round of latencies (64 rows of 5120: 2.5, 4 warps per row 3.4; 740 rows of
  //   to 2048 channels      2048: 3.3 and 3.4).  Above, the blocks of a second round cost more than they save (592 rows of 3072: 5.1, 4 warps 3.9)
  //   more than 5120        from the second row per SM on 8 warps per row, since blocks of 512 threads fit an SM twice at most: 592 rows of 6144
  //                         6.2 (block per row 9.7, 4 warps 6.5), 8192 rows of 8192 60.6 (127, 62.5); 4 warps where they need at most 6
  //                         chunks per lane and rows are many: 8192 rows of 6144 46.5 (8 warps 48.2)
  //   many, of up to 3072   2 warps per row: fewer warps that wait for one another (8192 rows of 2048: 16.1, 4 warps 18.1, one warp 17.5; 4096 rows of
  //                         3072: 12.6 and 13.1; below the limits 4 warps: 2048 rows of 3072 8.6, 2 warps 9.7)
  //   else                  4 warps per row (1183 rows of 4096: 6.7, block per row 10.0)
  const long sms = sm_count();
  if (nchunk <= 64) OMNI_NM_WARP(2, 1);
  else if (nchunk <= 128) OMNI_NM_WARP(4, 1);
  else if (rows <= (nchunk <= 256 ? 5 : nchunk <= 640 ? 2 : 1) * sms)
    launch_overlapped(norm_modulate_kernel<2>, rows, ((nchunk + 1) / 2 + 31) / 32 * 32, 0, st, xx, yy, D, ldx, ldy, w, bb, sh, sc, mod_stride,
                                                                               rows_per_batch, rms, eps);
  else if (nchunk > 768) OMNI_NM_WARP(4, 8);
  else if (nchunk > 640) {
    if (rows <= 4 * sms) OMNI_NM_WARP(3, 8);
    else OMNI_NM_WARP(6, 4);
  } else if (nchunk <= 384 && rows > (nchunk <= 256 ? 12 : 16) * sms) {
    if (nchunk <= 256) OMNI_NM_WARP(4, 2);
    else if (nchunk <= 320) OMNI_NM_WARP(5, 2);
    else OMNI_NM_WARP(6, 2);
  } else {
    if (nchunk <= 256) OMNI_NM_WARP(2, 4);
    else if (nchunk <= 384) OMNI_NM_WARP(3, 4);
    else if (nchunk <= 512) OMNI_NM_WARP(4, 4);
    else OMNI_NM_WARP(5, 4);
  }
#undef OMNI_NM_WARP
  return (int)cudaGetLastError();
}

// `sync` (may be null, head_dim 128 only): arrivals from the peers' QKV epilogues that the kernel
// waits for before it touches the buffer (see peer_signal.cuh); `status` receives a timeout code.
// `kc`, `vc` (both or neither; head_dim 128): pages [slots, Hkv, D] that the key heads, as they leave the kernel, and the value
// heads of row r are written to at slots[r] (< 0: not).
extern "C" int omni_qk_norm_rope_pages(void* qkv, int B, int S, int H, int Hkv, int D, int ld, const void* wq,
                                       const void* wk, const void* wq_alt, const void* wk_alt, int s_alt,
                                       const float* cosb, const float* sinb, int interleaved, float eps,
                                       const int* positions, void* kc, void* vc, const int* slots, const OmniSync* sync,
                                       int* status, void* stream) {
  const long total = (long)B * S * (H + Hkv);
  if (total <= 0) return sync ? RC_BAD_ARG : RC_OK;
  PeerSignal unused;
  PeerWait wt;
  unpack_sync(sync, unused, wt);
  const bool fast = D == 128 && (ld & 7) == 0 && (wq != nullptr) == (wk != nullptr);
  if ((wt.counter || kc) && !fast) return RC_BAD_ARG;
  if ((kc != nullptr) != (vc != nullptr) || (kc && !slots)) return RC_BAD_ARG;
  const int wpb = 8;
  const unsigned grid = (unsigned)((total + wpb - 1) / wpb);
  auto q = (__nv_bfloat16*)qkv;
  auto a = (const __nv_bfloat16*)wq; auto b = (const __nv_bfloat16*)wk;
  auto c = (const __nv_bfloat16*)wq_alt; auto d = (const __nv_bfloat16*)wk_alt;
  cudaStream_t st = (cudaStream_t)stream;
  if (fast) {
    const long rows = (long)B * S;
    const HeadRows r = {q, rows, S, H, Hkv, ld, a, b, c, d, s_alt, cosb, sinb, interleaved, eps, positions,
                        {(__nv_bfloat16*)kc, (__nv_bfloat16*)vc, slots}};
    const int all = H + Hkv + (kc ? Hkv : 0);
    const long pairs = rows * ((all + 1) / 2);
    // (a launch that waits for peers starts when its own predecessor has ended)
    // two heads to a warp up to about 600 rows of 48 heads; from there on a warp per row, which loads the coefficients once
    if (pairs <= 2L * 64 * sm_count())
      launch_with(!wt.counter, 1, qk_norm_rope128_kernel, (unsigned)((pairs + 7) / 8), 256, 0, st, r, wt, status);
    else
      // An ordinary launch: with many blocks, those that start while the last of a GEMM still hold their SMs are dealt out unevenly
      // (projection and this kernel, in brackets overlapped: 2000 rows of 32 / 4 heads 45.0 us (46.5), 8192 of 32 / 8 181.1 (184.7); two
      // heads to a warp 50.0 and 206)
      launch_with(false, 1, qk_norm_rope128_rows_kernel, (unsigned)((rows + 7) / 8), 256, 0, st, r, wt, status);
  } else if (D == 128)
    qk_norm_rope_kernel<128><<<grid, wpb * 32, 0, st>>>(q, B, S, H, Hkv, ld, a, b, c, d, s_alt, cosb, sinb, interleaved, eps, positions);
  else if (D == 64)
    qk_norm_rope_kernel<64><<<grid, wpb * 32, 0, st>>>(q, B, S, H, Hkv, ld, a, b, c, d, s_alt, cosb, sinb, interleaved, eps, positions);
  else
    return RC_BAD_ARG;
  return (int)cudaGetLastError();
}

extern "C" int omni_qk_norm_rope_sync(void* qkv, int B, int S, int H, int Hkv, int D, int ld, const void* wq,
                                      const void* wk, const void* wq_alt, const void* wk_alt, int s_alt,
                                      const float* cosb, const float* sinb, int interleaved, float eps,
                                      const int* positions, const OmniSync* sync, int* status, void* stream) {
  return omni_qk_norm_rope_pages(qkv, B, S, H, Hkv, D, ld, wq, wk, wq_alt, wk_alt, s_alt, cosb, sinb, interleaved, eps,
                                 positions, nullptr, nullptr, nullptr, sync, status, stream);
}

extern "C" int omni_qk_norm_rope(void* qkv, int B, int S, int H, int Hkv, int D, int ld, const void* wq,
                                 const void* wk, const void* wq_alt, const void* wk_alt, int s_alt,
                                 const float* cosb, const float* sinb, int interleaved, float eps,
                                 const int* positions, void* stream) {
  return omni_qk_norm_rope_sync(qkv, B, S, H, Hkv, D, ld, wq, wk, wq_alt, wk_alt, s_alt, cosb, sinb, interleaved, eps,
                                positions, nullptr, nullptr, stream);
}

extern "C" int omni_cfg_euler_step(const void* pos, const void* neg, float* lat, void* lat_bf16, long rows,
                                   int C, float guidance, float dt, int renorm, void* stream) {
  if (rows <= 0) return RC_OK;
  const int wpb = 8;
  const unsigned grid = (unsigned)((rows + wpb - 1) / wpb);
  launch_overlapped(cfg_euler_kernel, grid, wpb * 32, 0, (cudaStream_t)stream, (const __nv_bfloat16*)pos, (const __nv_bfloat16*)neg, lat, (__nv_bfloat16*)lat_bf16, rows, C, guidance, dt, renorm);
  return (int)cudaGetLastError();
}

extern "C" int omni_silu_mul(const void* x, void* y, long rows, int N, int ldx, int ldy, void* stream) {
  if (rows <= 0) return RC_OK;
  if ((N & 7) || (ldx & 7) || (ldy & 7)) return RC_BAD_ARG;
  const long nchunk = rows * (N >> 3);
  long blocks = (nchunk + 255) / 256;
  const bool full = blocks > 148 * 16;
  if (full) blocks = 148 * 16;
  // More blocks than the device holds at once: an ordinary launch, because blocks that start while a GEMM's last ones hold their SMs are dealt out
  // unevenly (norm, 2048 -> 2 x 6144, this, 6144 -> 2048, 4096 rows: 258 us, overlapped 266; 600 rows 70.5 and 70.0)
  launch_with(!full, 1, silu_mul_kernel, (unsigned)blocks, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)x, (__nv_bfloat16*)y, rows, N, ldx, ldy);
  return (int)cudaGetLastError();
}

extern "C" int omni_silu_mul_f32(const float* x, float* y, long rows, int N, long ldx, long ldy, void* stream) {
  if (rows <= 0 || N <= 0) return RC_OK;
  long blocks = (rows * N + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  silu_mul_f32_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(x, y, rows, N, ldx, ldy);
  return (int)cudaGetLastError();
}

// Number of partial pairs omni_rel_l1 writes for n elements (scratch needs 2x floats).
extern "C" int omni_rel_l1_parts(long n) {
  long blocks = ((n >> 3) + RL_THREADS - 1) / RL_THREADS;
  if (blocks > 148 * 4) blocks = 148 * 4;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

// scratch: >= 2 * omni_rel_l1_parts(n) floats of device memory owned by the caller.
extern "C" int omni_rel_l1(const void* a, const void* b, long n, float* scratch, float* state,
                           const float* coef, int ncoef, float thresh, int force_compute,
                           float* sums_out, void* stream) {
  if (n <= 0 || (n & 7) || a == nullptr || b == nullptr || scratch == nullptr) return RC_BAD_ARG;
  if (ncoef < 0 || (state != nullptr && ncoef > 0 && coef == nullptr)) return RC_BAD_ARG;
  const int parts = omni_rel_l1_parts(n);
  rel_l1_partial_kernel<<<parts, RL_THREADS, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b, n >> 3, scratch);
  rel_l1_finish_kernel<<<1, RL_THREADS, 0, (cudaStream_t)stream>>>(scratch, parts, state, coef, ncoef, thresh, force_compute, sums_out);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Allocation-free variant of omni_rel_l1 (declared in omni_noalloc.h).
//
// The two-stage reduction needs 2 floats of scratch per stage-1 CTA.  The general entry
// point takes that scratch from the caller; this one keeps it in a file-scope device array
// so that a caller which owns no allocator can still use the kernel.
constexpr int RL_NOALLOC_MAX_PARTS = 148 * 4;                 // same cap as omni_rel_l1_parts()
constexpr long RL_NOALLOC_MAX_ELEMS = 1L << 28;               // 268,435,456 elements per operand
static __device__ __align__(256) float g_rel_l1_scratch[2 * RL_NOALLOC_MAX_PARTS];  // 4,736 bytes

namespace {
constexpr int RL_MAX_DEVICES = 64;
std::mutex g_noalloc_mu;
float* g_noalloc_ptr[RL_MAX_DEVICES] = {nullptr};
}  // namespace

extern "C" long omni_rel_l1_noalloc_max_elems(void) { return RL_NOALLOC_MAX_ELEMS; }

extern "C" const char* omni_rel_l1_noalloc_strerror(int rc) {
  switch (rc) {
    case 0: return "ok";
    case RC_BAD_ARG: return "bad argument: n must be a positive multiple of 8, the pointers non-null, ncoef >= 0 and coef non-null when state and ncoef are given";
    case RC_TOO_LARGE: return "n exceeds omni_rel_l1_noalloc_max_elems() (2^28 elements per operand)";
    default: return rc > 0 ? "CUDA runtime error (the value is the cudaError_t)" : "unknown error";
  }
}

extern "C" int omni_rel_l1_noalloc(const void* a, const void* b, long n, float* sums_out, float* state,
                                   const float* coef, int ncoef, float thresh, int force_compute,
                                   void* stream) {
  if (a == nullptr || b == nullptr || n <= 0 || (n & 7)) return RC_BAD_ARG;
  if (sums_out == nullptr && state == nullptr) return RC_BAD_ARG;
  if (ncoef < 0 || (state != nullptr && ncoef > 0 && coef == nullptr)) return RC_BAD_ARG;
  if (n > RL_NOALLOC_MAX_ELEMS) return RC_TOO_LARGE;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= RL_MAX_DEVICES) return RC_BAD_ARG;
  float* scratch = nullptr;
  {
    // First call on this device: resolve the device address of the static array.  The array's
    // name is only a host-side handle here; a kernel must be given the address the runtime
    // reports for the current device.
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (g_noalloc_ptr[dev] == nullptr) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_rel_l1_scratch);
      if (e != cudaSuccess) return (int)e;
      g_noalloc_ptr[dev] = static_cast<float*>(p);
    }
    scratch = g_noalloc_ptr[dev];
  }
  const int parts = omni_rel_l1_parts(n);  // <= RL_NOALLOC_MAX_PARTS by construction
  // Stage 1 overwrites scratch[0 .. 2*parts) completely and stage 2 reads exactly that range,
  // so nothing left over from an earlier call is ever read and nothing needs clearing.
  rel_l1_partial_kernel<<<parts, RL_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, n >> 3, scratch);
  e = cudaGetLastError();                 // report a failed first launch, not only the second
  if (e != cudaSuccess) return (int)e;
  rel_l1_finish_kernel<<<1, RL_THREADS, 0, (cudaStream_t)stream>>>(scratch, parts, state, coef, ncoef, thresh,
                                                                   force_compute, sums_out);
  return (int)cudaGetLastError();
}
