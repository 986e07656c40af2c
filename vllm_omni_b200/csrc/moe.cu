// K10: mixture-of-experts routing, dispatch and combine around the tcgen05 expert GEMM.
//
//   omni_moe_route     softmax over expert logits, top-k, optional renormalisation
//   omni_moe_router    router product and choice in one launch: fp32 logits with a bias, the top-k largest, softmax
//                      among them, or sigmoid scores divided by their sum, of the best groups of experts (bf16 rows)
//   omni_moe_topk      the same choice from fp32 logits
//   omni_moe_pairs_f32 y[p] = act(W[expert of pair p] x[p / per]) in true fp32 (exact mode)
//   omni_moe_few_plan  few tokens: tiles of at most 16 rows per expert, from router logits (route included) or chosen ids
//   omni_moe_few_rows  few tokens: y[pair] = act(W[expert] x[pair / per]) with rows gathered in place, SwiGLU included
//   omni_moe_plan_tiles  rows of every expert back to back, its tiles of rows, and the row of every (token, k) pair
//   omni_moe_plan      the same with segments padded to 128 rows
//   omni_moe_dispatch  copy token rows into the expert-major buffer
//   omni_moe_combine   out[t] = sum_k w[t,k] * y[row(t,k)]  (+ optional residual / shared expert); omni_moe_combine_norm: and its RMS norm
//
// Every tile of rows lies inside one expert, so the GEMM of all experts is ONE launch with a per-tile expert index (moe_gemm.cuh;
// gemm_sm100.cu for padded segments).  The reference reaches vLLM's Triton fused_moe or a Python loop over experts
// (vllm_omni/model_executor/models/qwen3_omni/qwen3_moe.py).
#include "host_util.h"
#include "ptx_sm100.cuh"

namespace omni {

constexpr int MOE_TILE = 128;

// Limits for the checked build (OMNI_IN_BOUNDS in ptx_sm100.cuh; 0 = unknown / unchecked), set by the host
// through omni_moe_set_bounds and passed to the kernels by value: the rows the expert-major buffers hold.
struct MoeBounds {
  long max_rows;
  int* status;
};
static MoeBounds g_moe_bounds = {0, nullptr};
enum { KID_MOE_PLAN = 3, KID_MOE_DISPATCH = 4, KID_MOE_COMBINE = 5 };

// Softmax over the logits of one token, its k largest and their weights, by one warp; E <= 256 (8 per lane), k <= 16.  Lane j
// returns choice j.
__device__ __forceinline__ void route_token(const __nv_bfloat16* __restrict__ logits, int E, int k, int renorm, int lane, int& id,
                                            float& weight) {
  float v[8];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = lane + i * 32;
    v[i] = i * 32 < E && e < E ? __bfloat162float(logits[e]) : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i * 32 < E) { v[i] = v[i] == -INFINITY ? 0.f : __expf(v[i] - mx); sum += v[i]; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.0f / sum;
  float picked = 0.f;
  id = 0;
  weight = 0.f;
  // numbers that are not negative compare like their bit patterns, so the best of the warp is one integer reduction
#pragma unroll 1
  for (int j = 0; j < k; ++j) {
    int best = -1, bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i * 32 < E && __float_as_int(v[i]) > best) { best = __float_as_int(v[i]); bi = lane + i * 32; }
    const int top = __reduce_max_sync(0xffffffffu, best);
    bi = __reduce_min_sync(0xffffffffu, best == top ? bi : 0x7fffffff);
    const float w = __int_as_float(top) * inv;
    if (lane == j) { id = bi; weight = w; }
    picked += w;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (bi == lane + i * 32) v[i] = __int_as_float(0x80000000);     // remove the winner: negative as an integer
  }
  if (renorm) weight *= 1.0f / fmaxf(picked, 1e-20f);
}

// one warp per token
__global__ void __launch_bounds__(256)
moe_route_kernel(const __nv_bfloat16* logits, int ld, int T, int E, int k, int renorm,
                 int* __restrict__ ids, float* __restrict__ weights) {
  pdl_begin();
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  int id;
  float w;
  route_token(logits + (size_t)t * ld, E, k, renorm, lane, id, w);
  if (lane < k) { ids[(size_t)t * k + lane] = id; weights[(size_t)t * k + lane] = w; }
}

// What turns logits into a choice.  sigmoid = 0: softmax among the k largest.  sigmoid = 1: scores 1 / (1 + e^-z); with
// groups > 0 only the `keep` groups of neighbours with the largest sums of their two best scores take part; weights are
// scale * score / (sum of the chosen scores + 1e-20).
struct RouterRule {
  int sigmoid, groups, keep;
  float scale;
};

// the largest of n <= 256 values, value lane + 32 i in v[i]; ties go to the lower index
__device__ __forceinline__ void warp_best(const float (&v)[8], int n, int lane, float& best, int& bi) {
  best = -INFINITY;
  bi = 0x7fffffff;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i * 32 < n) {
      const int e = lane + i * 32;
      if (v[i] > best || (v[i] == best && v[i] != -INFINITY && e < bi)) { best = v[i]; bi = e; }
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
  }
}

// Leaves the experts of the kept groups in v (scores), -inf elsewhere.  `sh`: 256 floats of this warp.
__device__ __forceinline__ void keep_groups(float (&v)[8], int E, const RouterRule& rule, int lane, float* sh) {
  const int size = E / rule.groups;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (lane + i * 32 < E) sh[lane + i * 32] = v[i];
  __syncwarp();
  float sum[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int g = lane + i * 32;
    sum[i] = -INFINITY;
    if (i * 32 < rule.groups && g < rule.groups) {
      float a = sh[g * size], b = size > 1 ? -INFINITY : 0.f;
      for (int j = 1; j < size; ++j) {
        const float x = sh[g * size + j];
        b = fmaxf(b, fminf(a, x));
        a = fmaxf(a, x);
      }
      sum[i] = a + b;
    }
  }
  __syncwarp();
  unsigned live = 0u;
  for (int j = 0; j < rule.keep; ++j) {
    float best;
    int g;
    warp_best(sum, rule.groups, lane, best, g);
    if (g >= rule.groups) break;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = lane + i * 32;
      if (e == g) sum[i] = -INFINITY;
      if (i * 32 < E && e >= g * size && e < (g + 1) * size) live |= 1u << i;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (!(live & (1u << i))) v[i] = -INFINITY;
}

// Choice of one token by one warp from logits v (lane + 32 i holds expert lane + 32 i, -inf past the last), ties to the
// lower index.  E <= 256, k <= 16.  `sh`: 256 floats of this warp (groups only).
__device__ __forceinline__ void choose_experts(float (&v)[8], int E, int k, const RouterRule& rule, int lane, float* sh, int* ids,
                                               float* weights) {
  if (rule.sigmoid) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i * 32 < E) v[i] = lane + i * 32 < E ? 1.0f / (1.0f + expf(-v[i])) : -INFINITY;
    if (rule.groups > 0) keep_groups(v, E, rule, lane, sh);
  }
  float top = 0.f, sum = 0.f, mine = 0.f;
  int mine_id = 0;
  for (int j = 0; j < k; ++j) {
    float best;
    int bi;
    warp_best(v, E, lane, best, bi);
    if (bi >= E) bi = j;                       // no finite value left: any index inside the range
    if (j == 0) top = best;
    const float w = rule.sigmoid ? best : expf(best - top);
    sum += w;
    if (lane == j) { mine = w; mine_id = bi; }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (bi == lane + i * 32) v[i] = -INFINITY;
  }
  if (lane < k) {
    ids[lane] = mine_id;
    weights[lane] = rule.sigmoid ? mine / (sum + 1e-20f) * rule.scale : mine / sum;
  }
}

__global__ void __launch_bounds__(256)
moe_topk_kernel(const float* __restrict__ logits, long ld, int T, int E, int k, RouterRule rule, int* __restrict__ ids,
                float* __restrict__ weights) {
  __shared__ float sh[8][256];
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = lane + i * 32;
    v[i] = e < E ? logits[t * ld + e] : -INFINITY;
  }
  choose_experts(v, E, k, rule, lane, sh[threadIdx.x >> 5], ids + (long)t * k, weights + (long)t * k);
}

// Router of MT * 16 tokens per block: NW warps share the contraction (each takes every NW-th 32-channel chunk), 64 experts
// at a time; partial sums meet in shared memory in a fixed order.  A warp reads 16 bytes per row and chunk: lane group j
// of a quad owns channels 8 j .. 8 j + 7 of the chunk for both operands, which permutes the contraction alike on both
// sides.
template <int MT, int NW>
__global__ void __launch_bounds__(32 * NW)
moe_router_kernel(const __nv_bfloat16* x, long ldx, const __nv_bfloat16* w, long ldw,
                  const float* bias, int T, int D, int E, int Ep, int k, RouterRule rule,
                  int* __restrict__ ids, float* __restrict__ weights) {
  pdl_begin();
  extern __shared__ float sm[];
  float* part = sm;                            // [NW][MT * 16][64]
  float* logit = sm + NW * MT * 16 * 64;        // [MT * 16][256]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  const int t0 = blockIdx.x * (MT * 16);
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int e0 = 0; e0 < E; e0 += 64) {
    float acc[MT][8][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.f;
#pragma unroll(MT == 1 ? 2 : 1)
    for (int c = warp * 32; c < D; c += 32 * NW) {
      const int ch = c + j * 8;
      const bool in = ch < D;                  // D is a multiple of 8
      uint4 a[MT][2];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int t = t0 + m * 16 + h * 8 + g;
          a[m][h] = in && t < T ? *reinterpret_cast<const uint4*>(x + (long)t * ldx + ch) : zero;
        }
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const int e = e0 + n * 8 + g;
        const uint4 b = in && e < Ep ? *reinterpret_cast<const uint4*>(w + (long)e * ldw + ch) : zero;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                       "{%0, %1, %2, %3};"
                       : "+f"(acc[m][n][0]), "+f"(acc[m][n][1]), "+f"(acc[m][n][2]), "+f"(acc[m][n][3])
                       : "r"(a[m][0].x), "r"(a[m][1].x), "r"(a[m][0].y), "r"(a[m][1].y), "r"(b.x), "r"(b.y));
          asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                       "{%0, %1, %2, %3};"
                       : "+f"(acc[m][n][0]), "+f"(acc[m][n][1]), "+f"(acc[m][n][2]), "+f"(acc[m][n][3])
                       : "r"(a[m][0].z), "r"(a[m][1].z), "r"(a[m][0].w), "r"(a[m][1].w), "r"(b.z), "r"(b.w));
        }
      }
    }
    __syncthreads();                           // the previous group's sums are read
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float2*>(part + ((long)warp * MT * 16 + m * 16 + h * 8 + g) * 64 + n * 8 + j * 2) =
              make_float2(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
    __syncthreads();
    for (int i = threadIdx.x; i < MT * 16 * 64; i += 32 * NW) {
      const int e = e0 + (i & 63);
      if (e < E) {
        float s = bias ? bias[e] : 0.f;
#pragma unroll
        for (int q = 0; q < NW; ++q) s += part[q * MT * 16 * 64 + i];
        logit[(i >> 6) * 256 + e] = s;
      }
    }
  }
  __syncthreads();
  for (int r = warp; r < MT * 16; r += NW) {
    const int t = t0 + r;
    if (t >= T) break;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = lane + i * 32 < E ? logit[r * 256 + lane + i * 32] : -INFINITY;
    __syncwarp();                              // the row's logits become scratch
    choose_experts(v, E, k, rule, lane, logit + r * 256, ids + (long)t * k, weights + (long)t * k);
  }
}

// Exact mode: one warp per (pair, output); a result is one fixed-order chain plus a fixed-order sum over lanes.
__global__ void __launch_bounds__(256)
moe_pairs_f32_kernel(const float* __restrict__ x, long ldx, int per, const int* __restrict__ ids, const float* __restrict__ w,
                     int E, float* __restrict__ y, long ldy, long pairs, int N, int K, int relu2) {
  const long i = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= pairs * N) return;
  const long p = i / N;
  const int n = (int)(i - p * N);
  const int e = min(max(ids[p], 0), E - 1);
  const float* a = x + (p / per) * ldx;
  const float* b = w + ((long)e * N + n) * K;
  float s = 0.f;
  for (int c = lane; c < K; c += 32) s = fmaf(a[c], b[c], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (relu2) {
    s = fmaxf(s, 0.f);
    s *= s;
  }
  if (lane == 0) y[p * ldy + n] = s;
}

// single CTA: histogram, padded prefix sum, tile->expert table, (token,k)->row map.
// counts/cursor live in shared memory (E <= 1024).
__global__ void __launch_bounds__(1024)
moe_plan_kernel(const int* __restrict__ ids, int n_pairs, int E, int e_lo, int e_hi, int max_tiles,
                int* __restrict__ row_of_pair, int* __restrict__ tile_expert, int* __restrict__ offsets,
                int* __restrict__ n_rows_out, MoeBounds bd) {
  __shared__ int cnt[1024];
  __shared__ int off[1025];
  for (int e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) {
    const int e = ids[i];
    if (!OMNI_IN_BOUNDS(e >= 0 && e < E, bd.status, KID_MOE_PLAN)) continue;
    if (e >= e_lo && e < e_hi) atomicAdd(&cnt[e], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E; ++e) {
      off[e] = acc;
      acc += (cnt[e] + MOE_TILE - 1) / MOE_TILE * MOE_TILE;
    }
    off[E] = acc;
    *n_rows_out = acc;
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) offsets[e] = off[e];
  for (int tile = threadIdx.x; tile < max_tiles; tile += blockDim.x) {
    // expert owning row tile*128: the last e with off[e] <= row (binary search)
    const int row = tile * MOE_TILE;
    int ex = -1;
    if (row < off[E]) {
      int lo = 0, hi = E - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= row) lo = mid; else hi = mid - 1;
      }
      ex = lo;
    }
    tile_expert[tile] = ex;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;   // reuse as cursors
  __syncthreads();
  // deterministic placement: pairs are placed in index order per expert by one thread per expert
  // when the batch is small, otherwise by atomics (order inside an expert does not affect results)
  for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) {
    const int e = ids[i];
    row_of_pair[i] = (e >= e_lo && e < e_hi) ? off[e] + atomicAdd(&cnt[e], 1) : -1;
  }
}

// Exclusive sums over the block's 1024 threads of two counts at once; totals in the last two references.
__device__ __forceinline__ void block_scan2(int& a, int& b, int& total_a, int& total_b) {
  __shared__ int wa[32], wb[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, a0 = a, b0 = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ua = __shfl_up_sync(0xffffffffu, a, o), ub = __shfl_up_sync(0xffffffffu, b, o);
    if (lane >= o) { a += ua; b += ub; }
  }
  if (lane == 31) { wa[warp] = a; wb[warp] = b; }
  __syncthreads();
  int sa = wa[lane], sb = wb[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ua = __shfl_up_sync(0xffffffffu, sa, o), ub = __shfl_up_sync(0xffffffffu, sb, o);
    if (lane >= o) { sa += ua; sb += ub; }
  }
  total_a = __shfl_sync(0xffffffffu, sa, 31);
  total_b = __shfl_sync(0xffffffffu, sb, 31);
  const int before = (warp + 31) & 31;
  const int pa = __shfl_sync(0xffffffffu, sa, before), pb = __shfl_sync(0xffffffffu, sb, before);
  a = a - a0 + (warp ? pa : 0);
  b = b - b0 + (warp ? pb : 0);
}

// Plan without padding: the rows of expert e are [off[e], off[e] + cnt[e]); expert e owns c = ceil(cnt[e] / tile)
// tiles of about cnt[e] / c rows (rounded up to 16); tile t = (expert as the local weights number them, first row, rows).  Unused tiles get
// expert -1.  The place of a pair among its expert's rows is what its atomic add to the expert's count returns (the order
// inside an expert does not affect results).  One cluster of CL blocks: each counts its share of the pairs, reads the others' counts where they lie and
// numbers its own; bound by the chain of loads and
// atomic adds of a thread.
constexpr int PLAN_CLUSTER = 8;
__device__ __forceinline__ int ld_cluster_i32(uint32_t addr) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
template <int CL>
__global__ void __launch_bounds__(1024)
moe_plan_tiles_kernel(const int* ids, int n_pairs, int E, int e_lo, int e_hi, int tile_cap, int max_tiles,
                        int* __restrict__ row_of_pair, int* __restrict__ tile_expert, int* __restrict__ tile_row0,
                        int* __restrict__ tile_rows, int* __restrict__ n_rows_out, MoeBounds bd) {
  __shared__ int cnt[1024];
  __shared__ int off[1024];
  const int rank = CL > 1 ? (int)cluster_ctarank() : 0, first = rank * 1024 + threadIdx.x;
  cnt[threadIdx.x] = 0;
  __syncthreads();
  pdl_begin();
#pragma unroll 4
  for (int i = first; i < n_pairs; i += CL * 1024) {
    const int e = ids[i];
    int r = -1;
    if (OMNI_IN_BOUNDS(e >= 0 && e < E, bd.status, KID_MOE_PLAN) && e >= e_lo && e < e_hi) r = atomicAdd(&cnt[e], 1);
    row_of_pair[i] = r;
  }
  if (CL > 1) cluster_sync_all(); else __syncthreads();
  const int e = threadIdx.x;                            // experts past E have no rows
  int mine = cnt[e], before = 0;
  if (CL > 1) {
    mine = 0;
#pragma unroll
    for (int q = 0; q < CL; ++q) {
      const int n = ld_cluster_i32(mapa_shared(smem_u32(&cnt[e]), q));
      if (q < rank) before += n;
      mine += n;
    }
  }
  const int own = (mine + tile_cap - 1) / tile_cap, size = own ? ((mine + own - 1) / own + 15) / 16 * 16 : 0;
  int row = mine, tile = own, rows, tiles;
  block_scan2(row, tile, rows, tiles);
  off[e] = row + before;
  if (rank == 0) {
    if (e == 0) *n_rows_out = rows;
    for (int i = 0; i < own; ++i) {                     // never empty: (own - 1) * size < mine, as tile_cap is a multiple of 64
      tile_expert[tile + i] = e - e_lo;
      tile_row0[tile + i] = row + i * size;
      tile_rows[tile + i] = min(size, mine - i * size);
    }
    for (int t = tiles + threadIdx.x; t < max_tiles; t += 1024) {
      tile_expert[t] = -1;
      tile_row0[t] = 0;
      tile_rows[t] = 0;
    }
  }
  __syncthreads();
#pragma unroll 4
  for (int i = first; i < n_pairs; i += CL * 1024) {
    const int r = row_of_pair[i];
    if (r >= 0) row_of_pair[i] = off[ids[i]] + r;
  }
  if (CL > 1) cluster_sync_all();                       // counts stay until everyone has read them
}

// ------------------------------------------------------------------------------------------------------ few tokens
// Up to a few hundred (token, choice) pairs the chain is the streaming of the chosen experts' weights plus launches, so it has three
// instead of seven: plan (with the choice, from router logits), up projection with SwiGLU, down projection.  Rows are gathered
// where they are read and results lie at their pair's index, so nothing is copied; a tile is at most 16 rows of one expert.
constexpr int FEW_TILE = 16, FEW_PAIRS = 1024;          // no more pairs than experts (ops/moe.py), of which the plan takes 1024
struct FewPlan {
  int *ids;                       // [pairs]: read, or written when the choice is made here
  float* weights;                 // [pairs], written with the choice
  int *pair_of_row, *row_of_pair; // rows of an expert back to back; row_of_pair is the pair's own index, -1 = not local
  int *tile_expert, *tile_row0, *tile_rows;
  int max_tiles;
};

__global__ void __launch_bounds__(1024)
moe_few_plan_kernel(const __nv_bfloat16* logits, int ld, int T, int E, int k, int renorm, int e_lo, int e_hi,
                    const FewPlan p, MoeBounds bd) {
  pdl_begin();
  __shared__ int sid[FEW_PAIRS];
  __shared__ int cnt[1024];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_pairs = T * k;
  cnt[threadIdx.x] = 0;
  if (logits) {
    for (int t = warp; t < T; t += 32) {
      int id;
      float w;
      route_token(logits + (size_t)t * ld, E, k, renorm, lane, id, w);
      if (lane < k) {
        sid[t * k + lane] = id;
        p.ids[t * k + lane] = id;
        p.weights[t * k + lane] = w;
      }
    }
  } else if (threadIdx.x < n_pairs) {
    sid[threadIdx.x] = p.ids[threadIdx.x];
  }
  __syncthreads();
  const int i = threadIdx.x;
  int place = -1;
  if (i < n_pairs) {
    const int e = sid[i];
    if (OMNI_IN_BOUNDS(e >= 0 && e < E, bd.status, KID_MOE_PLAN) && e >= e_lo && e < e_hi) place = atomicAdd(&cnt[e], 1);
    p.row_of_pair[i] = place >= 0 ? i : -1;
  }
  __syncthreads();
  const int e = threadIdx.x, mine = cnt[e];
  int row = mine, tile = (mine + FEW_TILE - 1) / FEW_TILE, rows, tiles;
  block_scan2(row, tile, rows, tiles);
  for (int q = 0; q * FEW_TILE < mine; ++q) {
    p.tile_expert[tile + q] = e - e_lo;                 // the weights hold the local experts
    p.tile_row0[tile + q] = row + q * FEW_TILE;
    p.tile_rows[tile + q] = min(FEW_TILE, mine - q * FEW_TILE);
  }
  for (int t = tiles + threadIdx.x; t < p.max_tiles; t += 1024) p.tile_expert[t] = -1;
  __syncthreads();                                      // everyone has its count: the array becomes the first rows
  cnt[e] = row;
  __syncthreads();
  if (place >= 0) p.pair_of_row[cnt[sid[i]] + place] = i;
}

// y[pair, n] = act(sum_c W[e, n, c] x[pair / per, c]) for a tile of one expert and 16 columns (GATED: 8 columns n of silu(gate) * lift, rows
// n and N + n of W are the two halves of the MMA's 16).  The block's NW warps share the contraction.
template <int NW, bool GATED>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
moe_few_rows_kernel(const __nv_bfloat16* x, long ldx, int per, const __nv_bfloat16* w, int N, int K,
                    const int* tile_expert, const int* tile_row0, const int* tile_rows,
                    const int* pair_of_row, __nv_bfloat16* __restrict__ y, long ldy, int relu2) {
  pdl_begin();
  __shared__ float part[NW][FEW_TILE][16];
  constexpr int COLS = GATED ? 8 : 16;
  const int e = tile_expert[blockIdx.y];
  if (e < 0) return;
  const int row0 = tile_row0[blockIdx.y], rows = tile_rows[blockIdx.y];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  const int n0 = blockIdx.x * COLS;
  const __nv_bfloat16* base = w + (size_t)e * (GATED ? 2 : 1) * N * K;
  const __nv_bfloat16* w0 = base + (size_t)min(n0 + g, N - 1) * K;
  const __nv_bfloat16* w1 = base + (size_t)(GATED ? N + min(n0 + g, N - 1) : min(n0 + 8 + g, N - 1)) * K;
  auto row_of = [&](int r) { return r < rows ? x + (size_t)(pair_of_row[row0 + r] / per) * ldx : nullptr; };
  float (*mine)[16] = part[warp];
  if (rows <= 8) {
    float acc[1][4] = {};
    const __nv_bfloat16* const xr[1] = {row_of(g)};
    few_rows_products<1, NW, 8>(acc, w0, w1, xr, K, warp, j);
#pragma unroll
    for (int i = 0; i < 4; ++i) mine[j * 2 + (i & 1)][g + 8 * (i >> 1)] = acc[0][i];
  } else {
    float acc[2][4] = {};
    const __nv_bfloat16* const xr[2] = {row_of(g), row_of(8 + g)};
    few_rows_products<2, NW, 4>(acc, w0, w1, xr, K, warp, j);
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) mine[t * 8 + j * 2 + (i & 1)][g + 8 * (i >> 1)] = acc[t][i];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rows * COLS; i += 32 * NW) {
    const int m = i / COLS, c = i % COLS;
    if (n0 + c >= N) continue;
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int q = 0; q < NW; ++q) {
      a += part[q][m][c];
      if (GATED) b += part[q][m][8 + c];
    }
    if (GATED) a = silu(a) * b;
    else if (relu2) a = fmaxf(a, 0.f) * fmaxf(a, 0.f);
    y[(size_t)pair_of_row[row0 + m] * ldy + n0 + c] = __float2bfloat16(a);
  }
}

// x: [T, D] (pitch ldx) -> xp[row_of_pair[t*k+j], :] ; rows not written stay as they are (the GEMM
// output rows of padding are never read back).  A block per token, which is read once; bound by the writes: 2463 x 8 rows of 2048 channels 12.2 us (a thread per
// 16 bytes of a row, with the division that takes: 20.4), 64 x 8 1.7 us (2.1).
__global__ void __launch_bounds__(256)
moe_dispatch_kernel(const __nv_bfloat16* x, long ldx, const int* row_of_pair, int n_pairs,
                    int k, int D, __nv_bfloat16* __restrict__ xp, MoeBounds bd) {
  pdl_begin();
  const long p0 = (long)blockIdx.x * k;
  const int choices = (int)min((long)k, n_pairs - p0);
  for (int c = threadIdx.x * 8; c < D; c += blockDim.x * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(x + (size_t)blockIdx.x * ldx + c);
    for (int j0 = 0; j0 < choices; j0 += 4) {
      int r[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = j0 + j < choices ? row_of_pair[p0 + j0 + j] : -1;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (r[j] >= 0 && OMNI_IN_BOUNDS(bd.max_rows == 0 || r[j] < bd.max_rows, bd.status, KID_MOE_DISPATCH))
          *reinterpret_cast<uint4*>(xp + (size_t)r[j] * D + c) = v;
    }
  }
}

// acc += sum_j w[j] * y[row(j), c .. c + 7], four rows on their way at a time; pairs with row < 0 contribute nothing.
__device__ __forceinline__ void add_pairs(float (&acc)[8], const __nv_bfloat16* __restrict__ y, const int* __restrict__ rows,
                                          const float* __restrict__ w, int k, int D, int c, const MoeBounds& bd) {
#pragma unroll 1
  for (int j0 = 0; j0 < k; j0 += 4) {
    uint4 u[4];
    float wj[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = j0 + i < k ? rows[j0 + i] : -1;
      const bool in = r >= 0 && OMNI_IN_BOUNDS(bd.max_rows == 0 || r < bd.max_rows, bd.status, KID_MOE_COMBINE);
      wj[i] = in ? w[j0 + i] : 0.f;
      u[i] = in ? ld_stream(y + (size_t)r * D + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = unpack_bf16(u[i].x), b = unpack_bf16(u[i].y), cc = unpack_bf16(u[i].z), d = unpack_bf16(u[i].w);
      acc[0] += wj[i] * a.x; acc[1] += wj[i] * a.y; acc[2] += wj[i] * b.x; acc[3] += wj[i] * b.y;
      acc[4] += wj[i] * cc.x; acc[5] += wj[i] * cc.y; acc[6] += wj[i] * d.x; acc[7] += wj[i] * d.y;
    }
  }
}

// out[t, :] = (residual[t, :]) + sum_j w[t,j] * y[row(t,j), :]; pairs with row < 0 (experts of
// another rank) contribute nothing.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __nv_bfloat16* y, const int* row_of_pair,
                   const float* weights, int T, int k, int D, const __nv_bfloat16* residual,
                   long ldr, __nv_bfloat16* __restrict__ out, long ldo, MoeBounds bd) {
  pdl_begin();
  const int chunks = D >> 3;
  const long total = (long)T * chunks;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int t = (int)(i / chunks);
    const int c = (int)(i % chunks) * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (residual) {
      const uint4 u = *reinterpret_cast<const uint4*>(residual + (size_t)t * ldr + c);
      const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), cc = unpack_bf16(u.z), d = unpack_bf16(u.w);
      acc[0] = a.x; acc[1] = a.y; acc[2] = b.x; acc[3] = b.y; acc[4] = cc.x; acc[5] = cc.y; acc[6] = d.x; acc[7] = d.y;
    }
    add_pairs(acc, y, row_of_pair + (size_t)t * k, weights + (size_t)t * k, k, D, c, bd);
    uint4 o;
    o.x = pack_bf16(acc[0], acc[1]); o.y = pack_bf16(acc[2], acc[3]);
    o.z = pack_bf16(acc[4], acc[5]); o.w = pack_bf16(acc[6], acc[7]);
    *reinterpret_cast<uint4*>(out + (size_t)t * ldo + c) = o;
  }
}

// The same followed by the RMS norm of the sums (of the values as stored, in bf16), which the layer after reads: a block per token, a
// chunk of 8 channels per thread.  A norm of its own is one more dependent launch, 3 of a layer's 50 us for one token, and reads the
// rows again for many.  Four layers of 128 experts (2048 -> 768, top 8) and their attention: one sequence 249 -> 239 us per step, 64 sequences
// 1190 -> 1159 us.
__global__ void __launch_bounds__(1024)
moe_combine_norm_kernel(const __nv_bfloat16* y, const int* row_of_pair, const float* weights, int k, int D,
                        const __nv_bfloat16* residual, long ldr, __nv_bfloat16* __restrict__ out, long ldo,
                        const __nv_bfloat16* gain, float eps, __nv_bfloat16* __restrict__ normed, long ldn, MoeBounds bd) {
  pdl_begin();
  __shared__ float red[32];
  const int t = blockIdx.x, c = threadIdx.x * 8, warps = blockDim.x >> 5;
  const bool in = c < D;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  uint4 w = make_uint4(0u, 0u, 0u, 0u), o = w;
  if (in) {
    w = *reinterpret_cast<const uint4*>(gain + c);
    if (residual) {
      const uint4 u = *reinterpret_cast<const uint4*>(residual + (size_t)t * ldr + c);
      const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), cc = unpack_bf16(u.z), d = unpack_bf16(u.w);
      acc[0] = a.x; acc[1] = a.y; acc[2] = b.x; acc[3] = b.y; acc[4] = cc.x; acc[5] = cc.y; acc[6] = d.x; acc[7] = d.y;
    }
    add_pairs(acc, y, row_of_pair + (size_t)t * k, weights + (size_t)t * k, k, D, c, bd);
    o = make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
    *reinterpret_cast<uint4*>(out + (size_t)t * ldo + c) = o;
  }
  uint32_t v[4] = {o.x, o.y, o.z, o.w};
  const uint32_t g[4] = {w.x, w.y, w.z, w.w};
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16(v[j]);
    ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
  }
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, i);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
  for (int i = 0; i < warps; ++i) ss += red[i];
  const float rstd = rsqrtf(ss * (1.0f / (float)D) + eps);
  if (!in) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16(v[j]), m = unpack_bf16(g[j]);
    v[j] = pack_bf16(f.x * rstd * m.x, f.y * rstd * m.y);
  }
  *reinterpret_cast<uint4*>(normed + (size_t)t * ldn + c) = make_uint4(v[0], v[1], v[2], v[3]);
}

// Expert-parallel combine: the weighted sum of THIS rank's experts for token t is a partial result;
// it is stored straight into the slot this rank owns on the rank that owns token t's row block
// (peer_out[t / rows_per_owner], local row t % rows_per_owner, pitch D), so the cross-rank sum needs
// no separate all-reduce of a [T, D] tensor: a local reduce kernel finishes it (tp_reduce.cu).
struct MoePeers {
  __nv_bfloat16* out[16];
};
__global__ void __launch_bounds__(256)
moe_combine_scatter_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ row_of_pair,
                           const float* __restrict__ weights, int T, int k, int D, int rows_per_owner, MoePeers peers,
                           MoeBounds bd) {
  const int chunks = D >> 3;
  const long total = (long)T * chunks;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int t = (int)(i / chunks);
    const int c = (int)(i % chunks) * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    add_pairs(acc, y, row_of_pair + (size_t)t * k, weights + (size_t)t * k, k, D, c, bd);
    uint4 o;
    o.x = pack_bf16(acc[0], acc[1]); o.y = pack_bf16(acc[2], acc[3]);
    o.z = pack_bf16(acc[4], acc[5]); o.w = pack_bf16(acc[6], acc[7]);
    const int owner = t / rows_per_owner;
    *reinterpret_cast<uint4*>(peers.out[owner] + (size_t)(t - owner * rows_per_owner) * D + c) = o;
  }
}

}  // namespace omni

using namespace omni;
typedef __nv_bfloat16 bf16;

// 1 when this library was compiled with -DOMNI_BOUNDS_CHECK
extern "C" int omni_moe_bounds_check_enabled(void) {
#ifdef OMNI_BOUNDS_CHECK
  return 1;
#else
  return 0;
#endif
}

extern "C" void omni_moe_set_bounds(long max_rows, int* status) {
  g_moe_bounds.max_rows = max_rows;
  g_moe_bounds.status = status;
}

extern "C" int omni_moe_combine_scatter(const void* y, const int* row_of_pair, const float* weights, int T, int k, int D,
                                        int rows_per_owner, void* const* peer_out, void* stream) {
  if (T <= 0) return RC_OK;
  if ((D & 7) || rows_per_owner <= 0 || peer_out == nullptr) return RC_BAD_ARG;
  const int owners = (T + rows_per_owner - 1) / rows_per_owner;
  if (owners > 16) return RC_BAD_ARG;
  MoePeers peers;
  for (int i = 0; i < 16; ++i) peers.out[i] = i < owners ? static_cast<__nv_bfloat16*>(peer_out[i]) : nullptr;
  long blocks = ((long)T * (D >> 3) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  moe_combine_scatter_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)y, row_of_pair, weights, T, k, D, rows_per_owner, peers, g_moe_bounds);
  return (int)cudaGetLastError();
}

extern "C" int omni_moe_route(const void* logits, int ld, int T, int E, int k, int renorm, int* ids, float* weights,
                              void* stream) {
  if (T <= 0) return RC_OK;
  if (E > 256 || k > 16 || k > E) return RC_BAD_ARG;
  launch_overlapped(moe_route_kernel, (T + 7) / 8, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)logits, ld, T, E, k, renorm, ids, weights);
  return (int)cudaGetLastError();
}

static bool router_rule_ok(const RouterRule& r, int E, int k) {
  if (E > 256 || E < 1 || k > 16 || k > E || k < 1) return false;
  return r.groups == 0 || (r.sigmoid && r.groups > 0 && E % r.groups == 0 && r.keep >= 1 && r.keep <= r.groups && r.keep * (E / r.groups) >= k);
}

extern "C" int omni_moe_topk(const float* logits, long ld, int T, int E, int k, const RouterRule* rule, int* ids, float* weights,
                             void* stream) {
  if (T <= 0) return RC_OK;
  if (!router_rule_ok(*rule, E, k)) return RC_BAD_ARG;
  moe_topk_kernel<<<(T + 7) / 8, 256, 0, (cudaStream_t)stream>>>(logits, ld, T, E, k, *rule, ids, weights);
  return (int)cudaGetLastError();
}

// x [T, D] and w [Ep >= E, D] bf16 (D, pitches multiples of 8), bias [E] fp32 or null.
extern "C" int omni_moe_router(const void* x, long ldx, const void* w, long ldw, const float* bias, int T, int D, int E, int Ep,
                               int k, const RouterRule* rule, int* ids, float* weights, void* stream) {
  if (T <= 0) return RC_OK;
  if (!router_rule_ok(*rule, E, k) || D <= 0 || (D & 7) || (ldx & 7) || (ldw & 7)) return RC_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const bf16* xb = (const bf16*)x;
  const bf16* wb = (const bf16*)w;
  static unsigned long long prep[2] = {0, 0};
  if (T > 148 * 16) {
    const int smem = (8 * 32 * 64 + 32 * 256) * 4;
    if (int e = ensure_dynamic_smem((const void*)moe_router_kernel<2, 8>, smem, prep[0])) return e;
    launch_overlapped(moe_router_kernel<2, 8>, (T + 31) / 32, 256, smem, st, xb, ldx, wb, ldw, bias, T, D, E, Ep, k, *rule, ids, weights);
  } else {
    const int smem = (16 * 16 * 64 + 16 * 256) * 4;
    if (int e = ensure_dynamic_smem((const void*)moe_router_kernel<1, 16>, smem, prep[1])) return e;
    launch_overlapped(moe_router_kernel<1, 16>, (T + 15) / 16, 512, smem, st, xb, ldx, wb, ldw, bias, T, D, E, Ep, k, *rule, ids, weights);
  }
  return (int)cudaGetLastError();
}

// Pair p reads row p / per of x.
extern "C" int omni_moe_pairs_f32(const float* x, long ldx, int per, const int* ids, const float* w, int E, float* y, long ldy,
                                  long pairs, int N, int K, int relu2, void* stream) {
  if (pairs <= 0 || N <= 0) return RC_OK;
  if (per < 1 || E < 1 || K < 1) return RC_BAD_ARG;
  const long blocks = (pairs * N + 7) / 8;
  if (blocks > 0x7fffffffL) return RC_BAD_ARG;
  moe_pairs_f32_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(x, ldx, per, ids, w, E, y, ldy, pairs, N, K, relu2);
  return (int)cudaGetLastError();
}

// Experts [e_lo, e_hi) are local (expert parallelism); others get row -1.
// max_tiles: capacity of tile_expert = ceil((n_pairs + E*127) / 128).
extern "C" int omni_moe_plan(const int* ids, int n_pairs, int E, int e_lo, int e_hi, int max_tiles, int* row_of_pair,
                             int* tile_expert, int* offsets, int* n_rows_out, void* stream) {
  if (E > 1024) return RC_BAD_ARG;
  moe_plan_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(ids, n_pairs, E, e_lo, e_hi, max_tiles, row_of_pair, tile_expert, offsets, n_rows_out,
                                                        g_moe_bounds);
  return (int)cudaGetLastError();
}

// Even tiles of at most tile_cap (64, 128 or 256) rows for omni_gemm_bf16_experts; max_tiles: at least min(E, n_pairs) + n_pairs / tile_cap.
extern "C" int omni_moe_plan_tiles(const int* ids, int n_pairs, int E, int e_lo, int e_hi, int tile_cap, int max_tiles, int* row_of_pair,
                                   int* tile_expert, int* tile_row0, int* tile_rows, int* n_rows_out, void* stream) {
  if (E > 1024 || (tile_cap != 64 && tile_cap != 128 && tile_cap != 256)) return RC_BAD_ARG;
  // 128 experts, one block against eight: 512 pairs 2.6 and 4.4 us (the cluster's barriers), 8000 4.8 and 4.9, 19704 9.3 and 6.1, 64000 29 and 7.9
  if (n_pairs > 8192)
    launch_with(true, PLAN_CLUSTER, moe_plan_tiles_kernel<PLAN_CLUSTER>, PLAN_CLUSTER, 1024, 0, (cudaStream_t)stream, ids, n_pairs, E, e_lo, e_hi, tile_cap, max_tiles,
                row_of_pair, tile_expert, tile_row0, tile_rows, n_rows_out, g_moe_bounds);
  else
    launch_overlapped(moe_plan_tiles_kernel<1>, 1, 1024, 0, (cudaStream_t)stream, ids, n_pairs, E, e_lo, e_hi, tile_cap, max_tiles, row_of_pair,
                      tile_expert, tile_row0, tile_rows, n_rows_out, g_moe_bounds);
  return (int)cudaGetLastError();
}

// Plan of at most FEW_PAIRS pairs.  `logits` bf16 [T, E] (E <= 256, k <= 16): the choice is made here, ids and weights are outputs; null:
// ids [T * k] are given, E <= 1024.
extern "C" int omni_moe_few_plan(const void* logits, int ld, int T, int E, int k, int renorm, int e_lo, int e_hi, int* ids, float* weights,
                                 int* pair_of_row, int* row_of_pair, int* tile_expert, int* tile_row0, int* tile_rows, int max_tiles,
                                 void* stream) {
  if (T <= 0) return RC_OK;
  if (E > (logits ? 256 : 1024) || (logits && (k > 16 || k > E)) || T * k > FEW_PAIRS) return RC_BAD_ARG;
  const FewPlan p = {ids, weights, pair_of_row, row_of_pair, tile_expert, tile_row0, tile_rows, max_tiles};
  launch_overlapped(moe_few_plan_kernel, 1, 1024, 0, (cudaStream_t)stream, (const bf16*)logits, ld, T, E, k, renorm, e_lo, e_hi, p, g_moe_bounds);
  return (int)cudaGetLastError();
}

// Pair p reads row p / per of x [.., K] and writes row p of y; w [experts, N or 2 N (gated), K].  act: 0 none, 3 relu2, 5 SwiGLU.
extern "C" int omni_moe_few_rows(const void* x, long ldx, int per, const void* w, int N, int K, const int* tile_expert,
                                 const int* tile_row0, const int* tile_rows, int max_tiles, const int* pair_of_row, void* y, long ldy,
                                 int act, void* stream) {
  if (max_tiles <= 0 || N <= 0) return RC_OK;
  if (per < 1 || K <= 0 || (K & 7) || (ldx & 7) || max_tiles > 65535 || (act != 0 && act != 3 && act != 5)) return RC_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return RC_BAD_ARG;
  const bool gated = act == 5;
  const dim3 grid((unsigned)((N + (gated ? 7 : 15)) / (gated ? 8 : 16)), (unsigned)max_tiles);
  cudaStream_t st = (cudaStream_t)stream;
#define OMNI_FEW(NW, G)                                                                                                             \
  launch_overlapped(moe_few_rows_kernel<NW, G>, grid, 32 * NW, 0, st, (const bf16*)x, ldx, per, (const bf16*)w, N, K, tile_expert, tile_row0, tile_rows, \
                                                      pair_of_row, (bf16*)y, ldy, act == 3)
  // 8 warps have up to 2048 channels in flight at once; short contractions keep more blocks per SM instead
  if (K > 1024) {
    if (gated) OMNI_FEW(8, true); else OMNI_FEW(8, false);
  } else {
    if (gated) OMNI_FEW(4, true); else OMNI_FEW(4, false);
  }
#undef OMNI_FEW
  return (int)cudaGetLastError();
}

extern "C" int omni_moe_dispatch(const void* x, long ldx, const int* row_of_pair, int n_pairs, int k, int D, void* xp,
                                 void* stream) {
  if (n_pairs <= 0) return RC_OK;
  if ((D & 7) || k < 1) return RC_BAD_ARG;
  const int threads = min((D / 8 + 31) / 32 * 32, 256);
  launch_overlapped(moe_dispatch_kernel, (unsigned)((n_pairs + k - 1) / k), threads, 0, (cudaStream_t)stream, (const __nv_bfloat16*)x, ldx, row_of_pair, n_pairs, k, D, (__nv_bfloat16*)xp,
                                                                          g_moe_bounds);
  return (int)cudaGetLastError();
}

extern "C" int omni_moe_combine(const void* y, const int* row_of_pair, const float* weights, int T, int k, int D,
                                const void* residual, long ldr, void* out, long ldo, void* stream) {
  if (T <= 0) return RC_OK;
  if (D & 7) return RC_BAD_ARG;
  long blocks = ((long)T * (D >> 3) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  launch_overlapped(moe_combine_kernel, (unsigned)blocks, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)y, row_of_pair, weights, T, k, D, (const __nv_bfloat16*)residual, ldr, (__nv_bfloat16*)out, ldo,
      g_moe_bounds);
  return (int)cudaGetLastError();
}

// Also normed[t] = out[t] / rms(out[t]) * gain; D at most 8192, as for the norms of rows (elementwise.cu).
extern "C" int omni_moe_combine_norm(const void* y, const int* row_of_pair, const float* weights, int T, int k, int D, const void* residual,
                                     long ldr, void* out, long ldo, const void* gain, float eps, void* normed, long ldn, void* stream) {
  if (T <= 0) return RC_OK;
  if (D <= 0 || (D & 7) || D > 8192 || ((ldr | ldo | ldn) & 7)) return RC_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(gain) |
       reinterpret_cast<uintptr_t>(normed)) & 15)
    return RC_BAD_ARG;
  launch_overlapped(moe_combine_norm_kernel, (unsigned)T, (D / 8 + 31) / 32 * 32, 0, (cudaStream_t)stream, (const bf16*)y, row_of_pair, weights, k, D,
                    (const bf16*)residual, ldr, (bf16*)out, ldo, (const bf16*)gain, eps, (bf16*)normed, ldn, g_moe_bounds);
  return (int)cudaGetLastError();
}
