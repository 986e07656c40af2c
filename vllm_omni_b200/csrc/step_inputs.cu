// What a decoder step does before its first layer, in one launch each.
//
//   omni_fill_step    a step's values into the static tensors that a captured graph reads: up to 16 row copies with the
//                     padding rows of a larger batch (csrc side of engine/graph_runner.py)
//   omni_token_rows   embedding rows (or given rows where a mask says so) and the rotation tables cos / sin of every token
//
// Both move a few kilobytes; what they save is launches: ten to fifteen and ten, 2 us each on the device and 4 us each on the
// host, of a step that takes 250 us at one token.
#include "host_util.h"
#include "ptx_sm100.cuh"

namespace omni {

constexpr int FILL_JOBS = 16;

// Row i < n of `dst` takes row order[i] (ordered) or i of `src`; rows past n repeat row 0's source or become int32 -1, 1 or 0 (pad 1, 2, 3).  Bytes past
// src_bytes of a row are zero.  src == nullptr: zeros everywhere.
struct FillJob {
  const unsigned char* src;
  unsigned char* dst;
  long src_pitch, dst_pitch;
  int src_bytes, dst_bytes;
  int ordered, pad;
};
struct FillStep {
  FillJob jobs[FILL_JOBS];
  const long* order;
  int n_jobs, n, rows;
};

__global__ void __launch_bounds__(128)
fill_step_kernel(const __grid_constant__ FillStep p) {
  pdl_begin();
  const FillJob& j = p.jobs[blockIdx.y];
  const int i = blockIdx.x;
  const bool live = i < p.n;
  const long from = j.ordered ? p.order[live ? i : 0] : (live ? i : 0);
  const unsigned char* s = j.src ? j.src + from * j.src_pitch : nullptr;
  unsigned char* d = j.dst + (long)i * j.dst_pitch;
  const int pad = live ? 0 : j.pad;
  const bool words = ((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(d) | (unsigned)j.src_bytes | (unsigned)j.dst_bytes) & 3) == 0;
  if (words) {
    for (int c = threadIdx.x; c < j.dst_bytes / 4; c += 128)
      reinterpret_cast<uint32_t*>(d)[c] = pad ? (pad == 1 ? 0xffffffffu : (uint32_t)(pad == 2)) : (s && c < j.src_bytes / 4 ? reinterpret_cast<const uint32_t*>(s)[c] : 0u);
  } else {
    for (int c = threadIdx.x; c < j.dst_bytes; c += 128) d[c] = pad ? (pad == 1 ? 0xff : (unsigned char)(pad == 2 && (c & 3) == 0)) : (s && c < j.src_bytes ? s[c] : 0);
  }
}

struct TokenRows {
  const long* ids;
  const uint4* table;                  // [vocab, vecs]
  const uint4* given;                  // [T, vecs] or nullptr
  const unsigned char* mask;           // [T]: where the given row counts; nullptr = everywhere
  uint4* out;
  const long* pos;                     // [T], or [axes, T] at axis_pitch
  const float* freq;                   // [half]
  const int* axis;                     // [half] or nullptr (axis 0)
  float *cosv, *sinv;                  // [T, half]
  long axis_pitch;
  int vocab, vecs, half;
};

__global__ void __launch_bounds__(256)
token_rows_kernel(const __grid_constant__ TokenRows p) {
  pdl_begin();
  const long t = blockIdx.x;
  const bool given = p.given && (!p.mask || p.mask[t]);
  long id = p.ids[t];
  id = id < 0 ? 0 : (id >= p.vocab ? p.vocab - 1 : id);
  const uint4* src = given ? p.given + t * p.vecs : p.table + id * p.vecs;
  for (int c = threadIdx.x; c < p.vecs; c += 256) p.out[t * p.vecs + c] = src[c];
  for (int i = threadIdx.x; i < p.half; i += 256) {
    const float a = __fmul_rn((float)p.pos[(p.axis ? p.axis[i] * p.axis_pitch : 0) + t], p.freq[i]);
    p.cosv[t * p.half + i] = cosf(a);
    p.sinv[t * p.half + i] = sinf(a);
  }
}

}  // namespace omni

using namespace omni;

extern "C" int omni_fill_step(const FillStep* p, void* stream) {
  if (p->rows <= 0 || p->n_jobs <= 0) return RC_OK;
  if (p->n_jobs > FILL_JOBS || p->n < 1 || p->n > p->rows) return RC_BAD_ARG;
  launch_overlapped(fill_step_kernel, dim3((unsigned)p->rows, (unsigned)p->n_jobs), 128, 0, (cudaStream_t)stream, *p);
  return (int)cudaGetLastError();
}

extern "C" int omni_token_rows(const TokenRows* p, long T, void* stream) {
  if (T <= 0) return RC_OK;
  if (p->vocab <= 0 || p->vecs <= 0 || T > 0x7fffffffL) return RC_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(p->table) | reinterpret_cast<uintptr_t>(p->given) | reinterpret_cast<uintptr_t>(p->out)) & 15) return RC_BAD_ARG;
  launch_overlapped(token_rows_kernel, (unsigned)T, 256, 0, (cudaStream_t)stream, *p);
  return (int)cudaGetLastError();
}
