// NaN/Inf check of up to three 16-bit tensors of a call in one launch.
//
// The eager cache calls refuse inputs that are not finite before they touch the cache (the reference's contract), so the
// host has to wait for an answer.  torch.isfinite(t).all() per tensor is five launches, a copy and a wait for each of q, k
// and v, and it was most of an eager call's time (eight requests, four new tokens each: 3 x 70 of 450 us).  Here one launch looks at all of
// them and writes straight into the caller's pinned words, so a call waits once and copies nothing.  Bound: the launch
// and the wait for small inputs, HBM for whole prompts (every element is read once, 16 bytes a load, four loads in flight per thread).
#include <cuda_runtime.h>
#include <stdint.h>

#include "moba_b200.h"

namespace moba {
namespace {

struct FiniteView {
  const uint16_t* ptr[3];
  long long rows[3], st_t[3], st_h[3];  // rows = tokens * heads; element strides of token and head
  int heads[3], vec[3];                 // vec: every row starts on a 16-byte boundary
  int dim, count;
  uint32_t exponent;                    // the all-ones exponent of the format, in both halves of a word
  int* flags;
};

// true when one of the two values of a word has an all-ones exponent (Inf or NaN); the halves are tested one at a time
__device__ __forceinline__ bool not_finite2(uint32_t w, uint32_t e) {
  return (w & e & 0xFFFFu) == (e & 0xFFFFu) || (w & e & 0xFFFF0000u) == (e & 0xFFFF0000u);
}
__device__ __forceinline__ bool not_finite8(const uint4& w, uint32_t e) {
  return not_finite2(w.x, e) || not_finite2(w.y, e) || not_finite2(w.z, e) || not_finite2(w.w, e);
}

__global__ void __launch_bounds__(256) finite_kernel(FiniteView f) {
  const int which = blockIdx.y;
  if (which >= f.count) return;
  const uint16_t* base = f.ptr[which];
  const int heads = f.heads[which];
  bool bad = false;
  auto row_of = [&](long long r) {
    const long long t = r / heads;
    return base + t * f.st_t[which] + (r - t * heads) * f.st_h[which];
  };
  const long long first = (long long)blockIdx.x * 256 + threadIdx.x, step = (long long)gridDim.x * 256;
  if (f.vec[which]) {
    const int upr = f.dim >> 3;
    const long long units = f.rows[which] * upr;
    for (long long i = first; i < units; i += 4 * step) {
      uint4 w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long long at = i + j * step;
        w[j] = make_uint4(0u, 0u, 0u, 0u);
        if (at < units) {
          const long long r = at / upr;
          w[j] = *reinterpret_cast<const uint4*>(row_of(r) + (at - r * upr) * 8);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) bad |= not_finite8(w[j], f.exponent);
    }
  } else {
    const long long n = f.rows[which] * f.dim;
    for (long long i = first; i < n; i += step) {
      const long long r = i / f.dim;
      bad |= not_finite2(row_of(r)[i - r * f.dim], f.exponent);  // the upper half is zero: finite
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) f.flags[which] = 1;
}

}  // namespace
}  // namespace moba

using namespace moba;

extern "C" int moba_check_finite(const moba_finite_input* inputs, int count, int dim, int fp16, int32_t* flags, void* stream) {
  if (!inputs || !flags || count < 1 || count > 3 || dim < 1) return MOBA_ERR_INVALID;
  FiniteView f = {};
  long long most = 0;
  for (int i = 0; i < count; ++i) {
    const moba_finite_input& in = inputs[i];
    if (!in.data || in.tokens < 1 || in.heads < 1) return MOBA_ERR_INVALID;
    f.ptr[i] = static_cast<const uint16_t*>(in.data);
    f.rows[i] = in.tokens * in.heads;
    f.heads[i] = in.heads;
    f.st_t[i] = in.stride_t;
    f.st_h[i] = in.stride_h;
    f.vec[i] = dim % 8 == 0 && !((uintptr_t)in.data & 15) && (in.tokens == 1 || in.stride_t % 8 == 0) && (in.heads == 1 || in.stride_h % 8 == 0);
    const long long units = f.vec[i] ? f.rows[i] * (dim / 8) : f.rows[i] * dim;
    most = units > most ? units : most;
  }
  f.dim = dim;
  f.count = count;
  f.exponent = fp16 ? 0x7C007C00u : 0x7F807F80u;
  f.flags = flags;
  // a thread takes up to four units at once; eight CTAs per SM are enough to fill the memory pipeline
  const long long blocks = (most + 1023) / 1024;
  finite_kernel<<<dim3((unsigned)(blocks < 1184 ? blocks : 1184), count), 256, 0, (cudaStream_t)stream>>>(f);
  return cudaGetLastError() == cudaSuccess ? MOBA_OK : MOBA_ERR_CUDA;
}
