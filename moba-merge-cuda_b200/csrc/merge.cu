// Standalone global-softmax merge of a self branch with scattered remote contributions: the operator the
// reference exposes as merge_forward (src/moba_opt/ops/merge_cuda.py:32-60, ops/bindings.cpp:6-22,
// ops/merge.cu:27-288).  The prefill path does not use it (there the merge is the epilogue of the forward
// kernel); it exists for callers that hold the two branches themselves.
//   row p of the self branch (P = T*H rows) and every remote row m with mapping[m] == p are combined as
//   mx = max l, w = exp(l - mx), z = sum w, O = sum w o / z, L = mx + log z      (natural-log LSE, FP32 math)
// Two kernels: contributions are ticketed into per-row slot lists (atomic counters), then every row sorts
// its at most 32 contribution indices and reduces them in ascending order, so the result does not depend
// on the ticket order.  HBM-bound: every input byte is read once, every output byte written once.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "launch.cuh"
#include "moba_b200.h"
#include "sm100.cuh"

namespace moba {
namespace {

// Clears the counters.  A kernel, not a memset, so that the ticket pass can be a dependent launch behind it, its mapping read by
// then (229376 rows, 619 thousand contributions: 36.9 -> 33.8 us a merge).
__global__ void __launch_bounds__(256) merge_clear_kernel(int* counts, long long P) {
  dependents_may_start();
  const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
  if (i + 4 <= P && !(reinterpret_cast<uintptr_t>(counts) & 15)) *reinterpret_cast<int4*>(counts + i) = make_int4(0, 0, 0, 0);
  else for (long long j = i; j < min(i + 4, P); ++j) counts[j] = 0;
}

__global__ void __launch_bounds__(256) merge_ticket_kernel(const int64_t* __restrict__ mapping, long long M, long long P, int kmax,
                                                           int* counts, int* slots, unsigned* status) {
  const long long m = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long p = m < M ? mapping[m] : 0;   // an input of the call, read beside the clearing
  wait_for_predecessor();                       // the counters are clear, and whoever used this scratch before is done
  dependents_may_start();                       // the row kernel's self rows do not depend on the lists
  if (m >= M) return;
  if (p < 0 || p >= P) { atomicOr(status, kErrBadIndex); return; }
  const int slot = atomicAdd(counts + p, 1);
  if (slot < kmax) slots[p * kmax + slot] = (int)m;
  else atomicOr(status, kErrCapacity);
}

// 16 bytes of a row as eight (bf16, half) or four (fp32) FP32 values.
template <typename T> struct Chunk;
template <> struct Chunk<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void load(const __nv_bfloat16* p, float (&v)[8]) { unpack(*reinterpret_cast<const uint4*>(p), v); }
  __device__ static void unpack(const uint4& raw, float (&v)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
  }
  __device__ static void store(__nv_bfloat16* p, const float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <> struct Chunk<__half> {
  static constexpr int N = 8;
  __device__ static void load(const __half* p, float (&v)[8]) { unpack(*reinterpret_cast<const uint4*>(p), v); }
  __device__ static void unpack(const uint4& raw, float (&v)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
  }
  __device__ static void store(__half* p, const float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <> struct Chunk<float> {
  static constexpr int N = 4;
  __device__ static void load(const float* p, float (&v)[4]) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
  }
  __device__ static void unpack(const uint4& raw, float (&v)[4]) {
    v[0] = __uint_as_float(raw.x); v[1] = __uint_as_float(raw.y); v[2] = __uint_as_float(raw.z); v[3] = __uint_as_float(raw.w);
  }
  __device__ static void store(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};

// Rows with at most KM <= 16 contributions, in two stages per warp.
//   lists   a lane owns a row: count, contribution indices sorted in registers by an odd-even transposition network, their
//           LSEs, the weights.  These are three dependent trips to memory, and what bounded the kernel when every group of
//           lanes made them for its own row: a warp had 4 rows (head_dim 64) in flight per chain of trips, not 32.
//   rows    LPR lanes share a row, 16 bytes of it each per pass; the owner's indices and weights come through shared memory.
//           Two rows per group and up to four contributions of each are loaded before any is added, in ascending index order.
// rpw: rows per warp, 32 / LPR or 32.  Bound by memory: self row, remote rows and output once each; the registers are held
// to seven CTAs per SM (four above four contributions) because loads in flight are what counts - raw 16-byte values wait in
// registers, not their FP32 forms.  229376 rows of 64 bf16 with 2.7 contributions on average, 138 MB: 27 us = 5.1 TB/s; with
// lists per lane group in local memory 66 us, with this split but FP32 values and lists in registers (134 of them) 56 us.
// The kernel is a dependent launch.
template <typename T, int LPR, int KM>
__global__ void __launch_bounds__(128, KM <= 4 ? 7 : 4) merge_rows_kernel(const T* __restrict__ self_out, const float* __restrict__ self_lse,
                                                         const T* __restrict__ remote_out, const float* __restrict__ remote_lse,
                                                         const int* counts, const int* slots, long long P, int D, int kmax, int rpw,
                                                         T* __restrict__ out, float* __restrict__ lse) {
  constexpr int N = Chunk<T>::N;
  constexpr int GROUPS = 32 / LPR;
  constexpr int B = KM < 4 ? KM : 4;   // contributions loaded together
  constexpr int U = 2;                 // rows of a group in flight
  __shared__ int s_idx[128][KM | 1];   // lists of the CTA's rows, 32 per warp
  __shared__ float s_w[128][KM | 1];
  __shared__ float4 s_row[128];        // weight of the self row, 1 / denominator, contributions
  const int lane = threadIdx.x & 31, sub = lane % LPR;
  const long long row0 = ((long long)blockIdx.x * 4 + (threadIdx.x >> 5)) * rpw;
  if (row0 >= P) return;
  // ---- lists: lane r owns row r of the warp (the lanes past rpw repeat its rows)
  const long long own = row0 + (lane & (rpw - 1));
  const float l_self = own < P ? self_lse[own] : -INFINITY;
  wait_for_predecessor();   // the lists of the ticket pass
  const int cnt = own < P ? min(__ldcg(counts + own), kmax) : 0;
  int idx[KM];
#pragma unroll
  for (int i = 0; i < KM; ++i) idx[i] = i < cnt ? __ldcg(slots + own * kmax + i) : 0x7FFFFFFF;
#pragma unroll
  for (int pass = 0; pass < KM; ++pass) {
#pragma unroll
    for (int i = pass & 1; i + 1 < KM; i += 2) {
      const int lo = min(idx[i], idx[i + 1]), hi = max(idx[i], idx[i + 1]);
      idx[i] = lo; idx[i + 1] = hi;
    }
  }
  float w[KM];
  float mx = l_self;
#pragma unroll
  for (int i = 0; i < KM; ++i) w[i] = i < cnt ? remote_lse[idx[i]] : -INFINITY;
#pragma unroll
  for (int i = 0; i < KM; ++i) mx = fmaxf(mx, w[i]);
  const bool empty = mx == -INFINITY;  // no branch saw a key: zero output, LSE stays -inf
  const float w_self = empty ? 0.f : expf(l_self - mx);
  float z = w_self;
#pragma unroll
  for (int i = 0; i < KM; ++i) {
    w[i] = empty || i >= cnt ? 0.f : expf(w[i] - mx);
    z += w[i];
  }
  const float inv = z > 0.f ? 1.f / z : 0.f;
  if (own < P && lane < rpw) lse[own] = empty ? -INFINITY : mx + logf(z);
  if (lane < rpw) {
    const int wl = (threadIdx.x >> 5) * 32 + lane;
#pragma unroll
    for (int i = 0; i < KM; ++i) { s_idx[wl][i] = idx[i]; s_w[wl][i] = w[i]; }
    s_row[wl] = make_float4(w_self, inv, __int_as_float(own < P ? cnt : -1), 0.f);
  }
  __syncwarp();
  // ---- rows
  for (int r0 = lane / LPR; r0 < rpw; r0 += U * GROUPS) {
    const int* ix[U];
    const float* ww[U];
    int n[U];
    float ws[U], iv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = (threadIdx.x >> 5) * 32 + min(r0 + u * GROUPS, 31);
      const float4 head = s_row[r];
      ws[u] = head.x; iv[u] = head.y;
      n[u] = r0 + u * GROUPS < rpw ? __float_as_int(head.z) : -1;   // -1: no such row
      ix[u] = s_idx[r];
      ww[u] = s_w[r];
    }
    for (int d = sub * N; d < D; d += LPR * N) {
      uint4 self[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (n[u] >= 0) self[u] = *reinterpret_cast<const uint4*>(self_out + (row0 + r0 + u * GROUPS) * D + d);
      float acc[U][N];
#pragma unroll
      for (int i0 = 0; i0 < KM; i0 += B) {
        uint4 raw[U][B];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
          for (int i = 0; i < B; ++i)
            if (i0 + i < KM && i0 + i < n[u]) raw[u][i] = *reinterpret_cast<const uint4*>(remote_out + (long long)ix[u][i0 + i] * D + d);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (i0 == 0) {
            Chunk<T>::unpack(self[u], acc[u]);
#pragma unroll
            for (int e = 0; e < N; ++e) acc[u][e] *= ws[u];
          }
#pragma unroll
          for (int i = 0; i < B; ++i)
            if (i0 + i < KM && i0 + i < n[u]) {
              float v[N];
              Chunk<T>::unpack(raw[u][i], v);
#pragma unroll
              for (int e = 0; e < N; ++e) acc[u][e] = fmaf(ww[u][i0 + i], v[e], acc[u][e]);
            }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (n[u] < 0) continue;
#pragma unroll
        for (int e = 0; e < N; ++e) acc[u][e] *= iv[u];
        Chunk<T>::store(out + (row0 + r0 + u * GROUPS) * D + d, acc[u]);
      }
    }
  }
}

// The same for 17 to 32 contributions per row: the index list sits in local memory.
template <typename T, int LPR>
__global__ void __launch_bounds__(256) merge_rows_many_kernel(const T* __restrict__ self_out, const float* __restrict__ self_lse,
                                                         const T* __restrict__ remote_out, const float* __restrict__ remote_lse,
                                                         const int* __restrict__ counts, const int* __restrict__ slots, long long P,
                                                         int D, int kmax, T* __restrict__ out, float* __restrict__ lse) {
  constexpr int N = Chunk<T>::N;
  const int lane = threadIdx.x & 31, sub = lane % LPR;
  const long long row = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 / LPR) + lane / LPR;
  if (row >= P) return;
  const int cnt = min(counts[row], kmax);
  int idx[32];
  float w[32];
  for (int i = 0; i < cnt; ++i) {  // insertion sort of the contribution indices (ascending)
    const int v = slots[row * kmax + i];
    int j = i;
    while (j > 0 && idx[j - 1] > v) { idx[j] = idx[j - 1]; --j; }
    idx[j] = v;
  }
  const float l_self = self_lse[row];
  float mx = l_self;
  for (int i = 0; i < cnt; ++i) { w[i] = remote_lse[idx[i]]; mx = fmaxf(mx, w[i]); }
  const bool empty = mx == -INFINITY;  // no branch saw a key: zero output, LSE stays -inf
  const float w_self = empty ? 0.f : expf(l_self - mx);
  float z = w_self;
  for (int i = 0; i < cnt; ++i) { w[i] = empty ? 0.f : expf(w[i] - mx); z += w[i]; }
  const float inv = z > 0.f ? 1.f / z : 0.f;
  for (int d = sub * N; d < D; d += LPR * N) {
    float acc[N], v[N];
    Chunk<T>::load(self_out + row * D + d, v);
#pragma unroll
    for (int e = 0; e < N; ++e) acc[e] = w_self * v[e];
    for (int i = 0; i < cnt; ++i) {
      Chunk<T>::load(remote_out + (long long)idx[i] * D + d, v);
#pragma unroll
      for (int e = 0; e < N; ++e) acc[e] = fmaf(w[i], v[e], acc[e]);
    }
#pragma unroll
    for (int e = 0; e < N; ++e) acc[e] *= inv;
    Chunk<T>::store(out + row * D + d, acc);
  }
  if (sub == 0) lse[row] = empty ? -INFINITY : mx + logf(z);
}

// Fallback for head dimensions whose rows are not multiples of 16 bytes: one warp per row, scalar accesses.
template <typename T>
__global__ void __launch_bounds__(256) merge_rows_scalar_kernel(const T* __restrict__ self_out, const float* __restrict__ self_lse,
                                                                const T* __restrict__ remote_out, const float* __restrict__ remote_lse,
                                                                const int* __restrict__ counts, const int* __restrict__ slots,
                                                                long long P, int D, int kmax, T* __restrict__ out,
                                                                float* __restrict__ lse) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= P) return;
  const int cnt = min(counts[row], kmax);
  int idx[32];
  float w[32];
  for (int i = 0; i < cnt; ++i) {
    const int v = slots[row * kmax + i];
    int j = i;
    while (j > 0 && idx[j - 1] > v) { idx[j] = idx[j - 1]; --j; }
    idx[j] = v;
  }
  const float l_self = self_lse[row];
  float mx = l_self;
  for (int i = 0; i < cnt; ++i) { w[i] = remote_lse[idx[i]]; mx = fmaxf(mx, w[i]); }
  const bool empty = mx == -INFINITY;
  const float w_self = empty ? 0.f : expf(l_self - mx);
  float z = w_self;
  for (int i = 0; i < cnt; ++i) { w[i] = empty ? 0.f : expf(w[i] - mx); z += w[i]; }
  const float inv = z > 0.f ? 1.f / z : 0.f;
  for (int d = lane; d < D; d += 32) {
    float acc = w_self * (float)self_out[row * D + d];
    for (int i = 0; i < cnt; ++i) acc = fmaf(w[i], (float)remote_out[(long long)idx[i] * D + d], acc);
    out[row * D + d] = (T)(acc * inv);
  }
  if (lane == 0) lse[row] = empty ? -INFINITY : mx + logf(z);
}

// The list length in registers is the smallest of 1, 2, 3, 4, 8, 16 that holds kmax: an unused entry still costs its
// comparators in the sorting network.
template <typename T, int LPR>
void launch_rows_as(const T* so, const float* self_lse, const T* ro, const float* remote_lse, const int* counts, const int* slots,
                    long long rows, int dim, int kmax, T* o, float* lse, cudaStream_t st) {
  // A warp takes 32 rows where that still gives every SM a few warps; below that its groups take one row each.
  const int rpw = rows >= 32ll * 4 * device_sms() ? 32 : 32 / LPR;
  const long long per_cta = 4ll * rpw;
  auto go = [&](auto kernel) {
    launch_dependent(32u, kernel, dim3((unsigned)((rows + per_cta - 1) / per_cta)), dim3(128), 0, st, so, self_lse, ro, remote_lse, counts,
                     slots, rows, dim, kmax, rpw, o, lse);
  };
  if (kmax == 1) go(merge_rows_kernel<T, LPR, 1>);
  else if (kmax == 2) go(merge_rows_kernel<T, LPR, 2>);
  else if (kmax == 3) go(merge_rows_kernel<T, LPR, 3>);
  else if (kmax == 4) go(merge_rows_kernel<T, LPR, 4>);
  else if (kmax <= 8) go(merge_rows_kernel<T, LPR, 8>);
  else if (kmax <= 16) go(merge_rows_kernel<T, LPR, 16>);
  else merge_rows_many_kernel<T, LPR><<<(unsigned)((rows * LPR + 255) / 256), 256, 0, st>>>(so, self_lse, ro, remote_lse, counts, slots, rows, dim, kmax, o, lse);
}

template <typename T>
void launch_rows(const void* self_out, const float* self_lse, const void* remote_out, const float* remote_lse, const int* counts,
                 const int* slots, long long rows, int dim, int kmax, void* out, float* lse, cudaStream_t st) {
  const T* so = static_cast<const T*>(self_out);
  const T* ro = static_cast<const T*>(remote_out);
  T* o = static_cast<T*>(out);
  constexpr int N = Chunk<T>::N;
  const bool vec = dim % N == 0 && (reinterpret_cast<uintptr_t>(so) | reinterpret_cast<uintptr_t>(ro) | reinterpret_cast<uintptr_t>(o)) % 16 == 0;
  if (!vec) {
    merge_rows_scalar_kernel<T><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(so, self_lse, ro, remote_lse, counts, slots, rows, dim, kmax, o, lse);
    return;
  }
  const int chunks = dim / N;
  if (chunks <= 4) launch_rows_as<T, 4>(so, self_lse, ro, remote_lse, counts, slots, rows, dim, kmax, o, lse, st);
  else if (chunks <= 8) launch_rows_as<T, 8>(so, self_lse, ro, remote_lse, counts, slots, rows, dim, kmax, o, lse, st);
  else if (chunks <= 16) launch_rows_as<T, 16>(so, self_lse, ro, remote_lse, counts, slots, rows, dim, kmax, o, lse, st);
  else launch_rows_as<T, 32>(so, self_lse, ro, remote_lse, counts, slots, rows, dim, kmax, o, lse, st);
}

inline size_t align256m(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace
}  // namespace moba

using namespace moba;

extern "C" size_t moba_merge_scratch_bytes(long long rows, int kmax) {
  if (rows < 1 || kmax < 1 || kmax > 32) return 0;
  return align256m((size_t)rows * 4) + align256m((size_t)rows * kmax * 4);
}

extern "C" int moba_merge_forward(const void* self_out, const float* self_lse, const void* remote_out, const float* remote_lse,
                                  const int64_t* mapping, long long rows, long long remote_rows, int dim, int kmax, int dtype,
                                  void* scratch, size_t scratch_bytes, void* out, float* lse, unsigned* status, void* stream) {
  if (rows < 1 || remote_rows < 0 || dim < 1 || !self_out || !self_lse || !out || !lse || !status || !scratch) return MOBA_ERR_INVALID;
  if (remote_rows > 0 && (!remote_out || !remote_lse || !mapping)) return MOBA_ERR_INVALID;
  if (kmax < 1 || kmax > 32 || dtype < 0 || dtype > 2) return MOBA_ERR_UNSUPPORTED;
  if (scratch_bytes < moba_merge_scratch_bytes(rows, kmax)) return MOBA_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  int* counts = static_cast<int*>(scratch);
  int* slots = reinterpret_cast<int*>(static_cast<char*>(scratch) + align256m((size_t)rows * 4));
  merge_clear_kernel<<<(unsigned)((rows + 1023) / 1024), 256, 0, st>>>(counts, rows);
  if (remote_rows > 0)
    launch_dependent(32u, merge_ticket_kernel, dim3((unsigned)((remote_rows + 255) / 256)), dim3(256), 0, st, mapping, remote_rows, rows, kmax, counts, slots,
                     status);
  if (dtype == 0)
    launch_rows<__nv_bfloat16>(self_out, self_lse, remote_out, remote_lse, counts, slots, rows, dim, kmax, out, lse, st);
  else if (dtype == 2)
    launch_rows<__half>(self_out, self_lse, remote_out, remote_lse, counts, slots, rows, dim, kmax, out, lse, st);
  else
    launch_rows<float>(self_out, self_lse, remote_out, remote_lse, counts, slots, rows, dim, kmax, out, lse, st);
  return cudaGetLastError() == cudaSuccess ? MOBA_OK : MOBA_ERR_CUDA;
}
