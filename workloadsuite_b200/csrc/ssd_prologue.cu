// dt discretisation of SSDLayer.forward ahead of the core (model_ref.py:94, 102-103):
//   dt   = softplus(dt_raw + dt_bias[head])          in the layer's 16-bit (or fp32) dtype
//   A_dt = -exp(A_log[head]) * float(dt)             fp32, the per-token log-decay the core consumes
// dt_raw is read in place as a column slice of the projection output; both results are written contiguously.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ssd_b200.h"
#include "ssd_common.cuh"

namespace ssd {
namespace {

// The reference adds in the layer's dtype, then takes softplus in that dtype (threshold 20, as torch).
template <typename T>
__device__ __forceinline__ T discretise(T raw, T bias) {
  const float v = Cvt<T>::to_f(Cvt<T>::from_f(Cvt<T>::to_f(raw) + Cvt<T>::to_f(bias)));
  return Cvt<T>::from_f(v > 20.f ? v : log1pf(expf(v)));
}

// V consecutive heads per thread (V = 8: 16-byte pieces of 16-bit rows; V = 1 where rows are not aligned), the same heads
// in every row of the grid's stride, so that bias and rate are read once and nothing is divided per element.
// I: int where the row counter stays within it to the end (a division of 64 bits per row is dear), else int64_t.
template <typename T, int V, typename I>
__global__ void __launch_bounds__(128)
dt_prologue_kernel(const T* __restrict__ dt_raw, int64_t sb, int64_t sl, const T* __restrict__ dt_bias,
                   const float* __restrict__ A_log, T* __restrict__ dt_out, float* __restrict__ A_dt, I rows,
                   int seqlen, int nheads) {
  const I vecs = nheads / V;
  const I first = (I)blockIdx.x * blockDim.x + threadIdx.x;
  const I step = (I)gridDim.x * blockDim.x / vecs;   // rows per pass; threads past step * vecs have none
  if (first >= step * vecs) return;
  const int h0 = (int)(first % vecs) * V;
  float rate[V];
  T bias[V];
#pragma unroll
  for (int e = 0; e < V; ++e) {
    rate[e] = -expf(A_log[h0 + e]);
    bias[e] = dt_bias ? dt_bias[h0 + e] : Cvt<T>::from_f(0.f);
  }
  for (I r = first / vecs; r < rows; r += step) {
    const I b = r / seqlen;
    const T* src = dt_raw + b * sb + (int64_t)(r - b * seqlen) * sl + h0;
    const int64_t o = (int64_t)r * nheads + h0;
    alignas(16) T in[V], d[V];
    alignas(16) float a[V];
    constexpr int kWords = sizeof(T) * V / 16;
    if constexpr (V > 1) {
#pragma unroll
      for (int k = 0; k < kWords; ++k) reinterpret_cast<uint4*>(in)[k] = reinterpret_cast<const uint4*>(src)[k];
    } else {
      in[0] = src[0];
    }
#pragma unroll
    for (int e = 0; e < V; ++e) {
      d[e] = discretise<T>(in[e], bias[e]);
      a[e] = rate[e] * Cvt<T>::to_f(d[e]);
    }
    if constexpr (V > 1) {
#pragma unroll
      for (int k = 0; k < kWords; ++k) reinterpret_cast<uint4*>(dt_out + o)[k] = reinterpret_cast<const uint4*>(d)[k];
#pragma unroll
      for (int k = 0; k < V / 4; ++k) reinterpret_cast<float4*>(A_dt + o)[k] = reinterpret_cast<const float4*>(a)[k];
    } else {
      dt_out[o] = d[0];
      A_dt[o] = a[0];
    }
  }
}

template <typename T>
int launch_prologue(const void* dt_raw, int64_t sb, int64_t sl, const void* dt_bias, const float* A_log, void* dt_out,
                    float* A_dt, int batch, int seqlen, int nheads, cudaStream_t stream) {
  constexpr int V = 8, per16 = 16 / (int)sizeof(T);
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  // (a few rows: one head per thread, so that the functions of the eight do not run one after the other)
  const int64_t rows = (int64_t)batch * seqlen;
  const bool vec = nheads % V == 0 && rows >= ((1LL << 17) + nheads - 1) / nheads && al(dt_raw) && al(dt_out) && al(A_dt) &&
                   sb % per16 == 0 && sl % per16 == 0;
  const int vecs = vec ? nheads / V : nheads;
  // up to sixteen small CTAs per SM (as many as there is work for), and at least one pass of whole rows
  const int64_t most = 148 * 16, wanted = rows >= most * 128 ? most : std::min<int64_t>((rows * vecs + 127) / 128, most);
  const int64_t ctas = std::max<int64_t>(wanted, (vecs + 127LL) / 128);
  const bool small = rows + ctas * 128 <= 0x7fffffffLL;   // (a pass is at most ctas * 128 rows)
  auto go = [&](auto kern, auto nrows) {
    return launch(kern, (unsigned)ctas, 128, 0, stream, static_cast<const T*>(dt_raw), sb, sl, static_cast<const T*>(dt_bias),
                  A_log, static_cast<T*>(dt_out), A_dt, nrows, seqlen, nheads);
  };
  if (small) return vec ? go(dt_prologue_kernel<T, V, int>, (int)rows) : go(dt_prologue_kernel<T, 1, int>, (int)rows);
  return vec ? go(dt_prologue_kernel<T, V, int64_t>, rows) : go(dt_prologue_kernel<T, 1, int64_t>, rows);
}

}  // namespace
}  // namespace ssd

extern "C" int ssd_b200_dt_prologue(const void* dt_raw, int64_t stride_b, int64_t stride_l, const void* dt_bias,
                                    const float* A_log, void* dt_out, float* A_dt_out, int32_t batch, int32_t seqlen,
                                    int32_t nheads, int32_t dtype, void* stream) {
  if (!dt_raw || !A_log || !dt_out || !A_dt_out) return SSD_ERR_NULL_POINTER;
  if (batch <= 0 || seqlen <= 0 || nheads <= 0) return SSD_ERR_BAD_SHAPE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case SSD_DTYPE_F32:
      return ssd::launch_prologue<float>(dt_raw, stride_b, stride_l, dt_bias, A_log, dt_out, A_dt_out, batch, seqlen,
                                         nheads, s);
    case SSD_DTYPE_F16:
      return ssd::launch_prologue<__half>(dt_raw, stride_b, stride_l, dt_bias, A_log, dt_out, A_dt_out, batch, seqlen,
                                          nheads, s);
    case SSD_DTYPE_BF16:
      return ssd::launch_prologue<__nv_bfloat16>(dt_raw, stride_b, stride_l, dt_bias, A_log, dt_out, A_dt_out, batch,
                                                 seqlen, nheads, s);
    default:
      return SSD_ERR_UNSUPPORTED;
  }
}
