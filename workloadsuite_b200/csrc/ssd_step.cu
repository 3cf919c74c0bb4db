// One token of the SSD recurrence per call, the state carried in place: the decode-style use of the carry of
// model_ref.py:152-157 (the reference itself only has the chunked forward; one token of it reduces to this):
//   H[b,h] <- exp(a[b,h]) * H[b,h] + B[b,g] (x) (dt[b,h] * x[b,h])        H is [n, p] fp32
//   y[b,h] <- C[b,g] . H[b,h]   (+ x * D[h], then * silu(z), as model_ref.py:116-118, when given)
// HBM-bound: the fp32 state is read and written once (2 * n * p * 4 bytes per (b, h)); everything else is small.
// One CTA of 128 threads per (batch, head) and half of the columns, or of 256 threads and all of them (columns are independent,
// rows are what y sums over): thread (r, c) owns four state columns of the rows r, r + 16, ...; all of its state loads are
// issued before the first use (n / 16 sixteen-byte loads in flight per thread), y is reduced over the sixteen row groups
// through shared memory.  Contiguous operands have an instance of their own, whose offsets follow from the unit: with few state
// rows the 64-bit products of the strides are a third of a CTA's time (5120 heads, n 16: 11.7 us with them, 8.2 without).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ssd_b200.h"
#include "ssd_common.cuh"

namespace ssd {
namespace {

constexpr int kHeadDim = 64;
constexpr int kMaxRowsPerThread = 16;           // dstate <= 256

// ROWS = dstate / 16; COLS: columns of a CTA; DENSE: every operand contiguous.
template <typename T, int ROWS, int COLS, bool DENSE>
__global__ void __launch_bounds__(4 * COLS)
ssd_step_kernel(const SsdStepArgs p) {
  constexpr int kCols = COLS, kLanes = COLS / 4, kStepThreads = 16 * kLanes, kParts = kHeadDim / COLS;
  __shared__ float ypart[16][kCols];
  __shared__ float bs[16 * ROWS], cs[16 * ROWS];
  constexpr int n = 16 * ROWS;
  const int unit = blockIdx.x / kParts;      // b * nheads + h
  const int col0 = (blockIdx.x % kParts) * kCols;
  const int b = unit / p.nheads, h = unit - b * p.nheads;
  const int g = h / (p.nheads / p.ngroups);
  const int tid = threadIdx.x, r = tid / kLanes, c = tid % kLanes;
  float4* S = reinterpret_cast<float4*>(p.state + (int64_t)unit * n * kHeadDim + col0) + c;
  float4 hv[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) hv[i] = S[(int64_t)(i * 16 + r) * (kHeadDim / 4)];   // all loads first
  const int64_t row_bc = (int64_t)(b * p.ngroups + g) * n;
  const T* Bg = static_cast<const T*>(p.B) + (DENSE ? row_bc : b * p.b_stride[0] + g * p.b_stride[1]);
  const T* Cg = static_cast<const T*>(p.C) + (DENSE ? row_bc : b * p.c_stride[0] + g * p.c_stride[1]);
  for (int i = tid; i < n; i += kStepThreads) {
    bs[i] = Cvt<T>::to_f(Bg[i]);
    cs[i] = Cvt<T>::to_f(Cg[i]);
  }
  const T* xr = static_cast<const T*>(p.x) + (DENSE ? (int64_t)unit * kHeadDim : b * p.x_stride[0] + h * p.x_stride[1]) + col0;
  const bool has_dt = p.dt != nullptr;
  const float dtv = has_dt ? Cvt<T>::to_f(static_cast<const T*>(p.dt)[DENSE ? unit : b * p.dt_stride[0] + h * p.dt_stride[1]]) : 1.f;
  const float av = p.a[DENSE ? unit : b * p.a_stride[0] + h * p.a_stride[1]];
  // x * dt in the layer's precision, as the reference forms it (model_ref.py:144)
  float xd[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float xv = Cvt<T>::to_f(xr[4 * c + e]);
    xd[e] = has_dt ? Cvt<T>::to_f(Cvt<T>::from_f(xv * dtv)) : xv;
  }
  // what the epilogue needs, fetched while the state is on its way
  float xs = 0.f, ds = 0.f, zs = 0.f;
  if (tid < kCols) {
    if (p.D) {
      xs = Cvt<T>::to_f(xr[tid]);
      ds = p.d_in_dtype ? Cvt<T>::to_f(static_cast<const T*>(p.D)[h]) : static_cast<const float*>(p.D)[h];
    }
    if (p.z) zs = Cvt<T>::to_f(static_cast<const T*>(p.z)[(DENSE ? (int64_t)unit * kHeadDim : b * p.z_stride[0] + h * p.z_stride[1]) + col0 + tid]);
  }
  const float decay = __expf(av);
  __syncthreads();
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int row = i * 16 + r;
    const float bn = bs[row], cn = cs[row];
    float4 v = hv[i];
    v.x = fmaf(decay, v.x, bn * xd[0]); v.y = fmaf(decay, v.y, bn * xd[1]);
    v.z = fmaf(decay, v.z, bn * xd[2]); v.w = fmaf(decay, v.w, bn * xd[3]);
    S[(int64_t)row * (kHeadDim / 4)] = v;
    acc[0] = fmaf(cn, v.x, acc[0]); acc[1] = fmaf(cn, v.y, acc[1]);
    acc[2] = fmaf(cn, v.z, acc[2]); acc[3] = fmaf(cn, v.w, acc[3]);
  }
  *reinterpret_cast<float4*>(&ypart[r][4 * c]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  __syncthreads();
  if (tid < kCols) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) s += ypart[k][tid];
    if (p.D) s = fmaf(xs, ds, s);
    if (p.z) s *= zs / (1.f + __expf(-zs));
    static_cast<T*>(p.y)[(int64_t)unit * kHeadDim + col0 + tid] = Cvt<T>::from_f(s);
  }
}

bool dense(const SsdStepArgs& p) {
  const int64_t h = p.nheads, g = p.ngroups, n = p.dstate;
  auto is = [&](const int64_t* st, int64_t heads, int64_t inner) {
    return (p.batch == 1 || st[0] == heads * inner) && (heads == 1 || st[1] == inner);
  };
  return is(p.x_stride, h, kHeadDim) && is(p.a_stride, h, 1) && is(p.b_stride, g, n) && is(p.c_stride, g, n) &&
         (!p.dt || is(p.dt_stride, h, 1)) && (!p.z || is(p.z_stride, h, kHeadDim));
}

template <typename T, int ROWS>
int launch_step(const SsdStepArgs& p, cudaStream_t stream) {
  // Half of the columns per CTA where that reaches more SMs, and for n = 64 and 128 (1024 heads, n 128, states in L2: 7.1 us, 7.6
  // with all columns; from memory 12.7 and 12.4).  With fewer rows a CTA has too little to do (5120 heads, n 16: 9.8 and 8.2;
  // n 32: 10.7 and 10.0, but strided 14.4 and 15.3), with more the loads of half the columns are enough in flight (20480
  // heads, n 256: 393 and 388).
  const int units = p.batch * p.nheads;
  const bool d = dense(p), half = ROWS == 4 || ROWS == 8 || (ROWS == 2 && !d) || 2 * units <= 148;
  if (d)
    return half ? launch(ssd_step_kernel<T, ROWS, 32, true>, 2 * units, 128, 0, stream, p)
                : launch(ssd_step_kernel<T, ROWS, 64, true>, units, 256, 0, stream, p);
  return half ? launch(ssd_step_kernel<T, ROWS, 32, false>, 2 * units, 128, 0, stream, p)
              : launch(ssd_step_kernel<T, ROWS, 64, false>, units, 256, 0, stream, p);
}

template <typename T>
int launch_rows(const SsdStepArgs& p, cudaStream_t stream) {
  switch (p.dstate / 16) {
    case 1: return launch_step<T, 1>(p, stream);
    case 2: return launch_step<T, 2>(p, stream);
    case 4: return launch_step<T, 4>(p, stream);
    case 8: return launch_step<T, 8>(p, stream);
    case 16: return launch_step<T, 16>(p, stream);
    default: return SSD_ERR_UNSUPPORTED;
  }
}

}  // namespace
}  // namespace ssd

extern "C" int ssd_b200_step_strided(const SsdStepArgs* p, void* stream) {
  if (!p || !p->x || !p->a || !p->B || !p->C || !p->state || !p->y) return SSD_ERR_NULL_POINTER;
  if (p->batch <= 0 || p->nheads <= 0 || p->headdim <= 0 || p->dstate <= 0 || p->ngroups <= 0 || p->nheads % p->ngroups != 0)
    return SSD_ERR_BAD_SHAPE;
  if (p->headdim != ssd::kHeadDim || p->dstate % 16 != 0 || p->dstate / 16 > ssd::kMaxRowsPerThread)
    return SSD_ERR_UNSUPPORTED;
  if ((int64_t)p->batch * p->nheads > 0x3fffffffLL) return SSD_ERR_TOO_LARGE;
  if (reinterpret_cast<uintptr_t>(p->state) & 15) return SSD_ERR_MISALIGNED;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (p->dtype) {
    case SSD_DTYPE_F32: return ssd::launch_rows<float>(*p, s);
    case SSD_DTYPE_F16: return ssd::launch_rows<__half>(*p, s);
    case SSD_DTYPE_BF16: return ssd::launch_rows<__nv_bfloat16>(*p, s);
    default: return SSD_ERR_UNSUPPORTED;
  }
}

extern "C" int ssd_b200_step(const void* x, const float* a, const void* B, const void* C, const void* dt,
                             const float* D, const void* z, float* state, void* y, int32_t batch, int32_t nheads,
                             int32_t headdim, int32_t dstate, int32_t ngroups, int32_t dtype, void* stream) {
  const int64_t h = nheads, p = headdim, g = ngroups, n = dstate;
  const SsdStepArgs s = {x, a, B, C, dt, D, z, state, y, batch, nheads, headdim, dstate, ngroups, dtype, 0, 0,
                         {h * p, p}, {h, 1}, {g * n, n}, {g * n, n}, {h, 1}, {h * p, p}};
  return ssd_b200_step_strided(&s, stream);
}
