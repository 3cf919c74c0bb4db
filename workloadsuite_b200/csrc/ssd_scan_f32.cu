// fp32 CUDA-core SSD scan: the token-by-token recurrence
//   H_t = exp(a_t) H_{t-1} + B_t (x) (x_t dt_t),   y_t = C_t . H_t
// which the chunked form of the reference (model_ref.py:135-162) is
// algebraically equal to.  It is the exact-arithmetic path (fp32 inputs, the
// 1e-4 tolerance; from 64 tokens on mostly in chunked form, see
// launch_scan_f32()) and the fallback for shapes the tensor-core kernel does not
// cover.  One CTA walks one (batch, head[, segment]) with the n x p state held
// in registers: thread (j, sl) owns column j of the state and the rows
// n_i = (k*SL + sl)*4 + q, so the B/C rows are read from shared memory as
// conflict-free float4 broadcasts and y_t is finished by a shuffle over the SL
// lanes that share a column.
#include <algorithm>
#include <type_traits>
#include "chunk_f32.cuh"
#include "ssd_common.cuh"

namespace ssd {

namespace {

constexpr int kThreads = 256;
constexpr int kTile = 32;  // tokens staged in shared memory per step: a multiple of this, see tile_tokens()

template <typename T>
__device__ __forceinline__ void load8(const T* src, float* dst);

template <>
__device__ __forceinline__ void load8<__half>(const __half* src, float* dst) {
  uint4 v = *reinterpret_cast<const uint4*>(src);
  const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __half22float2(h[i]);
    dst[2 * i] = f.x;
    dst[2 * i + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* src, float* dst) {
  uint4 v = *reinterpret_cast<const uint4*>(src);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __bfloat1622float2(h[i]);
    dst[2 * i] = f.x;
    dst[2 * i + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void load8<float>(const float* src, float* dst) {
  float4 a = *reinterpret_cast<const float4*>(src);
  float4 b = *reinterpret_cast<const float4*>(src + 4);
  dst[0] = a.x; dst[1] = a.y; dst[2] = a.z; dst[3] = a.w;
  dst[4] = b.x; dst[5] = b.y; dst[6] = b.z; dst[7] = b.w;
}

template <typename T>
__device__ __forceinline__ void store8(T* dst, const float* src);
template <>
__device__ __forceinline__ void store8<__half>(__half* dst, const float* src) {
  uint4 v;
  __half2* h = reinterpret_cast<__half2*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(src[2 * i], src[2 * i + 1]);
  *reinterpret_cast<uint4*>(dst) = v;
}
template <>
__device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16* dst, const float* src) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(src[2 * i], src[2 * i + 1]);
  *reinterpret_cast<uint4*>(dst) = v;
}
template <>
__device__ __forceinline__ void store8<float>(float* dst, const float* src) {
  *reinterpret_cast<float4*>(dst) = make_float4(src[0], src[1], src[2], src[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(src[4], src[5], src[6], src[7]);
}

// Copies `rows` rows of `width` elements (row r at src + r*row_stride) into a
// dense fp32 [rows][width] shared-memory tile, optionally scaling row r by
// scale[r].
template <typename T, int UNROLL>
__device__ __forceinline__ void stage_rows(const T* src, int64_t row_stride, int rows, int width, float* dst,
                                           bool vec_ok, int tid) {
  if (sizeof(T) == 4 && vec_ok) {   // no conversion: asynchronous copies, waited for once all tensors' are under way
    const int per_row = width >> 2;
    for (int i = tid; i < rows * per_row; i += kThreads) {
      const int r = i / per_row, c = (i - r * per_row) << 2;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * width + c)),
                   "l"(src + r * row_stride + c)
                   : "memory");
    }
  } else if (vec_ok) {
    const int per_row = width >> 3;
#pragma unroll UNROLL
    for (int i = tid; i < rows * per_row; i += kThreads) {
      const int r = i / per_row, c = (i - r * per_row) << 3;
      load8<T>(src + r * row_stride + c, dst + r * width + c);
    }
  } else {
    for (int i = tid; i < rows * width; i += kThreads) {
      const int r = i / width, c = i - r * width;
      dst[r * width + c] = Cvt<T>::to_f(src[r * row_stride + c]);
    }
  }
}

// Sums v[0..U) over the SL lanes of an aligned group; lane sl is left with the sums of elements sl * U / SL + i in v[i].
template <int U, int SL>
__device__ __forceinline__ void reduce_scatter(float (&v)[U], int sl) {
  int left = U;
#pragma unroll
  for (int m = SL / 2; m >= 1; m >>= 1) {
    left >>= 1;
    const bool upper = sl & m;
#pragma unroll
    for (int i = 0; i < U / 2; ++i) {
      if (i < left) {
        const float send = upper ? v[i] : v[i + left];
        v[i] = (upper ? v[i + left] : v[i]) + __shfl_xor_sync(0xffffffffu, send, m);
      }
    }
  }
}

// FULL: the state has exactly NS * SL rows (the strides of B and C in shared memory are then constants).
// LINE: tokens worked on in line (1: one after the other).  CTAS: as many of an SM the registers have to leave room for (0: as
// it comes).  Tokens in line take 64 to 126 registers, one after the other 32 to 80; see launch_one().
// REDO: behind the tensor-core kernel at fp32 precision (ssd_split.cu), and only if that kernel says so; see Jobs.
// A piece of a scan.
struct Job {
  int unit, seg;
  bool compute_y;
  const float* init;   // or null
  float* fin;          // or null
  float* fin_ld;       // or null
};

// What the two passes and the fold of cut sequences do (or whole sequences one after the other), in one launch of as many CTAs as
// the chip holds, which take numbers from a counter: first every segment from a zero state, then the states entering the
// segments (256 elements a time, written over what they are made of), then every segment again.  What a number waits for has
// lower ones, which CTAs that run already have taken, so no wait needs a CTA that is still to come.  The counters are behind the
// words that say whether there is anything to do (RedoWords), cleared by the kernel ahead.  (1 x 131 001 tokens of 8 heads 3.65 ms,
// as three launches 3.38; whole sequences 41.2.  Two more launches would cost every call that need not be done again.)
struct Jobs {
  const ScanParams& p;
  unsigned* number;   // of the present job, in shared memory: what a job is is worked out again at its end, for the registers

  __device__ __forceinline__ bool cut() const { return p.nseg > 1; }
  __device__ __forceinline__ int64_t np() const { return (int64_t)p.n * p.p; }
  __device__ __forceinline__ unsigned units() const { return (unsigned)(p.batch * p.nheads); }
  __device__ __forceinline__ unsigned segs() const { return units() * (unsigned)p.nseg; }
  __device__ __forceinline__ unsigned parts() const { return (unsigned)((np() + kThreads - 1) / kThreads); }
  __device__ __forceinline__ unsigned first() const { return cut() ? segs() : 0; }             // number of the first fold,
  __device__ __forceinline__ unsigned second() const { return cut() ? segs() + units() * parts() : 0; }   // of the second pass
  // To the next one, or false.  All threads of the CTA.
  __device__ __forceinline__ bool next() const {
    while (true) {
      if (threadIdx.x == 0) {
        unsigned t = atomicAdd(reinterpret_cast<unsigned*>(p.redo + RedoWords::kNext), 1u);
        if (t >= second() + segs()) t = ~0u;
        else if (cut() && t >= second()) t = finished(RedoWords::kFolded, second() - first()) ? t : ~0u;
        else if (cut() && t >= first()) t = finished(RedoWords::kScanned, first()) ? t : ~0u;
        *number = t;
      }
      __syncthreads();
      const unsigned t = *number;
      if (t == ~0u) return false;
      if (t < first() || t >= second()) return true;
      fold((t - first()) / parts(), (t - first()) % parts());
      done(RedoWords::kFolded);
    }
  }
  __device__ __forceinline__ Job job() const {
    const unsigned t = *static_cast<volatile unsigned*>(number);
    const bool again = t >= second();
    const unsigned i = again ? t - second() : t, seg = i / units(), unit = i - seg * units();   // (the units of a segment share B and C)
    Job j = {(int)unit, (int)seg, again, nullptr, nullptr, nullptr};
    const int64_t at = (int64_t)unit * p.nseg + seg;
    if (!again) {
      j.fin = p.chain_state + at * np();
      j.fin_ld = p.chain_ld + at;
    } else if (cut()) {
      j.init = p.chain_state + at * np();
    } else {
      if (p.init) j.init = p.init + unit * np();
      if (p.fin) j.fin = p.fin + unit * np();
      if (p.fin_ld) j.fin_ld = p.fin_ld + unit;
    }
    return j;
  }
  // Behind the last write of a job.  All threads of the CTA.
  __device__ __forceinline__ void scanned() const {
    if (*number < first()) done(RedoWords::kScanned);
  }
  __device__ __forceinline__ void done(int word) const {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.redo + word) : "memory");
  }
  // (bounded: by what a wait may take, and ten microseconds for each token of a segment)
  __device__ __forceinline__ bool finished(int word, unsigned count) const {
    const long long t0 = clock64(), limit = p.wait_clocks + 20000LL * p.seg_len;
    while (true) {
      unsigned n;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(p.redo + word) : "memory");
      if (n >= count) return true;
      __nanosleep(100);
      if (clock64() - t0 > limit) {
        if (p.status) atomicCAS(p.status, 0, (int)STATUS_WAIT_TIMEOUT_CHAIN);
        return false;
      }
    }
  }
  // As ssd_fold_kernel below.
  __device__ __forceinline__ void fold(unsigned unit, unsigned part) const {
    const int64_t e = (int64_t)part * kThreads + threadIdx.x;
    const float* D = p.chain_ld + (int64_t)unit * p.nseg;
    const int64_t np = this->np();
    if (e < np) {
      float run = p.init ? p.init[unit * np + e] : 0.f;
      float* F = p.chain_state + (int64_t)unit * p.nseg * np + e;
      for (int s = 0; s < p.nseg; ++s) {
        const float f = __ldcg(F + s * np);
        F[s * np] = run;
        run = fmaf(run, expf(__ldcg(D + s)), f);
      }
      if (p.fin) p.fin[unit * np + e] = run;
    }
    if (p.fin_ld && part == 0 && threadIdx.x == 0) {
      double tot = 0.0;
      for (int s = 0; s < p.nseg; ++s) tot += (double)__ldcg(D + s);
      p.fin_ld[unit] = (float)tot;
    }
  }
};

template <typename T, int NS, int P, bool FULL, int LINE, int CTAS, bool REDO>
__global__ void __launch_bounds__(kThreads, CTAS) ssd_scan_f32_kernel(const ScanParams prm, const int tile) {
  constexpr int SL = kThreads / P;  // lanes sharing one state column
  constexpr int NS4 = NS / 4;
  extern __shared__ __align__(16) float smem[];
  const int n = FULL ? NS * SL : prm.n;
  float* Xs = smem;                  // [tile][P]   x_t * dt_t
  float* Bs = Xs + tile * P;         // [tile][n]
  float* Cs = Bs + tile * n;         // [tile][n]
  float* Ys = Cs + tile * n;         // [tile][P]
  float* dec = Ys + tile * P;        // [tile]  exp(a_t)
  float* araw = dec + tile;          // [tile]  a_t

  if constexpr (REDO) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int any = 0;
    for (int i = threadIdx.x; i < prm.redo_n; i += kThreads) any |= __ldcg(prm.redo + i);
    if (!__syncthreads_or(any)) {   // (that kernel leaves the sum of the log-decays to this one: in 64 bits, as below)
      if (!prm.fin_ld) return;
      double* part = reinterpret_cast<double*>(smem);
      for (int unit = blockIdx.x; unit < prm.batch * prm.nheads; unit += gridDim.x) {
        const float* A = prm.A + (int64_t)(unit / prm.nheads) * prm.as[0] + (int64_t)(unit % prm.nheads) * prm.as[2];
        double sum = 0.0;
        for (int t = threadIdx.x; t < prm.seqlen; t += kThreads) sum += (double)A[(int64_t)t * prm.as[1]];
        for (int d = 16; d >= 1; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
          for (int w = 1; w < kThreads / 32; ++w) sum += part[w];
          prm.fin_ld[(int64_t)unit * prm.finld_unit_stride] = (float)sum;
        }
        __syncthreads();
      }
      return;
    }
  }
  __shared__ unsigned number;
  const Jobs jobs = {prm, &number};
  Job job = {};
  int unit = blockIdx.x, seg = blockIdx.y;
  if (REDO && !jobs.next()) return;
  do {
  if constexpr (REDO) {
    job = jobs.job();
    unit = job.unit;
    seg = job.seg;
  }
  const int bi = unit / prm.nheads, hi = unit - bi * prm.nheads;
  const int gi = hi / (prm.nheads / prm.ngroups);
  const int tid = threadIdx.x;
  const int j = tid / SL, sl = tid - j * SL;
  const bool vec_ok = prm.vec_ok != 0;

  const int t_begin = seg * prm.seg_len;
  const int t_end = min(prm.seqlen, t_begin + prm.seg_len);

  const T* Xg = static_cast<const T*>(prm.X) + bi * prm.xs[0] + hi * prm.xs[2];
  const T* Bg = static_cast<const T*>(prm.B) + bi * prm.bs[0] + gi * prm.bs[2];
  const T* Cg = static_cast<const T*>(prm.C) + bi * prm.cs[0] + gi * prm.cs[2];
  const float* Ag = prm.A + bi * prm.as[0] + hi * prm.as[2];
  const T* Dg = prm.dt ? static_cast<const T*>(prm.dt) + bi * prm.dts[0] + hi * prm.dts[2] : nullptr;
  T* Yg = prm.Y ? static_cast<T*>(prm.Y) + bi * prm.ys[0] + hi * prm.ys[2] : nullptr;

  float h[NS];
  if (REDO ? job.init != nullptr : prm.init != nullptr) {
    const float* I = REDO ? job.init : prm.init + unit * prm.init_unit_stride + seg * prm.init_seg_stride;
#pragma unroll
    for (int k = 0; k < NS4; ++k)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int ni = (k * SL + sl) * 4 + q;
        h[k * 4 + q] = (ni < n) ? (REDO ? __ldcg(I + (int64_t)ni * P + j) : I[(int64_t)ni * P + j]) : 0.f;
      }
  } else {
#pragma unroll
    for (int k = 0; k < NS; ++k) h[k] = 0.f;
  }
  double asum = 0.0;

  for (int t0 = t_begin; t0 < t_end; t0 += tile) {
    const int rows = min(tile, t_end - t0);
    __syncthreads();  // previous tile fully consumed (Ys stored, Xs/Bs/Cs read)
    constexpr int kAhead = LINE == 1 ? 1 : 4;
    stage_rows<T, kAhead>(Xg + (int64_t)t0 * prm.xs[1], prm.xs[1], rows, P, Xs, vec_ok, tid);
    stage_rows<T, kAhead>(Bg + (int64_t)t0 * prm.bs[1], prm.bs[1], rows, n, Bs, vec_ok, tid);
    if (REDO ? job.compute_y : prm.compute_y) stage_rows<T, kAhead>(Cg + (int64_t)t0 * prm.cs[1], prm.cs[1], rows, n, Cs, vec_ok, tid);
    if (tid < rows) {
      const float a = Ag[(int64_t)(t0 + tid) * prm.as[1]];
      araw[tid] = a;
      dec[tid] = expf(a);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (Dg) {  // x~ = x * dt (model_ref.py:144)
      for (int i = tid; i < rows * P; i += kThreads) {
        const int r = i / P;
        Xs[i] *= Cvt<T>::to_f(Dg[(int64_t)(t0 + r) * prm.dts[1]]);
      }
      __syncthreads();
    }
    // U tokens in line: only the state's fma chain links them, so the shared-memory reads, the sums over the row groups and the
    // stores of one token run under those of the others (kept apart by hand: the compiler may not move a read of X, B or C
    // over a store of Y).
    auto tokens = [&](int t, auto ucount, auto want_y) {
      constexpr int U = decltype(ucount)::value;
      constexpr bool kY = decltype(want_y)::value;   // (a branch inside would end what the compiler may interleave)
      float x[U], d[U], y[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        x[u] = Xs[(t + u) * P + j];
        d[u] = dec[t + u];
        y[u] = 0.f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float4* B4 = reinterpret_cast<const float4*>(Bs + (t + u) * n);
        const float4* C4 = reinterpret_cast<const float4*>(Cs + (t + u) * n);
#pragma unroll
        for (int k = 0; k < NS4; ++k) {
          if ((k * SL) * 4 < n) {
            const float4 bv = B4[k * SL + sl];
            h[k * 4 + 0] = fmaf(h[k * 4 + 0], d[u], bv.x * x[u]);
            h[k * 4 + 1] = fmaf(h[k * 4 + 1], d[u], bv.y * x[u]);
            h[k * 4 + 2] = fmaf(h[k * 4 + 2], d[u], bv.z * x[u]);
            h[k * 4 + 3] = fmaf(h[k * 4 + 3], d[u], bv.w * x[u]);
            if constexpr (kY) {
              const float4 cv = C4[k * SL + sl];
              y[u] = fmaf(cv.x, h[k * 4 + 0], y[u]);
              y[u] = fmaf(cv.y, h[k * 4 + 1], y[u]);
              y[u] = fmaf(cv.z, h[k * 4 + 2], y[u]);
              y[u] = fmaf(cv.w, h[k * 4 + 3], y[u]);
            }
          }
        }
      }
      if constexpr (kY && U > 1) {
        reduce_scatter<U, SL>(y, sl);
#pragma unroll
        for (int i = 0; i < U / SL; ++i) {
          const int u = sl * (U / SL) + i;
          if constexpr (sizeof(T) == 4) Yg[(int64_t)(t0 + t + u) * prm.ys[1] + j] = y[i];   // (whole sectors: no staging)
          else Ys[(t + u) * P + j] = y[i];
        }
      } else if constexpr (kY) {
#pragma unroll
        for (int m = 1; m < SL; m <<= 1) y[0] += __shfl_xor_sync(0xffffffffu, y[0], m);
        if (sl == 0) {
          if constexpr (sizeof(T) == 4) Yg[(int64_t)(t0 + t) * prm.ys[1] + j] = y[0];
          else Ys[t * P + j] = y[0];
        }
      }
    };
    auto all = [&](auto want_y) {
      int t = 0;
      if constexpr (LINE > 1)
        for (; t + LINE <= rows; t += LINE) tokens(t, std::integral_constant<int, LINE>{}, want_y);
      for (; t < rows; ++t) tokens(t, std::integral_constant<int, 1>{}, want_y);
    };
    if (REDO ? job.compute_y : prm.compute_y) all(std::true_type{});
    else all(std::false_type{});
    if (tid == 0 && (REDO && prm.nseg > 1 ? !job.compute_y : prm.fin_ld != nullptr)) {
      for (int t = 0; t < rows; ++t) asum += (double)araw[t];
    }
    if (sizeof(T) < 4 && (REDO ? job.compute_y : prm.compute_y)) {
      __syncthreads();
      T* Yt = Yg + (int64_t)t0 * prm.ys[1];
      if constexpr (REDO) {   // with the skip and the gate, which that kernel applies too
        const T* Zg = prm.Z ? static_cast<const T*>(prm.Z) + bi * prm.zs[0] + hi * prm.zs[2] + (int64_t)t0 * prm.zs[1] : nullptr;
        if (prm.D || Zg) {
          for (int i = tid; i < rows * P; i += kThreads) {
            const int r = i / P, c = i - r * P;
            float v = Ys[i];
            if (prm.D) v = fmaf(Cvt<T>::to_f(Xg[(int64_t)(t0 + r) * prm.xs[1] + c]), load_skip<T>(prm, hi), v);
            if (Zg) {
              const float z = Cvt<T>::to_f(Zg[(int64_t)r * prm.zs[1] + c]);
              v *= z / (1.f + __expf(-z));
            }
            Ys[i] = v;
          }
          __syncthreads();
        }
      }
      if (vec_ok) {
        constexpr int per_row = P >> 3;
        for (int i = tid; i < rows * per_row; i += kThreads) {
          const int r = i / per_row, c = (i - r * per_row) << 3;
          store8<T>(Yt + r * prm.ys[1] + c, Ys + r * P + c);
        }
      } else {
        for (int i = tid; i < rows * P; i += kThreads) {
          const int r = i / P, c = i - r * P;
          Yt[r * prm.ys[1] + c] = Cvt<T>::from_f(Ys[i]);
        }
      }
    }
  }

  if constexpr (REDO) job = jobs.job();
  if (REDO ? job.fin != nullptr : prm.fin != nullptr) {
    float* F = REDO ? job.fin : prm.fin + unit * prm.fin_unit_stride + seg * prm.fin_seg_stride;
#pragma unroll
    for (int k = 0; k < NS4; ++k)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int ni = (k * SL + sl) * 4 + q;
        if (ni < n) F[(int64_t)ni * P + j] = h[k * 4 + q];
      }
  }
  if ((REDO ? job.fin_ld : prm.fin_ld) && tid == 0)
    *(REDO ? job.fin_ld : prm.fin_ld + unit * prm.finld_unit_stride + seg * prm.finld_seg_stride) = (float)asum;
  if constexpr (REDO) jobs.scanned();
  } while (REDO && jobs.next());
}

// H_in(seg) for every segment of every unit, from the zero-start final states:
//   run = init; for seg: emit run; run = run * exp(D_seg) + F_seg.
__global__ void ssd_fold_kernel(const float* states, int64_t st_unit_stride, int64_t st_seg_stride, const float* ld,
                                int64_t ld_unit_stride, int64_t ld_seg_stride, const float* init, float* out_single,
                                float* out_final, float* out_ld, int upto, float* incoming, int64_t np) {
  const int64_t unit = blockIdx.x;
  const int64_t e = (int64_t)blockIdx.y * blockDim.x + threadIdx.x;
  if (e >= np) return;
  float run = init ? init[unit * np + e] : 0.f;
  const float* F = states + unit * st_unit_stride + e;
  float* G = incoming ? incoming + unit * st_unit_stride + e : nullptr;   // same layout as `states`
  const float* D = ld + unit * ld_unit_stride;
  for (int s = 0; s < upto; ++s) {
    const float f = F[(int64_t)s * st_seg_stride];
    if (G) G[(int64_t)s * st_seg_stride] = run;
    run = fmaf(run, expf(D[(int64_t)s * ld_seg_stride]), f);
  }
  if (out_single) out_single[unit * np + e] = run;
  if (out_final) out_final[unit * np + e] = run;
  if (out_ld && e == 0) {
    double tot = 0.0;
    for (int s = 0; s < upto; ++s) tot += (double)D[(int64_t)s * ld_seg_stride];
    out_ld[unit] = (float)tot;
  }
}

size_t smem_bytes(int tile, int p, int n) { return sizeof(float) * (size_t)(2 * tile * p + 2 * tile * n + 2 * tile); }

// Tokens per step.  A step costs a round trip to memory and three barriers whatever its length, which other CTAs of the SM
// cover where there are some: so the longest step (up to 128 tokens) that still leaves room for as many CTAs as an SM
// gets, or for four.
int tile_tokens(const ScanParams& prm, int p) {
  const int64_t ctas = (int64_t)prm.batch * prm.nheads * prm.nseg;
  const int64_t per_sm = std::min<int64_t>(4, (ctas + 147) / 148);
  int tile = kTile;
  while (tile < 128 && tile < prm.seg_len && per_sm * (smem_bytes(2 * tile, p, prm.n) + 1024) <= 227 * 1024) tile *= 2;
  return tile;
}

template <typename T, int NS, int P>
int launch_one(const ScanParams& prm, cudaStream_t stream) {
  const int tile = tile_tokens(prm, P);
  const size_t smem = smem_bytes(tile, P, prm.n);
  // Tokens in line hide what links one to the next, but their registers leave an SM two CTAs (16-bit inputs, whose staging takes
  // them too, and any with 32 rows a thread).  Where more CTAs than that are waiting, they hide it as well:
  //  - fewer tokens than go in line: one after the other, in registers for one CTA more than the 64 or 80 that this takes leave
  //    room for where there are as many (bf16, 5120 sequences of one token, n 64: 43 us with the registers of the others, 22 so);
  //  - fp32 with 32 rows a thread, up to four CTAs per SM: one after the other (384 sequences of 200 tokens, n 128: 230 us in
  //    line, 178 so);
  //  - 16-bit, up to 16 rows a thread: in line in registers for four CTAs (444 sequences of 200 tokens, n 32: 88 us with two, 67
  //    so); 32 rows a thread and few tokens: for three.
  constexpr int SL = kThreads / P, kLine = NS >= 16 && SL <= 4 ? 4 : 8;   // (at least SL; fewer where the state fills the registers)
  constexpr bool k16 = sizeof(T) == 2;
  constexpr int kMany = !k16 ? 0 : NS >= 32 ? 3 : 4, kMost = !k16 || NS == 4 ? 0 : (NS >= 32 ? 4 : 5) - (P == 128 ? 1 : 0);
  const int64_t ctas = (int64_t)prm.batch * prm.nheads * prm.nseg;
  const int tokens = std::min(prm.seqlen, prm.seg_len);
  const bool many = ctas > 2 * 148, full = prm.n == NS * SL;
  auto kern = full ? ssd_scan_f32_kernel<T, NS, P, true, kLine, 0, false> : ssd_scan_f32_kernel<T, NS, P, false, kLine, 0, false>;
  if (k16 && full && tokens < kLine && ctas > kMany * 148)
    kern = ssd_scan_f32_kernel<T, NS, P, true, 1, kMost, false>;
  else if (tokens < kLine || (!k16 && NS == 32 && many && ctas <= 4 * 148))
    kern = full ? ssd_scan_f32_kernel<T, NS, P, true, 1, 0, false> : ssd_scan_f32_kernel<T, NS, P, false, 1, 0, false>;
  else if (k16 && many && (NS <= 16 || tokens < 16))
    kern = full ? ssd_scan_f32_kernel<T, NS, P, true, kLine, kMany, false> : ssd_scan_f32_kernel<T, NS, P, false, kLine, kMany, false>;
  bool early = false;
  if constexpr (k16 && P == 64 && NS >= 16) {
    if (prm.redo) {
      if (!full || tokens < kLine) return SSD_ERR_UNSUPPORTED;
      kern = many && (NS <= 16 || tokens < 16) ? ssd_scan_f32_kernel<T, NS, P, true, kLine, kMany, true>
                                               : ssd_scan_f32_kernel<T, NS, P, true, kLine, 0, true>;
      early = true;
    }
  }
  if (prm.redo && !early) return SSD_ERR_UNSUPPORTED;
  if (smem > 48 * 1024) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return SSD_ERR_CUDA;
  }
  // (As many CTAs as the chip holds: one for each of 5 120 heads that only look whether there is work take 20 us, these 1.)
  if (early) return launch_early(kern, (unsigned)std::min<int64_t>(ctas, 4 * 148), kThreads, smem, stream, prm, tile);
  dim3 grid((unsigned)(prm.batch * prm.nheads), (unsigned)prm.nseg);
  return launch(kern, grid, kThreads, smem, stream, prm, tile);
}

template <typename T, int P>
int launch_p(const ScanParams& prm, cudaStream_t stream) {
  constexpr int SL = kThreads / P;
  const int per_thread = prm.n / SL;
  if (per_thread <= 4) return launch_one<T, 4, P>(prm, stream);
  if (per_thread <= 16) return launch_one<T, 16, P>(prm, stream);
  return launch_one<T, 32, P>(prm, stream);
}

template <typename T>
int launch_t(const ScanParams& prm, cudaStream_t stream) {
  switch (prm.p) {
    case 32: return launch_p<T, 32>(prm, stream);
    case 64: return launch_p<T, 64>(prm, stream);
    case 128: return launch_p<T, 128>(prm, stream);
    default: return SSD_ERR_UNSUPPORTED;
  }
}

}  // namespace

bool scan_f32_supports(int p, int n) {
  if (p != 32 && p != 64 && p != 128) return false;
  const int sl = kThreads / p;
  return n > 0 && n % (4 * sl) == 0 && n / sl <= 32;
}

int scan_f32_tile_tokens() { return kTile; }

int launch_scan_f32(const ScanParams& prm, int dtype, cudaStream_t stream, bool in_line) {
  if (!scan_f32_supports(prm.p, prm.n)) return SSD_ERR_UNSUPPORTED;
  // fp32 tensors, unless the caller asks for this kernel by name: tokens side by side, where that is faster
  if (!in_line && dtype == SSD_DTYPE_F32 && chunk_f32_takes(prm) && chunk_f32_pays(prm)) return launch_chunk_f32(prm, stream);
  switch (dtype) {
    case SSD_DTYPE_F32: return launch_t<float>(prm, stream);
    case SSD_DTYPE_F16: return launch_t<__half>(prm, stream);
    case SSD_DTYPE_BF16: return launch_t<__nv_bfloat16>(prm, stream);
    default: return SSD_ERR_UNSUPPORTED;
  }
}

// ---------------------------------------------------------------------------------------------
// Skip and gate of SSDLayer.forward after the core (model_ref.py:116-118), for the kernels that do
// not fuse it:  Y <- (Y + x * D[head]) * silu(z), fp32 arithmetic, one rounding.  One thread per
// 8 consecutive head-dim elements (16 bytes of a 16-bit row; rows are 16-byte aligned when vec_ok),
// one block per token.
template <typename T>
__global__ void __launch_bounds__(256)
ssd_epilogue_kernel(const ScanParams p) {
  // one block per token row (b, t); its threads walk the row's (head, 8-element vector) pairs: 32-bit index math only
  const int vec = p.p / 8;
  const int b = blockIdx.x / p.seqlen, t = blockIdx.x - b * p.seqlen;
  for (int i = threadIdx.x; i < p.nheads * vec; i += blockDim.x) {
    const int hh = i / vec, v = i - hh * vec;
    T* y = static_cast<T*>(p.Y) + b * p.ys[0] + (int64_t)t * p.ys[1] + hh * p.ys[2] + 8 * v;
    const T* x = static_cast<const T*>(p.X) + b * p.xs[0] + (int64_t)t * p.xs[1] + hh * p.xs[2] + 8 * v;
    const T* z = p.Z ? static_cast<const T*>(p.Z) + b * p.zs[0] + (int64_t)t * p.zs[1] + hh * p.zs[2] + 8 * v : nullptr;
    const float d = p.D ? load_skip<T>(p, hh) : 0.f;
    // eight elements per thread, moved as whole 16-byte (32-byte for fp32) vectors when the rows allow it
    T yv[8], xv[8], zv[8];
    constexpr int kVecs = sizeof(T) * 8 / 16;
    if (p.vec_ok) {
#pragma unroll
      for (int k = 0; k < kVecs; ++k) {
        reinterpret_cast<uint4*>(yv)[k] = reinterpret_cast<const uint4*>(y)[k];
        if (p.D) reinterpret_cast<uint4*>(xv)[k] = reinterpret_cast<const uint4*>(x)[k];
        if (z) reinterpret_cast<uint4*>(zv)[k] = reinterpret_cast<const uint4*>(z)[k];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        yv[e] = y[e];
        if (p.D) xv[e] = x[e];
        if (z) zv[e] = z[e];
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float acc = Cvt<T>::to_f(yv[e]);
      if (p.D) acc = fmaf(Cvt<T>::to_f(xv[e]), d, acc);
      if (z) {
        const float zz = Cvt<T>::to_f(zv[e]);
        acc *= zz / (1.f + __expf(-zz));
      }
      yv[e] = Cvt<T>::from_f(acc);
    }
    if (p.vec_ok) {
#pragma unroll
      for (int k = 0; k < kVecs; ++k) reinterpret_cast<uint4*>(y)[k] = reinterpret_cast<const uint4*>(yv)[k];
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = yv[e];
    }
  }
}

int launch_epilogue(const ScanParams& p, int dtype, cudaStream_t stream) {
  if (!p.D && !p.Z) return SSD_OK;
  if (p.p % 8 != 0) return SSD_ERR_UNSUPPORTED;
  const int64_t rows = (int64_t)p.batch * p.seqlen;
  if (rows > 0x7fffffffLL) return SSD_ERR_TOO_LARGE;
  const int grid = (int)rows;
  const int work = p.nheads * (p.p / 8);
  const int threads = work >= 256 ? 256 : (work >= 128 ? 128 : 64);
  if (dtype == SSD_DTYPE_F32) return launch(ssd_epilogue_kernel<float>, grid, threads, 0, stream, p);
  if (dtype == SSD_DTYPE_F16) return launch(ssd_epilogue_kernel<__half>, grid, threads, 0, stream, p);
  return launch(ssd_epilogue_kernel<__nv_bfloat16>, grid, threads, 0, stream, p);
}

int launch_fold(const float* states, int64_t st_unit_stride, int64_t st_seg_stride, const float* ld,
                int64_t ld_unit_stride, int64_t ld_seg_stride, const float* init, float* out_single,
                float* out_final, float* out_ld, int upto, float* incoming, int64_t units, int64_t np,
                cudaStream_t stream) {
  if (units <= 0 || np <= 0) return SSD_ERR_BAD_SHAPE;
  if (units > 0x7fffffff || (np + 255) / 256 > 65535) return SSD_ERR_TOO_LARGE;
  dim3 grid((unsigned)units, (unsigned)((np + 255) / 256));
  return launch(ssd_fold_kernel, grid, 256, 0, stream, states, st_unit_stride, st_seg_stride, ld, ld_unit_stride, ld_seg_stride,
                init, out_single, out_final, out_ld, upto, incoming, np);
}

}  // namespace ssd
