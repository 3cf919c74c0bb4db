// fp32 SSD forward in chunked form (model_ref.py:135-162) on the CUDA cores: the tokens of a sequence side by side instead of one
// after the other as in ssd_scan_f32.cu.
//
// A tile of tokens is cut into pieces of 16, a warp or two for each.  With E_t the product of the decays from the piece's first token
// to t, and B^_s = B_s dt_s / E_s, a piece is plain products of small matrices:
//   F = sum_s B^_s (x) x_s             what it adds to the state, in units of E at its end
//   H <- E_end (H + F)                 from piece to piece (the only serial part: one step per piece)
//   Y_t = E_t (C_t . H + sum_{s <= t} (C_t . B^_s) x_s)
// What bounds it: the reads of shared memory, whose 128 bytes a cycle are words that arrive in registers, so that a word that all lanes
// read costs as much as one each.  Hence the register tiles of 8 x 4: a word serves 2.7 multiply-adds (in the recurrence one, and each
// token waits for the one before).  16 x 8 heads of 128 tokens, n 16, on 128 SMs: 9.9 -> 7.1 us (1 000 cycles to begin, 1 500 for the
// tile to arrive, 2 000 F, 750 G, 650 for the pieces' states, 1 600 and 2 100 the two sums of Y, 900 its stores); n 64 27.2 -> 17.7,
// n 128 and 64 heads 40.4 -> 28.8; 4 096 heads, n 128, 1 058 -> 827.  Two pieces a warp with tiles of 8 x 8 (four multiply-adds a word) were
// slower for want of warps (7.8).
// Against 64 bits (relative error of Y, recurrence in brackets): log-decays N(0, 1) 1.8e-7 (8.9e-7), of a Mamba layer 1.2e-7 (1.4e-7).
//
// E and its inverse stay near one only while the decays of a piece do.  A tile with a piece in which log-decays sum to less than -40 or more
// than 20 (decays of some nats a token, a reset between packed documents) is taken by the decays between its tokens instead, D(s, t) being
// those after s up to t, as good as one exponential too (resets are counted, not summed: -inf would take the sums behind it with it):
//   F = sum_s D(s, end) dt_s B_s (x) x_s,   H <- E_end H + F,   Y_t = E_t (C_t . H) + sum_{s <= t} D(s, t) (C_t . dt_s B_s) x_s
// 16 x 8 heads of 128 tokens, n 16, with decays of 3 nats a token or a reset 8.4 us (the recurrence 10.2), 2 048 heads, n 64, 272 and 258
// (290), 4 x 1 024 tokens of 32 heads, n 128, 388 and 371 (466); token by token, as such tiles first were, 30, 808 and 526, 1 379 and 989.
// A tile that comes out with a number that is not finite (an overflow of the scaled numbers, a NaN or an infinity that belongs to other
// tokens) is done again token by token, before any of it is written, and those behind it at once while the state is not finite
// (17, 494 and 577 us where that is so from the beginning).
#include <type_traits>

#include "chunk_f32.cuh"

namespace ssd {
namespace {

constexpr int kP = 64;      // head dim
constexpr int kQ = 16;      // tokens of a piece
constexpr float kLeast = -40.f, kMost = 20.f;
constexpr float kReset = -104.f;   // e^-104 = 2^-150: a factor of zero

// NP pieces a tile, WPP warps for each.
template <int N, int NP, int WPP>
struct ChunkLayout {
  static constexpr int kThreads = 32 * NP * WPP, kTokens = kQ * NP;
  static constexpr int kStride = N + 4;            // of B and C: rows that lanes read at once start in different banks
  static constexpr int oX = 0;                     // [token][64]
  static constexpr int oB = oX + kTokens * kP;     // [token][kStride]
  static constexpr int oC = oB + kTokens * kStride;
  static constexpr int oF = oC + kTokens * kStride;      // [piece][n][64]: F, then the state entering the piece
  static constexpr int oG = oF + NP * N * kP;            // [piece][s][t]: C_t . B^_s, t so that a thread's are side by side
  static constexpr int oE = oG + NP * kQ * kQ;           // [token]
  static constexpr int oSum = oE + kTokens;              // [token]: sum of log-decays, what rounding leaves of it, resets
  static constexpr int oOdd = oSum + 3 * kTokens;        // [piece]
  static constexpr int kBytes = (oOdd + NP) * 4;
  static_assert(kBytes <= 227 * 1024, "shared memory of one SM exceeded");
};

// d += f * v
__device__ __forceinline__ void axpy(float (&d)[4], float f, float4 v) {
  d[0] = fmaf(f, v.x, d[0]); d[1] = fmaf(f, v.y, d[1]); d[2] = fmaf(f, v.z, d[2]); d[3] = fmaf(f, v.w, d[3]);
}
__device__ __forceinline__ float dot(float4 a, float4 b) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x))); }
// Sums of 16 neighbouring lanes' numbers up to each lane, with what rounding leaves (Knuth's sum of two), so that their exponential is as
// good as one of a single number.
__device__ __forceinline__ void prefix(float& sum, float& rest, int lane) {
#pragma unroll
  for (int d = 1; d < kQ; d <<= 1) {
    const float ps = __shfl_up_sync(0xffffffffu, sum, d, kQ), pr = __shfl_up_sync(0xffffffffu, rest, d, kQ);
    if ((lane & 15) >= d) {
      const float s = sum + ps, b = s - sum;
      rest += pr + ((sum - (s - b)) + (ps - b));
      sum = s;
    }
  }
}
__device__ __forceinline__ float exp_of(float sum, float rest) {
  const float e = expf(sum);
  return fmaf(e, rest, e);
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }

template <int N, int NP, int WPP>
__global__ void __launch_bounds__(32 * NP * WPP) ssd_chunk_f32_kernel(const ScanParams prm) {
  using L = ChunkLayout<N, NP, WPP>;
  constexpr int kThreads = L::kThreads, S = L::kStride, kHeld = N * kP / 4 / kThreads;
  constexpr int kTok = 8 / WPP, kTG = kQ / kTok, kCG = 32 / kTG;   // of Y a thread has kTok tokens (tg, tg + kTG, ...) x 4 columns
  static_assert(kHeld * 4 * kThreads == N * kP && 4 * kCG * WPP == kP, "tiles");
  extern __shared__ __align__(16) float smem[];
  float *Xs = smem + L::oX, *Bs = smem + L::oB, *Cs = smem + L::oC, *Fs = smem + L::oF, *Es = smem + L::oE;
  const int tid = threadIdx.x, lane = tid & 31;
  const int piece = tid / (32 * WPP), part = (tid >> 5) % WPP;
  const int hi = blockIdx.x, bi = blockIdx.y, seg = blockIdx.z, gi = hi / (prm.nheads / prm.ngroups);
  const int64_t unit = (int64_t)bi * prm.nheads + hi;
  const int t_begin = seg * prm.seg_len, t_end = min(prm.seqlen, t_begin + prm.seg_len);
  const float* Xg = static_cast<const float*>(prm.X) + bi * prm.xs[0] + hi * prm.xs[2];
  const float* Bg = static_cast<const float*>(prm.B) + bi * prm.bs[0] + gi * prm.bs[2];
  const float* Cg = static_cast<const float*>(prm.C) + bi * prm.cs[0] + gi * prm.cs[2];
  const float* Ag = prm.A + bi * prm.as[0] + hi * prm.as[2];
  const float* Dg = prm.dt ? static_cast<const float*>(prm.dt) + bi * prm.dts[0] + hi * prm.dts[2] : nullptr;
  const bool want_y = prm.compute_y != 0;

  // `rows` rows of 4 * PER columns, the rest of the tile's last piece as zeros
  auto fetch = [&](float* dst, int stride, const float* src, int64_t step, int rows, int padded, auto per) {
    constexpr int PER = decltype(per)::value, kRows = kThreads / PER;
    static_assert(kThreads % PER == 0, "");
    const int r0 = tid / PER, c = tid % PER * 4;
    const float* p = src + r0 * step + c;
    uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + r0 * stride + c);
#pragma unroll 4
    for (int r = r0; r < padded; r += kRows, p += kRows * step, d += kRows * stride * 4)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(r < rows ? p : src), "r"(r < rows ? 16 : 0) : "memory");
  };

  // the state, between tiles: vector tid + i * kThreads of its rows
  float4 held[kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i) held[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (prm.init) {
    const float4* I = reinterpret_cast<const float4*>(prm.init + unit * prm.init_unit_stride + seg * prm.init_seg_stride);
#pragma unroll
    for (int i = 0; i < kHeld; ++i) held[i] = I[tid + i * kThreads];
  }
  double asum = 0.0;
  bool in_line = false;   // the state is not finite

#pragma unroll 1
  for (int t0 = t_begin; t0 < t_end; t0 += L::kTokens) {
    const int rows = min(L::kTokens, t_end - t0);
    const int pieces = (rows + kQ - 1) / kQ, padded = pieces * kQ;
    if (t0 > t_begin) __syncthreads();   // (the tile before is done with shared memory)
    // past the end: decay 1 and B = 0, the state stays as it is
    const int own = piece * kQ + (lane & 15);
    const float a = own < rows ? Ag[(int64_t)(t0 + own) * prm.as[1]] : 0.f;
    const float dt = Dg && own < rows ? Dg[(int64_t)(t0 + own) * prm.dts[1]] : 1.f;
    fetch(Bs, S, Bg + (int64_t)t0 * prm.bs[1], prm.bs[1], rows, padded, std::integral_constant<int, N / 4>{});
    fetch(Xs, kP, Xg + (int64_t)t0 * prm.xs[1], prm.xs[1], rows, padded, std::integral_constant<int, kP / 4>{});
    if (want_y) fetch(Cs, S, Cg + (int64_t)t0 * prm.cs[1], prm.cs[1], rows, padded, std::integral_constant<int, N / 4>{});
    // E of the piece's tokens, in lanes 0 .. 15 (the others do the same)
    float sum = a, rest = 0.f;
    prefix(sum, rest, lane);
    const float back = expf(-sum);
    const bool strong = !(sum > kLeast && sum < kMost);   // (NaN too)
    if (part == 0 && lane < kQ) Es[own] = exp_of(sum, rest);
    const bool odd = __any_sync(0xffffffffu, strong || in_line);
    if (part == 0 && lane == 0) smem[L::oOdd + piece] = odd ? 1.f : 0.f;
    __syncthreads();   // (under the loads; a vote takes 1 % more)
    float odds = 0.f;
#pragma unroll
    for (int k = 0; k < NP; k += 4) odds += dot(ld4(smem + L::oOdd + k), make_float4(1.f, 1.f, 1.f, 1.f));
    const bool by_pairs = odds != 0.f;

    const int tg = lane / kCG, col = part * (kP / WPP) + 4 * (lane % kCG);   // of Y
    const float* Xp = Xs + piece * kQ * kP;
    const float* Cp = Cs + piece * kQ * S;
    float* Bp = Bs + piece * kQ * S;
    float* Fp = Fs + piece * N * kP;
    float* Gp = smem + L::oG + piece * kQ * kQ;
    float4 start[kHeld];
    float y[kTok][4] = {};
    bool again = false;
    auto tile = [&](auto pairs) {
      constexpr bool kPairs = decltype(pairs)::value;
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      float w = dt * fmaf(-back, rest, back), to_end = 1.f;
      float *Sum = smem + L::oSum + piece * kQ, *Rest = Sum + L::kTokens, *Resets = Rest + L::kTokens;
      auto between = [&](int s, int t) {
        const float d = Sum[t] - Sum[s], b = d - Sum[t];
        return Resets[s] == Resets[t] ? exp_of(d, (Rest[t] - Rest[s]) + ((Sum[t] - (d - b)) - (Sum[s] + b))) : 0.f;
      };
      if constexpr (kPairs) {
        w = dt;
        const uint32_t upto = (2u << (lane & 15)) - 1, resets = __ballot_sync(0xffffffffu, a < kReset) & upto;
        float sm = a < kReset ? 0.f : a, rs = 0.f;
        prefix(sm, rs, lane);
        __syncwarp();
        if (lane < kQ && part == 0) {
          Sum[lane] = sm;
          Rest[lane] = rs;
          Resets[lane] = (float)__popc(resets);
          Es[own] = resets ? 0.f : exp_of(sm, rs);
        }
        if (WPP > 1) __syncthreads();
        else __syncwarp();
        to_end = between(lane & 15, kQ - 1);
      }
      {
        // B^, in place (warps without tokens have nothing that is read)
        constexpr int kRows = kQ / WPP;
#pragma unroll
        for (int i = 0; i < kRows * N / 4 / 32; ++i) {
          const int v = lane + 32 * i, r = part * kRows + v / (N / 4);
          const float s = __shfl_sync(0xffffffffu, w, r, 16);
          if (piece < pieces) {
            float* b = Bp + r * S + v % (N / 4) * 4;
            const float4 o = ld4(b);
            st4(b, o.x * s, o.y * s, o.z * s, o.w * s);
          }
        }
      }
      if (WPP > 1) __syncthreads();
      else __syncwarp();
      if (piece < pieces) {
        // F: 8 rows x 4 columns a thread
        const int fg = lane >> 4, fc = 4 * (lane & 15);
#pragma unroll 1
        for (int nb = part * (N / WPP); nb < (part + 1) * (N / WPP); nb += 16) {
          float f[8][4] = {};
          const float* b = Bp + nb + 8 * fg;
#pragma unroll 4
          for (int s = 0; s < kQ; ++s) {
            const float4 b0 = ld4(b + s * S), b1 = ld4(b + s * S + 4);
            float4 x = ld4(Xp + s * kP + fc);
            if constexpr (kPairs) {
              const float d = __shfl_sync(0xffffffffu, to_end, s);
              x = make_float4(x.x * d, x.y * d, x.z * d, x.w * d);
            }
            axpy(f[0], b0.x, x); axpy(f[1], b0.y, x); axpy(f[2], b0.z, x); axpy(f[3], b0.w, x);
            axpy(f[4], b1.x, x); axpy(f[5], b1.y, x); axpy(f[6], b1.z, x); axpy(f[7], b1.w, x);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) st4(Fp + (nb + 8 * fg + i) * kP + fc, f[i][0], f[i][1], f[i][2], f[i][3]);
        }
        if (want_y) {
          // G, of the warp's share of the piece's tokens: t = gt + kGT i, s = gs + kGS j
          constexpr int kGS = 8, kJ = kQ / kGS, kGT = 32 / kGS, kI = kQ / WPP / kGT;
          const int gt = lane / kGS + part * (kQ / WPP), gs = lane % kGS;
          float g[kI][kJ] = {};
#pragma unroll 4
          for (int n = 0; n < N; n += 4) {
            float4 b[kJ];
#pragma unroll
            for (int j = 0; j < kJ; ++j) b[j] = ld4(Bp + (gs + kGS * j) * S + n);
#pragma unroll
            for (int i = 0; i < kI; ++i) {
              const float4 c = ld4(Cp + (gt + kGT * i) * S + n);
#pragma unroll
              for (int j = 0; j < kJ; ++j) g[i][j] += dot(c, b[j]);
            }
          }
#pragma unroll
          for (int i = 0; i < kI; ++i)
#pragma unroll
            for (int j = 0; j < kJ; ++j) {
              const int t = gt + kGT * i, s = gs + kGS * j;
              if (kPairs && s <= t) g[i][j] *= between(s, t);
              Gp[s * kQ + t % kTG * kTok + t / kTG] = s <= t ? g[i][j] : 0.f;
            }
        }
      }
      __syncthreads();
      // the state entering each piece
#pragma unroll
      for (int i = 0; i < kHeld; ++i) {
        float4 run = start[i] = held[i];
        float* f = Fs + 4 * (tid + i * kThreads);
        float4 v[NP];
        float end[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
          v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
          end[k] = 1.f;
          if (k < pieces) {
            v[k] = ld4(f + k * (N * kP));
            end[k] = Es[k * kQ + kQ - 1];
          }
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) {
          *reinterpret_cast<float4*>(f + k * (N * kP)) = run;
          if constexpr (kPairs)
            run = make_float4(fmaf(end[k], run.x, v[k].x), fmaf(end[k], run.y, v[k].y), fmaf(end[k], run.z, v[k].z), fmaf(end[k], run.w, v[k].w));
          else
            run = make_float4(end[k] * (run.x + v[k].x), end[k] * (run.y + v[k].y), end[k] * (run.z + v[k].z), end[k] * (run.w + v[k].w));
        }
        held[i] = run;
        again = again || !(fabsf(run.x) + fabsf(run.y) + fabsf(run.z) + fabsf(run.w) < INFINITY);
      }
      if (want_y && piece < pieces) {
#pragma unroll 4
        for (int s = 0; s < kQ; ++s) {
          const float4 x = ld4(Xp + s * kP + col);
#pragma unroll
          for (int i = 0; i < kTok; i += 4) {
            const float4 g = ld4(Gp + s * kQ + tg * kTok + i);
            axpy(y[i], g.x, x); axpy(y[i + 1], g.y, x); axpy(y[i + 2], g.z, x); axpy(y[i + 3], g.w, x);
          }
        }
      }
      __syncthreads();
      if (want_y && piece < pieces) {
#pragma unroll 1
        for (int n = 0; n < N; n += 8) {
          float4 h[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) h[r] = ld4(Fp + (n + r) * kP + col);
#pragma unroll
          for (int i = 0; i < kTok; ++i) {
            const float* c = Cp + (tg + kTG * i) * S + n;
            const float4 c0 = ld4(c), c1 = ld4(c + 4);
            // (eight products at a time: a sum over n is then as short as the recurrence's)
            float p[4] = {c0.x * h[0].x, c0.x * h[0].y, c0.x * h[0].z, c0.x * h[0].w};
            axpy(p, c0.y, h[1]); axpy(p, c0.z, h[2]); axpy(p, c0.w, h[3]);
            axpy(p, c1.x, h[4]); axpy(p, c1.y, h[5]); axpy(p, c1.z, h[6]); axpy(p, c1.w, h[7]);
            const float et = kPairs ? Es[piece * kQ + tg + kTG * i] : 1.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) y[i][e] = kPairs ? fmaf(et, p[e], y[i][e]) : y[i][e] + p[e];
          }
        }
#pragma unroll
        for (int i = 0; i < kTok; ++i) {
          const float et = kPairs ? 1.f : Es[piece * kQ + tg + kTG * i];
          float all = 0.f;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            y[i][c] *= et;
            all += fabsf(y[i][c]);
          }
          again = again || !(all < INFINITY);
        }
      }
    };
    if (__builtin_expect(!by_pairs, 1)) {
      tile(std::false_type{});
    } else if (!in_line) {
      tile(std::true_type{});
    } else {
      again = true;
      asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
      for (int i = 0; i < kHeld; ++i) start[i] = held[i];
    }
    float* Yg = prm.Y ? static_cast<float*>(prm.Y) + bi * prm.ys[0] + hi * prm.ys[2] + t0 * prm.ys[1] : nullptr;
    if (__builtin_expect(!__syncthreads_or(again), 1)) {
      if (want_y) {
        float* p = Yg + (piece * kQ + tg) * prm.ys[1] + col;
#pragma unroll
        for (int i = 0; i < kTok; ++i, p += kTG * prm.ys[1]) {
          if (piece * kQ + tg + kTG * i < rows) st4(p, y[i][0], y[i][1], y[i][2], y[i][3]);
        }
      }
    } else {
      // token by token, some of them in line: thread (j, sl) has column j and the rows 16 i + 4 sl .. 16 i + 4 sl + 3
      constexpr int kGroup = kThreads / kP, kMine = N / kGroup, kLine = N <= 32 ? 8 : 4;
      static_assert(kGroup == 4 && 2 * L::kTokens <= NP * kQ * kQ && kQ % kLine == 0, "");
      const int j = tid / kGroup, sl = tid % kGroup;
      float *H = Fs, *decay = smem + L::oG, *step = decay + L::kTokens;
#pragma unroll
      for (int i = 0; i < kHeld; ++i) reinterpret_cast<float4*>(H)[tid + i * kThreads] = start[i];
      if (!in_line)
        for (int i = tid; i < rows * N; i += kThreads) Bs[i / N * S + i % N] = Bg[(int64_t)(t0 + i / N) * prm.bs[1] + i % N];
      for (int i = tid; i < padded; i += kThreads) {   // (past the end: nothing is added)
        decay[i] = i < rows ? expf(Ag[(int64_t)(t0 + i) * prm.as[1]]) : 1.f;
        step[i] = Dg && i < rows ? Dg[(int64_t)(t0 + i) * prm.dts[1]] : 1.f;
      }
      if (!in_line)
        for (int i = rows * N + tid; i < padded * N; i += kThreads) Bs[i / N * S + i % N] = 0.f;
      __syncthreads();
      float h[kMine];
#pragma unroll
      for (int i = 0; i < kMine; ++i) h[i] = H[(i / 4 * 16 + 4 * sl + i % 4) * kP + j];
#pragma unroll 1
      for (int t = 0; t < padded; t += kLine) {
        float s[kLine];
#pragma unroll
        for (int k = 0; k < kLine; ++k) {
          const float x = Xs[(t + k) * kP + j] * step[t + k], d = decay[t + k];
          const float *b = Bs + (t + k) * S + 4 * sl, *c = Cs + (t + k) * S + 4 * sl;
          s[k] = 0.f;
#pragma unroll
          for (int i = 0; i < kMine; i += 4) {
            const float4 bv = ld4(b + 4 * i);
            h[i] = fmaf(h[i], d, bv.x * x); h[i + 1] = fmaf(h[i + 1], d, bv.y * x);
            h[i + 2] = fmaf(h[i + 2], d, bv.z * x); h[i + 3] = fmaf(h[i + 3], d, bv.w * x);
            if (want_y) {
              const float4 cv = ld4(c + 4 * i);
              s[k] = fmaf(cv.w, h[i + 3], fmaf(cv.z, h[i + 2], fmaf(cv.y, h[i + 1], fmaf(cv.x, h[i], s[k]))));
            }
          }
        }
#pragma unroll
        for (int k = 0; k < kLine; ++k) {
          s[k] += __shfl_xor_sync(0xffffffffu, s[k], 1);
          s[k] += __shfl_xor_sync(0xffffffffu, s[k], 2);
        }
#pragma unroll
        for (int k = 0; k < kLine; ++k)
          if (want_y && sl == 0 && t + k < rows) Yg[(t + k) * prm.ys[1] + j] = s[k];
      }
      __syncthreads();
      in_line = false;
#pragma unroll
      for (int i = 0; i < kMine; ++i) {
        H[(i / 4 * 16 + 4 * sl + i % 4) * kP + j] = h[i];
        in_line = in_line || !(fabsf(h[i]) < INFINITY);
      }
      in_line = __syncthreads_or(in_line);
#pragma unroll
      for (int i = 0; i < kHeld; ++i) held[i] = reinterpret_cast<float4*>(H)[tid + i * kThreads];
    }
    if (prm.fin_ld && tid < 32) {
      double s = 0.0;
      for (int r = lane; r < rows; r += 32) s += (double)Ag[(int64_t)(t0 + r) * prm.as[1]];
      for (int d = 16; d >= 1; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      asum += s;
    }
  }
  if (prm.fin) {
    float4* F = reinterpret_cast<float4*>(prm.fin + unit * prm.fin_unit_stride + seg * prm.fin_seg_stride);
#pragma unroll
    for (int i = 0; i < kHeld; ++i) F[tid + i * kThreads] = held[i];
  }
  if (prm.fin_ld && tid == 0) prm.fin_ld[unit * prm.finld_unit_stride + seg * prm.finld_seg_stride] = (float)asum;
}

template <int N, int NP, int WPP>
int launch_chunk(const ScanParams& prm, cudaStream_t stream) {
  using L = ChunkLayout<N, NP, WPP>;
  auto kern = ssd_chunk_f32_kernel<N, NP, WPP>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes) != cudaSuccess) return SSD_ERR_CUDA;
  dim3 grid((unsigned)prm.nheads, (unsigned)prm.batch, (unsigned)prm.nseg);
  return launch(kern, grid, L::kThreads, L::kBytes, stream, prm);
}

}  // namespace

bool chunk_f32_takes(const ScanParams& prm) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return prm.p == kP && (prm.n == 16 || prm.n == 32 || prm.n == 64 || prm.n == 128) && prm.vec_ok && al(prm.init) && al(prm.fin) && prm.batch <= 65535;
}

// A tile costs much the same whatever is in it, so what counts is what is left for the last one.  Times of 3 984 heads in microseconds (start,
// tile, 16 tokens of a tile; start, 64 tokens one after the other): n 32: 65, 80, 112 and 129 tokens 221, 225, 241 and 388, the recurrence 166,
// 194, 262 and 303; n 64: 64, 65, 96 and 129 245, 375, 393 and 594, there 279, 293, 405 and 545; n 128: 32, 34, 48 and 65 279, 369, 372 and 619,
// there 282, 305, 409 and 543.  With up to eight heads an SM the recurrence is a tenth slower than that (not with n 128), with up to one 1.4
// times (n 128: a tenth).
bool chunk_f32_pays(const ScanParams& prm) {
  struct Cost { int tokens, start, tile, piece, start_in_line, in_line; };
  const Cost c = prm.n == 16 ? Cost{128, 2, 60, 7, 8, 83} : prm.n == 32 ? Cost{128, 20, 115, 15, 11, 144} : prm.n == 64 ? Cost{64, 20, 100, 30, 12, 262}
                                                                                                            : Cost{64, 30, 160, 55, 25, 500};
  const int64_t tokens = prm.seqlen < prm.seg_len ? prm.seqlen : prm.seg_len, ctas = (int64_t)prm.batch * prm.nheads * prm.nseg;
  if (tokens < (prm.n == 128 ? 32 : 64)) return false;
  const int64_t side_by_side = c.start + (tokens + c.tokens - 1) / c.tokens * c.tile + (tokens + kQ - 1) / kQ * c.piece;
  const int64_t in_line = c.start_in_line + tokens * c.in_line / 64;
  const int percent = ctas <= 148 ? (prm.n == 128 ? 110 : 140) : ctas <= 8 * 148 && prm.n != 128 ? 110 : 100;
  return 100 * side_by_side <= percent * in_line;
}

int launch_chunk_f32(const ScanParams& prm, cudaStream_t stream) {
  switch (prm.n) {
    case 16: return launch_chunk<16, 8, 1>(prm, stream);
    case 32: return launch_chunk<32, 8, 1>(prm, stream);
    case 64: return launch_chunk<64, 4, 2>(prm, stream);
    case 128: return launch_chunk<128, 4, 2>(prm, stream);
    default: return SSD_ERR_UNSUPPORTED;
  }
}

}  // namespace ssd
