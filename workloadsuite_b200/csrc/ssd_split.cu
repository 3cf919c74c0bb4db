// Tensor-core SSD forward at fp32 precision for 16-bit tensors, one head at a time: what lengths that are no whole tiles are
// given, whose results are rounded once.  The fp32 recurrence (ssd_scan_f32.cu) computes the same numbers token by token.
//
// Of each product one operand is a caller's tensor, exact in 16 bits; the other (the masked products P, the decayed X, the
// state) is an fp32 number, taken as the sum of 16-bit ones (split below): three bf16 numbers, which hold it exactly, or two
// fp16 numbers, which are off by up to 2^-23 of it (fp32 by 2^-24).  Those of Xd and of the state are in units from the largest of
// the tile, those of P in units of the tile's largest step, so that P below 2^-13 is off by up to 2^-36 instead; Y, which is all
// that comes of P, is rounded to 2^-11 of it or 2^-25.  So P.X is three (two) products with X, and S = B^T.Xd and C.H take the
// pieces side by side as columns; all products are exact, the sums fp32, the state is carried in fp32 registers, and Y is
// rounded once.  Log-decays are summed from the place they count from (the end of the tile for the
// state's weights, the borders of 32-token blocks for P's, and see kStrong), so a weight's error is that of its own exponent,
// however much has decayed before.  Against 64 bits (2 x 3001 tokens, 80 heads, n 128, bf16): Y 1.66e-3, its own rounding,
// here and in the recurrence; final state 8.4e-8 here, 1.29e-7 there.
//
// What cannot be done this way is left to the recurrence: a CTA that meets a number that is not finite (0 * inf in a masked
// place would reach tokens before its own; an fp16 piece overflows at 65 504) or a log-decay above zero that a tile's factors
// may not carry says so in `redo`, and the recurrence, launched behind this kernel, does the call again; otherwise that
// launch ends at once (and sums the log-decays over the sequence where the caller wants that).  It cuts sequences as it would
// have by itself.
//
// Roles (768 threads), one tile of 128 tokens after the other as one pipeline:
//   warp 0        TMA producer
//   warp 1        MMA issuer: G = C.B^T, S = B^T.Xd, C.H, P.X of a tile, in this order
//   warp 2        sums of the log-decay and every factor derived from them, up to four tiles ahead
//   warp 3        (fp16) units of Xd's pieces
//   warps 4-19    thread = tile row = TMEM lane; every four warps have 32 tokens as columns of P and 16 columns of the state:
//     state entering the tile, in pieces -> shared memory -> C.H
//     P = G o exp(segsum) o causal, in pieces -> TMEM (into the columns that G is read from) -> P.X
//     H <- exp(cs_last) H + S
//   warps 20-23   Xd = exp(cs_last - cs) x~ of the next tile, in pieces -> shared memory -> S
//     Y = P.X + exp(cs) C.H [+ skip and gate] -> shared memory -> TMA store
//
// What bounds it (bf16, n = 128): a 128 x N x 16 MMA takes 55 cycles at N = 64, 62 at 128, some 90 at 192, a tile 3 900 (G 8 of 128, S 8 of
// 192, C.H and P.X 24 of 64 each); G, S and C.H read both operands from shared memory, which moves 560 KB a tile, 4 400
// cycles.  The MMA issuer goes round in some 5 000.  P on eight warps instead of sixteen: 104 us instead of 98.7 (2 x 3001
// tokens, 80 heads; the recurrence takes 1 895); the pieces unpacked by integer instructions: 98.7 instead of 97.2.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "tile_walk.cuh"

namespace ssd {
namespace {

using namespace tc;

constexpr int kThreadsS = 768;
constexpr int kFactorsS = 4;   // tiles that the factors may be ahead

template <int N, int kPieces>
struct LayoutS {
  static constexpr int NB = N / 64;
  static constexpr int kBC = N == 128 ? 1 : 2;           // B and C tiles in flight
  static constexpr int kXSlots = N == 128 && kPieces == 3 ? 3 : 4;   // X tiles in flight; a consumed one is where Y is staged
  static constexpr int oB = 0;
  static constexpr int oC = oB + kBC * NB * kBlk;
  static constexpr int oX = oC + kBC * NB * kBlk;
  static constexpr int oXd = oX + kXSlots * kBlk;        // [piece]
  static constexpr int oH = oXd + kPieces * kBlk;        // [piece], N rows of 128 B
  static constexpr int oMisc = oH + kPieces * N * 128;
  static constexpr int kMiscBytes = 16384;
  static constexpr int kBytes = oMisc + kMiscBytes;
};

// Tensor memory.  P's pieces (8 columns each per 16 tokens) stand where G was: two of them fill its columns, of three those of
// 32 tokens take the same 32 columns and 16 more behind G, so that a thread writes over nothing that another one reads.
template <int kPieces>
struct Columns {
  static constexpr uint32_t G = 0, S = kPieces == 3 ? 192 : 128, Yo = S + 64 * kPieces, Yd = kPieces == 3 ? 448 : 384;
  // the first piece of k-step ks (16 tokens), and the second (the third is 8 columns behind it)
  static __device__ __forceinline__ uint32_t first(uint32_t ks) { return kPieces == 3 ? 16 * ks + 8 * (ks & 1) : 16 * ks; }
  static __device__ __forceinline__ uint32_t second(uint32_t ks) { return kPieces == 3 && (ks & 1) ? 128 + 8 * (ks - 1) : 16 * ks + 8; }
};

// Factors of one tile.
struct alignas(16) FactorsS {
  float n2[T];     // minus the log-decay from the start of the token's 32-token block to the token, * log2(e)
  float cf[T];     // exp(log-decay from the token to the end of its block) * dt
  float xw[T];     // exp(log-decay from the token to the end of the tile) * dt
  float dt[T];     // (of a tile with strong decays / exp(what the sum in n2 lacks))
  float row[T];    // of a tile with strong decays: exp(what the sum in n2 lacks)
  float blk2[4];   // log-decay of each block, * log2(e)
  float g;         // exp(log-decay of the tile)
  float unit;      // cf, xw and dt are in units of this (a power of two)
  float x_scale, x_unit;   // (fp16) Xd * x_scale is taken to pieces, which are in units of x_unit
  float ld;        // its log-decay as given
  int strong;      // a block decays by more than kStrong
};

struct MiscS {
  Work work;
  FactorsS f[kFactorsS];
  uint64_t full_b[2], full_c[2], empty_b[2], empty_c[2];   // [stage]
  uint64_t full_x[4], empty_x[4];
  uint64_t full_f[kFactorsS], empty_f[kFactorsS], full_u[kFactorsS];   // (full_u, fp16: with the unit of Xd's pieces)
  uint64_t bar_g, bar_s, bar_ch, bar_y;   // tcgen05.commit arrivals
  uint64_t bar_h, bar_p, bar_u;           // the state's pieces, P's pieces are stored; S has been read (16 warps)
  uint64_t bar_xd, bar_e;                 // Xd's pieces are stored; C.H and P.X have been read (4 warps)
  uint64_t bar_drain;
  uint64_t full_h[4];        // (fp16) [tile % 4]: the unit of the state's pieces is there
  float h_unit[4];
  uint32_t h_max[4];         // the largest |H| that enters the tile, as bits
  uint32_t tmem_base;
  int bad;                   // the recurrence has to do this call again
  long long wait_clocks;
  volatile int abort_flag;
  Look<1> look;
};
static_assert(sizeof(MiscS) <= LayoutS<128, 3>::kMiscBytes, "MiscS outgrew its shared-memory slot");
static_assert(LayoutS<128, 3>::kBytes <= 232448 && LayoutS<64, 3>::kBytes <= 232448, "shared memory budget of one SM exceeded");
static_assert(LayoutS<128, 2>::kBytes <= 232448 && LayoutS<64, 2>::kBytes <= 232448, "shared memory budget of one SM exceeded");

constexpr float kLowestS = -104.f;   // as in ssd_tc2.cu: a factor of zero either way
// Log-decays above zero: up to this in each token (4 in a tile) the product of two factors loses nothing that matters.
constexpr float kGrowth = 1.f / 32.f;
// On the diagonal a weight is 2^(difference of two sums from the start of the block), and what both hold from before takes bits of it:
// 150 behind one reset 2e-5 of it, 3 600 behind 24 of them 5e-4.  Where a block decays by more than this much (up to which they take
// 3.4e-6 of it at most, 7e-7 in the mean), the sums are taken in 64 bits too, and the factors of a row and a column carry what their
// 32 bits lack.  (2 x 3001 tokens, 80 heads, bf16 and fp16: 85.0 and 90.2 us without, 85.9 and 92.5 so, 88.7 and 92.7 with 64 bits
// in every tile.)
constexpr float kStrong = 16.f;

// Two fp32 numbers as sums of 16-bit ones, packed.
// bf16: high, middle, low, eight bits at a time from the top, so all subtractions are exact.  (The multiply-add that takes
// 16-bit factors spares the unpacking, which is the integer pipe's, of half the rate.)
// fp16: high (11 bits, rounded) and UP times the rest (rounded to 11 bits; the factor keeps it out of the subnormal numbers).
__device__ __forceinline__ uint32_t top_pair(uint64_t v) {
  const float2 f = unpair(v);
  return __byte_perm(__float_as_uint(f.x), __float_as_uint(f.y), 0x7632);
}
template <typename T16>
__device__ __forceinline__ uint64_t less(uint64_t v, uint32_t packed) {
  const float2 f = unpair(v);
  float x, y;
  if constexpr (std::is_same<T16, __nv_bfloat16>::value)
    asm("{\n\t.reg .b16 l, h, m;\n\tmov.b32 {l, h}, %2;\n\tmov.b16 m, 0xBF80;\n\t"
        "fma.rn.f32.bf16 %0, l, m, %3;\n\tfma.rn.f32.bf16 %1, h, m, %4;\n\t}"
        : "=f"(x), "=f"(y)
        : "r"(packed), "f"(f.x), "f"(f.y));
  else
    asm("{\n\t.reg .b16 l, h, m;\n\tmov.b32 {l, h}, %2;\n\tmov.b16 m, 0xBC00;\n\t"
        "fma.rn.f32.f16 %0, l, m, %3;\n\tfma.rn.f32.f16 %1, h, m, %4;\n\t}"
        : "=f"(x), "=f"(y)
        : "r"(packed), "f"(f.x), "f"(f.y));
  return pair(x, y);
}
template <typename T16, int UP>
__device__ __forceinline__ void split(uint64_t v, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  if constexpr (std::is_same<T16, __nv_bfloat16>::value) {
    p0 = top_pair(v);
    const uint64_t r = less<T16>(v, p0);
    p1 = top_pair(r);
    p2 = top_pair(less<T16>(r, p1));
  } else {
    p0 = pack_pair<T16>(v);
    p1 = pack_pair<T16>(mul_pair(less<T16>(v, p0), pair((float)UP, (float)UP)));
    p2 = 0;
  }
}
// With 2^11 the low piece does not overflow where the high one does not.  With 2^14 it does from 4 096 on, and a number in units that make
// the largest 2^11 to 2^12 is held to 2^-23 of it, or to 2^-50 of the largest.
constexpr int kUp = 1 << 11, kUpX = 1 << 14;

// The larger magnitudes of two pairs of fp16 numbers (of a NaN the other's), with some sign.
__device__ __forceinline__ uint32_t max_abs2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// (fp16) What the accumulators of the pieces hold together, times `unit`.
template <int UP>
__device__ __forceinline__ uint64_t low_and_high(uint64_t low, uint64_t high, float unit) {
  return mul_pair(fma_pair(low, pair(1.f / UP, 1.f / UP), high), pair(unit, unit));
}

// The power of two at or below x >= 0, but 2^-100 at least, and 1 for what is too large to have a unit (2^127 and more, infinity,
// NaN: what comes of those is not finite); and 1 / 2^k.
__device__ __forceinline__ float power_below(float x) {
  const uint32_t e = __float_as_uint(x) & 0x7f800000u;
  return e >= 0x7f000000u ? 1.f : __uint_as_float(max(e, 27u << 23));
}
__device__ __forceinline__ float inverse_power(float x) { return __uint_as_float(0x7f000000u - __float_as_uint(x)); }

// EPI: skip and gate of model_ref.py:116-118 (sp.D / sp.Z; either may be null) applied to Y in fp32 ahead of its one rounding.
// LB: sequences cut in look-back mode, an instance of its own as in ssd_tc2.cu (615 heads of 27 tokens, fp16: 30.6 us without).
template <typename T16, int N, bool EPI, bool LB>
__global__ void __launch_bounds__(kThreadsS, 1)
ssd_split_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmY, const TileParams prm) {
  constexpr bool kF16 = std::is_same<T16, __half>::value;
  constexpr int kPieces = kF16 ? 2 : 3;
  using L = LayoutS<N, kPieces>;
  using Cursor = CursorOf<1, LB>;
  using Col = Columns<kPieces>;
  constexpr uint32_t tG = Col::G, tYo = Col::Yo, tS = Col::S, tYd = Col::Yd;
  constexpr int NB = L::NB, KN = N / 16, KT = T / 16, BC = L::kBC, XS = L::kXSlots;
  extern __shared__ __align__(1024) uint8_t smem[];
  MiscS* m = reinterpret_cast<MiscS*>(smem + L::oMisc);
  const ScanParams& sp = prm.sp;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int32_t* status = sp.status;
  if (blockIdx.x == 0 && tid == 0) sp.redo[RedoWords::kNext] = sp.redo[RedoWords::kScanned] = sp.redo[RedoWords::kFolded] = 0;
  if (smem_u32(smem) & 1023u) {
    if (tid == 0) {
      if (status) atomicCAS(status, 0, (int)STATUS_BAD_SMEM_ALIGNMENT);
      sp.redo[blockIdx.x] = 0;
    }
    return;
  }
  if (sp.inject_lost_handover && sp.chain && blockIdx.x == 0) {   // (as in ssd_tc2.cu)
    if (tid == 0) sp.redo[0] = 0;
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < BC; ++s) {
      mbar_init(&m->full_b[s], 1); mbar_init(&m->full_c[s], 1);
      mbar_init(&m->empty_b[s], 1); mbar_init(&m->empty_c[s], 1);
    }
    for (int s = 0; s < XS; ++s) { mbar_init(&m->full_x[s], 1); mbar_init(&m->empty_x[s], 4); }
    for (int s = 0; s < kFactorsS; ++s) { mbar_init(&m->full_f[s], 1); mbar_init(&m->empty_f[s], 20); mbar_init(&m->full_u[s], 1); }
    mbar_init(&m->bar_g, 1); mbar_init(&m->bar_s, 1); mbar_init(&m->bar_ch, 1); mbar_init(&m->bar_y, 1);
    mbar_init(&m->bar_h, 16); mbar_init(&m->bar_p, 16); mbar_init(&m->bar_u, 16);
    mbar_init(&m->bar_xd, 4); mbar_init(&m->bar_e, 4);
    mbar_init(&m->bar_drain, 1);
    for (int s = 0; s < 4; ++s) {
      mbar_init(&m->full_h[s], 1);
      m->h_max[s] = 0;
    }
    m->abort_flag = 0;
    m->bad = 0;
    m->wait_clocks = sp.wait_clocks;
    work_list(prm, m->work);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&m->tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  if constexpr (LB) {
    find_beginning<1>(prm, m->work, m->look, kThreadsS / 32);
    __syncthreads();
  }
  tc_fence_after();
  // The recurrence's CTAs may come once all of these are on their SMs: they wait for the end of this kernel, but not to be launched.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t sB = smem_u32(smem + L::oB), sC = smem_u32(smem + L::oC), sX = smem_u32(smem + L::oX);
  const uint32_t sXd = smem_u32(smem + L::oXd), sH = smem_u32(smem + L::oH);
  const Work& wk = m->work;
  const uint32_t total = m->tmem_base == 0 ? (uint32_t)wk.total : 0u, npre = (uint32_t)wk.npre;
  auto warp_arrive = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };

  if (warp == 0 && lane == 0) {
    // ------------------------------------------------------------------ TMA producer (holds the clock: see guarded_wait)
    const uint64_t once = policy_evict_first(), again = policy_evict_last();
    prefetch_tmap(&tmX); prefetch_tmap(&tmB); prefetch_tmap(&tmC); prefetch_tmap(&tmY);
    bool ok = true;
    uint32_t xi = 0, xph = 0, bs = 0, bph = 0, cs = 0, cph = 0;
    Cursor c;
#pragma unroll 1
    for (uint32_t n = 0; n < total && ok; ++n) {
      c.next(prm, wk);
#pragma unroll 1
      for (int k = 0; k < (n < npre ? 2 : 3); ++k) {   // X, B, then C (not for a state-only tile)
        const CUtensorMap* tm = k == 0 ? &tmX : k == 1 ? &tmB : &tmC;
        uint64_t* full = k == 0 ? &m->full_x[xi] : k == 1 ? &m->full_b[bs] : &m->full_c[cs];
        uint64_t* empty = k == 0 ? &m->empty_x[xi] : k == 1 ? &m->empty_b[bs] : &m->empty_c[cs];
        const uint32_t ph = k == 0 ? xph : k == 1 ? bph : cph;
        uint32_t dst = k == 0 ? sX + xi * kBlk : k == 1 ? sB + bs * (NB * kBlk) : sC + cs * (NB * kBlk);
        const int blocks = k == 0 ? 1 : NB;
        ok = guarded_wait(empty, ph ^ 1, m, STATUS_WAIT_TIMEOUT_MMA);
        if (!ok) break;
        mbar_expect_tx(full, blocks * kBlk);
#pragma unroll 1
        for (int kb = 0; kb < blocks; ++kb, dst += kBlk)
          tma_load_5d(dst, tm, full, 64 * kb, k == 0 ? c.q : 0, c.g, c.t0, c.b, k == 0 ? once : again);
        if (k == 0) {
          if (++xi == XS) { xi = 0; xph ^= 1; }
        } else if (k == 1) {
          if (++bs == BC) { bs = 0; bph ^= 1; }
        } else {
          if (++cs == BC) { cs = 0; cph ^= 1; }
        }
      }
    }
    if (ok) ok = guarded_wait(&m->bar_drain, 0, m, STATUS_WAIT_TIMEOUT_SYNC);
    if (!ok) {
      const long long c0 = clock64();   // copies already in flight land before the shared memory is given back
      while (clock64() - c0 < 2000000LL) { }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // S has an accumulator for each piece, one product of 192 (128) columns.  bf16: C.H and P.X have one, products of 64 columns,
    // the low pieces first: an accumulator cuts off what it cannot hold (small ones last, the final state was off by 2.1e-7
    // instead of 8e-8).  (Shared memory is what the first three are short of: S as two products of 128 columns reads the B tile
    // twice.  2 x 3001 tokens, 80 heads: S and C.H that way 93.1 us, this way 86.0.)  fp16: two accumulators each.
    constexpr int fmt = kF16 ? 0 : 1;
    constexpr uint64_t kHi = umma_desc_base(0, 1024);
    constexpr uint32_t kMN = kBlk >> 4, kMNh = N * 128 >> 4, kRow16 = 2048 >> 4, kCol16 = 32 >> 4;
    constexpr uint32_t idG = umma_idesc(128, 128, fmt, 0, 0), idS = umma_idesc(128, 64 * kPieces, fmt, 1, 1);
    constexpr uint32_t idCH = umma_idesc(128, kF16 ? 128 : 64, fmt, 0, 1), idPX = umma_idesc(128, 64, fmt, 0, 1);
    uint32_t xb = 0;   // X slot of the tile, as a descriptor offset
#pragma unroll 1
    for (uint32_t n = 0; n < total; ++n) {
      const bool wy = n >= npre;
      const uint32_t py = n - npre;
      const uint32_t sb = n % BC, sc = py % BC;
      const uint32_t aB = (sB + sb * (NB * kBlk)) >> 4, aC = (sC + sc * (NB * kBlk)) >> 4;
      wait(&m->full_b[sb], (n / BC) & 1, m);
      if (wy) {
        wait(&m->full_c[sc], (py / BC) & 1, m);
        if (py > 0) wait(&m->bar_y, (py - 1) & 1, m);   // P of the tile before, which stands in G's columns, has been read
        tc_fence_after();
        if (elect_one()) {
#pragma unroll 1
          for (uint32_t k = 0; k < KN; k += 4) {
            const uint32_t o = (k >> 2) * kMN;
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i)
              umma_ss(tG, kHi | (1u << 16 | (aC + o + i * kCol16)), kHi | (1u << 16 | (aB + o + i * kCol16)), idG, k + i);
          }
          umma_commit(&m->bar_g);
        }
        __syncwarp();
      }
      wait(&m->bar_xd, n & 1, m);
      if (n > 0) wait(&m->bar_u, (n - 1) & 1, m);
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (uint32_t k = 0; k < KT; ++k)
          umma_ss(tS, kHi | (kMN << 16 | (aB + k * kRow16)), kHi | (kMN << 16 | ((sXd >> 4) + k * kRow16)), idS, k);
        umma_commit(&m->bar_s);
        umma_commit(&m->empty_b[sb]);
      }
      __syncwarp();
      if (wy) {
        wait(&m->bar_h, py & 1, m);
        if (py > 0) wait(&m->bar_e, (py - 1) & 1, m);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll 1
          for (uint32_t v = 0; v < (kF16 ? 1 : 3); ++v) {   // (low, middle, high)
            const uint32_t bh = (sH >> 4) + (kF16 ? 0 : 2 - v) * kMNh;
#pragma unroll
            for (uint32_t k = 0; k < KN; ++k)
              umma_ss(tYo, kHi | (1u << 16 | (aC + (k >> 2) * kMN + (k & 3) * kCol16)), kHi | (kMNh << 16 | (bh + k * kRow16)),
                      idCH, v + k);
          }
          umma_commit(&m->bar_ch);
          umma_commit(&m->empty_c[sc]);
        }
        __syncwarp();
        wait(&m->bar_p, py & 1, m);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll 1
          for (uint32_t k = 0; k < KT; ++k) {
            const uint64_t bx = kHi | (kMN << 16 | ((sX >> 4) + xb + k * kRow16));
            const uint32_t second = Col::second(k);
            if constexpr (kF16) {
              umma_ts(tYd, Col::first(k), bx, idPX, k);
              umma_ts(tYd + 64, second, bx, idPX, k);
            } else {
              umma_ts(tYd, second + 8, bx, idPX, k);   // (low, middle, high)
              umma_ts(tYd, second, bx, idPX, 1);
              umma_ts(tYd, Col::first(k), bx, idPX, 1);
            }
          }
          umma_commit(&m->bar_y);
        }
        __syncwarp();
      }
      xb = xb == (XS - 1) * kMN ? 0 : xb + kMN;
    }
    if (elect_one()) {
      umma_commit(&m->bar_drain);
      const long long t0 = clock64();
      while (!mbar_try_wait(&m->bar_drain, 0))
        if (clock64() - t0 > m->wait_clocks) break;
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ factors: lane i owns tokens 4i .. 4i+3
    const int64_t as1 = sp.as[1], ds1 = sp.dts[1], asT = T * as1, dsT = T * ds1;
    const float* Ag = nullptr;
    const T16* Dg = nullptr;
    bool growth = false;
    Cursor c;
#pragma unroll 1
    for (uint32_t n = 0; n < total; ++n) {
      c.next(prm, wk);
      if (c.first_tile()) {
        const int head = c.head(wk);
        const int64_t t = c.t0 + 4 * lane;
        Ag = sp.A + c.b * sp.as[0] + head * sp.as[2] + t * as1;
        Dg = static_cast<const T16*>(sp.dt) + c.b * sp.dts[0] + head * sp.dts[2] + t * ds1;
        if (sp.init && c.t_begin == 0) {   // the state that enters goes to L2
          const float* I = sp.init + ((int64_t)c.b * sp.nheads + head) * sp.init_unit_stride;
          for (int e = lane; e < N * P / 32; e += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(I + 32 * e));
        }
      }
      float a[4], dt[4];
      const int in = sp.seqlen - c.t0 - 4 * lane;   // past the end: decay 1 and x = 0, the state stays as it is (a step of 0: no unit of its own)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[e] = e < in ? Ag[e * as1] : 0.f;
        dt[e] = e >= in ? 0.f : sp.dt ? Cvt<T16>::to_f(Dg[e * ds1]) : 1.f;
      }
      Ag += asT;
      Dg += dsT;
      float ld = a[0] + a[1] + a[2] + a[3];
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, d);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (a[e] < kLowestS) a[e] = kLowestS;   // (NaN stays NaN)
        growth |= a[e] > kGrowth;
      }
      // sums within the block of 32 tokens (eight lanes): up to and with each token, and of what comes after it
      const float s01 = a[0] + a[1], s23 = a[2] + a[3];
      float up = s01 + s23, down = up;
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, up, d, 8), v = __shfl_down_sync(0xffffffffu, down, d, 8);
        if ((lane & 7) >= d) up += u;
        if ((lane & 7) + d < 8) down += v;
      }
      float before = __shfl_up_sync(0xffffffffu, up, 1, 8), after = __shfl_down_sync(0xffffffffu, down, 1, 8);
      if ((lane & 7) == 0) before = 0.f;
      if ((lane & 7) == 7) after = 0.f;
      float D[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) D[b] = __shfl_sync(0xffffffffu, up, 8 * b + 7);
      const int blk = lane >> 3;
      const float rest = blk == 0 ? D[3] + D[2] + D[1] : blk == 1 ? D[3] + D[2] : blk == 2 ? D[3] : 0.f;   // blocks after this one
      const float fr = expf(rest);
      const float n2[4] = {(before + a[0]) * -kLog2e, (before + s01) * -kLog2e, (before + (s01 + a[2])) * -kLog2e, up * -kLog2e};
      const bool strong = __any_sync(0xffffffffu, up < -kStrong);
      const float x[4] = {after + (s23 + a[1]), after + s23, after + a[3], after};
      float unit = 1.f;
      if constexpr (kF16) {   // weights of up to 2: what fp16 has to hold is then x, and G, and not their products with small steps
        float most = fmaxf(fmaxf(fabsf(dt[0]), fabsf(dt[1])), fmaxf(fabsf(dt[2]), fabsf(dt[3])));
        most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most)));
        unit = power_below(most);
        const float inv = inverse_power(unit);
#pragma unroll
        for (int e = 0; e < 4; ++e) dt[e] *= inv;
      }
      const uint32_t slot = n % kFactorsS;
      wait(&m->empty_f[slot], ((n / kFactorsS) & 1) ^ 1, m);
      FactorsS& f = m->f[slot];
      float cf[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) cf[e] = expf(x[e]) * dt[e];
      reinterpret_cast<float4*>(f.n2)[lane] = make_float4(n2[0], n2[1], n2[2], n2[3]);
      if (strong) {
        double from = 0.0, to = ((double)a[0] + (double)a[1]) + ((double)a[2] + (double)a[3]);
#pragma unroll 1
        for (int d = 1; d < 8; d <<= 1) {
          const double u = __shfl_up_sync(0xffffffffu, to, d, 8);
          if ((lane & 7) >= d) to += u;
        }
        from = __shfl_up_sync(0xffffffffu, to, 1, 8);
        if ((lane & 7) == 0) from = 0.0;
        float row[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          from += (double)a[e];
          const float lacks = (float)(from - (double)n2[e] * -0.6931471805599453);   // (2e-3 at most: exp by its series)
          row[e] = fmaf(lacks, fmaf(lacks, 0.5f, 1.f), 1.f);
          dt[e] *= fmaf(-lacks, fmaf(-lacks, 0.5f, 1.f), 1.f);
        }
        reinterpret_cast<float4*>(f.row)[lane] = make_float4(row[0], row[1], row[2], row[3]);
      }
      reinterpret_cast<float4*>(f.cf)[lane] = make_float4(cf[0], cf[1], cf[2], cf[3]);
      reinterpret_cast<float4*>(f.xw)[lane] = make_float4(cf[0] * fr, cf[1] * fr, cf[2] * fr, cf[3] * fr);
      reinterpret_cast<float4*>(f.dt)[lane] = make_float4(dt[0], dt[1], dt[2], dt[3]);
      if (lane < 4) f.blk2[lane] = (lane == 0 ? D[0] : lane == 1 ? D[1] : lane == 2 ? D[2] : D[3]) * kLog2e;
      if (lane == 4) {
        f.strong = strong;
        f.g = expf(((D[3] + D[2]) + D[1]) + D[0]);
        f.ld = ld;
        f.unit = unit;
      }
      warp_arrive(&m->full_f[slot]);
    }
    if (growth) m->bad = 1;
  } else if (kF16 && warp == 3) {
    // ------------------------------------------------------------------ (fp16) units of Xd's pieces
    // A power of two from the tile's largest |Xd| (up to 2^11: larger ones stay as they are), so that small numbers keep their
    // bits, and those that decay by far within the tile.  (2 x 3001 tokens, 80 heads: 92.8 us without units; 101.3 with them found by the
    // warps that make Xd; here 99.9 with eight lanes to a row, 94.9 with a row to a lane, which takes a third of the instructions.)
    uint32_t xi = 0, xph = 0;
#pragma unroll 1
    for (uint32_t n = 0; n < total; ++n) {
      const uint32_t slot = n % kFactorsS;
      wait(&m->full_f[slot], (n / kFactorsS) & 1, m);
      wait(&m->full_x[xi], xph, m);
      FactorsS& f = m->f[slot];
      float most = 0.f;
      const uint32_t at = sX + xi * kBlk + lane * 128 + ((lane & 7) << 4);   // (rows lane, lane + 32, ..., their pieces in an order without conflicts)
#pragma unroll 1
      for (int r = 0; r < T; r += 32) {
        uint32_t x2 = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
          const uint4 a = lds128((at + 128 * r) ^ (k << 4));
          x2 = max_abs2(x2, max_abs2(max_abs2(a.x, a.y), max_abs2(a.z, a.w)));
        }
        const float2 x = unpack2<T16>(x2);
        most = fmaxf(most, fmaxf(fabsf(x.x), fabsf(x.y)) * fabsf(f.xw[lane + r]));
      }
      most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most)));
      if (lane == 0) {
        const float unit = fminf(power_below(most), 2048.f);
        f.x_scale = inverse_power(unit) * 2048.f;
        f.x_unit = unit * (1.f / 2048.f) * f.unit;
        mbar_arrive(&m->full_u[slot]);
      }
      if (++xi == XS) { xi = 0; xph ^= 1; }
    }
  } else if (warp >= 4 && warp < 20) {
    // ------------------------------------------------------------------ warps 4-19: P and the state
    const int J = (warp - 4) >> 2;       // tokens 32 J .. 32 J + 31 as columns of P, columns 16 J .. 16 J + 15 of the state
    const int q = warp & 3, l = 32 * q + lane;
    const uint32_t tlane = (uint32_t)(32 * q) << 16;
    const uint32_t swz = (uint32_t)(l & 7);
    const bool owns_state = 32 * q < N;
    uint64_t H[8];                   // fp32 pairs
#pragma unroll
    for (int e = 0; e < 8; ++e) H[e] = 0;
    uint64_t odd = 0;                // 0 times every number that leaves: NaN if one is not finite
    const uint64_t zero2 = pair(0.f, 0.f);
    float asum0 = 0.f;               // log-decay summed over the earlier pieces of the sequence
    float asum = 0.f, acomp = 0.f;   // compensated sum of the tile totals
    Cursor c;
    bool fold = false;

    // P of this thread's row, 32 columns.  The block is below the diagonal (weight = decay from the block's end to the row * decay
    // to the block's end, both in one product), on it (an exponential per column), or above (zero).
    auto make_p = [&](const FactorsS& f) {
      float r = -f.n2[l];
#pragma unroll 1
      for (int b = J + 1; b < q; ++b) r += f.blk2[b];
      const float rf = ex2(r);
#pragma unroll 1
      for (int ks = 2 * J + 1; ks >= 2 * J; --ks) {   // (the second half of G first: see Columns)
        uint32_t p0[8], p1[8], p2[8];
        if (J > q) {
#pragma unroll
          for (int e = 0; e < 8; ++e) p0[e] = p1[e] = p2[e] = 0;
        } else {
          uint32_t g[16];
          uint64_t v[8];
          tmem_ld16(tG + tlane + 16 * ks, g);
          if (J < q) {
            const uint64_t rf2 = pair(rf, rf);
            const ulonglong2* cf = reinterpret_cast<const ulonglong2*>(f.cf + 16 * ks);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const ulonglong2 w = cf[e];
              v[2 * e] = mul_pair(rf2, w.x);
              v[2 * e + 1] = mul_pair(rf2, w.y);
            }
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = mul_pair(pair(g[2 * e], g[2 * e + 1]), v[e]);
          } else {
            const int last = lane - 16 * (ks & 1);   // columns up to this one are not after the row
            const ulonglong2* nn = reinterpret_cast<const ulonglong2*>(f.n2 + 16 * ks);
            const ulonglong2* dd = reinterpret_cast<const ulonglong2*>(f.dt + 16 * ks);
            const float row2 = -f.n2[l];
            const uint64_t rows2 = pair(row2, row2);
            auto weight = [&](uint64_t n2, uint64_t d) {
              const float2 x = unpair(add_pair(rows2, n2));
              return mul_pair(pair(ex2(x.x), ex2(x.y)), d);
            };
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const ulonglong2 n2 = nn[e], d = dd[e];
              v[2 * e] = weight(n2.x, d.x);
              v[2 * e + 1] = weight(n2.y, d.y);
            }
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float2 x = unpair(mul_pair(pair(g[2 * e], g[2 * e + 1]), v[e]));
              v[e] = pair(2 * e <= last ? x.x : 0.f, 2 * e + 1 <= last ? x.y : 0.f);
            }
            if (__builtin_expect(f.strong, 0)) {
              const float r = f.row[l];
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = mul_pair(v[e], pair(r, r));
            }
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) split<T16, kUp>(v[e], p0[e], p1[e], p2[e]);
        }
        tmem_st8(tlane + Col::first(ks), p0);
        tmem_st8(tlane + Col::second(ks), p1);
        if constexpr (!kF16) tmem_st8(tlane + Col::second(ks) + 8, p2);
      }
    };
    // The state's pieces, in shared memory; fp16 in units of h_unit / 2^14, which keeps the largest below 2^15.
    float h_unit = 1.f;
    auto store_h = [&]() {
      if (!owns_state) return;
      const float inv = kF16 ? inverse_power(h_unit) * 16384.f : 1.f;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        uint32_t p0[4], p1[4], p2[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split<T16, kUp>(kF16 ? mul_pair(H[4 * k + e], pair(inv, inv)) : H[4 * k + e], p0[e], p1[e], p2[e]);
        const uint32_t at = sH + l * 128 + (((2 * J + k) ^ swz) << 4);
        sts128(at, make_uint4(p0[0], p0[1], p0[2], p0[3]));
        sts128(at + N * 128, make_uint4(p1[0], p1[1], p1[2], p1[3]));
        if constexpr (!kF16) sts128(at + 2 * N * 128, make_uint4(p2[0], p2[1], p2[2], p2[3]));
      }
    };
    // (fp16) The unit is a power of two from the largest |H| of all sixteen warps.  A slot is cleared two tiles ahead: all warps
    // have read it, and none gets to use it again before the barrier of the tile between.
    auto find_h_unit = [&](uint32_t k) {
      uint32_t most = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 v = unpair(H[e]);
        most = max(most, max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu));
      }
      most = __reduce_max_sync(0xffffffffu, most);
      if (lane == 0) atomicMax(&m->h_max[k % 4], most);
      asm volatile("bar.sync 1, 512;" ::: "memory");
      h_unit = power_below(__uint_as_float(m->h_max[k % 4]));
      if (warp == 4 && lane == 0) {
        m->h_max[(k + 2) % 4] = 0;
        m->h_unit[k % 4] = h_unit;
        mbar_arrive(&m->full_h[k % 4]);
      }
    };
    // (bounded) wait until the sixteen warps of CTAs `from` .. `to` have published, a CTA per lane
    auto wait_published = [&](int to, int from) {
      grid_dependency_wait();
      const long long c0 = clock64();
      for (int k = to - lane; k >= from && !m->abort_flag; k -= 32) {
        while (true) {
          int f;
          asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(f) : "l"(sp.chain_flag + 2 * k) : "memory");
          if (f >= 16 || m->abort_flag) break;
          if (clock64() - c0 > m->wait_clocks) {
            m->abort_flag = (int)STATUS_WAIT_TIMEOUT_CHAIN;
            break;
          }
        }
      }
      __syncwarp();
    };
    auto enter_item = [&](bool wy) {
      if (c.goes_on(wk)) return;
      asum0 = asum = acomp = 0.f;
      const bool from_zero = sp.chain == 2 && !wy;               // (the look-back scan)
      fold = sp.chain && !from_zero && (c.t_begin > 0 || (LB && wk.again == 2));   // (the latter is to be looked at behind the fold)
      if (sp.init && !from_zero && !fold && owns_state) {
        const float* I = sp.init + ((int64_t)c.b * sp.nheads + c.head(wk)) * sp.init_unit_stride + (int64_t)l * P + 16 * J;
        if (prm.st32) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint64_t v[4];
            ldg256(I + 8 * e, v);
            H[4 * e] = v[0]; H[4 * e + 1] = v[1]; H[4 * e + 2] = v[2]; H[4 * e + 3] = v[3];
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const ulonglong2 v = reinterpret_cast<const ulonglong2*>(I)[e];
            H[2 * e] = v.x;
            H[2 * e + 1] = v.y;
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) H[e] = 0;
      }
    };
    // The state entering a piece from what the CTAs before published (see ssd_tc2.cu; slots [p / 4][n][4] of every other slot).
    auto fold_item = [&]() {
      const bool look_back = sp.chain == 2;
      const bool init = sp.init && look_back;
      int p = (int)blockIdx.x - 1;
      const int from = !look_back ? p : LB && c.t_begin == 0 ? (int)blockIdx.x : wk.from;
      wait_published(p, from);
      float lds = 0.f;   // look-back: log-decays of 32 pieces, one in each lane (asked for one by one they are a round trip to L2 each)
      int next = 0;
#pragma unroll 1
      for (;; --p) {
        const bool piece = p >= from;
        if (!piece && !init) break;
        const float* src = piece ? sp.chain_state + 2 * p * (int64_t)(N * P) + (4 * J * N + l) * 4
                                 : sp.init + ((int64_t)c.b * sp.nheads + c.head(wk)) * sp.init_unit_stride + (int64_t)l * P + 16 * J;
        const int step = piece ? N : 1;
        float ld = 0.f;
        if (!LB) ld = piece ? __ldcg(sp.chain_ld + 2 * p) : 0.f;
        else if (next == 0 && p - lane >= from) lds = __ldcg(sp.chain_ld + 2 * (p - lane));
        const float wgt = expf(asum0);           // asum0: log-decay between the end of the piece being added and this item
        if (owns_state && wgt != 0.f) {          // (an underflowed piece adds nothing)
          const ulonglong2* I = reinterpret_cast<const ulonglong2*>(src);
          const uint64_t w2 = pair(wgt, wgt);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const ulonglong2 v = __ldcg(I + e * step);   // (may be written by another SM: bypass L1)
            H[2 * e] = fma_pair(w2, v.x, H[2 * e]);
            H[2 * e + 1] = fma_pair(w2, v.y, H[2 * e + 1]);
          }
        }
        if (!piece) break;
        asum0 += LB ? __shfl_sync(0xffffffffu, lds, next) : ld;
        next = (next + 1) & 31;
      }
    };
    auto leave_item = [&](bool wy) {
#pragma unroll
      for (int e = 0; e < 8; ++e) odd = fma_pair(H[e], zero2, odd);
      const bool cut_back = sp.chain && c.t_begin / T + c.ntiles < wk.nt;
      const bool publish = cut_back && !(LB ? !c.scanned(wk) : sp.chain == 2 && wy);   // (look-back: the scan from zero)
      const int64_t slot = 2 * (int64_t)blockIdx.x;
      const int64_t unit = (int64_t)c.b * sp.nheads + c.head(wk);
      if (publish ? given_up(m) : cut_back) return;
      float* to = publish ? sp.chain_state + slot * (N * P) : (sp.fin ? sp.fin + unit * sp.fin_unit_stride : nullptr);
      if (to && owns_state) {
        float* F = to + (publish ? (4 * J * N + l) * 4 : l * P + 16 * J);
        const int step = publish ? N : 1;
        if (prm.st32 && !publish) {
#pragma unroll
          for (int e = 0; e < 2; ++e) stg256(F + 8 * e, H[4 * e], H[4 * e + 1], H[4 * e + 2], H[4 * e + 3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) reinterpret_cast<ulonglong2*>(F)[e * step] = make_ulonglong2(H[2 * e], H[2 * e + 1]);
        }
      }
      if (publish && l == 0 && J == 0) sp.chain_ld[slot] = asum0 + asum;
      if (publish) {
        __syncwarp();
        grid_dependency_wait();
        if (lane == 0) {
          const int one = 1;
          asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(sp.chain_flag + slot), "r"(one) : "memory");
        }
      }
    };

    uint32_t ky = 0;            // Y-producing tiles so far
    if (total > 0) {
      c.next(prm, wk);
      enter_item(npre == 0);
    }
#pragma unroll 1
    for (uint32_t n = 0; n < total; ++n) {
      const bool wy = n >= npre;
      const uint32_t slot = n % kFactorsS;
      if (__builtin_expect(fold, 0)) {
        fold_item();
        fold = false;
        if (LB && wk.again == 2) {   // (a beginning done again: from a state that does not vanish behind it?)
          bool gone = true;
#pragma unroll
          for (int e = 0; e < 8; ++e) gone = gone && vanishes(unpair(H[e]));
          if (!gone) m->bad = 1;
        }
      }
      if (wy) {
        if constexpr (kF16) find_h_unit(ky);
        wait(&m->bar_ch, (ky & 1) ^ 1, m);   // the C.H MMAs have read the pieces before these
        store_h();
        fence_proxy_async();
        warp_arrive(&m->bar_h);
      }
      wait(&m->full_f[slot], (n / kFactorsS) & 1, m);
      const FactorsS& f = m->f[slot];
      if (wy) {
        wait(&m->bar_g, ky & 1, m);
        tc_fence_after();
        make_p(f);
        tmem_st_wait();
        tc_fence_before();
        warp_arrive(&m->bar_p);
        ++ky;
      }
      {
        const float yk = f.ld - acomp, tk = asum + yk;
        acomp = (tk - asum) - yk;
        if (acomp != acomp) acomp = 0.f;   // (a sum of -inf stays that)
        asum = tk;
      }
      const float gs = f.g;
      float su = 1.f;
      if constexpr (kF16) {
        wait(&m->full_u[slot], (n / kFactorsS) & 1, m);
        su = f.x_unit;
      }
      wait(&m->bar_s, n & 1, m);
      tc_fence_after();
      if (owns_state) {
        const uint64_t g2 = pair(gs, gs);
        uint32_t s0[16], s1[16];
        tmem_ld16(tS + tlane + 64 + 16 * J, s0);
        tmem_ld16(tS + tlane + (kF16 ? 0 : 128) + 16 * J, s1);
        tmem_ld_wait();
        if constexpr (kF16) {
#pragma unroll
          for (int e = 0; e < 8; ++e) H[e] = fma_pair(H[e], g2, low_and_high<kUpX>(pair(s0[2 * e], s0[2 * e + 1]), pair(s1[2 * e], s1[2 * e + 1]), su));
        } else {   // (middle and low pieces, then the high ones: for the registers)
          uint64_t ml[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) ml[e] = add_pair(pair(s0[2 * e], s0[2 * e + 1]), pair(s1[2 * e], s1[2 * e + 1]));
          tmem_ld16(tS + tlane + 16 * J, s0);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 8; ++e) H[e] = fma_pair(H[e], g2, add_pair(pair(s0[2 * e], s0[2 * e + 1]), ml[e]));
        }
      }
      tc_fence_before();
      warp_arrive(&m->bar_u);
      if (lane == 0) mbar_arrive(&m->empty_f[slot]);
      const bool last = c.left == 0;
      if (__builtin_expect(last, 0)) leave_item(wy);
      if (n + 1 < total) c.next(prm, wk);
      if (__builtin_expect(last && n + 1 < total, 0)) enter_item(n + 1 >= npre);
    }
    const float2 o = unpair(odd);
    if (!(o.x == 0.f && o.y == 0.f)) m->bad = 1;
  } else if (warp >= 20) {
    // ------------------------------------------------------------------ warps 20-23: Xd, and read-out of Y
    const int q = warp & 3, l = 32 * q + lane;
    const uint32_t tlane = (uint32_t)(32 * q) << 16;
    const uint32_t swz = (uint32_t)(l & 7);
    const uint64_t zero2 = pair(0.f, 0.f);
    uint64_t odd = 0;
    Cursor c;
    uint32_t bi = 0, bph = 0;   // X slot of the next tile to make Xd of
    uint32_t xi = 0;            // X slot of the tile being read out
    uint32_t ky = 0;
    const uint64_t once = policy_evict_first();
    int pending = -1;           // (lane 0) X slot that this warp's last TMA store still reads
    auto release = [&]() {
      if (lane == 0 && pending >= 0) {
        bulk_wait_read_all();
        mbar_arrive(&m->empty_x[pending]);
        pending = -1;
      }
    };
#pragma unroll 1
    for (uint32_t k = 0; k <= total; ++k) {   // Xd of tile k, Y of tile k - 1
      if (k < total) {
        const uint32_t slot = k % kFactorsS;
        wait(kF16 ? &m->full_u[slot] : &m->full_f[slot], (k / kFactorsS) & 1, m);   // (warp 3 has waited for the others)
        wait(&m->full_x[bi], bph, m);
        if (k > 0) wait(&m->bar_s, (k - 1) & 1, m);   // the S MMAs have read the Xd before this one
        // eight lanes share a row (one 16-byte piece each), a warp moves four rows per instruction
        const uint32_t xb = sX + bi * kBlk, pc = (uint32_t)lane & 7u;
        const FactorsS& f = m->f[slot];
        const float scale = kF16 ? f.x_scale : 1.f;
#pragma unroll 2
        for (int i = 0; i < 8; ++i) {
          const uint32_t r = 32 * q + 4 * i + ((uint32_t)lane >> 3), at = r * 128 + ((pc ^ (r & 7u)) << 4);
          const uint4 a = lds128(xb + at);
          const float w = f.xw[r] * scale;
          const uint64_t w2 = pair(w, w);
          const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
          uint32_t p0[4], p1[4], p2[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 x = unpack2<T16>(aw[e]);
            split<T16, kUpX>(mul_pair(pair(x.x, x.y), w2), p0[e], p1[e], p2[e]);
          }
          sts128(sXd + at, make_uint4(p0[0], p0[1], p0[2], p0[3]));
          sts128(sXd + kBlk + at, make_uint4(p1[0], p1[1], p1[2], p1[3]));
          if constexpr (!kF16) sts128(sXd + 2 * kBlk + at, make_uint4(p2[0], p2[1], p2[2], p2[3]));
        }
        fence_proxy_async();
        warp_arrive(&m->bar_xd);
        if (k < npre && lane == 0) {   // nothing else reads X of a state-only tile
          mbar_arrive(&m->empty_x[bi]);
          mbar_arrive(&m->empty_f[slot]);
        }
        if (++bi == XS) { bi = 0; bph ^= 1; }
        release();
      }
      if (k == 0) continue;
      const uint32_t n = k - 1, slot = n % kFactorsS;
      c.next(prm, wk);
      if (n < npre) {
        if (++xi == XS) xi = 0;
        continue;
      }
      const FactorsS& f = m->f[slot];
      float r = -f.n2[l];
#pragma unroll 1
      for (int b = 0; b < q; ++b) r += f.blk2[b];
      float el = ex2(r);
      const float unit = f.unit;
      warp_arrive(&m->empty_f[slot]);
      if constexpr (kF16) {
        wait(&m->full_h[ky % 4], (ky / 4) & 1, m);
        el *= m->h_unit[ky % 4] * (1.f / 16384.f);
      }
      // (EPI) this thread's gate row, fetched some columns ahead
      constexpr int W = kF16 || EPI ? 8 : 16;   // columns at a time
      const int64_t tok = c.t0 + l;
      const bool gated = EPI && sp.Z && tok < sp.seqlen;
      const T16* zrow = static_cast<const T16*>(sp.Z) + c.b * sp.zs[0] + tok * sp.zs[1] + c.head(wk) * sp.zs[2];
      uint4 zn[W / 8];
      auto gate = [&](int i) {
        if (gated) {
#pragma unroll
          for (int k = 0; k < W / 8; ++k) zn[k] = __ldg(reinterpret_cast<const uint4*>(zrow + W * i) + k);
        }
      };
      float skip = 0.f;
      if constexpr (EPI) {
        gate(0);
        if (sp.D) skip = load_skip<T16>(sp, c.head(wk));
      }
      wait(&m->bar_y, ky & 1, m);
      tc_fence_after();
      release();
      const uint64_t el2 = pair(el, el);
      // X is consumed (its P.X MMAs are complete): the 16-bit Y rows are staged in its slot
      const uint32_t ystage = sX + xi * kBlk, yrow = ystage + l * 128;
      auto load = [](uint32_t at, uint32_t (&v)[W]) {
        if constexpr (W == 8) tmem_ld8(at, v);
        else tmem_ld16(at, v);
      };
#pragma unroll 1
      for (int i = 0; i < P / W; ++i) {
        uint32_t o[W], o1[W], d[W], d1[W];
        load(tYo + tlane + W * i, o);
        load(tYd + tlane + W * i, d);
        if constexpr (kF16) {
          load(tYo + 64 + tlane + W * i, o1);
          load(tYd + 64 + tlane + W * i, d1);
        }
        tmem_ld_wait();
        if (i == P / W - 1) {
          tc_fence_before();
          warp_arrive(&m->bar_e);
        }
        uint32_t w[W / 2];
        uint32_t xw[W / 2], zw[W / 2];
        if constexpr (EPI) {
#pragma unroll
          for (int k = 0; k < W / 8; ++k) {
            const uint4 x = lds128(yrow + (((W / 8 * i + k) ^ swz) << 4));   // (X's row, still in the slot)
            xw[4 * k] = x.x; xw[4 * k + 1] = x.y; xw[4 * k + 2] = x.z; xw[4 * k + 3] = x.w;
            zw[4 * k] = zn[k].x; zw[4 * k + 1] = zn[k].y; zw[4 * k + 2] = zn[k].z; zw[4 * k + 3] = zn[k].w;
          }
          if (i + 1 < P / W) gate(i + 1);
        }
#pragma unroll
        for (int e = 0; e < W / 2; ++e) {
          uint64_t yo = pair(o[2 * e], o[2 * e + 1]), yd = pair(d[2 * e], d[2 * e + 1]);
          if constexpr (kF16) {
            yo = low_and_high<kUp>(pair(o1[2 * e], o1[2 * e + 1]), yo, 1.f);
            yd = low_and_high<kUp>(pair(d1[2 * e], d1[2 * e + 1]), yd, unit);
          }
          uint64_t y = fma_pair(yo, el2, yd);
          odd = fma_pair(y, zero2, odd);
          if constexpr (EPI) {
            const float2 x = unpack2<T16>(xw[e]);
            if (sp.D) y = fma_pair(pair(x.x, x.y), pair(skip, skip), y);
            if (gated) {
              const float2 z = unpack2<T16>(zw[e]);
              y = mul_pair(y, pair(__fdividef(z.x, 1.f + __expf(-z.x)), __fdividef(z.y, 1.f + __expf(-z.y))));
            }
          }
          w[e] = pack_pair<T16>(y);
        }
#pragma unroll
        for (int k = 0; k < W / 8; ++k)
          sts128(yrow + (((W / 8 * i + k) ^ swz) << 4), make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]));
      }
      fence_proxy_async();         // staged rows -> visible to the TMA engine
      __syncwarp();
      if (lane == 0) {
        // each warp hands its own 32 rows to the TMA engine; rows past the end of the sequence are clipped
        if (c.t0 + 32 * q < sp.seqlen) {
          tma_store_5d(&tmY, ystage + 32 * q * 128, 0, c.q, c.g, c.t0 + 32 * q, c.b, once);
          bulk_commit();
        }
        pending = (int)xi;
      }
      if (++xi == XS) xi = 0;
      ++ky;
    }
    release();
    if (lane == 0) bulk_wait_all();   // the Y rows this warp stored must have landed before the CTA exits
    const float2 o = unpair(odd);
    if (!(o.x == 0.f && o.y == 0.f)) m->bad = 1;
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    if (status) {
      if (m->tmem_base != 0) atomicCAS(status, 0, (int)STATUS_TMEM_ALLOC);
      if (m->abort_flag) atomicCAS(status, 0, (int)m->abort_flag);
    }
    sp.redo[blockIdx.x] = m->abort_flag ? 0 : m->bad;   // (an incomplete result stays one: the status says so)
  }
  if (warp == 0) {
    __syncwarp();
    grid_dependency_wait();   // (where no sequence of this CTA was cut)
    tmem_dealloc(m->tmem_base, 512);
  }
}

template <typename T16, int N, bool EPI, bool LB>
int launch_typed(const CUtensorMap& tx, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& ty, const TileParams& prm,
                 int grid, cudaStream_t stream) {
  auto kern = ssd_split_kernel<T16, N, EPI, LB>;
  constexpr int smem = LayoutS<N, std::is_same<T16, __half>::value ? 2 : 3>::kBytes;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return SSD_ERR_CUDA;
  return launch_tiles(kern, grid, kThreadsS, smem, prm.sp, stream, tx, tb, tc, ty, prm);
}

}  // namespace

bool split_supports(const SsdArgs& a) {
  const int64_t units = (int64_t)a.batch * a.nheads;
  return tc_supports(a) && units * ((a.seqlen + T - 1) / T) <= 0x7fffffffLL;
}

// Skip and gate in the kernel: where that saves a launch of some 3 us (and its 4 us of host time) and costs less.  A tile takes
// 3.2 us longer with them (its four read-out warps have no time to spare), the epilogue kernel 1.7 us per tile and SM:
// 256 tiles 20.1 us with them and 21.0 without, 24 of them 12.1 and 13.7; 640 64 and 55; 16 384 706 and 543.
bool split_fuses_epilogue(const SsdArgs& a) {
  return (int64_t)a.batch * a.nheads * ((a.seqlen + T - 1) / T) <= 2 * kSms;
}

int split_grid(const SsdArgs& a, int chain) {
  const int64_t units = (int64_t)a.batch * a.nheads, nt = (a.seqlen + T - 1) / T;
  return chain ? dealt_grid(units, (int)nt, chain) : (int)std::min<int64_t>(units, kSms);
}

int launch_split(const SsdArgs& a, const ScanParams& sp, cudaStream_t stream) {
  TileParams prm;
  prm.sp = sp;
  prm.ppg = a.nheads / a.ngroups;
  prm.upairs = prm.nitems = a.batch * a.nheads;
  prm.st32 = ((reinterpret_cast<uintptr_t>(sp.init) | reinterpret_cast<uintptr_t>(sp.fin)) & 31) == 0;
  CUtensorMap tx, tb, tc, ty;
  const int hpg = a.nheads / a.ngroups;
  if (!make_map(&tx, a.X, a, P, hpg, a.x_stride, T) || !make_map(&tb, a.B, a, a.dstate, 1, a.b_stride, T) ||
      !make_map(&tc, a.C, a, a.dstate, 1, a.c_stride, T) || !make_map(&ty, a.Y, a, P, hpg, a.y_stride, 32))
    return SSD_ERR_UNSUPPORTED;
  const int grid = split_grid(a, sp.chain);
  auto go = [&](auto epilogue, auto look_back) {
    constexpr bool E = decltype(epilogue)::value, LB = decltype(look_back)::value;
    if (a.dtype == SSD_DTYPE_F16)
      return a.dstate == 128 ? launch_typed<__half, 128, E, LB>(tx, tb, tc, ty, prm, grid, stream)
                             : launch_typed<__half, 64, E, LB>(tx, tb, tc, ty, prm, grid, stream);
    return a.dstate == 128 ? launch_typed<__nv_bfloat16, 128, E, LB>(tx, tb, tc, ty, prm, grid, stream)
                           : launch_typed<__nv_bfloat16, 64, E, LB>(tx, tb, tc, ty, prm, grid, stream);
  };
  const bool epi = sp.D || sp.Z;
  if (sp.chain == 2) return epi ? go(std::true_type{}, std::true_type{}) : go(std::false_type{}, std::true_type{});
  return epi ? go(std::true_type{}, std::false_type{}) : go(std::false_type{}, std::false_type{});
}

}  // namespace ssd
