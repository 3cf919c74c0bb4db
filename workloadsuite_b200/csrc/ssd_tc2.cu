// Tensor-core SSD forward for sm_100a: one persistent CTA per SM walks work items (a run of 128-token tiles of one
// sequence of two heads) as one unbroken pipeline of tiles.
//
// The two heads of a pair read the same B and C (model_ref.py:97-99), so B, C and G = C.B^T (model_ref.py:143) are
// loaded and computed once per tile and shared, and S = B^T.[Xd0|Xd1] and C.[H0|H1] are single N = 128 MMAs.  A group
// with an odd number of heads leaves the second half of its last pair empty (zeros in, nothing out).
//
// Roles (512 threads):
//   warp 0        TMA producer
//   warp 1        MMA issuer: P.X(t) per head, then S(t+1), G(t+1), C.H(t+1)
//   warps 2, 3    prefix sum of the log-decay (model_ref.py:135) and every factor derived from it, one head each, up to
//                 four tiles ahead; the other roles read the factors from shared memory
//   warps 4-7     head 0, warps 8-11 head 1: thread = tile row = TMEM lane.  Per iteration, in this order:
//     A. P(t)   = G o exp(segsum) o causal  (:139-145)  -> TMEM, the A operand of Yd = P.X
//     D. 16-bit copy of the state entering tile t+1     -> shared memory -> Yo = C.H   (:160-161)
//     E. H <- exp(cs_last) H + S(t+1)       (:150,156)  in fp32 registers
//   warps 12-15   both heads, in this order (with skip and gate B is a step between A and D of the warps above, which then
//                 wait for this group):
//     B. Xd(t+1) = exp(cs_last - cs) x~     (:144,148)  -> shared memory -> S = B^T.Xd
//     Y(t) = Yd + exp(cs) Yo (:162) [+ skip and gate, :116-118] -> shared memory -> TMA store
//
// What bounds it.  A 128xNx16 tcgen05.mma takes 62 cycles at N = 128 and 55 at N = 64 (any operand layout), so the
// four contractions of a tile pair need 2 430 tensor-pipe cycles; HBM needs 2 800 cycles per SM for its 64 KB of X
// and Y.  The loop that sets the period is A -> P.X -> S -> E -> A, which is
// why Xd has other warps than P (a tile takes 5 200 to 5 500 cycles).  Tensor memory (512 columns) is what limits overlap: G 128,
// Yo 128, Yd 128 and 128 columns that S and P take turns in -- S(t+1) is consumed (step E) before P(t+1) is written
// (step A), and S(t+1) is issued once P.X(t) has read P(t).  Keeping Yo and Yd apart means that nothing has to be
// scaled in place between C.H and P.X, and that C.H(t+1) and the reloads of B and C run under steps A, B and D.
// All waits are bounded.
#include <cuda.h>

#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "ssd_common.cuh"
#include "tc_common.cuh"
#include "tc_ptx.cuh"
#include "tile_walk.cuh"

namespace ssd {
namespace {

using namespace ptx;
using namespace tc;

constexpr int kThreads2 = 512;

template <int N>
struct Layout2 {
  static constexpr int NB = N / 64;
  // B and C tiles in flight, and X tiles (one head each) in flight; an X slot whose tile is consumed doubles as the Y
  // staging buffer.  n = 64 leaves room for more of both.
  static constexpr int kBC = N == 128 ? 1 : 2;
  static constexpr int kXSlots = N == 128 ? 5 : 6;
  static constexpr int oB = 0;                           // [stage]
  static constexpr int oC = oB + kBC * NB * kBlk;        // [stage]
  static constexpr int oX = oC + kBC * NB * kBlk;        // [slot]
  static constexpr int oXd = oX + kXSlots * kBlk;        // [head]
  static constexpr int oH = oXd + 2 * kBlk;              // [head], N rows of 128 B
  static constexpr int oMisc = oH + 2 * N * 128;
  static constexpr int kMiscBytes = 16384;
  static constexpr int kBytes = oMisc + kMiscBytes;   // no slack: the dynamic segment must start 1024-byte aligned
};

// Factors of one tile of one head, written by the prefix-sum warp.
struct alignas(16) Factors {
  float cs2[T];       // cs * log2(e)
  float cf[T];        // exp(cs at the end of the row's 32-block - cs of the row) * dt: the row's factor as a column of P
  float dg[T];        // diagonal blocks: at columns 4i cs * log2(e) - log2(dt), at the three after it the ratio to the column before;
                      // dt in steep groups of four
  float tot;          // cs_last
  float ld;           // sum of the log-decays as given
  uint32_t steep;     // groups of four columns in which the factors of P span more than the ratios can carry
};

constexpr int kFactors = 4;   // tiles that the prefix sums may be ahead
constexpr int kReadBit = 8;   // of a ready flag: from there on it counts the warps that have read what enters their piece

// Log-decays below this count as this in the prefix sums: e^-104 is 2^-150, a factor of zero either way, while -inf (a
// reset) would make every difference of sums after it NaN, and a very large one would take their digits.
constexpr float kLowest = -104.f;
// A group of four columns of a diagonal block is steep if its ratios go through more than 2^40, or a dt is no ordinary positive
// number: the ratios start from the group's first column, and where that one underflows (2^-126) the three after it would
// be lost with it -- the diagonal, of factor dt, too.  So what is lost in the others is below 2^-86.
constexpr float kSteep = 40.f, kLeastLogDt = -60.f;

// What the MMA issuer does for one kind of product (see there).  `a` and `b` are the low words of the shared-memory
// descriptors (`a` a tensor-memory address for P.X), advanced by a_in / b_in per k-step and by a_out / b_out per four;
// the barriers are byte offsets within Misc2 (0: none).
struct alignas(16) Op {
  uint32_t a, b, id;
  uint16_t d, steps;
  uint16_t a_in, b_in, a_out, b_out;
  uint16_t wait0, wait1, commit0, commit1;
};
enum { kOpS, kOpG, kOpCH, kOpPX0, kOpPX1, kOps };

struct Misc2 {
  Work work;
  Op ops[2][kOps];                    // [tile parity] (the stage of B and C)
  uint4 causal[17][2];                // the first j of 16 columns kept, as masks of 16-bit pairs
  Factors f[2][kFactors];             // [head][tile ordinal % kFactors]
  uint64_t full_b[2], full_c[2], empty_b[2], empty_c[2];   // [stage]
  uint64_t full_x[6], empty_x[6];
  uint64_t full_f[2][kFactors], empty_f[2][kFactors];
  uint64_t bar_g, bar_s, bar_ch, bar_y[2];   // tcgen05.commit arrivals (S and C.H serve both heads at once)
  uint64_t bar_h, bar_e, bar_u;       // one arrival per warp and head (8); bar_u: S of a state-only tile is consumed
  uint64_t bar_xd;                    // one arrival per warp that makes Xd (4 of the read-out group; EPI: 8)
  uint64_t bar_p[2];                  // one arrival per warp of the head (4)
  uint64_t bar_drain;                 // all MMAs issued have completed
  uint32_t tmem_base;
  long long wait_clocks;     // bound of every wait (SM clock cycles)
  volatile int abort_flag;   // 0, or the status code of the first wait that gave up (every role then leaves)
  Look<2> look;
  float asum1[2];                 // log-decay of the piece that item 1 ended
};

static_assert(sizeof(Misc2) <= Layout2<128>::kMiscBytes, "Misc2 outgrew its shared-memory slot");
static_assert(Layout2<128>::kBytes <= 232448 && Layout2<64>::kBytes <= 232448, "shared memory budget of one SM exceeded");

// B. Xd = exp(cs_last - cs_l) * dt * x (model_ref.py:144,148) of rows 32 q .. 32 q + 31, in packed 16-bit arithmetic as the
// reference does it (WIDE: in fp32, rounded once).  Eight lanes share a row (one 16-byte piece each), a warp moves four rows
// per instruction.
template <typename T16, bool WIDE>
__device__ __forceinline__ void make_xd(uint32_t xb, uint32_t xd, const Factors& f, int q, int lane) {
  uint32_t r = 32 * q + ((uint32_t)lane >> 3);
  const uint32_t pc = (uint32_t)lane & 7u;
  const float g = ex2((f.tot * kLog2e) - f.cs2[32 * q + 31]);   // (cf goes as far as the end of the 32-row block)
#pragma unroll 1
  for (int i = 0; i < 2; ++i, r += 16) {
    uint4 a[4];
    float sc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = lds128(xb + (r + 4 * k) * 128 + ((pc ^ ((r + 4 * k) & 7u)) << 4));
      sc[k] = f.cf[r + 4 * k] * g;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint4 v;
      if constexpr (WIDE) {
        const uint64_t d = pair(sc[k], sc[k]);
        auto times = [&](uint32_t x) {
          const float2 xf = unpack2<T16>(x);
          return pack_pair<T16>(mul_pair(pair(xf.x, xf.y), d));
        };
        v.x = times(a[k].x); v.y = times(a[k].y); v.z = times(a[k].z); v.w = times(a[k].w);
      } else {
        const uint32_t d = pack2<T16>(sc[k], sc[k]);
        v.x = mul2<T16>(a[k].x, d); v.y = mul2<T16>(a[k].y, d); v.z = mul2<T16>(a[k].z, d); v.w = mul2<T16>(a[k].w, d);
      }
      sts128(xd + (r + 4 * k) * 128 + ((pc ^ ((r + 4 * k) & 7u)) << 4), v);
    }
  }
}

__device__ __forceinline__ int32_t* walk_bits(const ScanParams& sp) { return sp.chain_flag + 2 * kSms; }

// EPI: apply the skip and gate of model_ref.py:116-118 to Y on its way out (sp.D / sp.Z; either may be null).
// WIDE: Xd in fp32 arithmetic.  Groups with an odd number of heads have always had it so (bf16, final state against 64 bits:
// 1.65e-3, with the packed products 2.23e-3); those with an even number have the reference's packed products.
// LB: an instance for sequences cut in look-back mode (sp.chain == 2), as what a piece's beginning takes costs the walk of the others
// (see CursorOf).  The others keep their checks of sp.chain == 2, never true there: without them the compiler's registers spill 24 to 60
// bytes (8 x 2048 tokens of 24 heads 52.1 -> 55.3 us).
// (2: the final states lie on the initial ones; what that takes costs the others 0.5 to 1 us.)
template <typename T16, int N, bool EPI, bool WIDE, int LB>
__global__ void __launch_bounds__(kThreads2, 1)
ssd_tc2_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmY,
               const TileParams prm) {
  using L = Layout2<N>;
  using Cursor = CursorOf<2, (LB > 0)>;
  constexpr bool kCarry = LB == 2;
  constexpr int NB = L::NB;
  constexpr int KN = N / 16;
  constexpr int KT = T / 16;
  constexpr int BC = L::kBC;
  constexpr int XS = L::kXSlots;
  // State-only tiles of the look-back scan: C, the state's copy and their barriers are idle, so every other tile has its B and Xd there.
  // Nothing then waits for the MMA of the tile before but the accumulator (1 x 32 768 tokens of 24 and 64 heads 116 -> 112.5 and 271 -> 261 us).
  constexpr bool kTwo = LB && N == 128 && !EPI;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  Misc2* m = reinterpret_cast<Misc2*>(smem + L::oMisc);
  const ScanParams& sp = prm.sp;
  if (smem_u32(smem) & 1023u) {   // the 128-byte swizzle needs 1024-byte aligned tiles; give up cleanly otherwise
    if (threadIdx.x == 0 && sp.status) atomicCAS(sp.status, 0, (int)STATUS_BAD_SMEM_ALIGNMENT);
    return;
  }
  // (fault injection for the tests of the give-up path: the first CTA of a chained launch never publishes its
  //  hand-over, so the CTA that continues its sequence runs into the bound of its wait)
  if (sp.inject_lost_handover && sp.chain && blockIdx.x == 0) return;
  if constexpr (LB == 1) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (sp.walk_again) {
      grid_dependency_wait();
      if (!(walk_bits(sp)[blockIdx.x / 32] >> blockIdx.x % 32 & 1)) return;
    }
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int32_t* status = sp.status;

  if (tid == 0) {
    for (int s = 0; s < BC; ++s) {
      mbar_init(&m->full_b[s], 1); mbar_init(&m->full_c[s], 1);
      mbar_init(&m->empty_b[s], 1); mbar_init(&m->empty_c[s], 1);
    }
    // an X slot is handed back by four warps: those that read out Y from it, or those that made Xd of a state-only tile
    for (int s = 0; s < XS; ++s) { mbar_init(&m->full_x[s], 1); mbar_init(&m->empty_x[s], 4); }
    mbar_init(&m->bar_g, 1); mbar_init(&m->bar_s, 1); mbar_init(&m->bar_ch, 1);
    mbar_init(&m->bar_xd, EPI ? 8 : 4); mbar_init(&m->bar_h, 8); mbar_init(&m->bar_e, 8); mbar_init(&m->bar_u, 8);
    for (int h = 0; h < 2; ++h) {
      mbar_init(&m->bar_y[h], 1);
      mbar_init(&m->bar_p[h], 4);
      // factors are released by the head's four warps (P) and the four read-out warps
      for (int s = 0; s < kFactors; ++s) { mbar_init(&m->full_f[h][s], 1); mbar_init(&m->empty_f[h][s], 8); }
    }
    mbar_init(&m->bar_drain, 1);
    m->abort_flag = 0;
    m->wait_clocks = sp.wait_clocks;
    work_list(prm, m->work);
    if (LB == 1 && sp.walk_again) {   // one item: the piece, from the state that enters it
      m->work.again = m->work.npre = 0;
      m->work.total = m->work.hi - m->work.lo;
    }
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&m->tmem_base, 512);
  if (warp == 1 && lane < 17) {
    uint32_t k[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) k[e] = (2 * e < lane ? 0xffffu : 0u) | (2 * e + 1 < lane ? 0xffff0000u : 0u);
    m->causal[lane][0] = make_uint4(k[0], k[1], k[2], k[3]);
    m->causal[lane][1] = make_uint4(k[4], k[5], k[6], k[7]);
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (LB > 0) {   // (never with sp.fin_on_init; without the call kCarry's registers spill: 1 x 131 072 tokens of 32 heads 597 us, 510 so)
    if (!sp.walk_again) find_beginning<2>(prm, m->work, m->look, kThreads2 / 32);
    __syncthreads();
  }
  tc_fence_after();
  constexpr uint32_t tG = 0, tSP = 128, tYo = 256, tYd = 384;   // (all 512 columns are ours: the allocation starts at 0)
  const uint32_t sB = smem_u32(smem + L::oB), sC = smem_u32(smem + L::oC), sX = smem_u32(smem + L::oX);
  const uint32_t sXd = smem_u32(smem + L::oXd), sH = smem_u32(smem + L::oH);
  const Work& wk = m->work;
  const uint32_t total = m->tmem_base == 0 ? (uint32_t)wk.total : 0u, npre = (uint32_t)wk.npre;
  // One arrival per warp: every lane has issued its fences, the warp barrier orders their writes before
  // lane 0's arrive (128 per-thread arrivals on one mbarrier cost several hundred cycles per hand-off).
  auto warp_arrive = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  // Registers: 128 x 512 at launch, re-divided 64 | 168 | 168 | 112 (the sum may not exceed what was launched).
  if (warp < 4) {
    setmaxnreg_dec<64>();
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------------- TMA producer
      // X is read once; B and C again by every other pair of heads of the group, perhaps much later (where a CTA works on one
      // pair after the other, or the pairs' CTAs are at different places of the sequence)
      const uint64_t once = policy_evict_first(), again = policy_evict_last();
      prefetch_tmap(&tmX); prefetch_tmap(&tmB); prefetch_tmap(&tmC); prefetch_tmap(&tmY);
      bool ok = true;
      uint32_t xi = 0, xph = 0;              // next X slot and how often the ring has been walked (parity)
      uint32_t bs = 0, bph = 0, cs = 0, cph = 0;   // the same for B and C
      Cursor c;
#pragma unroll 1
      for (uint32_t n = 0; n < total && ok; ++n) {
        c.next(prm, wk);
        // X of both heads, B, then C (not for a state-only tile).  B before C: the B tile is free earlier, and the S MMA
        // that waits for it is on the state's chain.
#pragma unroll 1
        for (int k = 0; k < (n < npre ? 3 : 4); ++k) {
          const CUtensorMap* tm = k < 2 ? &tmX : k == 2 ? &tmB : &tmC;
          const bool to_b = k == 2 && !(kTwo && n < npre && (n & 1));
          uint64_t* full = k < 2 ? &m->full_x[xi] : to_b ? &m->full_b[bs] : &m->full_c[cs];
          uint64_t* empty = k < 2 ? &m->empty_x[xi] : to_b ? &m->empty_b[bs] : &m->empty_c[cs];
          const uint32_t ph = k < 2 ? xph : to_b ? bph : cph;
          uint32_t dst = k < 2 ? sX + xi * kBlk : to_b ? sB + bs * (NB * kBlk) : sC + cs * (NB * kBlk);
          const int blocks = k < 2 ? 1 : NB;
          ok = guarded_wait(empty, ph ^ 1, m, STATUS_WAIT_TIMEOUT_MMA);
          if (!ok) break;
          mbar_expect_tx(full, blocks * kBlk);
#pragma unroll 1
          for (int kb = 0; kb < blocks; ++kb, dst += kBlk)
            tma_load_5d(dst, tm, full, 64 * kb, k < 2 ? 2 * c.q + k : 0, c.g, c.t0, c.b, k < 2 ? once : again);
          if (k < 2) {
            if (++xi == XS) { xi = 0; xph ^= 1; }
          } else if (to_b) {
            if (++bs == BC) { bs = 0; bph ^= 1; }
          } else {
            if (++cs == BC) { cs = 0; cph ^= 1; }
          }
        }
      }
      if (ok) ok = guarded_wait(&m->bar_drain, 0, m, STATUS_WAIT_TIMEOUT_SYNC);   // (every MMA of the CTA: keeps the clock to the end)
      if (!ok) {
        // let copies already in flight land before the CTA gives its shared memory back (a millisecond)
        const long long c0 = clock64();
        while (clock64() - c0 < 2000000LL) { }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer (one elected thread issues)
      // Per tile S <- B^T.Xd, into the columns that P of the tile before was read from; for a tile that produces Y then
      // G <- C.B^T (both heads have read G of the tile before: their P is done), Yo <- C.H (both heads' Yo and Yd of the
      // tile before have been read out) and Yd <- P.X per head.  One copy of the code, driven by a table: a copy per kind
      // is 2 KB more of the instruction cache (the 2.7B layer's shape 272 -> 257 us; with one MMA per step of the loop
      // instead of four it is slower again).
      constexpr uint64_t kDescHi = umma_desc_base(0, 1024);
      constexpr uint32_t kMN = kBlk >> 4;
      const uint32_t npar = npre & 1, mb = smem_u32(m);
      if (lane < 2 * kOps) {
        constexpr int fmt = std::is_same<T16, __nv_bfloat16>::value ? 1 : 0;
        constexpr uint32_t kK = 1, kMNh = N * 128 >> 4;
        constexpr uint16_t kKi = 32 >> 4, kKo = kBlk >> 4, kMi = 2048 >> 4, kMo = 8192 >> 4;
        const uint32_t par = lane >= kOps, o = lane - (par ? kOps : 0);
        const uint32_t sb = par % BC, sc = ((par + npar) & 1) % BC;
        const uint32_t aB = (sB + sb * (NB * kBlk)) >> 4, aC = (sC + sc * (NB * kBlk)) >> 4;
        auto at = [&](const void* bar) { return (uint16_t)(smem_u32(bar) - mb); };
        Op op = {};
        if (o == kOpS) {
          op = {kMN << 16 | aB, kMN << 16 | sXd >> 4, umma_idesc(128, 128, fmt, 1, 1), (uint16_t)tSP, KT, kMi, kMi, kMo, kMo,
                at(&m->bar_xd), at(&m->bar_y[1]), at(&m->bar_s), at(&m->empty_b[sb])};
        } else if (o == kOpG) {
          op = {kK << 16 | aC, kK << 16 | aB, umma_idesc(128, 128, fmt, 0, 0), (uint16_t)tG, KN, kKi, kKi, kKo, kKo,
                at(&m->full_c[sc]), 0, at(&m->bar_g), at(&m->empty_b[sb])};
        } else if (o == kOpCH) {
          op = {kK << 16 | aC, kMNh << 16 | sH >> 4, umma_idesc(128, 128, fmt, 0, 1), (uint16_t)tYo, KN, kKi, kMi, kKo, kMo,
                at(&m->bar_h), at(&m->bar_e), at(&m->bar_ch), at(&m->empty_c[sc])};
        } else {
          const uint32_t h = o - kOpPX0;
          op = {tSP + 64 * h, kMN << 16 | sX >> 4, umma_idesc(128, 64, fmt, 0, 1), (uint16_t)(tYd + 64 * h), KT, 8, kMi, 32, kMo,
                at(&m->bar_p[h]), 0, at(&m->bar_y[h]), 0};
        }
        m->ops[par][o] = op;
      }
      __syncwarp();
      uint32_t xb = 0;                 // X slot of the tile, as a descriptor offset
#pragma unroll 1
      for (uint32_t n = 0; n < total; ++n) {
        const uint32_t py = n + npar;  // (its parity is that of the ordinal among the tiles that produce Y)
#pragma unroll 1
        for (int o = 0; o < kOps; ++o) {
          const uint4* op = reinterpret_cast<const uint4*>(&m->ops[n & 1][o]);
          uint4 lo = op[0];
          const uint4 hi = op[1];
          // S: Xd is there (and B: waited for by the warps that made Xd); P.X of the tile before is done (its commit for
          // head 1 covers head 0), or S of the state-only tile before has been consumed.
          // G: C.  C.H: the state copy; the read-out.  P.X: P (X is there: Xd was made of it).
          uint32_t w1 = hi.z >> 16, c1 = hi.w >> 16, p0 = py, p1 = py + 1;
          if (o == kOpS) {
            p0 = n;
            if (n <= npre) {
              w1 = n > 0 ? (uint32_t)offsetof(Misc2, bar_u) : 0u;
              p1 = n + 1;
            }
            if (n >= npre) {
              c1 = 0;
            } else if (kTwo && (n & 1)) {
              lo.x += (sC - sB) >> 4;
              lo.y += (sH - sXd) >> 4;
              c1 += (uint32_t)(offsetof(Misc2, empty_c) - offsetof(Misc2, empty_b));
            }
          }
          if (o == kOpG) p0 = kTwo ? (npre >> 1) + n - npre : (n - npre) / BC;
          wait_at(mb + (hi.z & 0xffffu), p0 & 1, m);
          if (w1) wait_at(mb + w1, p1 & 1, m);
          tc_fence_after();
          const uint32_t x = o >= kOpPX0 ? xb : 0;
          if (elect_one()) {
            uint32_t a = lo.x, b = lo.y + x, acc = 0;
            const uint32_t d = lo.w & 0xffffu, ai = hi.x & 0xffffu, bi = hi.x >> 16, ao = hi.y & 0xffffu, bo = hi.y >> 16;
            const uint32_t id = lo.z;
#pragma unroll 1
            for (uint32_t k = 0; k < lo.w >> 16; k += 4) {
              if (o < kOpPX0) {
                umma_ss(d, kDescHi | a, kDescHi | b, id, acc);
#pragma unroll
                for (int i = 1; i < 4; ++i) umma_ss(d, kDescHi | (a + i * ai), kDescHi | (b + i * bi), id, 1);
              } else {
                umma_ts(d, a, kDescHi | b, id, acc);
#pragma unroll
                for (int i = 1; i < 4; ++i) umma_ts(d, a + 8 * i, kDescHi | (b + i * (2048 >> 4)), id, 1);
              }
              a += ao; b += bo;
              acc = 1;
            }
            umma_commit_at(mb + (hi.w & 0xffffu));
            if (c1) umma_commit_at(mb + c1);
          }
          if (n < npre) break;
          if (o >= kOpPX0) xb = xb == (XS - 1) * kMN ? 0 : xb + kMN;
        }
        if (n < npre) xb = xb >= (XS - 2) * kMN ? xb - (XS - 2) * kMN : xb + 2 * kMN;
      }
      // Tensor memory is freed at the end of the kernel: the MMAs issued here must have completed by then (bounded).
      if (elect_one()) {
        umma_commit(&m->bar_drain);
        const long long t0 = clock64();
        while (!mbar_try_wait(&m->bar_drain, 0))
          if (clock64() - t0 > m->wait_clocks) break;
      }
      __syncwarp();
    } else if (warp >= 2) {
      // ---------------------------------------------------------------- prefix sums (warp 2: head 0, warp 3: head 1)
      // Lane i owns tokens 4i .. 4i+3; nothing is fetched for the tile after (this warp is ahead as it is).
      const int h = warp - 2;
      const int64_t as1 = sp.as[1], ds1 = sp.dts[1], asT = T * as1, dsT = T * ds1;
      const float* Ag = nullptr;
      const T16* Dg = nullptr;
      Cursor c;
#pragma unroll 1
      for (uint32_t n = 0; n < total; ++n) {
        c.next(prm, wk);
        if (__builtin_expect(c.first_tile(), 0)) {              // (later tiles of the item: where the last one ended)
          const int head = c.head(wk) + h, t = c.t0 + 4 * lane;
          Ag = sp.A + c.b * sp.as[0] + head * sp.as[2] + t * sp.as[1];
          Dg = static_cast<const T16*>(sp.dt) + c.b * sp.dts[0] + head * sp.dts[2] + t * sp.dts[1];
          // this warp is the first to know of an item: the state that enters it goes to L2
          if (sp.init && c.live(wk, h) && c.t_begin == 0) {
            const float* I = sp.init + ((int64_t)c.b * sp.nheads + head) * sp.init_unit_stride + c.seg * sp.init_seg_stride;
            for (int e = lane; e < N * P / 32; e += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(I + 32 * e));
          }
        }
        float a[4], dt[4] = {1.f, 1.f, 1.f, 1.f};
        if (__builtin_expect(c.t0 + T <= sp.seqlen && c.live(wk, h), 1)) {
          const float* p1 = Ag + as1;
          const float* p2 = p1 + as1;
          a[0] = *Ag; a[1] = *p1; a[2] = *p2; a[3] = p2[as1];
          if (sp.dt) {
            const T16* q1 = Dg + ds1;
            const T16* q2 = q1 + ds1;
            dt[0] = Cvt<T16>::to_f(*Dg); dt[1] = Cvt<T16>::to_f(*q1); dt[2] = Cvt<T16>::to_f(*q2); dt[3] = Cvt<T16>::to_f(q2[ds1]);
          }
        } else {
          const int in = c.live(wk, h) ? sp.seqlen - c.t0 - 4 * lane : 0;   // past the end: decay 1 and x = 0, the state stays as it is
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            a[e] = e < in ? Ag[e * as1] : 0.f;
            if (e < in && sp.dt) dt[e] = Cvt<T16>::to_f(Dg[e * ds1]);
          }
        }
        Ag += asT;
        Dg += dsT;
        float cs = a[0] + a[1] + a[2] + a[3], ld = cs;
        const bool low = __any_sync(0xffffffffu, fminf(fminf(a[0], a[1]), fminf(a[2], a[3])) < kLowest) != 0;
        if (__builtin_expect(low, 0)) {
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] = a[e] < kLowest ? kLowest : a[e];   // (NaN stays NaN)
          cs = a[0] + a[1] + a[2] + a[3];
#pragma unroll 1
          for (int d = 16; d >= 1; d >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, d);
        }
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const float t = __shfl_up_sync(0xffffffffu, cs, d);
          if (lane >= d) cs += t;
        }
        float c2[4];                                       // cs * log2(e)
        {
          float r = __shfl_up_sync(0xffffffffu, cs, 1);
          if (lane == 0) r = 0.f;
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            r += a[e];
            c2[e] = r * kLog2e;
          }
          c2[3] = cs * kLog2e;
        }
        const float ce = __shfl_sync(0xffffffffu, c2[3], lane | 7);   // at the end of the 32-token block
        const uint32_t slot = n % kFactors;
        wait(&m->empty_f[h][slot], ((n / kFactors) & 1) ^ 1, m);
        Factors& f = m->f[h][slot];
        reinterpret_cast<float4*>(f.cs2)[lane] = make_float4(c2[0], c2[1], c2[2], c2[3]);
        float cf[4], cc[4];
        float least = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          cf[e] = ex2(ce - c2[e]) * dt[e];
          // dt multiplies the columns of P instead of the rows of X (P.(dt o x) = (P o dt_s).x), so the X tile stays as
          // loaded.  The ratios are clamped: one above the diagonal may overflow, it is masked out.
          const float lg = lg2(dt[e]);                     // (lg2(1) is 0)
          least = fminf(least, lg);
          cc[e] = c2[e] - lg;
        }
        const float r0 = cc[0] - cc[1], r1 = cc[1] - cc[2], r2 = cc[2] - cc[3];
        const bool steep = !(fabsf(r0) + fabsf(r1) + fabsf(r2) <= kSteep && least > kLeastLogDt);   // (NaN: dt < 0, or dt = 0 throughout)
        const uint32_t all_steep = __ballot_sync(0xffffffffu, steep);
        float4 dg = make_float4(cc[0], ex2(fminf(r0, 126.f)), ex2(fminf(r1, 126.f)), ex2(fminf(r2, 126.f)));
        if (steep) dg = make_float4(dt[0], dt[1], dt[2], dt[3]);
        if (lane == 31) {
          f.tot = cs;
          f.ld = low ? ld : cs;
          f.steep = all_steep;
        }
        reinterpret_cast<float4*>(f.cf)[lane] = make_float4(cf[0], cf[1], cf[2], cf[3]);
        reinterpret_cast<float4*>(f.dg)[lane] = dg;
        warp_arrive(&m->full_f[h][slot]);
      }
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ warps 4-7: head 0, 8-11: head 1
    setmaxnreg_inc<168>();
    const int h = (warp - 4) >> 2;
    const int q = warp & 3;
    const int lane_base = q * 32;
    const int l = lane_base + lane;
    const uint32_t tlane = (uint32_t)lane_base << 16;
    const uint32_t swz = (uint32_t)(l & 7);
    const bool owns_state = lane_base < N;
    const uint32_t tS = tSP + 64 * h, tP = tSP + 64 * h;
    const uint32_t sHh = sH + h * (N * 128);

    uint64_t H[P / 2];               // fp32 pairs
#pragma unroll
    for (int e = 0; e < P / 2; ++e) H[e] = 0;
    float asum0 = 0.f;               // log-decay summed over the earlier pieces of the sequence
    float asum = 0.f, acomp = 0.f;   // compensated (Kahan) sum of the tile totals; FP64 is slow on this part

    // A. P = (C B^T) o exp(segsum), causal -> TMEM (A operand, 16-bit pairs).  Decay mask per 32-token column block J of
    // this warp's 32 rows (block q is the diagonal one):
    //   J == q: exp2(cs_l - cs_s), causal, one ex2 per four columns and the ratios between neighbours (steep groups: one ex2 per
    //           column, in a second pass);
    //   J <  q: exp(cs_l - cs_s) = rf_J[l] * cf[s] with both factors <= 1 for non-positive log-decays
    //           (rf_J[l] = exp(cs_l - cs_end(J)), cf[s] = exp(cs_end(J) - cs_s)): two multiplies;
    //   J >  q: zero.
    auto make_p = [&](const Factors& f) {
      const float cs2 = f.cs2[l];
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t g[16];
        tmem_ld16(tG + tlane + 32 * q + 16 * half, g);
        const float4* dv = reinterpret_cast<const float4*>(&f.dg[32 * q + 16 * half]);
        const uint4* keep = m->causal[max(0, min(16, lane - 16 * half + 1))];
        tmem_ld_wait();
        uint32_t pk[8];
#pragma unroll
        for (int e4 = 0; e4 < 4; ++e4) {
          const float4 d = dv[e4];
          const float w0 = ex2(cs2 - d.x), w1 = w0 * d.y, w2 = w1 * d.z, w3 = w2 * d.w;
          const float v0 = __uint_as_float(g[4 * e4]) * w0, v1 = __uint_as_float(g[4 * e4 + 1]) * w1;
          const float v2 = __uint_as_float(g[4 * e4 + 2]) * w2, v3 = __uint_as_float(g[4 * e4 + 3]) * w3;
          pk[2 * e4] = pack2<T16>(v0, v1);
          pk[2 * e4 + 1] = pack2<T16>(v2, v3);
        }
        const uint4 k0 = keep[0], k1 = keep[1];
        pk[0] &= k0.x; pk[1] &= k0.y; pk[2] &= k0.z; pk[3] &= k0.w;
        pk[4] &= k1.x; pk[5] &= k1.y; pk[6] &= k1.z; pk[7] &= k1.w;
        tmem_st8(tP + tlane + 16 * q + 8 * half, pk);
      }
#pragma unroll 1
      for (int J = 0; J < q; ++J) {   // strictly below the diagonal
        uint32_t g[32];
        tmem_ld32(tG + tlane + 32 * J, g);
        const float rf = ex2(cs2 - f.cs2[32 * J + 31]);
        const uint64_t rf2 = pair(rf, rf);
        const ulonglong2* fv = reinterpret_cast<const ulonglong2*>(&f.cf[32 * J]);
        tmem_ld_wait();
        uint32_t pk[16];
#pragma unroll
        for (int e4 = 0; e4 < 8; ++e4) {
          const ulonglong2 c = fv[e4];
          pk[2 * e4] = pack_pair<T16>(mul_pair(pair(g[4 * e4], g[4 * e4 + 1]), mul_pair(rf2, c.x)));
          pk[2 * e4 + 1] = pack_pair<T16>(mul_pair(pair(g[4 * e4 + 2], g[4 * e4 + 3]), mul_pair(rf2, c.y)));
        }
        tmem_st16(tP + tlane + 16 * J, pk);
      }
      const uint32_t steep = f.steep >> (8 * q) & 255u;
      if (__builtin_expect(steep != 0, 0)) {   // steep groups of the diagonal block, over what the ratios made of them
        tmem_st_wait();
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
          if (!(steep >> i & 1)) continue;
          uint32_t g[4];
          tmem_ld4(tG + tlane + 32 * q + 4 * i, g);
          const float4 d = reinterpret_cast<const float4*>(f.dg)[8 * q + i], c = reinterpret_cast<const float4*>(f.cs2)[8 * q + i];
          const float w[4] = {ex2(cs2 - c.x) * d.x, ex2(cs2 - c.y) * d.y, ex2(cs2 - c.z) * d.z, ex2(cs2 - c.w) * d.w};
          tmem_ld_wait();
          float v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = 4 * i + e <= lane ? __uint_as_float(g[e]) * w[e] : 0.f;
          tmem_st2(tP + tlane + 16 * q + 2 * i, pack2<T16>(v[0], v[1]), pack2<T16>(v[2], v[3]));
        }
      }
      if (q < 3) {
        uint32_t pz[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) pz[e] = 0u;
#pragma unroll 1
        for (int J = q + 1; J < 4; ++J) tmem_st16(tP + tlane + 16 * J, pz);
      }
    };
    auto store_hb = [&]() {
      if (owns_state) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4 v;
          v.x = pack_pair<T16>(H[4 * c]); v.y = pack_pair<T16>(H[4 * c + 1]);
          v.z = pack_pair<T16>(H[4 * c + 2]); v.w = pack_pair<T16>(H[4 * c + 3]);
          sts128(sHh + l * 128 + ((c ^ swz) << 4), v);
        }
      }
    };
    // (bounded) wait until the four warps of head h of CTAs `from` .. `to` have published, a CTA per lane (`read`: have read the state
    // that enters their piece, see settle()).  Every warp asks for itself: a barrier among the four would hang where one of them has given up.
    auto wait_published = [&](int to, int from, bool read = false) {
      grid_dependency_wait();
      const long long c0 = clock64();
      for (int c = to - lane; c >= from && !m->abort_flag; c -= 32) {
        while (true) {
          int f;
          asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(f) : "l"(sp.chain_flag + 2 * c + h) : "memory");
          if ((kCarry && read ? f >> kReadBit : kCarry ? f & ((1 << kReadBit) - 1) : f) >= 4 || m->abort_flag) break;
          if (clock64() - c0 > m->wait_clocks) {
            m->abort_flag = (int)STATUS_WAIT_TIMEOUT_CHAIN;
            break;
          }
        }
      }
      __syncwarp();
    };
    // The state entering an item: zero or the caller's, unless the item continues a sequence that another CTA works on.
    // Called as soon as the state of the item before has left, so that the loads are in flight during step A.
    Cursor c;
    bool fold = false;               // the state entering comes (also) from other CTAs: fold_item() before it is used
    auto enter_item = [&](bool wy) {
      if (c.goes_on(wk)) return;
      asum0 = asum = acomp = 0.f;
      const bool from_zero = sp.chain == 2 && !wy;               // (the look-back scan)
      fold = sp.chain && !from_zero && (c.t_begin > 0 || kCarry || (LB == 1 && wk.again == 2));   // (the latter two: settle() is to see it)
      if (sp.init && c.live(wk, h) && !from_zero && !fold && owns_state) {
        const float* I = sp.init + ((int64_t)c.b * sp.nheads + c.head(wk) + h) * sp.init_unit_stride + c.seg * sp.init_seg_stride +
                         (int64_t)l * P;
        if (prm.st32) {
#pragma unroll
          for (int e = 0; e < P / 8; ++e) {
            uint64_t v[4];
            ldg256(I + 8 * e, v);
            H[4 * e] = v[0]; H[4 * e + 1] = v[1]; H[4 * e + 2] = v[2]; H[4 * e + 3] = v[3];
          }
        } else {
#pragma unroll
          for (int e = 0; e < P / 4; ++e) {
            const ulonglong2 v = reinterpret_cast<const ulonglong2*>(I)[e];
            H[2 * e] = v.x;
            H[2 * e + 1] = v.y;
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < P / 2; ++e) H[e] = 0;
      }
    };
    // Chained: what the CTA before this one handed over.  Look-back: fold the pairs (state from zero, log-decay
    // sum) that the CTAs from .. before this one published for their pieces of this sequence, newest first:
    // H_in = sum_c exp(log-decay after c) F_c (+ the same for the caller's initial state).
    // Latency-bound, a piece after the other, so the flags are asked for by 32 lanes at once and in a slot the threads' 16
    // bytes stand side by side: rows of 256 bytes, as the caller's states have them, cost 32 cache lines a load.  One sequence
    // of 64 tiles on 64 SMs: 137 -> 37 us; 16 pairs of 16 tiles 54 -> 27; chained, 250 pairs of 16 tiles 103 -> 99.
    auto fold_item = [&]() {
      const bool look_back = sp.chain == 2;
      const bool init = sp.init && c.live(wk, h) && look_back;
      int p = (int)blockIdx.x - 1;
      const int from = !look_back ? p : LB && c.t_begin == 0 ? (int)blockIdx.x : wk.from;
      wait_published(p, from);
      float lds = 0.f;   // look-back: log-decays of 32 pieces, one in each lane (asked for one by one they are a round trip to L2 each)
      int next = 0;
#pragma unroll 1
      for (;; --p) {
        const bool piece = p >= from;
        if (!piece && !init) break;
        const float* src = piece ? sp.chain_state + (2 * p + h) * (int64_t)(N * P) + l * 4
                                 : sp.init + ((int64_t)c.b * sp.nheads + c.head(wk) + h) * sp.init_unit_stride +
                                       c.seg * sp.init_seg_stride + (int64_t)l * P;
        const int step = piece ? N : 1;
        float ld = 0.f;
        if (!LB) ld = piece ? __ldcg(sp.chain_ld + 2 * p + h) : 0.f;
        else if (next == 0 && p - lane >= from) lds = __ldcg(sp.chain_ld + 2 * (p - lane) + h);
        const float wgt = ex2(asum0 * kLog2e);   // asum0: log-decay between the end of the piece being added and this item
        if (owns_state && wgt != 0.f) {          // (an underflowed piece adds nothing)
          const ulonglong2* I = reinterpret_cast<const ulonglong2*>(src);
          const uint64_t w2 = pair(wgt, wgt);
#pragma unroll
          for (int e = 0; e < P / 4; ++e) {
            const ulonglong2 v = __ldcg(I + e * step);   // (may be written by another SM: bypass L1)
            H[2 * e] = fma_pair(w2, v.x, H[2 * e]);
            H[2 * e + 1] = fma_pair(w2, v.y, H[2 * e + 1]);
          }
        }
        if (!piece) break;
        asum0 += LB ? __shfl_sync(0xffffffffu, lds, next) : ld;
        next = (next + 1) & 31;
      }
      if (LB && asum0 != asum0) {   // (a log-decay that is NaN, in the sequence's first piece perhaps: nothing was added behind it)
        const uint64_t nan2 = pair(asum0, asum0);
#pragma unroll
        for (int e = 0; e < P / 2; ++e) H[e] = nan2;
      }
    };
    // Look-back, behind what enters an item that produces Y.  A beginning is done again: a state that does not vanish behind it has the piece
    // done again (a bit per CTA, see launch_tc2()).  And where the final states lie on the initial ones, the other pieces of the sequence are
    // told (in the upper bits of the flag: this warp has published by then, if it does) that this one has read.
    auto settle = [&]() {
      if (LB == 1 && wk.again == 2) {
        bool gone = true;
        if (owns_state) {
#pragma unroll
          for (int e = 0; e < P / 2; ++e) gone = gone && vanishes(unpair(H[e]));
        }
        if (!__all_sync(0xffffffffu, gone) && lane == 0 && !m->abort_flag) {
          grid_dependency_wait();
          atomicOr(walk_bits(sp) + blockIdx.x / 32, 1 << blockIdx.x % 32);
        }
      }
      if constexpr (kCarry) {
        __syncwarp();
        grid_dependency_wait();
        if (lane == 0) {
          const int one = 1 << kReadBit;
          asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(sp.chain_flag + 2 * blockIdx.x + h), "r"(one) : "memory");
        }
      }
    };
    // The state leaving an item: to this CTA's slot, or (last or only piece of the sequence) the caller's outputs.
    auto leave_item = [&](bool wy) {
      const bool cut_back = sp.chain && c.t_begin / T + c.ntiles < wk.nt;
      const bool publish = cut_back && !(LB ? !c.scanned(wk) : sp.chain == 2 && wy);   // (look-back: the scan from zero)
      const int64_t slot = 2 * (int64_t)blockIdx.x + h;
      const int64_t unit = (int64_t)c.b * sp.nheads + c.head(wk) + h;
      const int seg = sp.chain ? 0 : c.seg;
      const bool late = LB == 1 && wk.again == 2 && !cut_back && c.scanned(wk);   // (what came before is not known yet: item 2 knows)
      if (LB == 1 && wk.again == 2 && c.item <= 2) {
        if (c.item == 1 && l == 0) m->asum1[h] = asum;
        if (c.item == 2 && wk.hi % wk.nt == 0 && sp.fin_ld && l == 0 && c.live(wk, h)) sp.fin_ld[unit * sp.finld_unit_stride] = asum0 + m->asum1[h];
      }
      if (publish ? given_up(m) : (cut_back || !c.live(wk, h))) return;
      if (kCarry && !publish) wait_published((int)blockIdx.x - 1, wk.from, true);
      float* to = publish ? sp.chain_state + slot * (N * P)
                          : (sp.fin ? sp.fin + unit * sp.fin_unit_stride + seg * sp.fin_seg_stride : nullptr);
      float* ld = publish ? sp.chain_ld + slot
                          : (sp.fin_ld ? sp.fin_ld + unit * sp.finld_unit_stride + seg * sp.finld_seg_stride : nullptr);
      if (to && owns_state) {
        float* F = to + (publish ? l * 4 : l * P);
        const int step = publish ? N : 1;
        if (prm.st32 && !publish) {
#pragma unroll
          for (int e = 0; e < P / 8; ++e) stg256(F + 8 * e, H[4 * e], H[4 * e + 1], H[4 * e + 2], H[4 * e + 3]);
        } else {
#pragma unroll
          for (int e = 0; e < P / 4; ++e) reinterpret_cast<ulonglong2*>(F)[e * step] = make_ulonglong2(H[2 * e], H[2 * e + 1]);
        }
      }
      if (ld && l == 0 && !late) *ld = asum0 + asum;
      if (publish) {
        // Each warp publishes its own rows: a release-add by lane 0 after a warp barrier orders the
        // whole warp's stores before the count, and nobody has to wait for the stores to land.
        __syncwarp();
        grid_dependency_wait();
        if (lane == 0) {
          const int one = 1;
          asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(sp.chain_flag + slot), "r"(one) : "memory");
        }
      }
    };

    bool cur_y = false;
    uint32_t ky = 0;            // Y-producing tiles prepared
    uint32_t xi = h, xph = 0;   // (EPI) X slot of the tile being prepared
    if (total > 0) {
      c.next(prm, wk);
      enter_item(npre == 0);
    }
#pragma unroll 1
    for (uint32_t n = 0;; ++n) {   // tile n is prepared, P of tile n - 1 is made
      if (cur_y) {
        wait(&m->bar_g, (ky - 1) & 1, m);
        tc_fence_after();
        const uint32_t slot = (n - 1) % kFactors;
        make_p(m->f[h][slot]);
        tmem_st_wait();
        tc_fence_before();
        warp_arrive(&m->bar_p[h]);
        if (lane == 0) mbar_arrive(&m->empty_f[h][slot]);
      }
      if (n == total) break;
      const bool wy = n >= npre;   // this tile produces Y (a look-back launch starts with a state-only item)
      const uint32_t slot = n % kFactors;
      if constexpr (EPI) {
        // B. (the read-out warps have the skip and the gate to do; the S MMA that read the Xd before was waited for in E)
        wait(&m->full_f[h][slot], (n / kFactors) & 1, m);
        wait(&m->full_x[xi], xph, m);
        make_xd<T16, WIDE>(sX + xi * kBlk, sXd + h * kBlk, m->f[h][slot], q, lane);
        wait(&m->full_b[n % BC], (n / BC) & 1, m);   // (for the S MMA, which waits for these warps only)
        fence_proxy_async();
        warp_arrive(&m->bar_xd);
        if (!wy && lane == 0) mbar_arrive(&m->empty_x[xi]);
        xi += 2;
        if (xi >= XS) { xi -= XS; xph ^= 1; }
      }
      // D. 16-bit copy of the state for C.H
      if (__builtin_expect(fold, 0)) {
        fold_item();
        if constexpr (LB) settle();
        fold = false;
      }
      if (wy) {
        wait(&m->bar_ch, (ky & 1) ^ 1, m);   // the C.H MMA has read the copy before this one
        store_hb();
        fence_proxy_async();
        warp_arrive(&m->bar_h);
        ++ky;
      }
      // E. H <- exp(cs_last) H + S
      wait(&m->full_f[h][slot], (n / kFactors) & 1, m);
      const float gs = ex2(m->f[h][slot].tot * kLog2e);
      {
        const float yk = m->f[h][slot].ld - acomp, tk = asum + yk;
        acomp = (tk - asum) - yk;
        if (acomp != acomp) acomp = 0.f;   // (a sum of -inf stays that)
        asum = tk;
      }
      wait(&m->bar_s, n & 1, m);
      tc_fence_after();
      if (owns_state) {
        const uint64_t g2 = pair(gs, gs);
        uint32_t s0[32], s1[32];
        tmem_ld32(tS + tlane, s0);
        tmem_ld32(tS + tlane + 32, s1);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) H[e] = fma_pair(H[e], g2, pair(s0[2 * e], s0[2 * e + 1]));
#pragma unroll
        for (int e = 0; e < 16; ++e) H[16 + e] = fma_pair(H[16 + e], g2, pair(s1[2 * e], s1[2 * e + 1]));
      }
      if (!wy) {
        tc_fence_before();
        warp_arrive(&m->bar_u);
        if (lane == 0) mbar_arrive(&m->empty_f[h][slot]);
      }
      const bool last = c.left == 0;
      if (__builtin_expect(last, 0)) leave_item(wy);
      if (n + 1 < total) c.next(prm, wk);
      if (__builtin_expect(last && n + 1 < total, 0)) enter_item(n + 1 >= npre);
      cur_y = wy;
    }
  } else {
    // ------------------------------------------------------------------ warps 12-15: Xd, and read-out of Y, both heads
    setmaxnreg_dec<112>();
    const int q = warp & 3;
    const int lane_base = q * 32;
    const int l = lane_base + lane;
    const uint32_t tlane = (uint32_t)lane_base << 16;
    const uint32_t swz = (uint32_t)(l & 7);
    Cursor c;
    uint32_t bi = 0, bph = 0;   // X slot of the next tile to make Xd of
    uint32_t xi = 0;            // X slot of the tile being read out
    uint32_t ky = 0;
    const uint64_t once = policy_evict_first();
    uint32_t skip[2] = {0, 0};       // (EPI) D of both heads as loaded: a conversion there would hold the warp for the memory latency
    const T16* zp = nullptr;         // (EPI) gate of head 0, row lane / 4 of this warp's, piece lane % 4
    int pending = -1;    // (lane 0) X slot that this warp's last TMA store still reads
    auto release = [&]() {
      if (lane == 0 && pending >= 0) {
        bulk_wait_read_all();
        mbar_arrive(&m->empty_x[pending]);
        pending = -1;
      }
    };
#pragma unroll 1
    for (uint32_t k = 0; k <= total; ++k) {   // Xd of tile k, Y of tile k - 1
      if (EPI && k < npre) {   // (takes its turn in the factors' ring all the same)
        for (int h = 0; h < 2; ++h) {
          wait(&m->full_f[h][k % kFactors], (k / kFactors) & 1, m);
          warp_arrive(&m->empty_f[h][k % kFactors]);
        }
      }
      if (!EPI && k < total) {
        const bool two = kTwo && k < npre;
        const uint32_t xd = two && (k & 1) ? sH : sXd;
        if (k > 0 && !two) wait(&m->bar_s, (k - 1) & 1, m);   // the S MMA has read the Xd before this one
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          wait(&m->full_f[h][k % kFactors], (k / kFactors) & 1, m);
          wait(&m->full_x[bi], bph, m);
          make_xd<T16, WIDE>(sX + bi * kBlk, xd + h * kBlk, m->f[h][k % kFactors], q, lane);
          if (k < npre) {   // nothing else reads X and the factors of a state-only tile
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(&m->empty_x[bi]);
              mbar_arrive(&m->empty_f[h][k % kFactors]);
            }
          }
          if (++bi == XS) { bi = 0; bph ^= 1; }
        }
        // (for the S MMA, which waits for this group only)
        if constexpr (kTwo) {
          if (two && k > 0) wait(&m->bar_s, (k - 1) & 1, m);   // (the other Xd is free for the next tile)
          if (two) wait((k & 1) ? &m->full_c[0] : &m->full_b[0], (k >> 1) & 1, m);
          else wait(&m->full_b[0], (((npre + 1) >> 1) + k - npre) & 1, m);
        } else {
          wait(&m->full_b[k % BC], (k / BC) & 1, m);
        }
        fence_proxy_async();
        warp_arrive(&m->bar_xd);
        release();
      }
      if (k == 0) continue;
      const uint32_t n = k - 1, slot = n % kFactors;
      c.next(prm, wk);
      if (n < npre) {
        xi += 2;
        if (xi >= XS) xi -= XS;
        continue;
      }
      const int t0 = c.t0;
      if constexpr (EPI) {
        // (instructions are what this warp is short of: the gate's addresses are worked out once an item)
        if (__builtin_expect(c.first_tile(), 0)) {
          const int head = c.head(wk);
          if (sp.D) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (c.live(wk, h))
                skip[h] = sp.d_in_dtype ? reinterpret_cast<const uint16_t*>(sp.D)[head + h] : reinterpret_cast<const uint32_t*>(sp.D)[head + h];
          }
          zp = static_cast<const T16*>(sp.Z) + c.b * sp.zs[0] + head * sp.zs[2] + (int64_t)(t0 + lane_base + (lane >> 2)) * sp.zs[1] + 8 * (lane & 3);
        } else {
          zp += T * sp.zs[1];
        }
      }
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const bool live = c.live(wk, h);
        // (EPI) the gate rows of this warp's 32 tokens, fetched ahead of the wait for the MMA.  Four lanes read half a
        // 128-byte row per load, eight rows per instruction; the rows reach their threads through the staging buffer below.
        uint4 zr[8];
        const uint32_t dskip = h ? skip[1] : skip[0];
        const T16* zh = h ? zp + sp.zs[2] : zp;
        if constexpr (EPI) {
          if (sp.Z && live) {
            const int64_t s8 = 8 * sp.zs[1];
            if (__builtin_expect(t0 + T <= sp.seqlen, 1)) {
              const T16* r = zh;
#pragma unroll
              for (int i = 0; i < 4; ++i, r += s8) {
                zr[i] = __ldg(reinterpret_cast<const uint4*>(r));
                zr[4 + i] = __ldg(reinterpret_cast<const uint4*>(r) + 4);
              }
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (t0 + lane_base + 8 * i + (lane >> 2) < sp.seqlen) {
                  zr[i] = __ldg(reinterpret_cast<const uint4*>(zh + i * s8));
                  zr[4 + i] = __ldg(reinterpret_cast<const uint4*>(zh + i * s8) + 4);
                }
              }
            }
          }
        }
        if constexpr (EPI) {
          // the next gate rows, one per lane, as near as they go without registers
          const int tn = t0 + l + (h ? T : 0);
          if (sp.Z && tn < sp.seqlen && c.live(wk, h ^ 1))
            asm volatile("prefetch.global.L1 [%0];" ::"l"(zp + (h ? T * sp.zs[1] : sp.zs[2]) + (lane - (lane >> 2)) * sp.zs[1]));
          wait(&m->full_f[h][slot], (n / kFactors) & 1, m);
        }
        const float el = ex2(m->f[h][slot].cs2[l]);
        warp_arrive(&m->empty_f[h][slot]);
        wait(&m->bar_y[h], ky & 1, m);
        tc_fence_after();
        release();
        const uint64_t el2 = pair(el, el);
        // The X tile is dead (its P.X MMA is complete): the 16-bit Y rows are staged in its slot.
        const uint32_t ystage = sX + xi * kBlk;
        const uint32_t yrow = ystage + l * 128;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t o[32], d[32];
          tmem_ld32(tYo + 64 * h + tlane + 32 * half, o);
          tmem_ld32(tYd + 64 * h + tlane + 32 * half, d);
          tmem_ld_wait();
          if (half == 1) {
            tc_fence_before();
            warp_arrive(&m->bar_e);   // both accumulators are read out
          }
          uint64_t y[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) y[e] = fma_pair(pair(o[2 * e], o[2 * e + 1]), el2, pair(d[2 * e], d[2 * e + 1]));
          if constexpr (EPI) {
            // Y <- (Y + x * D) * silu(z) (model_ref.py:116-118) in fp32; x is this thread's row of the X tile, still in
            // the slot that the Y rows go to; silu(z) = z / 2 (1 + tanh(z / 2)), the tanh on 16-bit pairs.
            if (sp.D && live) {
              const float dsf = sp.d_in_dtype ? unpack2<T16>(dskip).x : __uint_as_float(dskip);
              const uint64_t ds = pair(dsf, dsf);
#pragma unroll
              for (int cc = 0; cc < 4; ++cc) {
                const uint4 xr = lds128(yrow + (((4 * half + cc) ^ swz) << 4));
                const uint32_t xw[4] = {xr.x, xr.y, xr.z, xr.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 xf = unpack2<T16>(xw[e]);
                  y[4 * cc + e] = fma_pair(pair(xf.x, xf.y), ds, y[4 * cc + e]);
                }
              }
            }
            if (sp.Z && live) {
              // x of this half is consumed: the warp's gate rows go through its 32 rows of the slot to the threads that
              // own them (four lanes hold the four 16-byte pieces of one row's half)
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int row = lane_base + 8 * i + (lane >> 2);
                sts128(ystage + row * 128 + (((4 * half + (lane & 3)) ^ (row & 7)) << 4), half ? zr[4 + i] : zr[i]);
              }
              __syncwarp();
              const uint32_t half2 = pack2<T16>(0.5f, 0.5f);
#pragma unroll
              for (int cc = 0; cc < 4; ++cc) {
                const uint4 zq = lds128(yrow + (((4 * half + cc) ^ swz) << 4));
                const uint32_t zw[4] = {zq.x, zq.y, zq.z, zq.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  // silu(z) = z / 2 + z / 2 tanh(z / 2) on the packed 16-bit pair, rounded once (model_ref.py:118 in half
                  // precision); the product with Y is taken in fp32
                  const uint32_t zz = mul2<T16>(zw[e], half2);
                  const float2 gf = unpack2<T16>(fma2<T16>(zz, tanh2<T16>(zz), zz));
                  y[4 * cc + e] = mul_pair(y[4 * cc + e], pair(gf.x, gf.y));
                }
              }
            }
          }
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            uint4 v;
            v.x = pack_pair<T16>(y[4 * cc]); v.y = pack_pair<T16>(y[4 * cc + 1]);
            v.z = pack_pair<T16>(y[4 * cc + 2]); v.w = pack_pair<T16>(y[4 * cc + 3]);
            sts128(yrow + (((4 * half + cc) ^ swz) << 4), v);
          }
        }
        fence_proxy_async();         // staged rows -> visible to the TMA engine
        __syncwarp();
        if (lane == 0) {
          // each warp hands its own 32 rows to the TMA engine; rows past the end of the sequence are clipped
          if (live && t0 + lane_base < sp.seqlen) {
            tma_store_5d(&tmY, ystage + lane_base * 128, 0, 2 * c.q + h, c.g, t0 + lane_base, c.b, once);
            bulk_commit();
          }
          pending = (int)xi;
        }
        if (++xi == XS) xi = 0;
      }
      ++ky;
    }
    release();
    if (lane == 0) bulk_wait_all();   // the Y rows this warp stored must have landed before the CTA exits
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && status) {
    if (m->tmem_base != 0) atomicCAS(status, 0, (int)STATUS_TMEM_ALLOC);
    if (m->abort_flag) atomicCAS(status, 0, (int)m->abort_flag);
  }
  if (warp == 0) {
    __syncwarp();
    grid_dependency_wait();   // (where no sequence of this CTA was cut)
    tmem_dealloc(m->tmem_base, 512);
  }
}

// The ready flags of a launch with cut sequences have to start at zero (the workspace keeps the call before's).  The forward
// starts beside this kernel, which itself starts when all work before it in the stream is done, and asks for its end
// (grid_dependency_wait) only where a flag is first used; a memset ahead of the forward cost 2.5 to 3.5 us of every such call.
__global__ void clear_flags_kernel(int* flags) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  flags[threadIdx.x] = 0;
}

template <typename T16, int N, bool EPI, bool WIDE, int LB>
int launch_typed2(const CUtensorMap& tx, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& ty,
                  const TileParams& prm, cudaStream_t stream) {
  auto kern = ssd_tc2_kernel<T16, N, EPI, WIDE, LB>;
  constexpr int smem = Layout2<N>::kBytes;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return SSD_ERR_CUDA;
  const int nt = (prm.sp.seqlen + T - 1) / T;
  const int grid = prm.sp.chain ? dealt_grid(prm.upairs, nt, prm.sp.chain) : std::min(prm.nitems, kSms);
  const int rc = launch_tiles(kern, grid, kThreads2, smem, prm.sp, stream, tx, tb, tc, ty, prm);
  if (LB != 1 || !prm.sp.beginnings || rc != SSD_OK) return rc;
  // What entered a piece and did not vanish (see find_beginning()): the piece again, from the states that the launch before left in scratch.
  // 1 us where there is none.  (As one more item of the same launch, or that launch's list again, 1.5 to 3 % of every look-back call.)
  TileParams again = prm;
  again.sp.walk_again = 1;
  return launch_early(kern, grid, kThreads2, smem, stream, tx, tb, tc, ty, again);
}

bool odd_groups(const SsdArgs& a) { return a.nheads / a.ngroups % 2 != 0; }

// Head pairs over the whole batch; a group with an odd number of heads has a half-empty pair.
int64_t unit_pairs(const SsdArgs& a) { return (int64_t)a.batch * a.ngroups * ((a.nheads / a.ngroups + 1) / 2); }

}  // namespace

int64_t tc2_units(const SsdArgs& a) { return unit_pairs(a); }

bool tc2_long_pieces(const SsdArgs& a) {
  const int64_t units = unit_pairs(a), nt = (a.seqlen + T - 1) / T;
  if (units >= kSms) return false;
  const int64_t pieces = dealt_grid(units, (int)nt, 2) / units;
  return dealt_grid(units, (int)nt, 2) % units == 0 && pieces > 1 && (nt + pieces - 1) / pieces >= kLeastBeginning;
}

int launch_clear_flags(int32_t* flags, int count, cudaStream_t stream) {
  return launch(clear_flags_kernel, 1, count, 0, stream, flags);
}

// Skip and gate in the kernel: with packed 16-bit gates, which groups with an odd number of heads have never had (bf16, Y
// against 64 bits: 2.9e-3 with the epilogue kernel's fp32 gate, 3.7e-3 with packed ones).
bool tc2_fuses_epilogue(const SsdArgs& a) { return !odd_groups(a); }

bool tc_supports(const SsdArgs& a) {
  if (a.dtype != SSD_DTYPE_F16 && a.dtype != SSD_DTYPE_BF16) return false;
  if (a.headdim != P || (a.dstate != 64 && a.dstate != 128)) return false;
  if (!ok16(a.X) || !ok16(a.B) || !stride_ok(a.x_stride) || !stride_ok(a.b_stride)) return false;
  const bool state_only = (a.flags & SSD_FLAG_STATE_ONLY) != 0;
  if (!state_only) {
    if (!a.C || !a.Y) return true;  // shape query without pointers (kernel_name / workspace_bytes)
    if (!ok16(a.C) || !ok16(a.Y) || !stride_ok(a.c_stride) || !stride_ok(a.y_stride)) return false;
  }
  return true;
}

// How a sequence that is cut (nseg > 1) is scanned by this kernel:
//   1  with at least one sequence per SM the tiles of all sequences are dealt out evenly over the CTAs inside one
//      launch; a sequence cut that way hands its state from CTA to CTA through scratch ("chained");
//   2  with fewer sequences than SMs the same even deal, but each CTA first scans the last piece of its range
//      from zero and publishes (state, log-decay sum), and a piece folds what the CTAs before it published
//      ("look-back"), still one launch;
//   0  two passes and a fold (three launches): kept for the state-only run and the run that reuses its segment
//      states, which a sequence-sharded forward makes around its exchange.
int tc_chain_mode(const SsdArgs& a, int nseg, int64_t upairs) {
  if (nseg <= 1) return 0;
  if (upairs >= kSms) return 1;
  return (a.flags & (SSD_FLAG_STATE_ONLY | SSD_FLAG_REUSE_SEGMENTS)) ? 0 : 2;
}

int tc_default_segments(const SsdArgs& a, int64_t upairs) {
  const int tiles = (a.seqlen + T - 1) / T;
  // Costs in tile times (2.7 to 3.1 us), fitted to forwards of 1 to 600 pairs and 2 to 64 tiles, each timed whole and cut; the
  // constants are what a launch takes beside its tiles.  16 pairs of 4, 8 and 32 tiles: whole 17, 29 and 95 us, cut 16, 18
  // and 33; 250 pairs of 4, 8 and 32 tiles: 31, 54 and 199, cut 33, 54 and 181.
  const double even = (double)upairs * tiles / kSms;   // tiles per SM under the even deal (any count above one selects it)
  if (upairs >= kSms) {
    const double rounds = (double)((upairs + kSms - 1) / kSms);
    return tiles >= 2 && even * 1.02 + 4.9 < 0.98 * (rounds * tiles + 2.4) ? 2 : 1;
  }
  if (!(a.flags & (SSD_FLAG_STATE_ONLY | SSD_FLAG_REUSE_SEGMENTS))) {
    // Look-back: the state-only scan of the last piece of every range, two start-ups and the round trip through scratch, and
    // the fold of the pieces before the last one of a sequence.
    const double pieces = std::min((double)kSms / upairs, (double)tiles);
    // With more than half as many pairs as SMs the deal saves little and every tile of a range's last piece is read twice: whole
    // sequences, unless the saving (at 1.55 of a tile's time for a dealt one) is more than the start-ups of a cut (96 pairs
    // of 64 tiles: 204 us dealt out, 185 whole; 80 pairs of 64: 174 and 185).
    if (pieces < 2 && even * 1.55 + 5 > tiles + 2.2) return 1;
    return tiles >= 2 && even * 1.4 + 4.9 + 0.12 * pieces < 0.98 * (tiles + 2.2) ? 2 : 1;
  }
  if (upairs >= 120) return 1;
  // Two passes: cutting the sequences into concurrently scanned segments costs a second pass
  // (about 0.4 of a full pass) and a per-item start-up (about 1.5 tile times).  Pick the count that
  // minimises the modelled time, in tile times, of the busiest CTA.
  double best_cost = (double)tiles + 1.5;   // one CTA per sequence
  int best = 1;
  for (int nseg = 2; nseg <= 32 && nseg * 2 <= tiles; ++nseg) {
    const int64_t rounds = (upairs * nseg + kSms - 1) / kSms;
    const int per_item = (tiles + nseg - 1) / nseg;
    const double cost = (double)rounds * (per_item * 1.4 + 3.0);
    if (cost < best_cost * 0.97) {
      best_cost = cost;
      best = nseg;
    }
  }
  return best;
}

int launch_tc2(const SsdArgs& a, const ScanParams& sp, cudaStream_t stream) {
  if (sp.seg_len % T != 0) return SSD_ERR_UNSUPPORTED;
  TileParams prm;
  prm.sp = sp;
  prm.ppg = (a.nheads / a.ngroups + 1) / 2;
  const int64_t upairs = unit_pairs(a);
  if (upairs * sp.nseg > 0x7fffffffLL || upairs * ((a.seqlen + T - 1) / T) > 0x7fffffffLL) return SSD_ERR_TOO_LARGE;
  prm.upairs = (int)upairs;
  prm.st32 = ((reinterpret_cast<uintptr_t>(sp.init) | reinterpret_cast<uintptr_t>(sp.fin)) & 31) == 0;   // (rows are 256 bytes)
  prm.nitems = prm.upairs * sp.nseg;
  CUtensorMap tx, tb, tc, ty;
  if (!make_map(&tx, a.X, a, P, a.nheads / a.ngroups, a.x_stride, T)) return SSD_ERR_CUDA;
  if (!make_map(&tb, a.B, a, a.dstate, 1, a.b_stride, T)) return SSD_ERR_CUDA;
  if (sp.compute_y) {
    if (!make_map(&tc, a.C, a, a.dstate, 1, a.c_stride, T)) return SSD_ERR_CUDA;
    if (!make_map(&ty, a.Y, a, P, a.nheads / a.ngroups, a.y_stride, 32)) return SSD_ERR_CUDA;
  } else {
    tc = tb;
    ty = tx;
  }
  const bool epi = sp.compute_y && (sp.D || sp.Z);
  if (epi) {
    // the gate rows are read with 16-byte loads
    if (sp.Z && ((reinterpret_cast<uintptr_t>(sp.Z) & 15) || sp.zs[0] % 8 || sp.zs[1] % 8 || sp.zs[2] % 8))
      return SSD_ERR_MISALIGNED;
  }
  auto go = [&](auto epilogue, auto wide, auto look_back) {
    constexpr bool E = decltype(epilogue)::value, W = decltype(wide)::value;
    constexpr int LB = decltype(look_back)::value;
    if (a.dtype == SSD_DTYPE_BF16)
      return a.dstate == 128 ? launch_typed2<__nv_bfloat16, 128, E, W, LB>(tx, tb, tc, ty, prm, stream)
                             : launch_typed2<__nv_bfloat16, 64, E, W, LB>(tx, tb, tc, ty, prm, stream);
    return a.dstate == 128 ? launch_typed2<__half, 128, E, W, LB>(tx, tb, tc, ty, prm, stream)
                           : launch_typed2<__half, 64, E, W, LB>(tx, tb, tc, ty, prm, stream);
  };
  auto one = [&](auto look_back) {
    if (epi) return go(std::true_type{}, std::false_type{}, look_back);
    return odd_groups(a) ? go(std::false_type{}, std::true_type{}, look_back) : go(std::false_type{}, std::false_type{}, look_back);
  };
  if (sp.chain != 2) return one(std::integral_constant<int, 0>{});
  return sp.fin_on_init ? one(std::integral_constant<int, 2>{}) : one(std::integral_constant<int, 1>{});
}

}  // namespace ssd
