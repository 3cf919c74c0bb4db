// What the tensor-core kernels share: how the 128-token tiles of all sequences are dealt out to the CTAs, bounded waits,
// products of fp32 pairs, launches.
#pragma once

#include "ssd_common.cuh"
#include "tc_common.cuh"
#include "tc_ptx.cuh"

namespace ssd {
namespace tc {

using namespace ptx;

constexpr int kSms = 148;

// Work list of this CTA.
//  - Regular mode: items blockIdx.x, blockIdx.x + gridDim.x, ... of the (segment, sequence) grid.
//  - Chained mode (sp.chain == 1): all tiles of all sequences, laid end to end, are cut into gridDim.x equal
//    ranges, so every CTA gets the same number of tiles (+-1) whatever the number of sequences.  A range holds
//    the tail of one sequence, whole sequences and the head of another; they are walked in reverse, head first:
//    the head's state is what the next CTA's tail piece waits for, and a tail piece (walked last) then finds
//    the state it needs already there when there is at least one sequence per CTA.
//  - Look-back mode (sp.chain == 2), for fewer sequences than CTAs: the same even cut, but a piece cannot wait
//    for the full scan of the piece before it (the pieces of one sequence would run one after the other).
//    Instead every CTA first scans the LAST piece of its range from a zero state, state and log-decay sum only
//    (item 0, skipped when that piece ends its sequence), and publishes the pair.  Then it walks its pieces like
//    the chained mode; a piece that starts inside a sequence folds the published pairs of the CTAs before it, back
//    to the one that holds the sequence's first tile (the recurrence is linear: H_in = sum_c exp(sum of the
//    log-decays after c) F_c), skipping those whose decay factor has underflowed.
//    Of a long piece only a beginning is scanned that way (find_beginning()): from where what enters the piece has decayed to nothing,
//    the scan from zero is the scan, and writes Y at once (and the sequence's final state, where the piece ends it).  Then the
//    beginning is done again, from the state that does enter -- and by a launch behind this one the whole piece, if that state turns out to
//    be one that does not decay to nothing (not finite, or of 2^67 and more).
// Computed once per CTA (thread 0, into shared memory): the 64-bit divisions are bulky code.
struct Work {
  int total;            // tiles of all items
  int npre;             // the first npre of them produce a state only
  int lo, hi, nt, first;   // chained modes: global tile range, tiles per sequence, first tile of item 0's sequence
  int from;             // look-back mode: the CTA that holds the first tile of the range's first sequence
  int hpg, ppg;         // heads per B/C group, head pairs per group
  // item 0 as (pair of the group, group, batch entry, segment), and the step from one item to the next in the same
  // mixed-radix digits: the walk needs no division
  int d0[4], step[4];
  int again;            // look-back mode: items of the range's last piece that follow item 0: 0 or 1 (after its state-only scan), or 2
                        // where only its beginning is scanned for the state (the rest of the piece, then the beginning again)
};

struct TileParams {
  ScanParams sp;
  int nitems;   // upairs * nseg
  int upairs;   // batch * pairs of heads (or heads, where a kernel works on one at a time; below too)
  int ppg;      // head pairs per B/C group
  int st32;     // the states that enter and leave start on 32-byte boundaries
};

// Item `i` of the (segment, batch, group, pair) grid as digits.
__device__ __forceinline__ void digits(int i, const TileParams& prm, int (&d)[4]) {
  d[0] = i % prm.ppg; i /= prm.ppg;
  d[1] = i % prm.sp.ngroups; i /= prm.sp.ngroups;
  d[2] = i % prm.sp.batch; d[3] = i / prm.sp.batch;
}

__device__ __forceinline__ void work_list(const TileParams& prm, Work& wk) {
  const ScanParams& sp = prm.sp;
  wk.nt = (sp.seqlen + T - 1) / T;
  wk.hpg = sp.nheads / sp.ngroups;
  wk.ppg = prm.ppg;
  wk.npre = sp.compute_y ? 0 : 0x7fffffff;
  wk.lo = wk.hi = wk.first = wk.from = wk.again = 0;
  if (sp.chain) {
    const long long total = (long long)prm.upairs * wk.nt;
    wk.lo = (int)((long long)blockIdx.x * total / gridDim.x);
    wk.hi = (int)((long long)(blockIdx.x + 1) * total / gridDim.x);
    wk.total = wk.hi - wk.lo;
    const int last = (wk.hi - 1) / wk.nt;     // (every CTA has at least one tile)
    wk.first = last * wk.nt;
    if (sp.chain == 2 && wk.hi % wk.nt != 0) {
      wk.npre = wk.hi - max(wk.lo, wk.first);
      wk.total += wk.npre;
      wk.again = 1;
    }
    // the largest c with lo(c) <= first tile of the range's first sequence
    const int first = wk.lo / wk.nt * wk.nt;
    int c = (int)((((long long)first + 1) * gridDim.x - 1) / total);
    while (c > 0 && (long long)c * total / gridDim.x > first) --c;
    while ((long long)(c + 1) * total / gridDim.x <= first) ++c;
    wk.from = c;
    digits(last, prm, wk.d0);
    wk.step[0] = -1;
    wk.step[1] = wk.step[2] = wk.step[3] = 0;
  } else {
    wk.total = 0;
    for (int i = blockIdx.x; i < prm.nitems; i += gridDim.x) {
      const int t = i / prm.upairs * sp.seg_len;
      wk.total += (min(sp.seqlen, t + sp.seg_len) - t + T - 1) / T;
    }
    digits(blockIdx.x, prm, wk.d0);
    digits(gridDim.x, prm, wk.step);
  }
}

// Walks the tiles of all items of this CTA, in order.  An item is a run of `ntiles` tiles of one (batch, head pair)
// sequence from token t_begin on.
// kLookBack: whether there are items of the look-back mode (asked for at run time it costs the walk of the others: 256 x 512 tokens of 48
// heads 560 -> 575 us, 8 x 2048 of 24 52.1 -> 52.6).
template <int kHeads, bool kLookBack>   // heads of an item
struct CursorOf {
  int t0, left;           // first token of the current tile, tiles of the item after it
  int t_begin, ntiles;
  int q, g, b, seg;       // pair of the group, group, batch entry, segment
  int first;              // chained modes: first tile of the sequence in the laid-out order
  int item;
  __device__ __forceinline__ CursorOf() : left(0), item(-1) {}
  __device__ __forceinline__ void next(const TileParams& prm, const Work& wk) {
    if (__builtin_expect(left > 0, 1)) {
      --left;
      t0 += T;
      return;
    }
    const ScanParams& sp = prm.sp;
    if (++item == 0) {
      q = wk.d0[0]; g = wk.d0[1]; b = wk.d0[2]; seg = wk.d0[3];
      first = wk.first;
    } else if (kLookBack ? item > wk.again : !(item == 1 && sp.chain == 2 && wk.npre > 0)) {   // (up to there: the piece scanned first again)
      first -= wk.nt;
      int c = 0;
      q += wk.step[0];
      if (q >= prm.ppg) { q -= prm.ppg; c = 1; }
      if (q < 0) { q += prm.ppg; c = -1; }
      g += wk.step[1] + c;
      c = 0;
      if (g >= sp.ngroups) { g -= sp.ngroups; c = 1; }
      if (g < 0) { g += sp.ngroups; c = -1; }
      b += wk.step[2] + c;
      c = 0;
      if (b >= sp.batch) { b -= sp.batch; c = 1; }
      seg += wk.step[3] + c;
    }
    if (sp.chain) {
      const int start = max(wk.lo, first), end = min(wk.hi, first + wk.nt);
      t_begin = (start - first) * T;
      ntiles = end - start;
      if (kLookBack && wk.again == 2 && item <= 2) {
        if (item == 1) t_begin += wk.npre * T;
        ntiles = item == 1 ? ntiles - wk.npre : wk.npre;
      }
    } else {
      t_begin = seg * sp.seg_len;
      ntiles = (min(sp.seqlen, t_begin + sp.seg_len) - t_begin + T - 1) / T;
    }
    t0 = t_begin;
    left = ntiles - 1;
  }
  // Look-back mode: an item that goes on from the state the last one left; one whose end is that of the scan from zero.
  __device__ __forceinline__ bool goes_on(const Work& wk) const { return kLookBack && wk.again == 2 && item == 1; }
  __device__ __forceinline__ bool scanned(const Work& wk) const { return kLookBack && wk.again > 0 && item == wk.again - 1; }
  __device__ __forceinline__ bool first_tile() const { return left == ntiles - 1; }
  __device__ __forceinline__ int head(const Work& wk) const { return g * wk.hpg + kHeads * q; }   // first of the item
  __device__ __forceinline__ bool live(const Work& wk, int h) const { return kHeads * q + h < wk.hpg; }
};

// Look-back mode, all threads of a CTA, behind a barrier after work_list() and ahead of one before the list is used: how much of the
// range's last piece needs the state that enters it.  Where the log-decays from its first token on sum to less than -150, e^-150 = 2^-216
// has taken any entering state below 2^67 (kVanishes) past the smallest fp32 number (2^-149): it is not there any more.  A layer's slowest heads (rate
// 1, steps of 0.03) get there after 40 tiles.  1 x 131 072 tokens, 32 heads, 114 tiles a CTA: 510 -> 432 us, bit by bit the same.
// A piece scanned so is through with its first pass later (n - 0.6 k tile times for a beginning of k tiles) than one scanned for the state
// only (0.4 n), and what waits for it waits longer.  So the pieces of a sequence all do it or none: if, by the sequence's first tiles, k is
// at most 0.6 of a piece (32 768 tokens, 64 heads, each piece for itself and up to 1.0: 271 -> 298 us); and only where every range is one
// piece, as other ranges may begin with one that waits (the same case: 270 -> 305).  A look takes 1.5 us, another where it says yes; pieces
// of less than 40 tiles are left alone.
constexpr float kVanishes = 0x1p67f;
__device__ __forceinline__ bool vanishes(float2 v) { return fabsf(v.x) < kVanishes && fabsf(v.y) < kVanishes; }
constexpr int kLookTiles = 32, kFirstTiles = 2, kLeastBeginning = 40;
template <int kHeads>   // heads of an item
struct Look {
  float sums[2][kLookTiles][kHeads], first[kFirstTiles][kHeads];
};
template <int kHeads>
__device__ __forceinline__ void find_beginning(const TileParams& prm, Work& wk, Look<kHeads>& m, int warps) {
  const ScanParams& sp = prm.sp;
  const int from = max(wk.lo, wk.first), tiles = wk.hi - from;
  if (!sp.beginnings || tiles < kLeastBeginning || (int)gridDim.x % prm.upairs != 0 || (wk.again == 0 && from == wk.first)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int heads = min(kHeads, wk.hpg - kHeads * wk.d0[0]);
  // A tile's sums by one warp, every 32 / kHeads lanes a head.  (A line holds a token's heads: reading it for one at a time, and 16 tiles of
  // the sequence's beginning, cost 14 to 25 us.)
  constexpr int kLanes = 32 / kHeads, kTokens = T / kLanes;
  const int h = lane / kLanes;
  const float* A = sp.A + wk.d0[2] * sp.as[0] + (wk.d0[1] * wk.hpg + kHeads * wk.d0[0] + min(h, heads - 1)) * sp.as[2];
  auto sum_of = [&](int tile, float (&to)[kHeads]) {
    const int64_t t = (int64_t)tile * T + kTokens * (lane % kLanes);
    float s = 0.f;
    if (t + kTokens <= sp.seqlen) {   // (less at the end: no harm)
      const float* a = A + t * sp.as[1];
#pragma unroll
      for (int e = 0; e < kTokens; ++e, a += sp.as[1]) s += *a;
    }
#pragma unroll
    for (int d = kLanes / 2; d >= 1; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane % kLanes == 0) to[h] = s;
  };
  if (warp < kFirstTiles) sum_of(warp, m.first[warp]);
  __syncthreads();
  const float usual = (float)prm.upairs * wk.nt / gridDim.x;
  bool all = true;
  for (int k = 0; k < heads; ++k) all = all && (m.first[0][k] + m.first[1][k]) * (0.6f * usual) < -150.f * kFirstTiles;
  int beginning = 0, gone[kHeads] = {};   // `gone`: tiles after which a head has nothing left
  float run[kHeads] = {};
  for (int done = 0; all && done < tiles && beginning == 0; done += kLookTiles) {
    float (&sums)[kLookTiles][kHeads] = m.sums[done / kLookTiles & 1];
    for (int i = warp; i < kLookTiles; i += warps) sum_of(from - wk.first + min(done + i, tiles - 1), sums[i]);
    __syncthreads();
    // every warp for itself, a tile to a lane
#pragma unroll
    for (int k = 0; k < kHeads; ++k) {
      if (k >= heads) continue;
      float v = done + lane < tiles ? sums[lane][k] : 0.f;
#pragma unroll
      for (int d = 1; d < kLookTiles; d <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
      }
      v += run[k];
      const unsigned below = __ballot_sync(0xffffffffu, v < -150.f);
      if (gone[k] == 0 && below) gone[k] = done + __ffs(below);
      run[k] = __shfl_sync(0xffffffffu, v, 31);
    }
    beginning = 0;
    bool both = true;
#pragma unroll
    for (int k = 0; k < kHeads; ++k) {
      if (k >= heads) continue;
      both = both && gone[k] > 0;
      beginning = max(beginning, gone[k]);
    }
    if (!both) beginning = 0;
  }
  __syncthreads();   // (everybody has read the list)
  if (threadIdx.x == 0 && beginning > 0 && beginning < tiles) {
    wk.again = 2;
    wk.npre = beginning;
    wk.total = wk.hi - wk.lo + beginning;
  }
}

// Waits.  Instructions are what this kernel is short of: a scheduler's own instruction cache holds a few KB, and code
// that streams past it from the SM's (about 24 KB) arrives at 2.7 cycles per instruction, past that one at five to ten.
// So a wait is only "until the phase is over, or the CTA has given up", and one thread -- the TMA producer, whose waits
// depend on everybody's progress -- holds the clock (guarded_wait).  A role that was released that way runs through
// its remaining tiles without waiting, on whatever is in the buffers, and leaves.
// (The phase before a fresh barrier's first counts as over: the parity of "free" in the first round.)
template <class Misc>
__device__ __forceinline__ void wait_at(uint32_t bar, uint32_t parity, const Misc* m) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .u32 a;\n"
      "AGAIN:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1;\n\t@p bra DONE;\n\t"
      "ld.volatile.shared.u32 a, [%2];\n\tsetp.eq.u32 p, a, 0;\n\t@p bra AGAIN;\n"
      "DONE:\n\t}"
      ::"r"(bar), "r"(parity), "r"(smem_u32(const_cast<int*>(&m->abort_flag)))
      : "memory");
}
template <class Misc>
__device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity, const Misc* m) { wait_at(smem_u32(bar), parity, m); }
// False when the CTA has given up; gives up with `code` when the bound runs out (twice that of the wait for another
// CTA's hand-over: everything inside the CTA may be waiting behind that one, and the cause should be what reports).
template <class Misc>
__device__ __forceinline__ bool guarded_wait(uint64_t* bar, uint32_t parity, Misc* m, int code) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (m->abort_flag) return false;
    if (clock64() - t0 > 2 * m->wait_clocks) {
      m->abort_flag = code;   // reported to the caller's status word at kernel end
      return false;
    }
  }
  return m->abort_flag == 0;
}
// (the same for all lanes of the warp)
template <class Misc>
__device__ __forceinline__ bool given_up(const Misc* m) { return __any_sync(0xffffffffu, m->abort_flag != 0) != 0; }

__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r));
  return r != 0;
}

// Products of fp32 pairs (one instruction for two elements).
__device__ __forceinline__ uint64_t pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t pair(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ float2 unpair(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t mul_pair(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_pair(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
template <typename T16>
__device__ __forceinline__ uint32_t pack_pair(uint64_t v) {
  const float2 f = unpair(v);
  return pack2<T16>(f.x, f.y);
}

// 32 bytes per thread (a whole sector: a thread's row of the state would otherwise be moved half a sector at a time, and
// the load/store unit takes a cycle per sector touched).
__device__ __forceinline__ void ldg256(const void* p, uint64_t (&v)[4]) {
  asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
}
__device__ __forceinline__ void stg256(void* p, uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
  asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// ---------------------------------------------------------------------------- host side

// Look-back and chained modes: one CTA per SM, at least a tile for each.  Look-back: where it leaves few SMs out, every
// sequence in the same number of pieces, so that all items are at the same tokens at the same time and find B and C in L2
// (one sequence of 131 072 tokens, 16 pairs: 9 pieces each on 144 SMs).
inline int dealt_grid(int64_t units, int tiles, int chain) {
  int grid = (int)(units * tiles < kSms ? units * tiles : kSms);
  if (chain == 2) {
    const int most = (int)(kSms / units), pieces = most < tiles ? most : tiles;
    if (pieces > 1 && pieces * units >= kSms * 93 / 100) grid = (int)(pieces * units);
  }
  return grid;
}

// Ready flags of a launch, and behind them a bit for each CTA whose piece is to be walked again.
constexpr int kFlags = 2 * kSms + (kSms + 31) / 32;

// Launches a kernel over the tiles; where sequences are cut, behind the clearing of their ready flags, which it starts beside.
template <typename... Params, typename... Args>
int launch_tiles(void (*kernel)(Params...), int grid, int threads, int smem, const ScanParams& sp, cudaStream_t stream,
                 const Args&... args) {
  if (!sp.chain) return launch(kernel, grid, threads, smem, stream, args...);
  if (launch_clear_flags(sp.chain_flag, kFlags, stream) != SSD_OK) return SSD_ERR_CUDA;
  return launch_early(kernel, grid, threads, smem, stream, args...);
}

}  // namespace tc
}  // namespace ssd
