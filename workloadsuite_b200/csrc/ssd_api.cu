// C ABI of the SSD forward (declared in include/ssd_b200.h): argument
// validation, kernel choice, sequence segmentation and the host-buffer pipeline.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "ssd_common.cuh"

namespace {

constexpr int kAbiVersion = 3;
constexpr int kSmCount = 148;  // B200
constexpr int kTcTile = 128;   // tokens of a tensor-core tile

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

int elem_size(int dtype) { return dtype == SSD_DTYPE_F32 ? 4 : 2; }

int validate(const SsdArgs* a) {
  if (!a) return SSD_ERR_NULL_POINTER;
  if (a->batch <= 0 || a->seqlen <= 0 || a->nheads <= 0 || a->headdim <= 0 || a->dstate <= 0 || a->ngroups <= 0)
    return SSD_ERR_BAD_SHAPE;
  if (a->nheads % a->ngroups != 0) return SSD_ERR_BAD_SHAPE;
  if (a->chunk <= 0 || a->seqlen % a->chunk != 0) return SSD_ERR_BAD_CHUNK;
  if (a->dtype != SSD_DTYPE_F32 && a->dtype != SSD_DTYPE_F16 && a->dtype != SSD_DTYPE_BF16)
    return SSD_ERR_UNSUPPORTED;
  if (a->kernel != SSD_KERNEL_AUTO && a->kernel != SSD_KERNEL_SCAN_F32 && a->kernel != SSD_KERNEL_TCGEN05)
    return SSD_ERR_UNSUPPORTED;
  if (a->nsegments < 0 || a->wait_limit_ms < 0) return SSD_ERR_BAD_SHAPE;
  if ((int64_t)a->batch * a->nheads > 0x7fffffffLL) return SSD_ERR_TOO_LARGE;
  return SSD_OK;
}

int validate_pointers(const SsdArgs* a) {
  if (!a->X || !a->A || !a->B) return SSD_ERR_NULL_POINTER;
  const bool state_only = (a->flags & SSD_FLAG_STATE_ONLY) != 0;
  if (!state_only && (!a->Y || !a->C)) return SSD_ERR_NULL_POINTER;
  if (state_only && !a->final_state) return SSD_ERR_NULL_POINTER;
  return SSD_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int resolve_kernel(const SsdArgs* a) {
  if (a->kernel == SSD_KERNEL_SCAN_F32) return SSD_KERNEL_SCAN_F32;
  if (a->kernel == SSD_KERNEL_TCGEN05) return SSD_KERNEL_TCGEN05;
  // (states that are only 4-byte aligned go to the fp32 scan, which moves them element by element)
  const bool st16 = aligned16(a->initial_state) && aligned16(a->final_state);
  // Whole tiles only.  The tensor-core kernel takes any length, but rounds P, Xd and the copy of the state to 16 bits; other
  // lengths stay in fp32 with one rounding of Y unless the caller asks for that kernel.  bf16, 2 x 3001 tokens, against 64
  // bits: Y 1.66e-3 here (its own rounding) and 2.42e-3 there, final state 1.4e-7 and 2.4e-3.
  return ssd::tc_supports(*a) && st16 && a->seqlen % kTcTile == 0 ? SSD_KERNEL_TCGEN05 : SSD_KERNEL_SCAN_F32;
}

// First and one past the last byte of a tensor's elements.
struct Range {
  uintptr_t lo, hi;
  bool on(const Range& o) const { return lo < o.hi && o.lo < hi; }
};
Range range(const void* p, int64_t bytes) {
  const uintptr_t lo = reinterpret_cast<uintptr_t>(p);
  return {lo, p ? lo + (uintptr_t)bytes : lo};
}
Range range(const SsdArgs* a, const void* p, const int64_t* st, int heads, int inner, int size) {
  return range(p, ((a->batch - 1) * st[0] + (a->seqlen - 1) * st[1] + (heads - 1) * st[2] + inner) * size);
}
Range output(const SsdArgs* a) { return range(a, a->Y, a->y_stride, a->nheads, a->headdim, elem_size(a->dtype)); }

// Whether an output may share memory with an input (but for Y and Z): a call that is done again (below) needs its inputs as they were.
bool outputs_on_inputs(const SsdArgs* a) {
  const int e = elem_size(a->dtype);
  const int64_t heads = (int64_t)a->batch * a->nheads, state = heads * a->dstate * a->headdim * 4;
  const Range fin = range(a->final_state, state), ld = range(a->final_logdecay, heads * 4), y = output(a);
  const Range in[] = {range(a, a->X, a->x_stride, a->nheads, a->headdim, e),  range(a, a->B, a->b_stride, a->ngroups, a->dstate, e),
                      range(a, a->C, a->c_stride, a->ngroups, a->dstate, e),  range(a, a->dt, a->dt_stride, a->nheads, 1, e),
                      range(a, a->A, a->a_stride, a->nheads, 1, 4),           range(a->initial_state, state),
                      range(a->D, a->nheads * (a->flags & SSD_FLAG_D_IN_DTYPE ? e : 4))};
  for (const Range& r : in)
    if (r.on(y) || r.on(fin) || r.on(ld)) return true;
  const Range z = range(a, a->Z, a->z_stride, a->nheads, a->headdim, e);
  return z.on(fin) || z.on(ld);
}

// A state carried in place (or nearly): of cut sequences, the last piece must not write before the others have read.
bool final_on_initial(const SsdArgs* a) {
  const int64_t state = (int64_t)a->batch * a->nheads * a->dstate * a->headdim * 4;
  return range(a->final_state, state).on(range(a->initial_state, state));
}

// Y written over the gates.  A kernel that reads each gate ahead of its place in Y may do that, but not for a second time.
bool output_on_gate(const SsdArgs* a) { return range(a, a->Z, a->z_stride, a->nheads, a->headdim, elem_size(a->dtype)).on(output(a)); }

// Look-back calls of the tensor-core kernel that scan only the beginnings of long pieces first: what is walked again after all needs its
// inputs as they were.
bool by_beginnings(const SsdArgs* a) { return ssd::tc2_long_pieces(*a) && !outputs_on_inputs(a) && !output_on_gate(a); }

// The fp32 scan of a call whose kernel is not chosen by the caller: on the tensor cores at fp32 precision where they can
// (ssd_split.cu), unless the sequences are so short that the recurrence is through before the other kernel's pipeline has
// filled.  Its time goes with tokens x state, bf16: 8 heads of 17, 33 and 100 tokens, n 128: 8.5, 13.6 and 33 us, there 9.3, 9.4
// and 9.5; n 64: 5.8, 8.9 and 19, there 8.5, 8.5 and 8.8.  With more heads than SMs it falls behind earlier: 296 heads of 17 tokens,
// n 128, and of 33, n 64: 13.4 and 14.0 us, there 13.8 and 13.2; 1 280 of 17 tokens, n 128 and 64: 54 and 29 us, there 35 and 33.
bool use_split(const SsdArgs* a, int kernel) {
  const int64_t heads = (int64_t)a->batch * a->nheads;
  const int64_t least = heads <= kSmCount ? 3072 : heads <= 4 * kSmCount ? 2112 : 1536;
  return kernel == SSD_KERNEL_SCAN_F32 && (int64_t)a->seqlen * a->dstate >= least && a->kernel == SSD_KERNEL_AUTO && a->nsegments <= 1 &&
         !(a->flags & (SSD_FLAG_STATE_ONLY | SSD_FLAG_REUSE_SEGMENTS)) && aligned16(a->initial_state) && aligned16(a->final_state) &&
         ssd::split_supports(*a) && !outputs_on_inputs(a);
}

// The same as a query without pointers sees it.
bool split_by_shape(const SsdArgs* a) {
  SsdArgs s = *a;
  s.X = s.B = s.C = s.dt = nullptr;
  s.A = s.initial_state = nullptr;
  s.Y = nullptr;
  s.final_state = nullptr;
  return use_split(&s, resolve_kernel(&s));
}

// What the kernels that run these arguments work on: pairs of heads, or heads.
int64_t tc_units(const SsdArgs* a, bool split) { return split ? (int64_t)a->batch * a->nheads : ssd::tc2_units(*a); }

// Number of independently scanned segments per sequence and their length.
void resolve_segments(const SsdArgs* a, int kernel, bool split, int* nseg, int* seg_len) {
  const bool tensor = split || kernel == SSD_KERNEL_TCGEN05;
  const int tile = tensor ? kTcTile : ssd::scan_f32_tile_tokens();
  int want = a->nsegments;
  if (want <= 0) {
    if (tensor) {
      want = ssd::tc_default_segments(*a, tc_units(a, split));
    } else {
      const int64_t units = (int64_t)a->batch * a->nheads;
      // Two passes cost about 1.5x the work of one, so split only when the
      // unsplit grid would leave most of the SMs idle.
      want = units >= (3 * kSmCount) / 2 ? 1 : (int)((4 * kSmCount + units - 1) / units);
      const int max_by_len = std::max(1, a->seqlen / 256);
      want = std::min(want, max_by_len);
    }
  }
  want = std::max(1, std::min(want, 65535));
  int len = (a->seqlen + want - 1) / want;
  len = (len + tile - 1) / tile * tile;
  *seg_len = len;
  *nseg = (a->seqlen + len - 1) / len;
}

// The segments of the recurrence behind the tensor-core kernel at fp32 precision: its own, up to a head for every other SM.  Beyond,
// whole sequences take less (n 128, 3001 tokens: 24, 48 and 64 heads 353, 685 and 839 us cut, 950, 1 019 and 1 037 whole; 80, 120 and
// 160: 1 156, 1 623 and 2 264 cut, 1 046, 1 057 and 1 946 whole; n 64, 20 001 tokens: 64 heads 3 551 and 3 940, 80 4 760 and 4 006).
void redo_segments(const SsdArgs* a, int* nseg, int* seg_len) {
  *nseg = 1;
  if (2 * (int64_t)a->batch * a->nheads <= kSmCount) resolve_segments(a, SSD_KERNEL_SCAN_F32, false, nseg, seg_len);
  if (*nseg == 1) *seg_len = (int)align_up(a->seqlen, ssd::scan_f32_tile_tokens());
}

int chain_mode(const SsdArgs* a, int kernel, bool split, int nseg) {
  return split || kernel == SSD_KERNEL_TCGEN05 ? ssd::tc_chain_mode(*a, nseg, tc_units(a, split)) : 0;
}

// Scratch of a launch that hands states from CTA to CTA: one slot per CTA and head of the pair -- state, log-decay sum, ready flag.
constexpr size_t kSlots = 2 * (size_t)kSmCount;
size_t chain_bytes(size_t np) { return align_up(kSlots * np * sizeof(float), 256) + 2 * align_up(kSlots * sizeof(float), 256); }

// Scratch of the two passes over cut sequences: segment states and log-decay sums, and the states entering the segments (`keep`) or
// those written over the former.
size_t two_pass_bytes(const SsdArgs* a, int nseg, bool keep) {
  const size_t units = (size_t)a->batch * a->nheads, np = (size_t)a->dstate * a->headdim;
  return (keep ? 2 : 1) * align_up(units * nseg * np * sizeof(float), 256) + align_up(units * nseg * sizeof(float), 256);
}

// Scratch of the tensor-core kernel at fp32 precision and the recurrence behind it, which do not need theirs at the same time.
size_t split_bytes(const SsdArgs* a, int chain, int redo_nseg) {
  const size_t np = (size_t)a->dstate * a->headdim;
  return ssd::RedoWords::kBytes +
         std::max(chain != 0 ? chain_bytes(np) : 0, redo_nseg > 1 ? two_pass_bytes(a, redo_nseg, false) : 0);
}

// What a call of the tensor-core kernel at fp32 precision asks for.
size_t ask_by_shape(const SsdArgs* a) {
  int nseg, seg_len, redo_nseg, redo_len;
  resolve_segments(a, SSD_KERNEL_SCAN_F32, true, &nseg, &seg_len);
  redo_segments(a, &redo_nseg, &redo_len);
  return split_bytes(a, chain_mode(a, SSD_KERNEL_SCAN_F32, true, nseg), redo_nseg);
}

bool strides_mult(const int64_t* s, int m) { return s[0] % m == 0 && s[1] % m == 0 && s[2] % m == 0; }

void fill_params(const SsdArgs* a, ssd::ScanParams* p) {
  std::memset(p, 0, sizeof(*p));
  p->X = a->X; p->A = a->A; p->B = a->B; p->C = a->C; p->dt = a->dt; p->Y = a->Y;
  p->D = a->D; p->Z = a->Z;
  p->d_in_dtype = (a->flags & SSD_FLAG_D_IN_DTYPE) ? 1 : 0;
  p->status = a->status;
  p->batch = a->batch; p->seqlen = a->seqlen; p->nheads = a->nheads; p->p = a->headdim; p->n = a->dstate;
  p->ngroups = a->ngroups;
  for (int i = 0; i < 3; ++i) {
    p->xs[i] = a->x_stride[i]; p->as[i] = a->a_stride[i]; p->bs[i] = a->b_stride[i];
    p->cs[i] = a->c_stride[i]; p->dts[i] = a->dt_stride[i]; p->ys[i] = a->y_stride[i];
    p->zs[i] = a->z_stride[i];
  }
  const int per16 = 16 / elem_size(a->dtype);
  bool v = aligned16(a->X) && aligned16(a->B) && strides_mult(a->x_stride, per16) &&
           strides_mult(a->b_stride, per16) && a->headdim % 8 == 0 && a->dstate % 8 == 0;
  if (a->C) v = v && aligned16(a->C) && strides_mult(a->c_stride, per16);
  if (a->Y) v = v && aligned16(a->Y) && strides_mult(a->y_stride, per16);
  if (a->Z) v = v && aligned16(a->Z) && strides_mult(a->z_stride, per16);
  p->vec_ok = v ? 1 : 0;
  // the bound of the device-side waits: about a second by default; SM clocks run at up to ~2 GHz
  p->wait_clocks = a->wait_limit_ms > 0 ? (long long)a->wait_limit_ms * 2000000LL : 2000000000LL;
  p->inject_lost_handover = (a->flags & SSD_FLAG_INJECT_LOST_HANDOVER) ? 1 : 0;
}

// The gate rows are read with 16-byte loads by the fused epilogue; the stand-alone kernel has a scalar path.
bool z_vector_friendly(const SsdArgs* a) {
  if (!a->Z) return true;
  const int per16 = 16 / elem_size(a->dtype);
  return aligned16(a->Z) && strides_mult(a->z_stride, per16);
}

// The tensor-core kernels move the fp32 states as 16-byte vectors.
bool states_aligned16(const SsdArgs* a) { return aligned16(a->initial_state) && aligned16(a->final_state); }

int launch_kernel(int kernel, const SsdArgs* a, const ssd::ScanParams& prm, cudaStream_t stream) {
  if (kernel == SSD_KERNEL_TCGEN05) return ssd::launch_tc2(*a, prm, stream);
  return ssd::launch_scan_f32(prm, a->dtype, stream, a->kernel != SSD_KERNEL_AUTO);
}

}  // namespace

extern "C" {

int ssd_b200_abi_version(void) { return kAbiVersion; }

const char* ssd_b200_strerror(int code) {
  switch (code) {
    case SSD_OK: return "ok";
    case SSD_ERR_NULL_POINTER: return "a required pointer is NULL";
    case SSD_ERR_BAD_SHAPE: return "invalid shape (sizes must be positive; n_heads must be divisible by n_groups)";
    case SSD_ERR_BAD_CHUNK: return "seq_len must be a positive multiple of chunk";
    case SSD_ERR_UNSUPPORTED: return "shape, dtype or kernel not supported by this build";
    case SSD_ERR_WORKSPACE: return "workspace missing or too small";
    case SSD_ERR_CUDA: return "a CUDA runtime call failed";
    case SSD_ERR_MISALIGNED: return "pointer or stride not aligned for the selected kernel";
    case SSD_ERR_TOO_LARGE: return "size beyond a fixed limit";
    case SSD_ERR_DEVICE_WAIT: return "a bounded device-side wait ran out; the results are incomplete";
    default: return "unknown error code";
  }
}

const char* ssd_b200_kernel_name(const SsdArgs* args) {
  if (validate(args) != SSD_OK) return "invalid";
  return resolve_kernel(args) == SSD_KERNEL_TCGEN05 ? "tcgen05" : "scan_f32";
}

int ssd_b200_plan(const SsdArgs* args, int32_t* kernel_out, int32_t* nsegments_out, int32_t* launches_out) {
  const int rc = validate(args);
  if (rc != SSD_OK) return rc;
  const int kernel = resolve_kernel(args);
  const bool split = use_split(args, kernel);
  int nseg, seg_len;
  resolve_segments(args, kernel, split, &nseg, &seg_len);
  const bool state_only = (args->flags & SSD_FLAG_STATE_ONLY) != 0;
  int launches = 1;
  if (nseg > 1) {
    const bool chained = chain_mode(args, kernel, split, nseg) != 0;
    launches = chained ? 1 : (state_only ? 2 : 3);
    if (!chained && (args->flags & SSD_FLAG_REUSE_SEGMENTS)) launches -= 1;
  }
  if (split) launches += 1;   // (the scan that does the call again where it has to)
  if (kernel_out) *kernel_out = kernel;
  if (nsegments_out) *nsegments_out = nseg;
  if (launches_out) *launches_out = launches;
  return SSD_OK;
}

size_t ssd_b200_workspace_bytes(const SsdArgs* args) {
  if (validate(args) != SSD_OK) return 0;
  const int kernel = resolve_kernel(args);
  const bool split = use_split(args, kernel);
  int nseg, seg_len;
  resolve_segments(args, kernel, split, &nseg, &seg_len);
  if (split) return ask_by_shape(args);
  if (nseg <= 1) return 0;
  return chain_mode(args, kernel, split, nseg) != 0 ? chain_bytes((size_t)args->dstate * args->headdim) : two_pass_bytes(args, nseg, true);
}

// The forward proper.  `fuse_epilogue`: the selected kernel applies D / Z itself; otherwise they are dropped here
// and ssd_b200_forward() runs the stand-alone epilogue kernel afterwards.
// `fold_in_place`: the states entering the segments are written over those they are made of, in half the scratch.
static int forward_impl(const SsdArgs* args, void* stream_v, bool fuse_epilogue, bool fold_in_place) {
  int rc = validate(args);
  if (rc != SSD_OK) return rc;
  rc = validate_pointers(args);
  if (rc != SSD_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  const int kernel = resolve_kernel(args);
  if (kernel == SSD_KERNEL_TCGEN05 && !ssd::tc_supports(*args)) return SSD_ERR_UNSUPPORTED;
  if (kernel == SSD_KERNEL_TCGEN05 && !states_aligned16(args)) return SSD_ERR_MISALIGNED;
  if (kernel == SSD_KERNEL_SCAN_F32 && !ssd::scan_f32_supports(args->headdim, args->dstate))
    return SSD_ERR_UNSUPPORTED;

  const bool split = use_split(args, kernel);
  int nseg, seg_len;
  resolve_segments(args, kernel, split, &nseg, &seg_len);
  const bool state_only = (args->flags & SSD_FLAG_STATE_ONLY) != 0;
  const int64_t units = (int64_t)args->batch * args->nheads;
  const int64_t np = (int64_t)args->dstate * args->headdim;

  ssd::ScanParams prm;
  fill_params(args, &prm);
  prm.seg_len = seg_len;
  prm.nseg = nseg;
  if (!fuse_epilogue || state_only) prm.D = nullptr, prm.Z = nullptr;
  // whole sequences, or pieces of them within one launch: the caller's states and sums directly
  ssd::ScanParams whole = prm;
  whole.compute_y = state_only ? 0 : 1;
  whole.init = args->initial_state;
  whole.init_unit_stride = np;
  whole.fin = args->final_state;
  whole.fin_unit_stride = np;
  whole.fin_ld = args->final_logdecay;
  whole.finld_unit_stride = 1;
  if (nseg <= 1 && !split) return launch_kernel(kernel, args, whole, stream);

  if (!args->workspace || args->workspace_bytes < (fold_in_place ? two_pass_bytes(args, nseg, false) : ssd::least_workspace(args)))
    return SSD_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(args->workspace) & 255) return SSD_ERR_MISALIGNED;
  const int chain = chain_mode(args, kernel, split, nseg);
  if (chain != 0 || split) {
    // one launch: the pieces of a sequence pass their state through the workspace (see chain_bytes())
    char* ws = static_cast<char*>(args->workspace);
    ssd::ScanParams pc = whole;
    if (split) {
      pc.redo = reinterpret_cast<int32_t*>(ws);
      ws += ssd::RedoWords::kBytes;
    }
    if (chain != 0) {
      pc.chain = chain;
      pc.fin_on_init = chain == 2 && !split && final_on_initial(args) ? 1 : 0;
      pc.beginnings = chain == 2 && (split || by_beginnings(args)) ? 1 : 0;
      pc.chain_state = reinterpret_cast<float*>(ws);
      pc.chain_ld = reinterpret_cast<float*>(ws + align_up(kSlots * np * sizeof(float), 256));
      pc.chain_flag = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(pc.chain_ld) + align_up(kSlots * sizeof(float), 256));   // (cleared by the launch)
    }
    if (!split) return launch_kernel(kernel, args, pc, stream);
    const bool scan_at_once = fuse_epilogue && output_on_gate(args);   // (by the words that say that it is to be done again)
    if (scan_at_once) {
      if (cudaMemsetAsync(pc.redo, 0, ssd::RedoWords::kBytes, stream) != cudaSuccess || cudaMemsetAsync(pc.redo, 1, sizeof(int32_t), stream) != cudaSuccess)
        return SSD_ERR_CUDA;
      rc = SSD_OK;
    } else {
      rc = ssd::launch_split(*args, pc, stream);
    }
    if (rc == SSD_OK) {
      // the recurrence, where the call has to be done again: in segments, if there is scratch for them
      redo_segments(args, &nseg, &seg_len);
      if (args->workspace_bytes < split_bytes(args, chain, nseg)) nseg = 1, seg_len = (int)align_up(args->seqlen, ssd::scan_f32_tile_tokens());
      whole.nseg = nseg;
      whole.seg_len = seg_len;
      whole.redo = pc.redo;
      whole.redo_n = scan_at_once ? 1 : ssd::split_grid(*args, chain);
      whole.chain_state = reinterpret_cast<float*>(ws);
      whole.chain_ld = reinterpret_cast<float*>(ws + align_up((size_t)units * nseg * np * sizeof(float), 256));
      return ssd::launch_scan_f32(whole, args->dtype, stream);
    }
    if (rc != SSD_ERR_UNSUPPORTED) return rc;
    SsdArgs scan = *args;   // (strides that a tensor map cannot have)
    scan.kernel = SSD_KERNEL_SCAN_F32;
    if (args->workspace_bytes < ssd_b200_workspace_bytes(&scan)) scan.nsegments = 1;
    if (!whole.D && !whole.Z) scan.D = nullptr, scan.Z = nullptr;   // (the caller of this applies them)
    return ssd_b200_forward(&scan, stream);
  }

  float* seg_states = static_cast<float*>(args->workspace);
  const size_t st_bytes = align_up((size_t)units * nseg * np * sizeof(float), 256);   // (see two_pass_bytes())
  float* seg_in = fold_in_place ? seg_states : reinterpret_cast<float*>(static_cast<char*>(args->workspace) + st_bytes);
  float* seg_ld = reinterpret_cast<float*>(static_cast<char*>(args->workspace) + (fold_in_place ? 1 : 2) * st_bytes);

  // pass 1: every segment from a zero state, state and log-decay sum only
  if (!(args->flags & SSD_FLAG_REUSE_SEGMENTS)) {
    ssd::ScanParams p1 = prm;
    p1.compute_y = 0;
    p1.Y = nullptr;
    p1.init = nullptr;
    p1.fin = seg_states;
    p1.fin_unit_stride = (int64_t)nseg * np;
    p1.fin_seg_stride = np;
    p1.fin_ld = seg_ld;
    p1.finld_unit_stride = nseg;
    p1.finld_seg_stride = 1;
    rc = launch_kernel(kernel, args, p1, stream);
    if (rc != SSD_OK) return rc;
  }

  // fold: state entering each segment (kept apart from the zero-start states, so that those can be
  // reused), final state, total log-decay
  rc = ssd::launch_fold(seg_states, (int64_t)nseg * np, np, seg_ld, nseg, 1, args->initial_state, nullptr,
                        args->final_state, args->final_logdecay, nseg, state_only ? nullptr : seg_in, units, np,
                        stream);
  if (rc != SSD_OK || state_only) return rc;

  // pass 2: every segment again, seeded with its incoming state, writing Y
  ssd::ScanParams p2 = prm;
  p2.compute_y = 1;
  p2.init = seg_in;
  p2.init_unit_stride = (int64_t)nseg * np;
  p2.init_seg_stride = np;
  p2.fin = nullptr;
  p2.fin_ld = nullptr;
  return launch_kernel(kernel, args, p2, stream);
}

int ssd_b200_forward(const SsdArgs* args, void* stream_v) {
  int rc = validate(args);
  if (rc != SSD_OK) return rc;
  const bool state_only = (args->flags & SSD_FLAG_STATE_ONLY) != 0;
  const int chosen = resolve_kernel(args);
  SsdArgs scan;
  bool in_place = false;
  if (chosen == SSD_KERNEL_SCAN_F32 && args->kernel == SSD_KERNEL_AUTO && args->dtype != SSD_DTYPE_F32) {
    const size_t given = args->workspace ? args->workspace_bytes : 0;
    if (use_split(args, chosen)) {
      // Without scratch that the tensor-core kernel can do with: the recurrence, which needs none for whole sequences.
      if (given < ssd::least_workspace(args) || (reinterpret_cast<uintptr_t>(args->workspace) & 255)) {
        scan = *args;
        scan.kernel = SSD_KERNEL_SCAN_F32;
        args = &scan;
      }
    } else if (split_by_shape(args) && given < ssd_b200_workspace_bytes(args) && given >= ask_by_shape(args)) {
      // An output on an input, or states that are not 16-byte aligned, make a call the recurrence's that by its shape is the
      // tensor-core kernel's: it does with the scratch that the shape asked for, in the segments that it would be done again in.
      int seg_len;
      scan = *args;
      scan.kernel = SSD_KERNEL_SCAN_F32;
      redo_segments(args, &scan.nsegments, &seg_len);
      in_place = scan.nsegments > 1;
      args = &scan;
    }
  }
  if (state_only || (!args->D && !args->Z)) return forward_impl(args, stream_v, false, in_place);
  // skip and gate of model_ref.py:116-118: fused into the tensor-core kernels, a kernel of their own otherwise
  const int kernel = resolve_kernel(args);
  const bool split = use_split(args, kernel);
  const bool can = kernel == SSD_KERNEL_TCGEN05 ? ssd::tc_supports(*args) && ssd::tc2_fuses_epilogue(*args) : split && ssd::split_fuses_epilogue(*args);
  // (Y over the gates: by the recurrence, with both in it, as a kernel behind it would read its results for gates)
  const bool fuse = (can && z_vector_friendly(args) && !(args->flags & SSD_FLAG_SEPARATE_EPILOGUE)) || (split && output_on_gate(args));
  rc = forward_impl(args, stream_v, fuse, in_place);
  if (rc != SSD_OK || fuse) return rc;
  ssd::ScanParams ep;
  fill_params(args, &ep);
  return ssd::launch_epilogue(ep, args->dtype, static_cast<cudaStream_t>(stream_v));
}

int ssd_b200_fold_states(const float* states, int64_t states_shard_stride, const float* logdecay,
                         int64_t logdecay_shard_stride, const float* initial, float* out, int32_t nshards,
                         int32_t rank, int64_t units, int64_t np, void* stream) {
  if (!states || !logdecay || !out) return SSD_ERR_NULL_POINTER;
  if (nshards <= 0 || rank < 0 || rank > nshards || units <= 0 || np <= 0) return SSD_ERR_BAD_SHAPE;
  return ssd::launch_fold(states, np, states_shard_stride, logdecay, 1, logdecay_shard_stride, initial, out, nullptr,
                          nullptr, rank, nullptr, units, np, static_cast<cudaStream_t>(stream));
}

}  // extern "C"

size_t ssd::least_workspace(const SsdArgs* args) {
  const size_t need = ssd_b200_workspace_bytes(args);
  if (need == 0) return 0;
  const int kernel = resolve_kernel(args);
  if (!use_split(args, kernel)) return need;
  int nseg, seg_len;
  resolve_segments(args, kernel, true, &nseg, &seg_len);
  return split_bytes(args, chain_mode(args, kernel, true, nseg), 1);
}

bool ssd::whole_without_scratch(const SsdArgs* args) {
  if (validate(args) != SSD_OK) return false;
  const int kernel = resolve_kernel(args);
  int nseg, seg_len;
  resolve_segments(args, SSD_KERNEL_SCAN_F32, false, &nseg, &seg_len);
  return use_split(args, kernel) && nseg == 1;
}
