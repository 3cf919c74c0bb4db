// Shared definitions of the SSD forward kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ssd_b200.h"

namespace ssd {

// Device status codes written to SsdArgs::status (0 = fine).
enum : int {
  STATUS_OK = 0,
  STATUS_WAIT_TIMEOUT_TMA = 1,   // a bounded wait for a TMA transfer ran out
  STATUS_WAIT_TIMEOUT_MMA = 2,   // a bounded wait for a tcgen05 commit ran out
  STATUS_WAIT_TIMEOUT_SYNC = 3,  // a bounded wait between warps of one CTA ran out
  STATUS_TMEM_ALLOC = 4,         // tensor memory could not be allocated
  STATUS_BAD_SMEM_ALIGNMENT = 5, // dynamic shared memory did not start on a 1024-byte boundary
  STATUS_WAIT_TIMEOUT_CHAIN = 6  // a bounded wait for the previous segment of a chained sequence ran out
};

// Words of ScanParams::redo: one per CTA of the tensor-core kernel at fp32 precision, and the counters of the scan behind it.
struct RedoWords {
  static constexpr int kNext = 148, kScanned = 149, kFolded = 150, kBytes = 768;
};

// One launch of a scan over [seg_begin, seg_end) of every (batch, head) unit.
// Strides are in elements.  "unit" = batch * nheads + head.
struct ScanParams {
  const void* X;
  const float* A;
  const void* B;
  const void* C;
  const void* dt;      // may be null
  void* Y;             // may be null when compute_y == 0
  const float* init;   // state entering segment (unit, seg); null = zeros
  int64_t init_unit_stride, init_seg_stride;
  float* fin;          // state leaving segment (unit, seg); may be null
  int64_t fin_unit_stride, fin_seg_stride;
  float* fin_ld;       // sum of A over the segment; may be null
  int64_t finld_unit_stride, finld_seg_stride;
  int32_t* status;     // may be null
  int batch, seqlen, nheads, p, n, ngroups;
  int seg_len, nseg;
  int compute_y;
  int vec_ok;          // all row starts 16-byte aligned
  long long wait_clocks;   // bound of every device-side wait, in SM clock cycles
  int inject_lost_handover;   // SSD_FLAG_INJECT_LOST_HANDOVER: CTA 0 of a chained launch leaves without working
  // Chained mode (tensor-core kernels; 1): a piece of a sequence starts from the state that the
  // piece before it (on the neighbouring CTA) left in chain_state, once chain_flag says it is there.
  // Look-back mode (2): chain_state / chain_ld hold each CTA's state-from-zero and log-decay sum of the last
  // piece of its range; a piece folds those of the CTAs before it.
  int chain;
  float* chain_state;     // [slot][p/4][n][4], slot = 2 * CTA + head of the pair (0 where a kernel works on one head)
  float* chain_ld;        // [slot] running sum of the log-decay up to the end of the piece
  int32_t* chain_flag;    // [slot], cleared by the launch
  int fin_on_init;        // look-back: `fin` and `init` share memory: a state is written once all pieces of its sequence have read theirs
  int beginnings;         // look-back: of long pieces only the beginning may be scanned first (no output on an input)
  int walk_again;         // the launch behind such a one: pieces that what entered them did not vanish in are walked again
  // The tensor-core kernel at fp32 precision writes a word per CTA: not 0 if the fp32 scan has to do the call again.  The scan, when
  // given them (redo_n of them), starts beside that kernel's end and leaves at once if all are 0; cut sequences' segment states and
  // log-decay sums are then in chain_state and chain_ld, [unit][segment].
  int32_t* redo;
  int redo_n;
  // Optional epilogue Y <- (Y + x * D[head]) * silu(z) (model_ref.py:116-118); either pointer may be null.
  const float* D;         // [h], fp32 or (d_in_dtype) elements of the tensors' type
  const void* Z;          // [b,s,h,p], strides zs
  int d_in_dtype;
  int64_t xs[3], as[3], bs[3], cs[3], dts[3], ys[3], zs[3];
};

template <typename T> struct Cvt;
template <> struct Cvt<float> {
  static __device__ __forceinline__ float to_f(float v) { return v; }
  static __device__ __forceinline__ float from_f(float v) { return v; }
};
template <> struct Cvt<__half> {
  static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f(float v) { return __float2half_rn(v); }
};
template <> struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
};

// Enqueues a kernel and says whether THIS launch failed: cudaGetLastError() behind a launch also reports (once) what an
// earlier call of the thread left, and a launch that is called failed is made again -- a step would be applied twice.
template <typename... Params, typename... Args>
inline int launch(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...) == cudaSuccess ? SSD_OK : SSD_ERR_CUDA;
}

// The same for a kernel that may start beside the end of the one ahead, and waits for that end itself.
template <typename... Params, typename... Args>
inline int launch_early(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...) == cudaSuccess ? SSD_OK : SSD_ERR_CUDA;
}

// D[head] of the skip term.
template <typename T>
__device__ __forceinline__ float load_skip(const ScanParams& p, int head) {
  return p.d_in_dtype ? Cvt<T>::to_f(reinterpret_cast<const T*>(p.D)[head]) : p.D[head];
}

// Launchers implemented in the kernel translation units.  Each returns an
// SSD_ERR_* code and enqueues on `stream`.
int launch_scan_f32(const ScanParams& prm, int dtype, cudaStream_t stream, bool in_line = true);   // in_line: as the token recurrence, not chunked
bool scan_f32_supports(int p, int n);
int scan_f32_tile_tokens();

// Y <- (Y + x * D[head]) * silu(z) in place over [b,s,h,p] (for the kernels that do not fuse it).
int launch_epilogue(const ScanParams& p, int dtype, cudaStream_t stream);

// `incoming` (nullable, may alias `states`) receives the state entering every segment, in the layout of `states`.
int launch_fold(const float* states, int64_t st_unit_stride, int64_t st_seg_stride, const float* ld,
                int64_t ld_unit_stride, int64_t ld_seg_stride, const float* init, float* out_single,
                float* out_final, float* out_ld, int upto, float* incoming, int64_t units, int64_t np,
                cudaStream_t stream);

// tensor-core kernel (ssd_tc2.cu)
bool tc_supports(const SsdArgs& a);
bool tc2_fuses_epilogue(const SsdArgs& a);
int64_t tc2_units(const SsdArgs& a);   // pairs of heads
int tc_default_segments(const SsdArgs& a, int64_t units);
int tc_chain_mode(const SsdArgs& a, int nseg, int64_t units);   // 1: chained, 2: look-back (one launch each); 0: two passes + fold
bool tc2_long_pieces(const SsdArgs& a);   // look-back, by shape: ScanParams::beginnings, and one more launch
int launch_tc2(const SsdArgs& a, const ScanParams& prm, cudaStream_t stream);
int launch_clear_flags(int32_t* flags, int count, cudaStream_t stream);   // to zero, beside what is launched next

// tensor-core kernel at fp32 precision (ssd_split.cu)
bool split_supports(const SsdArgs& a);
bool split_fuses_epilogue(const SsdArgs& a);
int split_grid(const SsdArgs& a, int chain);   // CTAs, each of which writes its word of ScanParams::redo
int launch_split(const SsdArgs& a, const ScanParams& prm, cudaStream_t stream);   // SSD_ERR_UNSUPPORTED: nothing was enqueued

size_t least_workspace(const SsdArgs* a);   // what the call can do with (ssd_b200_workspace_bytes(): what it asks for)
bool whole_without_scratch(const SsdArgs* a);   // asks for some, but without it is the recurrence over whole sequences

}  // namespace ssd
