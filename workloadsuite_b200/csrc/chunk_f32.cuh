// The fp32 scan in chunked form (ssd_chunk_f32.cu), which launch_scan_f32() takes where it is the faster one.
#pragma once

#include "ssd_common.cuh"

namespace ssd {

bool chunk_f32_takes(const ScanParams& prm);   // fp32 tensors of this shape and alignment
bool chunk_f32_pays(const ScanParams& prm);    // and is faster than the recurrence there
int launch_chunk_f32(const ScanParams& prm, cudaStream_t stream);

}  // namespace ssd
