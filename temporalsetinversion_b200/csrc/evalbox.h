// evalbox.h — interval evaluation of one tape on a list of space-time boxes:
// the tape as the kernels see it, and their launch.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_types.h"

namespace tsi {

struct EvalTape {
  const uint2 *code;
  uint32_t len, nregs, out_reg;
  WideDev wide;  // nbundles == 0: no bundled form
  int sm_count;
};

// Bytes of operand log a reverse call needs for n boxes.
inline size_t evalbox_log_bytes(size_t n, uint32_t len) { return n * (len ? len : 1u) * 16u; }

cudaError_t launch_evalbox(bool directed, const EvalTape &t, uint32_t n, const float *boxes, bool reverse, float *out,
                           float4 *log, cudaStream_t st);
// Loads the kernels on the current device and sets their shared memory
// limits, so that launches do neither.
cudaError_t evalbox_preload();

}  // namespace tsi
