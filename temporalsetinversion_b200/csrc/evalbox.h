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

// Bytes of operand log a reverse call needs for n boxes: an entry per box and
// instruction, and one for the lanes without a box.
inline size_t evalbox_log_bytes(size_t n, uint32_t len) { return n * (len ? len : 1u) * 16u + 16u; }

// A warp's register rows in shared memory: how many boxes it takes, the
// columns of a row and a lane's column.  A row's offset has 16 bits, that of
// the row past the last register included; the lanes that find no column of
// their own share one that no box has.
inline __host__ __device__ uint32_t narrow_boxes(uint32_t nregs) { return nregs < 256u ? 32u : 16u; }
inline __host__ __device__ uint32_t narrow_columns(uint32_t nregs) { return nregs < 256u ? 32u : 17u; }
inline __host__ __device__ uint32_t narrow_column(uint32_t nregs, uint32_t lane) {
  const uint32_t last = narrow_columns(nregs) - 1u;
  return lane < last ? lane : last;
}
inline size_t narrow_bytes(uint32_t nregs) {
  return (((size_t)(nregs + 1u) * narrow_columns(nregs) * 8u + 15u) & ~size_t(15)) + 32u * 16u;
}
// Most dynamic shared memory the narrow form is launched with.
constexpr size_t kNarrowMax = 66u << 10;

cudaError_t launch_evalbox(bool directed, const EvalTape &t, uint32_t n, const float *boxes, bool reverse, float *out,
                           float4 *log, cudaStream_t st);
// Loads the kernels on the current device and sets their shared memory
// limits, so that launches do neither.
cudaError_t evalbox_preload();

}  // namespace tsi
