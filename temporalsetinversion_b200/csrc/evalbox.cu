// evalbox.cu — interval evaluation of one tape on a list of space-time boxes.
//
// The body of compute.wgsl:3632-3970 without the octree: forward tape,
// reverse interval AD seeded with 1 at the output, sensitivities of the four
// arguments, by the interpreters of the refinement kernel.  With one thread
// per box, registers and log in global memory, every tape instruction waited
// for its operands from L2.
//
// Many boxes: a warp per 32 of them (narrow_interp.cuh), bound by the
// instructions it issues per tape instruction.  Few boxes on a long tape: a
// block per box (wide_interp.cuh), bound by the latency of a bundle's step.
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "evalbox.h"
#include "interval.cuh"
#include "narrow_interp.cuh"
#include "wide_interp.cuh"

namespace tsi {

// Shared memory of a block: the boxes' register rows and the instruction
// buffer, or a cell's values and sensitivities.
extern __shared__ __align__(16) unsigned char evalbox_smem[];

__device__ __forceinline__ void load_box(const float *b, Iv v[4]) {
  for (int q = 0; q < 4; ++q) v[q] = Iv{b[2 * q], b[2 * q + 1]};
}
__device__ __forceinline__ void store_box(float *o, Iv f, const Iv sens[4]) {
  o[0] = f.lo;
  o[1] = f.hi;
  for (int q = 0; q < 4; ++q) {
    o[2 + 2 * q] = sens[q].lo;
    o[3 + 2 * q] = sens[q].hi;
  }
}

// One warp, up to 32 boxes, each in a column of its own (evalbox.h).  The
// lanes without a box work on the last one in a column that no box has: a
// lane that ran ahead in a shared one would change what the others still
// read.  Their operands go to one place behind the log, read as anything.
// 60000 boxes on a 4697-instruction tape with sensitivities: a call takes
// 12.8 ms with a thread per box, 2.5 ms so.
template <bool D>
__global__ void __launch_bounds__(32) evalbox_narrow(EvalTape T, uint32_t n, const float *__restrict__ boxes,
                                                     int reverse, float *__restrict__ out, float4 *log) {
  const uint32_t lane = threadIdx.x, per = narrow_boxes(T.nregs);
  const size_t first = (size_t)blockIdx.x * per, len = max(T.len, 1u);
  const uint32_t cols = (uint32_t)min((size_t)per, (size_t)n - first);
  NarrowRows R;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(evalbox_smem);
  R.stride = narrow_columns(T.nregs) * 8u;
  R.rf = base + narrow_column(T.nregs, lane) * 8u;
  R.sink = T.nregs * R.stride;
  R.prog = base + ((R.sink + R.stride + 15u) & ~15u);
  R.log_step = lane < cols ? cols : 0u;
  const size_t box = first + min(lane, cols - 1u);
  Iv v[4], sens[4] = {iv(0.0f), iv(0.0f), iv(0.0f), iv(0.0f)};
  load_box(boxes + box * 8u, v);
  // `cols` columns of at most len entries
  float4 *lg = !reverse ? nullptr : lane < cols ? log + first * len + lane : log + n * len;
  uint32_t nlog = 0;
  const Iv f = narrow_forward<D>(T.code, T.len, T.out_reg, R, lane, v[0], v[1], v[2], v[3], lg, nullptr, nlog);
  if (reverse) {
    bool bad = false;
    narrow_reverse<D>(T.code, T.len, T.nregs, T.out_reg, R, lane, lg, nlog, true, false, sens, bad);
  }
  if (lane < cols) store_box(out + box * 10u, f, sens);
}

// One block per box at a time, on the bundled form.  511 boxes on a
// 1177-instruction tape, without sensitivities: a call takes 371 us with a
// thread per box, 164 with a warp per 32, 53 so (39 of them with one box).
template <bool D>
__global__ void __launch_bounds__(256) evalbox_wide(EvalTape T, uint32_t n, const float *__restrict__ boxes,
                                                    int reverse, float *__restrict__ out) {
  __shared__ float2 s_sens[4];
  const CellArray<false> V(evalbox_smem), G(evalbox_smem + (T.wide.nvalues + 2u) * 8u);
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    Iv v[4], sens[4] = {iv(0.0f), iv(0.0f), iv(0.0f), iv(0.0f)};
    load_box(boxes + (size_t)i * 8u, v);
    const Iv f = cell_forward<D, false>(T.wide, V, G, false, nullptr, nullptr, v[0], v[1], v[2], v[3], v[3]);
    if (reverse) {
      cell_reverse16<D>(T.wide, V, G, s_sens);
      for (int q = 0; q < 4; ++q) sens[q] = Iv{s_sens[q].x, s_sens[q].y};
    }
    if (threadIdx.x == 0) store_box(out + (size_t)i * 10u, f, sens);
    __syncthreads();  // the field and the sensitivities are read before the next box writes its values
  }
}

// elementwise checks of the f32 math and min/max (GPU math tests)
__global__ void math_kernel(int which, uint32_t n, const float *a, const float *b, float *out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float r;
  switch (which) {
    case 0: r = fm_sin(a[i]); break;
    case 1: r = fm_exp(a[i]); break;
    case 2: r = fm_log(a[i]); break;
    case 3: r = fm_atan2(a[i], b[i]); break;
    case 4: r = fm_powi(a[i], (int)b[i]); break;
    case 5: r = fm_min(a[i], b[i]); break;
    case 6: r = fm_max(a[i], b[i]); break;
    case 7: r = fminf(a[i], b[i]); break;
    case 8: r = fmaxf(a[i], b[i]); break;
    case 9: r = fm_rcp_in(a[i]); break;
    case 10: r = fm_div_in(a[i], b[i], fm_rcp_in(b[i])); break;
    case 11: r = fm_sqrt_in(a[i]); break;
    case 12: r = IA<false>::quadrant(a[i]); break;
    default: r = 0.0f; break;
  }
  out[i] = r;
}

constexpr size_t kWideMax = 200u << 10;  // most dynamic shared memory of a block per box

template <bool D>
static cudaError_t launch(const EvalTape &t, uint32_t n, const float *boxes, bool reverse, float *out, float4 *log,
                          cudaStream_t st) {
  const WideDev &W = t.wide;
  const size_t wide = ((size_t)W.nvalues + 2u) * 8u + (reverse ? (size_t)W.gslots * 8u : 0u);
  if (W.nbundles && wide <= kWideMax && (!reverse || W.rev16)) {
    int bps = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, evalbox_wide<D>, 256, wide);
    if (e != cudaSuccess) return e;
    const uint64_t grid = (uint64_t)bps * t.sm_count, waves = grid ? (n + grid - 1) / grid : 0;
    // A wave of blocks takes as long as four to five instructions per bundle
    // of the narrow form.  Both ways in microseconds (forward, reverse): 277
    // instructions in 27 bundles, 2000 boxes 100, 137 against 112, 148; 20000
    // boxes 418, 699 against 266, 306.  4697 in 34, 20000 boxes 619, 2080
    // against 765, 1923; 60000 boxes 1658, 6035 against 1224, 2541.
    if (waves && t.len >= 4u * (uint64_t)W.nbundles * waves) {
      evalbox_wide<D><<<(unsigned)(n < grid ? n : grid), 256, wide, st>>>(t, n, boxes, reverse, out);
      return cudaGetLastError();
    }
  }
  const uint32_t per = narrow_boxes(t.nregs);
  evalbox_narrow<D><<<(n + per - 1u) / per, 32, narrow_bytes(t.nregs), st>>>(t, n, boxes, reverse, out, log);
  return cudaGetLastError();
}

cudaError_t launch_evalbox(bool directed, const EvalTape &t, uint32_t n, const float *boxes, bool reverse, float *out,
                           float4 *log, cudaStream_t st) {
  return directed ? launch<true>(t, n, boxes, reverse, out, log, st) : launch<false>(t, n, boxes, reverse, out, log, st);
}

cudaError_t evalbox_preload() {
  static std::mutex mu;
  static bool done[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
  auto limit = [](auto *kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  e = limit(evalbox_narrow<true>, kNarrowMax);
  if (e == cudaSuccess) e = limit(evalbox_narrow<false>, kNarrowMax);
  if (e == cudaSuccess) e = limit(evalbox_wide<true>, kWideMax);
  if (e == cudaSuccess) e = limit(evalbox_wide<false>, kWideMax);
  if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
  return e;
}

cudaError_t launch_math(int which, uint32_t n, const float *a, const float *b, float *out, cudaStream_t st) {
  math_kernel<<<(n + 255) / 256, 256, 0, st>>>(which, n, a, b, out);
  return cudaGetLastError();
}

}  // namespace tsi
