// trace.cu — octree ray tracer, one thread per pixel (compute.wgsl `rt_main`
// 4650-4688 with `cinematic` off, `trace` 4189-4403).
//
// Each pixel walks the octree top-down (trace_walk.cuh) and is shaded by the
// age colour of the leaf it hits.  The cinematic path tracer is in
// cinematic.cu.  This file is compiled with --fmad=false so that the
// arithmetic is the plain f32 sequence of the reference (no FMA
// contraction).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "device_types.h"
#include "fmath.cuh"
#include "interp.cuh"
#include "trace_params.h"
#include "trace_walk.cuh"

namespace tsi {

constexpr uint32_t kTraceWarps = 4;  // of a block

// FAST: normals by finite differences of the tape (a separate instance, so
// the plain tracer carries no point-evaluation code).
template <bool FAST>
__device__ __forceinline__ void trace_pixels(const TraceParams *__restrict__ Tp) {
  const TraceParams &T = *Tp;
  // a block covers a 16x8 pixel tile and each warp a 4x8 column of it, so
  // the rays of a warp are close together and walk similar nodes (8x4 and
  // 8x8-per-two-warps tiles measured 1-2% slower on the benchmark frames).
  // Blocks of four warps leave the SMs more evenly than blocks of eight: a
  // 640x360 frame 0.168 to 0.162 ms, 1280x720 0.215 to 0.207, 1920x1080 the
  // same; one or two warps gain nothing more.
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t px = blockIdx.x * (4u * kTraceWarps) + warp * 4u + (lane & 3u);
  const uint32_t py = blockIdx.y * 8u + (lane >> 2);
  const bool valid = px < T.W && py < T.H;
  const uint64_t pix = (uint64_t)py * T.W + px;
  // ray_direction (4590-4594) and the view transform (4629-4631)
  const F3 rd = primary_dir(T, (float)px, (float)py - T.yshift);
  const F3 ro = f3(T.eye[0], T.eye[1], T.eye[2]);
  const F3 inv = rcp3(rd);  // the slab tests' reciprocal direction, once per ray

  Walk w;
  w.c = f3(1.0f, 1.0f, 1.0f);
  w.nrm = f3(0.0f, 0.0f, 0.0f);
  w.end = ro;
  w.since = 0.0f;
  w.tnorm = T.time;
  w.hit = false;
  w.visits = 0;
  if (valid && T.rendermode == 0.0f) walk_octree<true>(T, ro, rd, inv, w);
  if (FAST) {  // fast normals (compute.wgsl:4337-4342)
    const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x;
    if (__any_sync(0xffffffffu, w.hit)) {
      const F3 n = tape_normal(T, tid & 31u, tid >> 5, w.end, w.tnorm, w.hit);
      if (w.hit) w.nrm = n;
    }
  }
  F3 c = w.c;
  float dist = -1.0f;
  if (valid && T.rendermode == 0.0f) shade_walk(T, w, ro, c, dist);
  const bool intersected = w.hit;
  const F3 nrm = w.nrm;
  const uint32_t visits = w.visits;
  // get_color_single / get_color_supersample, non-cinematic (4444-4516, 4620-4648)
  float cr = c.x, cg = c.y, cb = c.z, ca = 1.0f;
  if (T.rendermode != 0.0f) {
    cr = cg = cb = ca = 0.0f;
  } else if (T.normal_viz && !intersected) {
    cr = cg = cb = 10.0f;
    ca = 0.0f;
  }
  if (T.rgba) {
    // the channels of a warp without a hit are one number each, the age
    // colour's green and blue are: a power costs some hundred instructions
    const float pr = fm_powf(cr, 0.45f);
    const float pg = __all_sync(FULL_MASK, cg == cr) ? pr : fm_powf(cg, 0.45f);
    const float pb = __all_sync(FULL_MASK, cb == cg) ? pg : fm_powf(cb, 0.45f);
    if (valid) T.rgba[pix] = make_float4(pr, pg, pb, ca);
  }
  if (valid && T.depth) T.depth[pix] = dist;
  if (valid && T.normal) {
    T.normal[pix * 3 + 0] = nrm.x;
    T.normal[pix * 3 + 1] = nrm.y;
    T.normal[pix * 3 + 2] = nrm.z;
  }
  if (T.visits) {
    // one atomic per warp
    unsigned long long v = visits;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x + threadIdx.y * blockDim.x) % 32 == 0) atomicAdd(T.visits, v);
  }
}

template <bool FAST>
__global__ void __launch_bounds__(32 * kTraceWarps, 32 / kTraceWarps) trace_kernel(const TraceParams *__restrict__ Tp) {
  trace_pixels<FAST>(Tp);
}
// One frame per blockIdx.z.  (A single frame through this kernel takes 2.6%
// longer at 1440p: its arguments are behind one more address.)
template <bool FAST>
__global__ void __launch_bounds__(32 * kTraceWarps, 32 / kTraceWarps)
    trace_batch_kernel(const __grid_constant__ TraceBatch B) {
  const TraceParams *Tp = B.T[blockIdx.z];
  // a smaller frame than the largest
  if (blockIdx.x * (4u * kTraceWarps) >= Tp->W || blockIdx.y * 8u >= Tp->H) return;
  trace_pixels<FAST>(Tp);
}

// Shared memory of a block with fast normals.
static size_t trace_smem_bytes(const TraceParams &T) { return T.code ? (size_t)kTraceWarps * normal_bytes(T.nregs) : 0; }

cudaError_t launch_cinematic(const TraceParams &T, const TraceParams *Tdev, cudaStream_t st);

// Frames of the same kind go into one launch: a frame of a few hundred
// thousand pixels leaves the GPU idle while its last rays end.
template <bool FAST>
static cudaError_t launch_kind(const TraceParams *const *T, const TraceParams *const *Tdev, uint32_t n,
                               cudaStream_t st) {
  for (uint32_t i = 0; i < n;) {
    TraceBatch B;
    uint32_t m = 0, w = 0, h = 0;
    size_t smem = 0;
    for (; i < n && m < kTraceBatch; ++i) {
      if (T[i]->cinematic || (T[i]->code != nullptr) != FAST) continue;
      B.T[m++] = Tdev[i];
      w = std::max(w, T[i]->W);
      h = std::max(h, T[i]->H);
      smem = std::max(smem, trace_smem_bytes(*T[i]));
    }
    if (m == 0) break;
    for (uint32_t q = m; q < kTraceBatch; ++q) B.T[q] = nullptr;
    if (smem > (48u << 10)) {  // the attribute is per kernel and device: only ever raise it
      static std::mutex mu;
      static size_t set_bytes[64] = {0};
      int dev = 0;
      cudaError_t e = cudaGetDevice(&dev);
      if (e != cudaSuccess) return e;
      std::lock_guard<std::mutex> lock(mu);
      if (dev < 0 || dev >= 64 || smem > set_bytes[dev]) {
        e = cudaFuncSetAttribute(trace_kernel<FAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
          e = cudaFuncSetAttribute(trace_batch_kernel<FAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) set_bytes[dev] = smem;
      }
    }
    const dim3 grid((w + 4 * kTraceWarps - 1) / (4 * kTraceWarps), (h + 7) / 8, m);
    if (m == 1) trace_kernel<FAST><<<grid, 32 * kTraceWarps, smem, st>>>(B.T[0]);
    else trace_batch_kernel<FAST><<<grid, 32 * kTraceWarps, smem, st>>>(B);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_traces(const TraceParams *const *T, const TraceParams *const *Tdev, uint32_t n, cudaStream_t st) {
  cudaError_t e = launch_kind<false>(T, Tdev, n, st);
  if (e == cudaSuccess) e = launch_kind<true>(T, Tdev, n, st);
  for (uint32_t i = 0; i < n && e == cudaSuccess; ++i)
    if (T[i]->cinematic) e = launch_cinematic(*T[i], Tdev[i], st);
  return e;
}

}  // namespace tsi
