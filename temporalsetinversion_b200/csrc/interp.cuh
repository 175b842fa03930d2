// interp.cuh — the plain one-warp tape interpreter: a cell or point per lane,
// one tape instruction at a time on the packed register tape (tape_format.h),
// interval registers in shared memory, forward only (compute.wgsl:3633-3772).
// It serves points whose values leave fix's range (trace_walk.cuh); cells and
// boxes take narrow_interp.cuh or wide_interp.cuh.  Beside it, what all of
// them share.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "interval.cuh"
#include "tape_format.h"

namespace tsi {

#define FULL_MASK 0xffffffffu

// Instruction j of a 32-instruction chunk held one per lane.
__device__ __forceinline__ uint2 chunk_word(uint2 c, uint32_t j) {
  return make_uint2(__shfl_sync(0xffffffffu, c.x, j), __shfl_sync(0xffffffffu, c.y, j));
}
// Chunk k of a tape: instruction 32k + lane (zero past the end).
__device__ __forceinline__ uint2 load_chunk(const uint2 *__restrict__ code, uint32_t len, int k, uint32_t lane) {
  const int i = 32 * k + (int)lane;
  return (k >= 0 && i < (int)len) ? code[i] : make_uint2(0u, 0u);
}

__device__ __forceinline__ bool finite2(Iv a) { return isfinite(a.lo) && isfinite(a.hi); }

__device__ __forceinline__ Iv ld_reg(const float2 *rf, uint32_t r, uint32_t lane) {
  const float2 v = rf[r * 32u + lane];
  return Iv{v.x, v.y};
}
__device__ __forceinline__ void st_reg(float2 *rf, uint32_t r, uint32_t lane, Iv v) {
  rf[r * 32u + lane] = make_float2(v.lo, v.hi);
}

// ---------------------------------------------------------------- handlers
// Rare handlers live out of line so the interpreter loop stays small.
template <bool D>
__device__ __noinline__ Iv cold_forward(uint32_t h, Iv A, Iv B, float lit) {
  return IA<D>::forward(h, A, B, lit);
}

template <bool D>
__device__ __forceinline__ Iv op_forward(uint32_t h, Iv A, Iv B, float lit) {
  using I = IA<D>;
  Iv v;
  switch (h) {
    case H_CONST: v = iv(lit); break;
    case H_COPY: v = A; break;
    case H_ADD_II: v = I::add(A, B); break;
    case H_SUB_II: v = I::sub(A, B); break;
    case H_MUL_II: v = I::mul(A, B); break;
    case H_MIN_II: v = I::min_(A, B); break;
    case H_MAX_II: v = I::max_(A, B); break;
    case H_ADD_IF: v = I::add_f(A, lit); break;
    case H_SUB_IF: v = I::sub_f(A, lit); break;
    case H_MUL_IF: v = I::mul_f(A, lit); break;
    case H_MIN_IF: v = Iv{fm_min(A.lo, lit), fm_min(A.hi, lit)}; break;
    case H_MAX_IF: v = Iv{fm_max(A.lo, lit), fm_max(A.hi, lit)}; break;
    case H_SQR: v = I::sqr(A); break;
    case H_SQRT: v = I::sqrt_(A); break;
    case H_NEG: v = I::neg(A); break;
    case H_ABS: v = I::abs_(A); break;
    case H_SUB_FI: v = I::sub(iv(lit), A); break;
    default: return cold_forward<D>(h, A, B, lit);  // fixed inside
  }
  return I::fix(v);
}

template <bool D>
__device__ __noinline__ int cold_reverse_rule(uint32_t h, Iv A, Iv B, float lit, Iv &r0, Iv &r1) {
  return IA<D>::reverse_rule(h, A, B, lit, r0, r1);
}

// ---------------------------------------------------------------- passes
// Forward pass over `len` instructions; returns the output register's value.
template <bool D>
__device__ __forceinline__ Iv forward_pass(const uint2 *__restrict__ code, uint32_t len, uint32_t out_reg, float2 *rf,
                                           uint32_t lane, Iv x, Iv y, Iv z, Iv t) {
  st_reg(rf, 0, lane, x);
  st_reg(rf, 1, lane, y);
  st_reg(rf, 2, lane, z);
  st_reg(rf, 3, lane, t);
  // the tape arrives 32 instructions per coalesced load, one chunk ahead
  uint2 cur = load_chunk(code, len, 0, lane), nxt = load_chunk(code, len, 1, lane);
  for (uint32_t c0 = 0; c0 < len; c0 += 32u) {
    const uint32_t n = min(32u, len - c0);
    for (uint32_t j = 0; j < n; ++j) {
      const uint2 w = chunk_word(cur, j);
      const uint32_t h = TSI_W0_H(w.x);
      const float lit = __uint_as_float(w.y);
      const Iv Av = ld_reg(rf, TSI_W0_A(w.x), lane);
      const Iv Bv = TSI_H_IS_II(h) ? ld_reg(rf, w.y & 255u, lane) : iv(lit);
      st_reg(rf, TSI_W0_DST(w.x), lane, op_forward<D>(h, Av, Bv, lit));
    }
    cur = nxt;
    nxt = load_chunk(code, len, (int)(c0 / 32u) + 2, lane);
  }
  return ld_reg(rf, out_reg, lane);
}

}  // namespace tsi
