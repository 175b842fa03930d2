// point_tape.cuh — a tape at two or four points per lane, for the finite-difference
// normals of the tracers: the values the interval interpreter gives on point
// boxes, in scalars.
//
// On a point every bound is the other one as long as no operation leaves the
// range that fix clamps to (compute.wgsl:3462-3472 then leaves the value
// alone; beyond it, or for a NaN, the bounds part).  So one number per point
// is computed, and a lane that met a value outside the range says so; the
// caller then evaluates the interval form.  The two points of a pair share
// packed operations, and all of a lane the decoded instruction
// (narrow_interp.cuh), its operand loads and its branches.
//
// Bound by instruction issue: per tape instruction some 20 instead of 4 x 100
// of the interval form.  640x360 frame of 16 spheres (277 instructions) 0.36
// to 0.16 ms, its path-traced image 6.3 to 3.4 ms.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fmath.cuh"
#include "interp.cuh"
#include "narrow_interp.cuh"

namespace tsi {

// Shared memory of a warp with P pairs of points per lane: the registers'
// rows, a row of zeros, 32 decoded instructions.
template <int P>
__host__ __device__ __forceinline__ uint32_t point_bytes(uint32_t nregs) {
  return (nregs + 1u) * (256u * P) + 512u;
}

template <int P>
struct Pts {
  F2 v[P];
};

__device__ __forceinline__ Pts<1> point_ld(uint32_t addr, Pts<1>) {
  Pts<1> p;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(p.v[0].v) : "r"(addr) : "memory");
  return p;
}
__device__ __forceinline__ Pts<2> point_ld(uint32_t addr, Pts<2>) {
  Pts<2> p;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(p.v[0].v), "=l"(p.v[1].v) : "r"(addr) : "memory");
  return p;
}
__device__ __forceinline__ void point_st(uint32_t addr, Pts<1> p) {
  asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(p.v[0].v) : "memory");
}
__device__ __forceinline__ void point_st(uint32_t addr, Pts<2> p) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(addr), "l"(p.v[0].v), "l"(p.v[1].v) : "memory");
}
template <int P>
__device__ __forceinline__ Pts<P> point_dup(float x) {
  Pts<P> r;
#pragma unroll
  for (int i = 0; i < P; ++i) r.v[i] = f2_dup(x);
  return r;
}
template <int P, typename F>
__device__ __forceinline__ Pts<P> point_map(Pts<P> x, Pts<P> y, F f) {
  Pts<P> r;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    float p, q, u, v;
    f2_unpack(x.v[i], p, q);
    f2_unpack(y.v[i], u, v);
    r.v[i] = f2_pack(f(p, u), f(q, v));
  }
  return r;
}

// The field at a lane's 2 P points (x, y, z: a value each), by the whole
// warp.  False in a lane whose values left the range.
template <int P>
static __device__ __noinline__ bool point_forward(const uint2 *__restrict__ code, uint32_t len_, uint32_t nregs,
                                                  uint32_t out_reg, uint32_t smem, uint32_t lane, Pts<P> x, Pts<P> y,
                                                  Pts<P> z, float t, float *f) {
  constexpr uint32_t kRow = 256u * P;
  const Pts<P> kind{};
  const uint32_t len = uniform_u32(len_);
  NarrowRows R;
  R.rf = smem + lane * (8u * P);
  R.sink = nregs * kRow;
  R.prog = smem + (nregs + 1u) * kRow;
  point_st(R.rf, x);
  point_st(R.rf + kRow, y);
  point_st(R.rf + 2u * kRow, z);
  point_st(R.rf + 3u * kRow, point_dup<P>(t));
  point_st(R.rf + R.sink, point_dup<P>(-0.0f));
  // NaN once a value is NaN, infinite or above 9.7e5 (the product overflows)
  Pts<P> bad = point_dup<P>(0.0f);
  bool odd = false;
  const F2 big = f2_dup(3.5e32f), nil = f2_dup(0.0f);
  auto keep = [&](uint32_t off, const Pts<P> &v) {
#pragma unroll
    for (int i = 0; i < P; ++i) bad.v[i] = f2_fma(f2_mul_alone(v.v[i], big), nil, bad.v[i]);
    point_st(R.rf + off, v);
  };
  uint2 nxt = load_chunk(code, len, 0, lane);
  for (uint32_t c0 = 0; c0 < len; c0 += 32u) {
    const uint32_t n = min(32u, len - c0);
    __syncwarp();
    const uint4 dec = decode_forward<false>(nxt, kRow, R.sink);
    prog_st(R, lane, dec);
    const uint32_t other = __ballot_sync(FULL_MASK, lane >= n || !(dec.x & NC_LIN));
    const NarrowKinds K = narrow_kinds(dec.x);
    nxt = load_chunk(code, len, (int)(c0 / 32u) + 1, lane);
    __syncwarp();
    uint32_t j = 0;
    uint4 w = prog_ld(R, 0);
    while (j < n) {
      const uint32_t rest = other >> j;
      const uint32_t end = rest ? j + (uint32_t)__ffs((int)rest) - 1u : 32u;
#pragma unroll 1
      for (; j < end; ++j) {
        const uint4 w1 = prog_ld(R, (j + 1u) & 31u);
        const Pts<P> X = point_ld(R.rf + (w.y & 0xffffu), kind), Y = point_ld(R.rf + (w.y >> 16), kind);
        const F2 m = f2_dup(__uint_as_float(w.z)), lit = f2_dup(__uint_as_float(w.w));
        Pts<P> v;
#pragma unroll
        for (int i = 0; i < P; ++i) v.v[i] = f2_add(f2_fma(m, X.v[i], lit), Y.v[i]);
        keep(w.x >> 16, v);
        w = w1;
      }
      if (j < n) {
        const uint4 w1 = prog_ld(R, (j + 1u) & 31u);
        const uint32_t c = w.x;
        const Pts<P> X = point_ld(R.rf + (w.y & 0xffffu), kind), Y0 = point_ld(R.rf + (w.y >> 16), kind);
        const float lit = __uint_as_float(w.w);
        const Pts<P> Y = (c & NC_YLIT) ? point_dup<P>(lit) : Y0;
        Pts<P> v;
        if ((K.sqr >> j) & 1u) {
#pragma unroll
          for (int i = 0; i < P; ++i) v.v[i] = f2_mul_alone(X.v[i], X.v[i]);
        } else if ((K.mm >> j) & 1u) {
          const bool mx = c & NC_MAX;
          v = point_map(X, Y, [&](float p, float q) {
            const float lo = fm_min(p, q), hi = fm_max(p, q);
            return mx ? hi : lo;
          });
        } else if ((K.mul >> j) & 1u) {
#pragma unroll
          for (int i = 0; i < P; ++i) v.v[i] = f2_mul_alone(X.v[i], Y.v[i]);
        } else if ((K.abs >> j) & 1u) {
          v = point_map(X, X, [](float p, float) { return fabsf(p); });
        } else {
          const uint32_t h = c & 63u;
          if (__any_sync(FULL_MASK, h == H_SQRT)) {
            v = point_map(X, X, [](float p, float) { return __fsqrt_rn(fm_max(p, 0.0f)); });
          } else if (__any_sync(FULL_MASK, h == H_SIN)) {
#pragma unroll
            for (int i = 0; i < P; ++i) {
              float p, q;
              f2_unpack(X.v[i], p, q);
              fm_sin2(p, q, p, q);
              v.v[i] = f2_pack(p, q);
            }
          } else {
            v = point_map(X, Y, [&](float p, float q) {
              const Iv r = cold_forward<false>(h, iv(p), iv(q), lit);
              odd |= !(r.lo == r.hi);
              return r.lo;
            });
          }
        }
        keep(c >> 16, v);
        w = w1;
        ++j;
      }
    }
  }
  const Pts<P> o = point_ld(R.rf + out_reg * kRow, kind);
  float b = 0.0f;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    float p, q;
    f2_unpack(o.v[i], f[2 * i], f[2 * i + 1]);
    f2_unpack(bad.v[i], p, q);
    b = b + (p + q);
  }
  return !odd && b == b;
}

}  // namespace tsi
