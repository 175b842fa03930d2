// trace_walk.cuh — the octree walk of one ray (compute.wgsl `trace`
// 4189-4403, `efficient_slabs` 4059-4070), shared by the frame tracer
// (trace.cu, rt_main) and the cinematic path tracer (cinematic.cu).
//
// The walk follows the reference's state machine step for step: slab test
// of the current node, a 2x2x2 DDA over its children, descent into children
// with f <= 0 whose eps-padded box the ray hits, hit at the first leaf,
// including its handling of the DDA leaving the node and of out-of-range
// child indices, with a 32-entry stack instead of 16 so octrees deeper than
// 8 levels do not overflow.  Compiled with --fmad=false: the arithmetic is
// the plain f32 sequence of the reference (no FMA contraction).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_types.h"
#include "fmath.cuh"
#include "interp.cuh"
#include "point_tape.cuh"
#include "trace_params.h"

namespace tsi {

struct F3 {
  float x, y, z;
};
__device__ __forceinline__ F3 f3(float a, float b, float c) { return F3{a, b, c}; }
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ F3 operator*(F3 a, F3 b) { return f3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ F3 operator/(F3 a, F3 b) { return f3(a.x / b.x, a.y / b.y, a.z / b.z); }
__device__ __forceinline__ F3 muls(F3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ F3 rcp3(F3 a) { return f3(1.0f / a.x, 1.0f / a.y, 1.0f / a.z); }
__device__ __forceinline__ float len3(F3 a) { return sqrtf((a.x * a.x + a.y * a.y) + a.z * a.z); }
__device__ __forceinline__ float sgn(float x) { return x > 0.0f ? 1.0f : (x < 0.0f ? -1.0f : 0.0f); }

__device__ __forceinline__ F3 slabs(F3 p0, F3 p1, F3 ro, F3 inv) {
  const F3 t0 = (p0 - ro) * inv, t1 = (p1 - ro) * inv;
  const float mnx = fm_min(t0.x, t1.x), mny = fm_min(t0.y, t1.y), mnz = fm_min(t0.z, t1.z);
  const float mxx = fm_max(t0.x, t1.x), mxy = fm_max(t0.y, t1.y), mxz = fm_max(t0.z, t1.z);
  const float d1 = fm_max(mnx, fm_max(mny, mnz));
  const float d2 = fm_min(mxx, fm_min(mxy, mxz));
  return f3((d1 <= d2 && d2 >= 0.0f) ? 1.0f : 0.0f, fm_max(d1, 0.0f), fm_max(d2, 0.0f));
}

__device__ __forceinline__ void node_box(const VoxelPoolDev &pool, uint32_t v, F3 &p0, F3 &p1) {
  const float4 a = pool.box_xy[v];
  const float2 b = pool.box_z[v];
  p0 = f3(a.x, a.z, b.x);
  p1 = f3(a.y, a.w, b.y);
}

// Dynamic shared memory of the tracers: with fast normals, per warp what
// point_forward takes (in the general form: a register file of intervals).
extern __shared__ __align__(16) unsigned char trace_smem[];

// Shared memory of a warp with fast normals: four points per lane while four
// blocks of four warps fit an SM's shared memory so, else two at a time.
__host__ __device__ __forceinline__ bool four_points(uint32_t nregs) { return point_bytes<2>(nregs) <= 14u << 10; }
__host__ __device__ __forceinline__ uint32_t normal_bytes(uint32_t nregs) {
  return four_points(nregs) ? point_bytes<2>(nregs) : point_bytes<1>(nregs);
}

// finite_diff_normal (compute.wgsl:4143-4184) for any tape: the tetrahedron
// of points p + k h (h = 0.01, k in {(1,-1,-1), (-1,-1,1), (-1,1,-1),
// (1,1,1)}) with f evaluated by the tape on point boxes (round to nearest),
// normalised as v / |v|.  The reference pastes a per-scene function here;
// the tape makes it work for every scene.  Called by the whole warp with at
// least one lane that hit; the others evaluate that lane's points.
constexpr float kNormalH = 0.01f;

// The four values by the interval interpreter, point by point: for values
// beyond fix's range.
static __device__ __noinline__ void tape_values_general(const TraceParams &T, uint32_t lane, float2 *rf, F3 p, float t,
                                                        float f[4]) {
  const float h = kNormalH;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    const float kx = (q == 0 || q == 3) ? 1.0f : -1.0f, ky = q >= 2 ? 1.0f : -1.0f, kz = (q & 1) ? 1.0f : -1.0f;
    __syncwarp();
    const Iv r = forward_pass<false>(T.code, T.len, T.out_reg, rf, lane, iv(p.x + kx * h), iv(p.y + ky * h),
                                     iv(p.z + kz * h), iv(t));
    f[q] = r.lo;
  }
}

static __device__ __forceinline__ F3 tape_normal(const TraceParams &T, uint32_t lane, uint32_t warp, F3 p, float t,
                                                 bool hit) {
  const uint32_t hits = __ballot_sync(FULL_MASK, hit);
  const int src = hit ? (int)lane : __ffs((int)hits) - 1;
  p = f3(__shfl_sync(FULL_MASK, p.x, src), __shfl_sync(FULL_MASK, p.y, src), __shfl_sync(FULL_MASK, p.z, src));
  t = __shfl_sync(FULL_MASK, t, src);
  unsigned char *mem = trace_smem + (size_t)warp * normal_bytes(T.nregs);
  const uint32_t smem = (uint32_t)__cvta_generic_to_shared(mem);
  const float h = kNormalH;
  const float xp = p.x + h, xm = p.x - h, yp = p.y + h, ym = p.y - h, zp = p.z + h, zm = p.z - h;
  const F2 x0 = f2_pack(xp, xm), x1 = f2_pack(xm, xp), y0 = f2_pack(ym, ym), y1 = f2_pack(yp, yp), z = f2_pack(zm, zp);
  float f[4];
  bool good;
  if (four_points(T.nregs)) {
    good = point_forward<2>(T.code, T.len, T.nregs, T.out_reg, smem, lane, Pts<2>{x0, x1}, Pts<2>{y0, y1}, Pts<2>{z, z},
                            t, f);
  } else {
    good = point_forward<1>(T.code, T.len, T.nregs, T.out_reg, smem, lane, Pts<1>{x0}, Pts<1>{y0}, Pts<1>{z}, t, f);
    __syncwarp();
    good &= point_forward<1>(T.code, T.len, T.nregs, T.out_reg, smem, lane, Pts<1>{x1}, Pts<1>{y1}, Pts<1>{z}, t, f + 2);
  }
  if (!__all_sync(FULL_MASK, good)) tape_values_general(T, lane, reinterpret_cast<float2 *>(mem), p, t, f);
  const float kx[4] = {1.0f, -1.0f, -1.0f, 1.0f}, ky[4] = {-1.0f, -1.0f, 1.0f, 1.0f};
  const float kz[4] = {-1.0f, 1.0f, -1.0f, 1.0f};
  F3 v = f3(kx[0] * f[0], ky[0] * f[0], kz[0] * f[0]);
  for (int q = 1; q < 4; ++q) v = v + f3(kx[q] * f[q], ky[q] * f[q], kz[q] * f[q]);
  const float l = len3(v);
  return f3(v.x / l, v.y / l, v.z / l);
}

// What the walk of one ray leaves: the colour darkened along the way
// (COLOR), the leaf's stored normal, where the walk ended, the time since
// the leaf was evaluated and the time of its finite-difference normal.
struct Walk {
  F3 c, nrm, end;
  float since, tnorm;
  bool hit;
  uint32_t visits;
};

// The walk for any ray and any boxes (parallel rays, infinities, NaN).
template <bool COLOR>
__device__ __noinline__ void walk_general(const TraceParams &T, F3 ro, F3 rd, F3 inv, Walk &w) {
  const VoxelPoolDev &pool = T.pool;
  const float TEPS = 0.0001f;
  F3 c = f3(1.0f, 1.0f, 1.0f);
  F3 nrm = f3(0.0f, 0.0f, 0.0f);
  uint32_t visits = 0;
  bool intersected = false;
  float hit_since = 0.0f;  // time since the leaf was evaluated
  float hit_t = T.time;    // time of the finite-difference normal
  uint32_t stack[32];
  uint32_t sp = 0;
  F3 ro2 = ro;
  stack[sp++] = 0u;
  uint32_t region = 0u;
  F3 p0, p1;
  node_box(pool, region, p0, p1);
  F3 hit = slabs(p0, p1, ro2, inv);
  bool done = (hit.x == 0.0f);
  for (uint32_t iter = 0; iter < 5000u && !done; ++iter) {
    if (intersected) break;
    if (sp == 0) {
      done = true;
      break;
    }
    region = stack[--sp];
    if (hit.x == 0.0f) {
      if (sp == 0) continue;
      node_box(pool, stack[sp - 1], p0, p1);
      hit = slabs(p0, p1, ro2, inv);
      continue;
    }
    const F3 two = f3(2.0f, 2.0f, 2.0f);
    const F3 rol = muls((ro2 + muls(rd, hit.y + TEPS)) - p0, 2.0f) / (p1 - p0);
    const F3 rdl = rd * (two / (p1 - p0));
    int mp0 = (int)floorf(rol.x), mp1 = (int)floorf(rol.y), mp2 = (int)floorf(rol.z);
    const float dd0 = 1.0f / fabsf(rdl.x), dd1 = 1.0f / fabsf(rdl.y), dd2 = 1.0f / fabsf(rdl.z);
    const float s0 = sgn(rdl.x), s1 = sgn(rdl.y), s2 = sgn(rdl.z);
    const int st0 = (int)s0, st1 = (int)s1, st2 = (int)s2;
    float sd0 = ((s0 * ((float)mp0 - rol.x) + s0 * 0.5f) + 0.5f) * dd0;
    float sd1 = ((s1 * ((float)mp1 - rol.y) + s1 * 0.5f) + 0.5f) * dd1;
    float sd2 = ((s2 * ((float)mp2 - rol.z) + s2 * 0.5f) + 0.5f) * dd2;
    float m0 = 0.0f, m1 = 0.0f, m2 = 0.0f;
    const F3 old_ro2 = ro2;
    // per node: the darkening of every DDA step and the children's brick
    const bool darken = !T.normal_viz && fm_max(p1.x - p0.x, fm_max(p1.y - p0.y, p1.z - p0.z)) < 1.0f;
    const uint32_t cbase = pool.child[region];
    // ro2 = old_ro2 + rd t after every step, as in the reference; it is
    // only read where a child is tested, where the walk leaves this node's
    // loop and at the end, so it is formed there (`moved`: not yet formed
    // for the last step)
    float t = 0.0f;
    bool moved = false;
    for (int i = 0; i < 32; ++i) {
      if (COLOR && darken) c = muls(c, T.darken);
      const F3 mv = f3(m0 * (sd0 - dd0), m1 * (sd1 - dd1), m2 * (sd2 - dd2));
      // the reference adds its sphere-march step here, which is always 0
      // (and t > 0 or NaN, so adding 0 changes no bit)
      t = (len3(mv) + hit.y) + TEPS;
      moved = true;
      if (t >= hit.z - TEPS) {  // left the node (4277-4292)
        ro2 = old_ro2 + muls(rd, hit.z);
        moved = false;
        if (sp == 0) {
          hit = f3(0.0f, 0.0f, 0.0f);
          break;
        }
        node_box(pool, stack[sp - 1], p0, p1);
        hit = slabs(p0, p1, ro2, inv);
        break;
      }
      const int ci = mp0 + 2 * mp1 + 4 * mp2;
      if (ci < 0 || ci >= 8) break;
      const uint32_t child = cbase + (uint32_t)ci;
      if (cbase != TSI_NONE) ++visits;
      if (cbase != TSI_NONE && pool.f[child] <= 0.0f) {
        ro2 = old_ro2 + muls(rd, t);
        moved = false;
        F3 q0, q1;
        node_box(pool, child, q0, q1);
        const F3 tp0 = f3(q0.x - TEPS, q0.y - TEPS, q0.z - TEPS);
        const F3 tp1 = f3(q1.x + TEPS, q1.y + TEPS, q1.z + TEPS);
        const F3 th = slabs(tp0, tp1, ro2, inv);
        if (th.x == 1.0f) {
          if (pool.child[child] != TSI_NONE) {
            if (sp < 32) stack[sp++] = region;
            if (sp < 32) stack[sp++] = child;
            p0 = tp0;
            p1 = tp1;
            hit = th;
            break;
          }
          // the leaf's colour is set after the walk (the fast normal is
          // evaluated by the whole warp there)
          intersected = true;
          const float4 nv = pool.normal[child];
          nrm = f3(nv.x, nv.y, nv.z);
          hit_since = T.time - pool.t[child];
          if (T.swept) hit_t = pool.t[region];  // compute.wgsl:4339-4341
          break;
        }
      }
      // 4389-4391
      const float n0 = (sd0 <= fm_min(sd1, sd2)) ? 1.0f : 0.0f;
      const float n1 = (sd1 <= fm_min(sd2, sd0)) ? 1.0f : 0.0f;
      const float n2 = (sd2 <= fm_min(sd0, sd1)) ? 1.0f : 0.0f;
      m0 = n0;
      m1 = n1;
      m2 = n2;
      sd0 = sd0 + m0 * dd0;
      sd1 = sd1 + m1 * dd1;
      sd2 = sd2 + m2 * dd2;
      mp0 = mp0 + (int)m0 * st0;
      mp1 = mp1 + (int)m1 * st1;
      mp2 = mp2 + (int)m2 * st2;
    }
    if (moved) ro2 = old_ro2 + muls(rd, t);
  }
  w.end = ro2;
  w.c = c;
  w.nrm = nrm;
  w.since = hit_since;
  w.tnorm = hit_t;
  w.hit = intersected;
  w.visits = visits;
}

// Whether a ray may take the fast walk: its direction's components and, by
// the caller, the boxes' extents are well inside the normal range.
__device__ __forceinline__ bool plain_ray(F3 ro, F3 rd) {
  const float lo = 9.094947e-13f, hi = 4.0f, far = 16777216.0f;  // 2^-40, 2^24
  const float ax = fabsf(rd.x), ay = fabsf(rd.y), az = fabsf(rd.z);
  return ax >= lo && ay >= lo && az >= lo && ax <= hi && ay <= hi && az <= hi && fabsf(ro.x) <= far &&
         fabsf(ro.y) <= far && fabsf(ro.z) <= far;
}

// A box as a pair of bounds per axis, the way the pool holds them: a bound
// and its opposite take one packed operation.
struct Box2 {
  F2 x, y, z;
};
__device__ __forceinline__ Box2 node_box2(const VoxelPoolDev &pool, uint32_t v) {
  const float4 a = pool.box_xy[v];
  const float2 b = pool.box_z[v];
  return Box2{f2_pack(a.x, a.y), f2_pack(a.z, a.w), f2_pack(b.x, b.y)};
}
// slabs, with the hit as a predicate; inv: the reciprocal direction, twice
// per axis.
__device__ __forceinline__ bool slab_range(const Box2 &b, F3 ro, const Box2 &inv, float &near, float &far) {
  float ax, bx, ay, by, az, bz;
  f2_unpack(f2_mul_alone(f2_add(b.x, f2_dup(-ro.x)), inv.x), ax, bx);
  f2_unpack(f2_mul_alone(f2_add(b.y, f2_dup(-ro.y)), inv.y), ay, by);
  f2_unpack(f2_mul_alone(f2_add(b.z, f2_dup(-ro.z)), inv.z), az, bz);
  const float d1 = fm_max(fm_min(ax, bx), fm_max(fm_min(ay, by), fm_min(az, bz)));
  const float d2 = fm_min(fm_max(ax, bx), fm_min(fm_max(ay, by), fm_max(az, bz)));
  near = fm_max(d1, 0.0f);
  far = fm_max(d2, 0.0f);
  return d1 <= d2 && d2 >= 0.0f;
}

// walk_general's results for such rays, bit for bit, in little more than a
// third of the instructions (the tracer is bound by instruction issue):
//  - the nine divisions of a node's set-up share a reciprocal per axis and
//    have no slow path (fm_rcp_in, fm_div_in);
//  - the signs of the local direction are those of rd;
//  - the march's mask is three predicates, its child index one integer that
//    the steps add to; the step length is |sd - dd| of the one axis that
//    stepped (the root of a square is the absolute value, exactly, without
//    over- or underflow; Boldo 2015), the root only when axes tie;
//  - a node entered has children: their brick is the child field that the
//    descent tested;
//  - the darkened colour is one number until the walk ends: its channels
//    start equal and are scaled alike.
// 1080p frame of the 256-primitive scene: 640 million warp instructions and
// 0.81 ms with walk_general, 0.53 ms with this form; 1440p: 1.11 and 0.67 ms
// (0.69 with x and y of the set-up in scalars).
template <bool COLOR>
__device__ __forceinline__ void walk_plain(const TraceParams &T, F3 ro, F3 rd, F3 inv, uint32_t cbase, Walk &w) {
  const VoxelPoolDev &pool = T.pool;
  const float TEPS = 0.0001f;
  float shade = 1.0f;
  F3 nrm = f3(0.0f, 0.0f, 0.0f);
  uint32_t visits = 0;
  bool intersected = false;
  float hit_since = 0.0f;  // time since the leaf was evaluated
  float hit_t = T.time;    // time of the finite-difference normal
  uint32_t stack[32];  // the ancestors of `region`
  uint32_t sp = 0;
  F3 ro2 = ro;
  uint32_t region = 0u;
  const Box2 inv2{f2_dup(inv.x), f2_dup(inv.y), f2_dup(inv.z)};
  Box2 box = node_box2(pool, region);
  float hy, hz;
  bool in = slab_range(box, ro2, inv2, hy, hz);
  const F3 sg = f3(rd.x > 0.0f ? 1.0f : -1.0f, rd.y > 0.0f ? 1.0f : -1.0f, rd.z > 0.0f ? 1.0f : -1.0f);
  const int st0 = rd.x > 0.0f ? 1 : -1, st1 = rd.y > 0.0f ? 2 : -2, st2 = rd.z > 0.0f ? 4 : -4;
  bool go = in;  // a node to visit
  for (uint32_t iter = 0; iter < 5000u && go; ++iter) {
    if (!in) {  // missed: on to its parent
      if (sp == 0) break;
      region = stack[--sp];
      cbase = pool.child[region];
      box = node_box2(pool, region);
      in = slab_range(box, ro2, inv2, hy, hz);
      continue;
    }
    float x0, x1, y0, y1, z0, z1;
    f2_unpack(box.x, x0, x1);
    f2_unpack(box.y, y0, y1);
    f2_unpack(box.z, z0, z1);
    const F3 half = f3((x1 - x0) * 0.5f, (y1 - y0) * 0.5f, (z1 - z0) * 0.5f);
    const F3 num = (ro2 + muls(rd, hy + TEPS)) - f3(x0, y0, z0);
    float cell0, cell1, cell2, sd0, sd1, sd2, dd0, dd1, dd2;
    // by the half extent h: 2 n / e = n / h and 2 / e = 1 / h, exactly
    auto axis = [](float n, float h, float d, float s, float &cell, float &sd, float &dd) {
      const float y = fm_rcp_in(h);
      const float rol = fm_div_in(n, h, y);
      dd = fm_rcp_in(fabsf(d * y));
      cell = floorf(rol);
      // (s (cell - rol) + s / 2) + 1/2: the sign comes out of the first sum
      sd = __fmaf_rn(s, (cell - rol) + 0.5f, 0.5f) * dd;
    };
    {  // x and y side by side, the same operations packed
      const F2 h2 = f2_pack(half.x, half.y), n2 = f2_pack(num.x, num.y), nh = f2_pack(-half.x, -half.y);
      const F2 one = f2_dup(1.0f);
      auto rcp2 = [&](F2 neg, float a, float b) {
        float p, q;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(p) : "f"(a));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(b));
        const F2 y = f2_pack(p, q);
        return f2_fma(f2_fma(neg, y, one), y, y);
      };
      const F2 y2 = rcp2(nh, half.x, half.y);
      const F2 q2 = f2_mul_alone(n2, y2);
      const F2 rol = f2_fma(f2_fma(nh, q2, n2), y2, q2);
      float ax, ay, r0, r1;
      f2_unpack(f2_mul_alone(f2_pack(rd.x, rd.y), y2), ax, ay);
      ax = fabsf(ax);
      ay = fabsf(ay);
      const F2 dd = rcp2(f2_pack(-ax, -ay), ax, ay);
      f2_unpack(rol, r0, r1);
      cell0 = floorf(r0);
      cell1 = floorf(r1);
      const F2 u = f2_add(f2_fma(rol, f2_dup(-1.0f), f2_pack(cell0, cell1)), f2_dup(0.5f));
      const F2 sd = f2_mul_alone(f2_fma(f2_pack(sg.x, sg.y), u, f2_dup(0.5f)), dd);
      f2_unpack(sd, sd0, sd1);
      f2_unpack(dd, dd0, dd1);
    }
    axis(num.z, half.z, rd.z, sg.z, cell2, sd2, dd2);
    // the cells are small whole numbers: their sum is exact, and adding
    // 1.5 2^23 leaves it in the low bits
    int ci = __float_as_int(__fmaf_rn(4.0f, cell2, __fmaf_rn(2.0f, cell1, cell0)) + 12582912.0f) - 0x4b400000;
    float len = 0.0f;  // |mask (sd - dd)| of the last step
    const F3 old_ro2 = ro2;
    // per node: the darkening of every DDA step and the exit distance
    const bool darken = COLOR && !T.normal_viz && fm_max(half.x, fm_max(half.y, half.z)) < 0.5f;
    const float leave = hz - TEPS;
    const float *cf = pool.f + cbase;
    go = false;
    float t = 0.0f;
    bool moved = false;
    for (int i = 0; i < 32; ++i) {
      if (darken) shade = shade * T.darken;
      t = (len + hy) + TEPS;
      moved = true;
      if (t >= leave) {  // left the node (4277-4292)
        ro2 = old_ro2 + muls(rd, hz);
        moved = false;
        if (sp == 0) break;
        region = stack[--sp];
        cbase = pool.child[region];
        box = node_box2(pool, region);
        in = slab_range(box, ro2, inv2, hy, hz);
        go = true;
        break;
      }
      if ((uint32_t)ci >= 8u) break;  // on with the parent, in this box
      ++visits;
      if (cf[ci] <= 0.0f) {
        const uint32_t child = cbase + (uint32_t)ci;
        ro2 = old_ro2 + muls(rd, t);
        moved = false;
        Box2 pad = node_box2(pool, child);
        const F2 eps = f2_pack(-TEPS, TEPS);
        pad.x = f2_add(pad.x, eps);
        pad.y = f2_add(pad.y, eps);
        pad.z = f2_add(pad.z, eps);
        float ty, tz;
        if (slab_range(pad, ro2, inv2, ty, tz)) {
          const uint32_t below = pool.child[child];
          if (below != TSI_NONE) {
            stack[sp++] = region;  // (at most a level each: fewer than 32)
            region = child;
            cbase = below;
            box = pad;
            hy = ty;
            hz = tz;
            go = true;
            break;
          }
          // the leaf's colour is set after the walk (the fast normal is
          // evaluated by the whole warp there)
          intersected = true;
          const float4 nv = pool.normal[child];
          nrm = f3(nv.x, nv.y, nv.z);
          hit_since = T.time - pool.t[child];
          if (T.swept) hit_t = pool.t[region];  // compute.wgsl:4339-4341
          break;
        }
      }
      // 4389-4391: every axis at the least distance steps
      const float m = fm_min(sd0, fm_min(sd1, sd2));
      const bool b0 = sd0 <= m, b1 = sd1 <= m, b2 = sd2 <= m;
      const float d = b0 ? dd0 : (b1 ? dd1 : dd2);
      len = fabsf((m + d) - d);
      if (b0) {
        sd0 = sd0 + dd0;
        ci += st0;
      }
      if (b1) {
        sd1 = sd1 + dd1;
        ci += st1;
      }
      if (b2) {
        sd2 = sd2 + dd2;
        ci += st2;
      }
      if ((b0 && (b1 || b2)) || (b1 && b2))
        len = len3(f3(b0 ? sd0 - dd0 : 0.0f, b1 ? sd1 - dd1 : 0.0f, b2 ? sd2 - dd2 : 0.0f));
    }
    if (moved) {  // out of the cells, or 32 steps: the parent, in this node's box
      ro2 = old_ro2 + muls(rd, t);
      if (sp != 0) {
        region = stack[--sp];
        cbase = pool.child[region];
        go = true;
      }
    }
  }
  w.end = ro2;
  w.c = f3(shade, shade, shade);
  w.nrm = nrm;
  w.since = hit_since;
  w.tnorm = hit_t;
  w.hit = intersected;
  w.visits = visits;
}

template <bool COLOR>
__device__ __forceinline__ void walk_octree(const TraceParams &T, F3 ro, F3 rd, F3 inv, Walk &w) {
  const uint32_t top = T.pool.child[0];
  if (T.plain_boxes && top != TSI_NONE && plain_ray(ro, rd)) walk_plain<COLOR>(T, ro, rd, inv, top, w);
  else walk_general<COLOR>(T, ro, rd, inv, w);
}

// The colour of `trace` at the end of a walk from ro (4322-4401): the age
// colour of the leaf (or its normal, normal_viz) on the darkened colour,
// clamped; the hit distance |end - ro|, -1 for a miss.
__device__ __forceinline__ void shade_walk(const TraceParams &T, const Walk &w, F3 ro, F3 &c, float &dist) {
  c = w.c;
  dist = -1.0f;
  if (w.hit) {
    if (T.normal_viz) {
      const float nl = len3(w.nrm);
      c = f3(w.nrm.x / nl * 0.5f + 0.5f, w.nrm.y / nl * 0.5f + 0.5f, w.nrm.z / nl * 0.5f + 0.5f);
    } else {
      // c - mix(1 - movement, 1 - base, clamp(60 t, 0, 1)), movement (1,0,0), base (1,1,1)
      const float tt = fm_min(fm_max(w.since * 60.0f, 0.0f), 1.0f);
      const F3 a = f3(0.0f, 1.0f, 1.0f), b = f3(0.0f, 0.0f, 0.0f);
      const F3 lerp = f3(a.x * (1.0f - tt) + b.x * tt, a.y * (1.0f - tt) + b.y * tt, a.z * (1.0f - tt) + b.z * tt);
      c = c - lerp;
    }
    c = f3(fm_max(fm_min(c.x, 1.0f), 0.0f), fm_max(fm_min(c.y, 1.0f), 0.0f), fm_max(fm_min(c.z, 1.0f), 0.0f));
    dist = fabsf(len3(w.end - ro));
  } else {
    c = f3(fm_max(fm_min(c.x, 1.0f), 0.0f), fm_max(fm_min(c.y, 1.0f), 0.0f), fm_max(fm_min(c.z, 1.0f), 0.0f));
  }
}

// The primary ray through pixel position (pxf, pyf), pyf already shifted for
// scene 0 (ray_direction 4590-4594, the view transform 4629-4631).
__device__ __forceinline__ F3 primary_dir(const TraceParams &T, float pxf, float pyf) {
  float xy0 = (pxf - (float)T.W / 2.0f) + 0.5f;
  float xy1 = (pyf - (float)T.H / 2.0f) + 0.5f;
  F3 d = f3(xy0, -xy1, -T.zdist);
  const float dl = len3(d);
  d = f3(d.x / dl, d.y / dl, d.z / dl);
  F3 rd;
  rd.x = ((T.m[0] * d.x + T.m[4] * d.y) + T.m[8] * d.z) + T.m[12] * 0.0f;
  rd.y = ((T.m[1] * d.x + T.m[5] * d.y) + T.m[9] * d.z) + T.m[13] * 0.0f;
  rd.z = ((T.m[2] * d.x + T.m[6] * d.y) + T.m[10] * d.z) + T.m[14] * 0.0f;
  return rd;
}

}  // namespace tsi
