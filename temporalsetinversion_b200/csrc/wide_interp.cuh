// wide_interp.cuh — the block-wide interpreter of the bundled tape
// (tape_compile.h WideTape): one cell per block, one thread per slot of a
// bundle, every SSA value in its own shared-memory slot.
//
// cell_forward follows compute.wgsl:3633-3772, cell_reverse
// compute.wgsl:3786-3900 with per-use contribution records for values with
// several users (their sensitivities are summed in the sequential order).
//
// A bundle step is a block barrier apart from the next and a cell is a chain
// of steps, so a step's latency is the cost: what a warp issues between two
// barriers, about four cycles an instruction.  The host therefore decodes
// every slot (wide_tape.h): a kind for the whole warp, operand indices that
// always name a value (an absent one the zero, a padding lane's result the
// dummy), sensitivity targets that are a value's or a record's place in one
// array.  A step then takes no test but those on its group's kind, which
// comes as a byte of a word made uniform for the compiler once in four
// steps; linear handlers are one fused form; a value with one user needs no
// accumulator; and the slots of the next four steps are on their way.  (Eight
// steps ahead hide a load's 900 cycles from L2 better for a lone cell, but
// the walk unrolled eight times costs levels that mix cells and items a fifth
// in instruction fetches; the slots out of line, 5% at every level.)
// 256-primitive tape (32 steps), levels of 64 cells: 31 thousand cycles
// forward and 58 thousand reverse with a switch over the handlers and slots
// found through the bundle table, 25 and 52 thousand with this form;
// inversions of the 256-primitive animation at localsubdiv 10 0.80 to 0.77
// ms, rotating swept scene 2.66 to 2.58 ms.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "device_types.h"
#include "interp.cuh"
#include "narrow_interp.cuh"
#include "wide_tape.h"

namespace tsi {

// A cell's array of intervals: shared memory by its 32-bit address, or (GM)
// the block's slice of the global scratch.
template <bool GM>
struct CellArray;
template <>
struct CellArray<false> {
  uint32_t base;
  __device__ __forceinline__ explicit CellArray(void *p) : base((uint32_t)__cvta_generic_to_shared(p)) {}
  __device__ __forceinline__ Iv ld(uint32_t i) const {
    Iv v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.lo), "=f"(v.hi) : "r"(base + i * 8u) : "memory");
    return v;
  }
  __device__ __forceinline__ void st(uint32_t i, Iv v) const {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(base + i * 8u), "f"(v.lo), "f"(v.hi) : "memory");
  }
};
template <>
struct CellArray<true> {
  unsigned long long base;
  __device__ __forceinline__ explicit CellArray(void *p) : base((unsigned long long)__cvta_generic_to_global(p)) {}
  __device__ __forceinline__ Iv ld(uint32_t i) const {
    Iv v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.lo), "=f"(v.hi) : "l"(base + i * 8ull) : "memory");
    return v;
  }
  __device__ __forceinline__ void st(uint32_t i, Iv v) const {
    asm volatile("st.global.v2.f32 [%0], {%1, %2};" ::"l"(base + i * 8ull), "f"(v.lo), "f"(v.hi) : "memory");
  }
};

// The barrier between two steps.  The warps arrive from different places of
// their walks (every warp arrives once per step); PTX counts the arrivals at
// the barrier, whichever instruction they come from.
__device__ __forceinline__ void step_barrier() { asm volatile("barrier.sync 0;" ::: "memory"); }

// One warp's walk through the steps: `step(q, kind)` runs on its slot of each
// step it has a group in.  The next kWideAhead steps' slots are on their way
// in registers, at addresses that depend on nothing loaded but the kinds (a
// load that waits for a test of a loaded table, or whose result is selected,
// is waited for at once); a step without a group reads the slot of the next
// one that has (an L1 hit).
// Steps are rounded up to a multiple of kWideAhead, for every warp alike.
template <typename Step>
__device__ __forceinline__ void walk_steps(const WideDev &W, uint32_t stream, const uint4 *__restrict__ recs,
                                           Step step) {
  const uint2 st = W.streams[stream];
  const uint32_t n = uniform_u32(W.nbundles);
  const uint32_t *__restrict__ ctl = W.ctl + st.y;
  const uint4 *ptr = recs + st.x + (threadIdx.x & 31u);
  constexpr uint32_t kWords = kWideAhead / 4u;
  const uint32_t last = (n + kWideAhead - 1u) / kWideAhead * kWords + kWords;
  uint32_t c[kWords], l[kWords];
  uint4 q[kWideAhead];
#pragma unroll
  for (uint32_t i = 0; i < kWords; ++i) c[i] = uniform_u32(ctl[i]);
#pragma unroll
  for (uint32_t i = 0; i < kWords; ++i) l[i] = ctl[kWords + i];
#pragma unroll
  for (uint32_t u = 0; u < kWideAhead; ++u) {
    q[u] = *ptr;
    ptr += ((c[u / 4u] >> (8u * (u & 3u))) & 31u) != WK_NONE ? 32 : 0;
  }
  for (uint32_t k = 0; k < n; k += kWideAhead) {
    uint32_t next[kWords];
#pragma unroll
    for (uint32_t i = 0; i < kWords; ++i) {
      next[i] = uniform_u32(l[i]);
      l[i] = ctl[min(k / 4u + 2u * kWords + i, last)];
    }
#pragma unroll
    for (uint32_t u = 0; u < kWideAhead; ++u) {
      const uint32_t kind = (c[u / 4u] >> (8u * (u & 3u))) & 31u;
      const uint32_t ahead = (next[u / 4u] >> (8u * (u & 3u))) & 31u;
      if (kind != WK_NONE) step(q[u], kind);
      q[u] = *ptr;
      ptr += ahead != WK_NONE ? 32 : 0;
      step_barrier();
    }
#pragma unroll
    for (uint32_t i = 0; i < kWords; ++i) c[i] = next[i];
  }
}

// 2-bit decision of a min/max over A and B (compute.wgsl:3660-3700): bit 0
// the A operand is always chosen, bit 1 the B operand is.
__device__ __forceinline__ uint32_t minmax_decision(bool amax, Iv A, Iv B) {
  const bool a_below = A.hi < B.lo, b_below = B.hi < A.lo;
  return ((amax ? b_below : a_below) ? 1u : 0u) | ((amax ? a_below : b_below) ? 2u : 0u);
}

// ---------------------------------------------------------------- forward
// Where a forward slot's operands are read and its value goes: an array with
// a place per value, or slots of shared memory and (keep) the place in the
// global scratch that the reverse pass reads.
template <bool GM>
struct ForwardPlaces {
  CellArray<GM> V;
  __device__ __forceinline__ Iv a(const uint4 &q) const { return V.ld(q.y); }
  __device__ __forceinline__ Iv b(const uint4 &q) const { return V.ld(q.z); }
  __device__ __forceinline__ void st(const uint4 &q, Iv v) const { V.st(q.x >> WC_DST_SHIFT, v); }
};
struct ForwardSlots {
  CellArray<false> S;
  CellArray<true> V;
  bool keep;
  __device__ __forceinline__ Iv a(const uint4 &q) const { return S.ld(q.y & 0xffffu); }
  __device__ __forceinline__ Iv b(const uint4 &q) const { return S.ld((q.x & WC_II) ? q.z : 0u); }
  __device__ __forceinline__ void st(const uint4 &q, Iv v) const {
    S.st(q.y >> 16, v);
    if (keep) V.st(q.x >> WC_DST_SHIFT, v);
  }
};

// One slot over one of the time intervals: its value to V, a min/max's
// decision to dec (a byte per min/max) when it is set.
template <bool D, typename Places>
__device__ __forceinline__ void wide_forward_slot(uint32_t kind_, uint4 q, Places V, uint8_t *dec) {
  using I = IA<D>;
  const Iv X = V.a(q), Y0 = V.b(q);
  const uint32_t kind = uniform_u32(kind_);
  const float f = __uint_as_float(q.w);
  Iv v;
  if (kind == WK_LIN) {
    // X or -X, plus the literal or Y (the other is the zero that changes no sum)
    const float m = (q.x & WC_NEG) ? -1.0f : 1.0f;
    const Iv S = (q.x & WC_SWAP) ? Iv{X.hi, X.lo} : X;
    if (!D) {
      const F2 r = f2_add(f2_fma(f2_dup(m), f2_pack(S.lo, S.hi), f2_dup(f)), f2_pack(Y0.lo, Y0.hi));
      f2_unpack(r, v.lo, v.hi);
    } else {
      const float lo = (q.x & WC_ZERO) ? 0.0f : f, hi = (q.x & WC_ZERO) ? -0.0f : f;
      v = Iv{__fadd_rd(__fmaf_rd(m, S.lo, lo), Y0.lo), __fadd_ru(__fmaf_ru(m, S.hi, hi), Y0.hi)};
    }
  } else if (kind == WK_SCALE) {
    v = I::mul_f(X, f);
  } else if (kind == WK_SQR) {
    v = I::sqr(X);
  } else if (kind == WK_MM) {
    const Iv B = (q.x & WC_II) ? Y0 : iv(f);
    const bool mx = q.x & WC_MAX;
    const Iv lo = I::min_(X, B), hi = I::max_(X, B);
    v = mx ? hi : lo;
    if (dec) dec[(q.x & WC_II) ? q.w : q.z] = (uint8_t)minmax_decision(mx, X, B);
  } else if (kind == WK_MUL) {
    v = I::mul(X, Y0);
  } else if (kind == WK_ABS) {
    v = I::abs_(X);
  } else if (kind == WK_SQRT) {
    v = I::sqrt_(X);
  } else if (kind == WK_SIN) {
    v = I::sin_(X);
  } else {
    const bool ii = q.x & WC_II;
    v = cold_forward<D>(ii ? q.w : q.z, X, ii ? Y0 : iv(f), f);
  }
  V.st(q, I::fix(v));
}

// Forward pass over the bundles (compute.wgsl:3633-3772); returns the field.
// dual: over two time intervals at once, V holding the values over `t` (the
// field and the reverse pass use them) and V2 those over `t2`, whose min/max
// decisions go to dec2 (those over `t` to dec); the second evaluation is
// independent of the first, so a step runs both.  Every min/max writes its
// decision byte when dec is set.
template <bool D, bool GM>
__device__ __forceinline__ Iv cell_forward(const WideDev &W, CellArray<GM> V, CellArray<GM> V2, bool dual, uint8_t *dec,
                                           uint8_t *dec2, Iv x, Iv y, Iv z, Iv t, Iv t2) {
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    const Iv zero = Iv{D ? 0.0f : -0.0f, -0.0f};
    V.st(0, x);
    V.st(1, y);
    V.st(2, z);
    V.st(3, t);
    V.st(W.nvalues, zero);
    if (dual) {
      V2.st(0, x);
      V2.st(1, y);
      V2.st(2, z);
      V2.st(3, t2);
      V2.st(W.nvalues, zero);
    }
  }
  __syncthreads();
  const bool both = __any_sync(FULL_MASK, dual);
  walk_steps(W, tid >> 5, W.fwd, [&](const uint4 &q, uint32_t kind) {
    wide_forward_slot<D>(kind, q, ForwardPlaces<GM>{V}, dec);
    if (both) wide_forward_slot<D>(kind, q, ForwardPlaces<GM>{V2}, dec2);
  });
  return V.ld(W.nvalues - 1u);
}

// The same for a cell whose values are in the global scratch, by slots of
// shared memory from S on (S2 behind them): a step then reads what the one
// before wrote without the round trip to L2, and the scratch is only written,
// where the reverse pass will read it (keep).  18777-instruction tape, 2360
// slots: 110 to 65 thousand cycles a cell, inversions of the 1024-primitive
// animation 2.01 and 2.68 to 1.60 and 2.26 ms.
template <bool D>
__device__ __forceinline__ Iv cell_forward_slots(const WideDev &W, unsigned char *S, CellArray<true> V, bool keep_,
                                                 bool dual, uint8_t *dec, uint8_t *dec2, Iv x, Iv y, Iv z, Iv t, Iv t2) {
  const uint32_t tid = threadIdx.x;
  const bool both = __any_sync(FULL_MASK, dual), keep = __any_sync(FULL_MASK, keep_);
  const ForwardSlots A{CellArray<false>(S), V, keep}, B{CellArray<false>(S + W.fslots * 8u), V, false};
  if (tid < 4u) {
    const Iv v = tid == 0u ? x : tid == 1u ? y : tid == 2u ? z : t;
    A.S.st(2u + tid, v);
    if (keep) V.st(tid, v);
    if (both) B.S.st(2u + tid, tid == 3u ? t2 : v);
  }
  if (tid == 4u) {
    const Iv zero = Iv{D ? 0.0f : -0.0f, -0.0f};
    A.S.st(0u, zero);
    if (keep) V.st(W.nvalues, zero);
    if (both) B.S.st(0u, zero);
  }
  __syncthreads();
  walk_steps(W, tid >> 5, W.fwd_slots, [&](const uint4 &q, uint32_t kind) {
    wide_forward_slot<D>(kind, q, A, dec);
    if (both) wide_forward_slot<D>(kind, q, B, dec2);
  });
  const Iv field = A.S.ld(W.f_field);
  __syncthreads();  // the slots' place is used again
  return field;
}

// Sum of a value's contribution records, last user first, onto +0: the
// accumulation order of the sequential reverse pass.  The sums are one
// dependent chain; the loads run ahead of it.
template <bool D, typename G>
__device__ __forceinline__ Iv gather_sens(G R, uint32_t base, uint32_t count) {
  Iv S = iv(0.0f);
  uint32_t i = 0;
  for (; i + 8u <= count; i += 8u) {
    Iv c[8];
#pragma unroll
    for (uint32_t u = 0; u < 8u; ++u) c[u] = R.ld(base + i + u);
#pragma unroll
    for (uint32_t u = 0; u < 8u; ++u) S = IA<D>::add(c[u], S);
  }
  for (; i < count; ++i) S = IA<D>::add(R.ld(base + i), S);
  return S;
}

// ---------------------------------------------------------------- reverse
// A slot of the reverse pass, unpacked (wide_tape.h).
struct WideRevSlot {
  uint32_t flags, a, b, lit, ta, tb, src, count;
};

// One slot of the reverse pass: its sensitivity (its own value's, or the sum
// of its contribution records), the handler's reverse rule and the
// operands' shares, each to its target in G: the operand's own place (one
// user: nothing else is added to it) or this use's record.
template <bool D, typename VArray, typename GArray>
__device__ __forceinline__ void wide_reverse_slot(uint32_t kind_, WideRevSlot p, VArray V, GArray G) {
  using I = IA<D>;
  const float f = __uint_as_float(p.lit);
  const Iv A = V.ld(p.a), B0 = V.ld(p.b);
  const uint32_t kg = uniform_u32(kind_), kind = kg & 15u;
  Iv s;
  if (kg & WK_GATHER) s = p.count ? gather_sens<D>(G, p.src, p.count) : G.ld(p.src);
  else s = G.ld(p.src);
  // a point factor's product (exact in the directed form: the factor is 0 or
  // +-1, so one rounding mode serves both bounds)
  auto point_mul = [&](float c) -> Iv {
    const float u = __fmul_rn(c, s.lo), w = __fmul_rn(c, s.hi);
    const Iv r = Iv{fm_min(u, w), fm_max(u, w)};
    if (D && (u != u || w != w)) return I::entire();
    return r;
  };
  Iv c0, c1 = iv(0.0f);
  if (kind == WK_LIN) {
    c0 = point_mul((p.flags & WC_NEG) ? -1.0f : 1.0f);
    c1 = point_mul((p.flags & WC_NEG2) ? -1.0f : 1.0f);
  } else if (kind == WK_SCALE) {
    c0 = I::mul(I::fix(iv(f)), s);
  } else if (kind == WK_SQR) {
    c0 = I::mul(I::fix(I::mul_f(A, 2.0f)), s);
  } else if (kind == WK_MM) {
    // a decided min/max passes the sensitivity to one operand, an undecided
    // one to both (directed: by a factor in [0, 1])
    const Iv B = (p.flags & WC_II) ? B0 : iv(f);
    const bool mx = p.flags & WC_MAX, a_below = A.hi < B.lo, b_below = !a_below && B.hi < A.lo;
    const bool a_out = mx ? a_below : b_below, b_out = mx ? b_below : a_below;
    c0 = point_mul(a_out ? 0.0f : 1.0f);
    c1 = point_mul(b_out ? 0.0f : 1.0f);
    if (D && !a_out && !b_out) c0 = c1 = I::mul(Iv{0.0f, 1.0f}, s);
  } else if (kind == WK_MUL) {
    c0 = I::mul(I::fix(B0), s);
    c1 = I::mul(I::fix(A), s);
  } else if (kind == WK_ABS) {
    c0 = I::mul(I::abs_rr(A), s);
  } else if (kind == WK_SQRT) {
    c0 = I::mul(I::fix(I::sqrt_rr(A)), s);
  } else if (kind == WK_SIN) {
    c0 = I::mul(I::fix(I::cos_(A)), s);
  } else {
    const bool ii = p.flags & WC_II;
    Iv r0 = iv(0.0f), r1 = iv(0.0f);
    cold_reverse_rule<D>((p.flags >> 8) & 63u, A, ii ? B0 : iv(f), f, r0, r1);
    c0 = I::mul(I::fix(r0), s);
    c1 = I::mul(I::fix(r1), s);
  }
  c0 = I::add(c0, iv(0.0f));
  c1 = I::add(c1, iv(0.0f));
  // the skip rule of compute.wgsl:3800-3806 (flagged operands of a zero
  // sensitivity receive zero); to nearest a finite factor's product with a
  // zero adds a zero anyway
  if (D && (p.flags & WC_SKIP) && s.lo == 0.0f && s.hi == 0.0f) c0 = c1 = iv(0.0f);
  G.st(p.ta, c0);
  G.st(p.tb, c1);
}

// Reverse interval AD over the bundles (compute.wgsl:3786-3900).  sens_out:
// the four arguments' sensitivities, in shared memory.  G: the sensitivities'
// slots, in shared memory also where the values are in the global scratch:
// a step reads and writes them, so their round trips to L2 are what it then
// waits for, while the values are only read.  18777-instruction tape, some
// 5000 slots for as many values and 7850 records: 315 to 125 thousand cycles
// a cell, inversions of the 1024-primitive animation 2.88 and 4.08 to 2.01
// and 2.68 ms.
template <bool D, typename VArray>
__device__ __forceinline__ void cell_reverse16(const WideDev &W, VArray V, CellArray<false> G, float2 *sens_out) {
  const uint32_t tid = threadIdx.x;
  if (tid < 4u && !W.arg_gcount[tid]) G.st(W.g_arg[tid], iv(0.0f));
  if (tid == 4u) G.st(0u, iv(0.0f));         // the zero
  if (tid == 5u) G.st(1u, iv(0.0f));         // the dummy
  if (tid == 6u) G.st(W.g_field, iv(1.0f));  // the field
  __syncthreads();
  const uint32_t nv = W.nvalues;
  walk_steps(W, kWideWarps + (tid >> 5), W.rev16, [&](const uint4 &p, uint32_t kind) {
    const bool ii = p.w & WC_II;
    wide_reverse_slot<D>(kind,
                         WideRevSlot{p.w & 0xffffu, p.x & 0xffffu, ii ? p.z : nv, p.z, p.y & 0xffffu, p.y >> 16,
                                     p.x >> 16, p.w >> 16},
                         V, G);
  });
  if (tid < 4u) {
    const uint32_t gc = W.arg_gcount[tid];
    const Iv s = gc ? gather_sens<D>(G, W.g_arg[tid], gc) : G.ld(W.g_arg[tid]);
    sens_out[tid] = make_float2(s.lo, s.hi);
  }
  __syncthreads();
}

// The same with everything in the global scratch, by indices of 32 bits (the
// second array's slot is read in the step).  G: the values' sensitivities and
// behind them the contribution records.
template <bool D>
__device__ __forceinline__ void cell_reverse(const WideDev &W, CellArray<true> V, CellArray<true> G, float2 *sens_out) {
  const uint32_t tid = threadIdx.x;
  if (tid < 4u) G.st(tid, iv(0.0f));
  if (tid == 4u) G.st(W.nvalues, iv(0.0f));       // the zero
  if (tid == 5u) G.st(W.nvalues + 1u, iv(0.0f));  // the dummy
  if (tid == 6u) G.st(W.nvalues - 1u, iv(1.0f));  // the field
  __syncthreads();
  const uint32_t stream = kWideWarps + (tid >> 5);
  const uint4 *t = W.rev + W.rev_slots + W.streams[stream].x + (tid & 31u);
  walk_steps(W, stream, W.rev, [&](const uint4 &p, uint32_t kind) {
    const uint4 r = *t;
    t += 32;
    wide_reverse_slot<D>(kind, WideRevSlot{p.x, p.y, p.z, p.w, r.x, r.y, r.z, r.w}, V, G);
  });
  if (tid < 4u) {
    const uint32_t gc = W.arg_gcount[tid];
    const Iv s = gc ? gather_sens<D>(G, W.nvalues + 2u + W.arg_gbase[tid], gc) : G.ld(tid);
    sens_out[tid] = make_float2(s.lo, s.hi);
  }
  __syncthreads();
}

}  // namespace tsi
