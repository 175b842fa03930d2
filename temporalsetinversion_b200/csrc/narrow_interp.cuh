// narrow_interp.cuh — the one-warp tape interpreter of the refinement
// kernel: 8, 16 or 32 cells per warp, one tape instruction at a time on the
// packed register tape (tape_format.h), interval registers in shared memory.
//
// narrow_forward follows compute.wgsl:3633-3772 (with the operand log and
// the min/max branch ballots that the reverse pass and the pruning need);
// narrow_reverse follows compute.wgsl:3785-3964.
//
// What bounds it: the instructions the warp issues per tape instruction
// (about four cycles each; a one-wave level lasts as long as its longest
// tape).  A switch over the handlers cost 170 cycles whichever handler it
// reached, and every branch the compiler takes for divergent 50, while the
// interval operation itself takes 10.  Hence
//  - each 32-instruction chunk is decoded once, one instruction per lane, to
//    16 bytes in shared memory (row offsets, a factor, a literal), and read
//    back by one broadcast load an instruction ahead;
//  - every handler that is linear in its operands (add, subtract, negate,
//    copy, multiply by a literal: two instructions in three) is
//    out = (m X + lit) + Y, where the product is exact or all else is the
//    zero that an addition leaves unchanged.  A ballot at the decode finds
//    the runs of such instructions; a run is a loop without a branch;
//  - the others are told apart by the bits of ballots taken at the decode,
//    which the compiler knows to be uniform;
//  - the reverse rules of linear handlers are factors of the sensitivity; an
//    absent second operand's share goes to a row that is never read, so one
//    and two operands take the same instructions;
//  - the operand log holds only what is not linear, packed densely, so that
//    the reverse pass reads it ahead.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_types.h"
#include "interp.cuh"

namespace tsi {

// Control word of a decoded instruction: handler in bits 0-5, single-use
// flags of the operands, the class, and the destination's row offset above.
constexpr uint32_t NC_FA = 1u << 6, NC_FB = 1u << 7;
constexpr uint32_t NC_LIN = 1u << 8;    // out = m X + Y
constexpr uint32_t NC_MUL = 1u << 9;
constexpr uint32_t NC_MM = 1u << 10;    // min/max
constexpr uint32_t NC_MAX = 1u << 11;   // ... max
constexpr uint32_t NC_SQR = 1u << 12;
constexpr uint32_t NC_ABS = 1u << 13;
constexpr uint32_t NC_SWAP = 1u << 14;  // X's bounds change places
constexpr uint32_t NC_YLIT = 1u << 15;  // Y is the literal
constexpr uint32_t NC_ZERO = NC_FA;     // (forward) the literal is the zero that changes no sum

// A warp's part of the shared memory: its register file (a row per register,
// a column of 8 bytes per cell), the chunk buffer, and a row that takes what
// nobody reads.  Items of one or two parents have 8 or 16 cells and one
// column more, which the lanes without a cell share (they compute along, on
// nothing that is read): the rows are then narrow enough for one
// shared-memory wavefront.
struct NarrowRows {
  uint32_t rf;      // shared address of this lane's column of row 0
  uint32_t prog;    // shared address of the 32 decoded instructions
  uint32_t stride;  // bytes of a row
  uint32_t sink;    // offset of the sink row
  uint32_t log_step;  // log entries from one instruction to the next (0: this lane's all go to one place)
};
// Of an item with so many parents: cells, then (below 32) the shared column.
__device__ __forceinline__ uint32_t narrow_cells(uint32_t parents) {
  return parents == 1u ? 8u : (parents == 2u ? 16u : 32u);
}
__device__ __forceinline__ NarrowRows narrow_rows(const void *base, uint32_t rcap, uint32_t lane, uint32_t parents) {
  NarrowRows R;
  const uint32_t cells = narrow_cells(parents);
  const uint32_t b = (uint32_t)__cvta_generic_to_shared(base);
  R.stride = cells < 32u ? (cells + 1u) * 8u : 256u;
  R.rf = b + min(lane, cells) * 8u;
  R.sink = rcap * 256u;
  R.log_step = R.stride / 8u;
  R.prog = b + rcap * 256u + 256u;
  return R;
}

__device__ __forceinline__ Iv row_ld(const NarrowRows &R, uint32_t off) {
  Iv v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.lo), "=f"(v.hi) : "r"(R.rf + off) : "memory");
  return v;
}
__device__ __forceinline__ void row_st(const NarrowRows &R, uint32_t off, Iv v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(R.rf + off), "f"(v.lo), "f"(v.hi) : "memory");
}
__device__ __forceinline__ uint4 prog_ld(const NarrowRows &R, uint32_t j) {
  uint4 w;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
               : "r"(R.prog + j * 16u)
               : "memory");
  return w;
}
__device__ __forceinline__ void prog_st(const NarrowRows &R, uint32_t j, uint4 w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(R.prog + j * 16u), "r"(w.x), "r"(w.y), "r"(w.z),
               "r"(w.w)
               : "memory");
}

// (m X + lit) + Y with one rounding: either the product is exact and one of
// the two terms, or both, the zero that an addition leaves unchanged (nz.lo,
// nz.hi), or both terms are.
template <bool D>
__device__ __forceinline__ Iv linear(float m, Iv X, Iv lit, Iv Y) {
  if (D) return Iv{__fadd_rd(__fmaf_rd(m, X.lo, lit.lo), Y.lo), __fadd_ru(__fmaf_ru(m, X.hi, lit.hi), Y.hi)};
  const F2 r = f2_add(f2_fma(f2_dup(m), f2_pack(X.lo, X.hi), f2_pack(lit.lo, lit.hi)), f2_pack(Y.lo, Y.hi));
  Iv v;
  f2_unpack(r, v.lo, v.hi);
  return v;
}

// Whether a product with the literal has a point as its factor: fix leaves
// the interval [lit, lit] alone.
__device__ __forceinline__ bool plain_factor(float lit) { return fabsf(lit) <= kBIG; }

// The zero that an addition leaves unchanged is -0 to nearest and rounding
// up, +0 rounding down (NC_ZERO: the bounds' literals are lit and, directed,
// -lit; the sink row holds it for Y).
template <bool D>
__device__ __forceinline__ uint4 decode_forward(uint2 w, uint32_t stride, uint32_t sink) {
  const uint32_t h = TSI_W0_H(w.x);
  const uint32_t a = TSI_W0_A(w.x) * stride, d = TSI_W0_DST(w.x) * stride;
  const bool ii = TSI_H_IS_II(h);
  const uint32_t b = ii ? (w.y & 255u) * stride : sink;
  uint32_t c = h | (ii ? 0u : NC_YLIT), x = a, y = b;
  float m = 1.0f, lit = __uint_as_float(w.y);
  const float zero = D ? 0.0f : -0.0f;
  switch ((w.x & TSI_W0_ODD) ? H_COUNT : h) {
    case H_ADD_II: c |= NC_LIN | NC_ZERO; lit = zero; break;
    case H_SUB_II: c |= NC_LIN | NC_ZERO | NC_SWAP; x = b; y = a; m = -1.0f; lit = zero; break;
    case H_ADD_IF: c |= NC_LIN; break;
    case H_SUB_IF: c |= NC_LIN; lit = -lit; break;
    case H_SUB_FI: c |= NC_LIN | NC_SWAP; m = -1.0f; break;
    case H_NEG: c |= NC_LIN | NC_SWAP | NC_ZERO; m = -1.0f; lit = zero; break;
    case H_COPY: c |= NC_LIN | NC_ZERO; lit = zero; break;
    case H_MUL_IF:
      if (!D && plain_factor(lit)) {  // bounds change places for a factor that is not >= 0
        c |= NC_LIN | NC_ZERO;
        if (!(lit >= 0.0f)) c |= NC_SWAP;
        m = lit;
        lit = zero;
      }
      break;
    case H_MUL_II: c |= NC_MUL; break;
    case H_SQR: c |= NC_SQR; break;
    case H_ABS: c |= NC_ABS; break;
    case H_MIN_II: case H_MIN_IF: c |= NC_MM; break;
    case H_MAX_II: case H_MAX_IF: c |= NC_MM | NC_MAX; break;
    default: break;
  }
  return make_uint4(c | (d << 16), x | (y << 16), __float_as_uint(m), __float_as_uint(lit));
}

// The classes agree with decode_forward's on what is linear: the forward
// pass logs the operands of everything else, the reverse pass pops them.
template <bool D>
__device__ __forceinline__ uint4 decode_reverse(uint2 w, uint32_t stride, uint32_t sink) {
  const uint32_t h = TSI_W0_H(w.x);
  const uint32_t d = TSI_W0_DST(w.x) * stride;
  const bool ii = TSI_H_IS_II(h);
  uint32_t a = TSI_W0_A(w.x) * stride, b = ii ? (w.y & 255u) * stride : sink;
  // one operand: both flags follow the first
  uint32_t c = h | (TSI_W0_FA(w.x) ? NC_FA : 0u) | ((ii ? TSI_W0_FB(w.x) : TSI_W0_FA(w.x)) ? NC_FB : 0u);
  const float lit = __uint_as_float(w.y);
  float c0 = 1.0f, c1 = 1.0f;
  switch ((w.x & TSI_W0_ODD) && h != H_CONST ? H_COUNT : h) {
    case H_ADD_II: case H_ADD_IF: case H_SUB_IF: case H_COPY: c |= NC_LIN; break;
    case H_SUB_II: c |= NC_LIN; c1 = -1.0f; break;
    case H_SUB_FI: case H_NEG: c |= NC_LIN; c0 = -1.0f; break;
    case H_CONST: a = sink; break;
    case H_MUL_IF:
      if (!D && plain_factor(lit)) {
        c |= NC_LIN;
        c0 = lit;
      }
      break;
    case H_MUL_II: c |= NC_MUL; break;
    case H_SQR: c |= NC_SQR; break;
    case H_ABS: c |= NC_ABS; break;
    case H_MIN_II: case H_MIN_IF: c |= NC_MM; break;
    case H_MAX_II: case H_MAX_IF: c |= NC_MM | NC_MAX; break;
    default: break;
  }
  // the literal of the handlers that are not linear travels in the factor
  // (directed, the lost operand's arguments in place of a copy's second factor,
  // which goes to the sink, and of a constant's literal)
  const bool deps = D && (h == H_COPY || h == H_CONST);
  return make_uint4(c | (d << 16), a | (b << 16), __float_as_uint(c0),
                    deps ? TSI_W0_DEPS(w.x) : (c & NC_LIN) ? __float_as_uint(c1) : w.y);
}

// Which instructions of a chunk are of a kind, by ballot (one instruction per
// lane): branches on these bits are uniform.
struct NarrowKinds {
  uint32_t sqr, mm, mul, abs;
};
__device__ __forceinline__ NarrowKinds narrow_kinds(uint32_t c) {
  NarrowKinds K;
  K.sqr = __ballot_sync(FULL_MASK, (c & NC_SQR) != 0u);
  K.mm = __ballot_sync(FULL_MASK, (c & NC_MM) != 0u);
  K.mul = __ballot_sync(FULL_MASK, (c & NC_MUL) != 0u);
  K.abs = __ballot_sync(FULL_MASK, (c & NC_ABS) != 0u);
  return K;
}

// A value equal in all lanes, known as such to the compiler.
__device__ __forceinline__ uint32_t uniform_u32(uint32_t v) { return __reduce_max_sync(FULL_MASK, v); }

// Forward pass over `len` instructions (compute.wgsl:3633-3772).  Pushes the
// operands of everything that is not linear on the log `lg` (this lane's
// column of it, an entry of 16 bytes every R.log_step; null: no log) and the
// min/max branch ballots to `dg` when they are set.  `nlog` is the number of
// log entries (0 in a lane whose log_step is 0).  Returns the output
// register's value.
template <bool D>
__device__ __noinline__ Iv narrow_forward(const uint2 *__restrict__ code, uint32_t len_, uint32_t out_reg,
                                          NarrowRows R, uint32_t lane, Iv x, Iv y, Iv z, Iv t, float4 *lg, uint2 *dg,
                                          uint32_t &nlog) {
  using I = IA<D>;
  const uint32_t len = uniform_u32(len_);
  const bool log_on = __any_sync(FULL_MASK, lg != nullptr), dec_on = __any_sync(FULL_MASK, dg != nullptr);
  row_st(R, 0, x);
  row_st(R, R.stride, y);
  row_st(R, 2u * R.stride, z);
  row_st(R, 3u * R.stride, t);
  const uint32_t cols = R.log_step;
  float4 *lp = lg;
  row_st(R, R.sink, Iv{D ? 0.0f : -0.0f, -0.0f});
  auto linear_step = [&](const uint4 &w) {
    const uint32_t c = w.x;
    const float lit = __uint_as_float(w.w);
    const Iv X = row_ld(R, w.y & 0xffffu), Y = row_ld(R, w.y >> 16);
    const Iv v = linear<D>(__uint_as_float(w.z), (c & NC_SWAP) ? Iv{X.hi, X.lo} : X,
                           Iv{lit, (D && (c & NC_ZERO)) ? -lit : lit}, Y);
    row_st(R, c >> 16, I::fix(v));
  };
  auto other_step = [&](const uint4 &w, const NarrowKinds &K, uint32_t j) {
    const uint32_t c = w.x;
    const float lit = __uint_as_float(w.w);
    const Iv X = row_ld(R, w.y & 0xffffu), Y0 = row_ld(R, w.y >> 16);
    const Iv Y = (c & NC_YLIT) ? iv(lit) : Y0;
    Iv v;
    if (log_on) {
      *lp = make_float4(X.lo, X.hi, Y.lo, Y.hi);
      lp += cols;
    }
    if ((K.sqr >> j) & 1u) {
      v = I::sqr(X);
    } else if ((K.mm >> j) & 1u) {
      const bool mx = c & NC_MAX;
      const Iv lo = I::min_(X, Y), hi = I::max_(X, Y);
      v = mx ? hi : lo;
      if (dec_on) {
        // bit 0: the first operand is always chosen, bit 1: the second
        const uint32_t ux = __ballot_sync(FULL_MASK, X.hi < Y.lo), uy = __ballot_sync(FULL_MASK, Y.hi < X.lo);
        if (lane == 0u) *dg = mx ? make_uint2(uy, ux) : make_uint2(ux, uy);
        ++dg;
      }
    } else if ((K.mul >> j) & 1u) {
      v = I::mul(X, Y);
    } else if ((K.abs >> j) & 1u) {
      v = I::abs_(X);
    } else {
      const uint32_t h = c & 63u;
      if (__any_sync(FULL_MASK, h == H_SQRT)) v = I::sqrt_(X);
      else if (__any_sync(FULL_MASK, h == H_SIN)) v = I::sin_(X);
      else v = cold_forward<D>(h, X, Y, lit);
    }
    row_st(R, c >> 16, I::fix(v));
  };
  uint2 nxt = load_chunk(code, len, 0, lane);
  for (uint32_t c0 = 0; c0 < len; c0 += 32u) {
    const uint32_t n = min(32u, len - c0);
    __syncwarp();
    const uint4 dec = decode_forward<D>(nxt, R.stride, R.sink);
    prog_st(R, lane, dec);
    // instructions that are not linear (one past the last ends the chunk)
    const uint32_t other = __ballot_sync(FULL_MASK, lane >= n || !(dec.x & NC_LIN));
    const NarrowKinds K = narrow_kinds(dec.x);
    nxt = load_chunk(code, len, (int)(c0 / 32u) + 1, lane);  // a chunk ahead
    __syncwarp();  // (votes order no memory)
    uint32_t j = 0;
    uint4 w = prog_ld(R, 0);
    while (j < n) {
      const uint32_t rest = other >> j;
      const uint32_t end = rest ? j + (uint32_t)__ffs((int)rest) - 1u : 32u;
#pragma unroll 1
      for (; j + 2u <= end; j += 2u) {
        const uint4 w1 = prog_ld(R, j + 1u);
        linear_step(w);
        w = prog_ld(R, (j + 2u) & 31u);
        linear_step(w1);
      }
      if (j < end) {
        const uint4 w1 = prog_ld(R, (j + 1u) & 31u);
        linear_step(w);
        w = w1;
        ++j;
      }
      if (j < n) {
        const uint4 w1 = prog_ld(R, (j + 1u) & 31u);
        other_step(w, K, j);
        w = w1;
        ++j;
      }
    }
  }
  nlog = log_on && cols ? (uint32_t)((lp - lg) / cols) : 0u;
  return row_ld(R, out_reg * R.stride);
}

// Reverse pass (compute.wgsl:3785-3964): sensitivities reuse the register
// file; a register's accumulator is consumed and cleared at the definition
// it holds.  `bad` tells of a non-finite sensitivity in a lane that takes
// the derivative: every accumulator is either consumed at a definition or
// one of the four arguments', and a sum that became infinite or NaN stays
// so, so testing what is consumed finds every one.
//
// Those are the cells whose full tape may give more than a pruned one: it
// adds what a decided min/max passes to the operand that lost, zero times its
// sensitivity.  The caller runs them on the full tape.
//
// Directed, a root at zero makes infinite sensitivities in ordinary cells,
// and the full tape on one warp took a level of 64-primitive cells 0.65 ms.
// But there zero times an infinite bound is the whole line, and so is every
// product and sum with it: what the full tape adds is known.  A copy or a
// constant that a decided min/max has become carries the arguments that its
// lost operand depends on; with a sensitivity that is not finite those are
// the whole line, and nothing else changes.  Unless `strict`: then a rule
// behind a lost operand may itself be infinite and turn a plain zero into
// more (directed rules are not clamped), and directed cells are treated like
// the others.  Inversions of the directed 64-primitive scene 0.95 to
// 0.42 ms.
template <bool D>
__device__ __noinline__ void narrow_reverse(const uint2 *__restrict__ code, uint32_t len_, uint32_t nregs,
                                            uint32_t out_reg, NarrowRows R, uint32_t lane, const float4 *lg,
                                            uint32_t nlog, bool take, bool strict_, Iv sens[4], bool &bad) {
  using I = IA<D>;
  const uint32_t len = uniform_u32(len_);
  __syncwarp();
  for (uint32_t r = 0; r < nregs; ++r) row_st(R, r * R.stride, iv(0.0f));
  row_st(R, R.sink, iv(0.0f));
  row_st(R, out_reg * R.stride, iv(1.0f));
  // the log from its end, three entries ahead
  const uint32_t cols = R.log_step;
  int lp = (int)uniform_u32(nlog);
  auto entry = [&](int i) { return i < 0 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : lg[(size_t)i * cols]; };
  float4 E0 = entry(lp - 1), E1 = entry(lp - 2), E2 = entry(lp - 3);
  float nonfinite = 0.0f;  // becomes NaN with the first infinite or NaN bound
  const bool all = !D || __any_sync(FULL_MASK, strict_);
  uint32_t lost = 0;  // arguments whose sensitivity is the whole line
  // a point factor's product: exact for the factors of the directed form (0
  // and +-1), so one rounding mode serves both bounds
  auto point_mul = [](float f, Iv s) -> Iv {
    const float x = __fmul_rn(f, s.lo), y = __fmul_rn(f, s.hi);
    const Iv r = Iv{fm_min(x, y), fm_max(x, y)};
    if (D && (x != x || y != y)) return I::entire();
    return r;
  };
  auto check = [&](Iv s, bool pruned, uint32_t deps) {
    if (D && !all) {
      lost |= pruned && !finite2(s) ? deps : 0u;
      return;
    }
    nonfinite = __fmaf_rn(s.lo, 0.0f, nonfinite);
    nonfinite = __fmaf_rn(s.hi, 0.0f, nonfinite);
  };
  // The skip rule of compute.wgsl:3800-3806 (flagged operands of a zero
  // sensitivity are set to zero instead of added to) changes nothing here: a
  // flagged operand has no other user, so its accumulator is +0, and a
  // finite factor's product with a zero adds a zero.
  auto linear_step = [&](const uint4 &w) {
    const uint32_t d = w.x >> 16, a = w.y & 0xffffu, b = w.y >> 16;
    const Iv s = row_ld(R, d);
    row_st(R, d, iv(0.0f));
    // both accumulators are read before either is written (an instruction
    // whose operands are one register keeps the second write)
    const Iv pa = row_ld(R, a), pb = row_ld(R, b);
    check(s, (w.x & 63u) == H_COPY, w.w);
    row_st(R, a, I::add(point_mul(__uint_as_float(w.z), s), pa));
    row_st(R, b, I::add(point_mul(__uint_as_float(w.w), s), pb));
  };
  auto other_step = [&](const uint4 &w, const NarrowKinds &K, int j) {
    const uint32_t c = w.x, d = w.x >> 16, a = w.y & 0xffffu, b = w.y >> 16;
    const Iv s = row_ld(R, d);
    row_st(R, d, iv(0.0f));
    const Iv pa = row_ld(R, a), pb = row_ld(R, b);
    check(s, (c & 63u) == H_CONST, w.w);
    const bool skip = (s.lo == 0.0f && s.hi == 0.0f) && (c & (NC_FA | NC_FB)) == (NC_FA | NC_FB);
    const Iv A = Iv{E0.x, E0.y}, B = Iv{E0.z, E0.w};
    --lp;
    E0 = E1;
    E1 = E2;
    E2 = entry(lp - 3);
    Iv n0, n1 = iv(0.0f);
    if ((K.sqr >> j) & 1u) {
      n0 = I::add(I::mul(I::fix(I::mul_f(A, 2.0f)), s), pa);
    } else if ((K.mm >> j) & 1u) {
      // a decided min/max passes the sensitivity to one operand, an
      // undecided one to both (directed: by a factor in [0, 1])
      const bool a_below = A.hi < B.lo, b_below = !a_below && B.hi < A.lo;
      const bool a_out = (c & NC_MAX) ? a_below : b_below, b_out = (c & NC_MAX) ? b_below : a_below;
      Iv r0 = point_mul(a_out ? 0.0f : 1.0f, s), r1 = point_mul(b_out ? 0.0f : 1.0f, s);
      if (D && !a_out && !b_out) r0 = r1 = I::mul(Iv{0.0f, 1.0f}, s);
      n0 = I::add(r0, pa);
      n1 = I::add(r1, pb);
    } else if ((K.mul >> j) & 1u) {
      n0 = I::add(I::mul(I::fix(B), s), pa);
      n1 = I::add(I::mul(I::fix(A), s), pb);
    } else if ((K.abs >> j) & 1u) {
      n0 = I::add(I::mul(I::abs_rr(A), s), pa);
    } else {
      const uint32_t h = c & 63u;
      Iv q0 = iv(0.0f), q1 = iv(0.0f);
      if (__any_sync(FULL_MASK, h == H_SQRT)) q0 = I::sqrt_rr(A);
      else if (__any_sync(FULL_MASK, h == H_SIN)) q0 = I::cos_(A);
      else cold_reverse_rule<D>(h, A, B, __uint_as_float(w.w), q0, q1);
      n0 = I::add(I::mul(I::fix(q0), s), pa);
      n1 = I::add(I::mul(I::fix(q1), s), pb);
    }
    if (skip) n0 = n1 = iv(0.0f);
    row_st(R, a, n0);
    row_st(R, b, n1);
  };
  const int nch = (int)((len + 31u) / 32u);
  uint2 nxt = load_chunk(code, len, nch - 1, lane);
  for (int k = nch - 1; k >= 0; --k) {
    __syncwarp();
    const uint4 dec = decode_reverse<D>(nxt, R.stride, R.sink);
    prog_st(R, lane, dec);
    const int n = min(32, (int)len - 32 * k);
    const uint32_t other = __ballot_sync(FULL_MASK, !(dec.x & NC_LIN));
    const NarrowKinds K = narrow_kinds(dec.x);
    nxt = load_chunk(code, len, k - 1, lane);
    __syncwarp();  // (votes order no memory)
    int j = n - 1;
    uint4 w = prog_ld(R, (uint32_t)j);
    while (j >= 0) {
      // the last instruction at or below j that is not linear, -1 if none is
      const int stop = 31 - __clz((int)(other & (0xffffffffu >> (31 - j))));
#pragma unroll 1
      for (; j - 2 >= stop; j -= 2) {
        const uint4 w1 = prog_ld(R, (uint32_t)(j - 1));
        linear_step(w);
        w = prog_ld(R, (uint32_t)(j - 2) & 31u);
        linear_step(w1);
      }
      if (j > stop) {
        const uint4 w1 = prog_ld(R, (uint32_t)(j - 1) & 31u);
        linear_step(w);
        w = w1;
        --j;
      }
      if (j >= 0) {
        const uint4 w1 = prog_ld(R, (uint32_t)(j - 1) & 31u);
        other_step(w, K, j);
        w = w1;
        --j;
      }
    }
  }
  for (uint32_t q = 0; q < 4u; ++q) {
    sens[q] = row_ld(R, q * R.stride);
    check(sens[q], false, 0u);
    if (D && ((lost >> q) & 1u)) sens[q] = I::entire();
  }
  bad |= take && nonfinite != nonfinite;
}

}  // namespace tsi
