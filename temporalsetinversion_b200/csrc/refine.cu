// refine.cu — octree refinement step kernel (compute.wgsl `main`, 3513-4056).
//
// One launch per octree level, over every scene of the launch.  A warp takes
// one work item: up to four sibling parents (children of one grandparent,
// sharing one tape record) x 8 octants, one child cell per lane
// (narrow_interp.cuh: interval registers in shared memory, a column per
// cell).  While a level has blocks enough for its cells, items of long tapes
// go to the wide path instead, one block per cell (wide_interp.cuh).
//
// Per child cell the lane runs, as in the reference:
//   cell setup and temporal interval         compute.wgsl:3582-3626
//   forward interval tape                    3632-3774
//   reverse interval AD (operand log replay) 3776-3970
//   temporal error bound, fast flag          3971-4009
//   classify, re-enqueue or deallocate       4011-4045
// then, per sibling group that re-enqueues cells, prunes the tape: min/max
// instructions whose branch is decided for every enqueued sibling become
// copies (or constants), instructions that no longer reach the output are
// dropped.  Pruning never changes a result: a decided MIN/MAX returns its
// chosen operand bit for bit, and the reverse pass falls back to the full
// tape when a sensitivity overflows (the only case where the dead branch of
// the full tape would contribute, through 0 * inf; narrow_reverse tells
// where).
//
// A pruned tape is valid for cells inside its group's boxes whose time
// interval lies inside the interval the decisions were taken on.  The
// children of a re-enqueued cell are evaluated over [child.t, time]; when
// that reaches further back than the cell's own evaluation interval (the
// cell was evaluated at a point in time), the branch decisions are taken
// again by a second forward pass over the widened interval, so the children
// can use the pruned tape instead of an ancestor's.
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "device_types.h"
#include "interp.cuh"
#include "narrow_interp.cuh"
#include "wide_interp.cuh"
#include "interval.cuh"
#include "opcost.h"

namespace tsi {

__constant__ uint32_t c_cost_fwd[H_COUNT] = TSI_OPCOST_FWD_INIT;
__constant__ uint32_t c_cost_rr[H_COUNT] = TSI_OPCOST_RR_INIT;

constexpr int kWarps = 8;  // warps per block (block of 256)

// Dynamic shared memory of refine_kernel: the narrow path's register files,
// or the working set of the wide path's cell.
extern __shared__ __align__(16) unsigned char tsi_dyn_smem[];

// Programmatic dependent launch (PTX griddepcontrol, sm_90 and later): the
// wait returns once the grids this launch depends on have completed and
// their writes are visible (at once for a launch without that dependency);
// the trigger lets the stream's next launch begin once every block of this
// one has issued it.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// First word of the copy that a decided min/max (first word w) becomes: of
// operand A, or else B, in register r.
__device__ __forceinline__ uint32_t copy_word(uint32_t w, bool of_a, uint32_t d, uint32_t r) {
  const uint32_t flag = of_a ? TSI_W0_FA(w) : TSI_W0_FB(w), raw = w & (of_a ? TSI_W0_RAW_A : TSI_W0_RAW_B);
  return TSI_W0(H_COPY, flag, 0u, d, r) | (w & TSI_W0_ODD) | (raw ? TSI_W0_RAW_A : 0u);
}

// Backward liveness scan of one sibling group (g, enqueued siblings E) by the
// whole warp: decided min/max become copies/constants, dead instructions
// vanish.  The kept instructions are written in reverse order to `tmp`;
// returns their count.  A chunk of 32 instructions is decoded one per lane
// (decision, operand and destination masks); what is left of the serial scan
// is three logic operations an instruction on the 64-bit mask of live
// registers, on masks read back by broadcast loads.  (One lane decoding and
// scanning took 300 cycles an instruction.  By the level counters the scans of
// the 64 and 256-primitive animations take 60 cycles per instruction of their
// items' forward passes, which take 320 to 340.)
template <bool D>
__device__ __forceinline__ uint32_t prune_group(const uint2 *__restrict__ code, uint32_t len_, uint32_t n_minmax_,
                                                uint32_t out_reg, const uint2 *dg, uint32_t g, uint32_t E, uint2 *tmp,
                                                const NarrowRows &R, uint32_t lane, uint32_t &mm_kept, uint32_t &fwd_cost,
                                                uint32_t &rev_cost) {
  const uint32_t len = uniform_u32(len_);
  uint32_t live_lo = out_reg < 32u ? 1u << out_reg : 0u, live_hi = out_reg >= 32u ? 1u << (out_reg - 32u) : 0u;
  uint32_t cnt = 0, kept_mm = 0, fc = 0, rc = 0;
  const int nch = (int)((len + 31u) / 32u);
  int m = (int)uniform_u32(n_minmax_);  // min/max ordinals from the end
  uint2 nxt = load_chunk(code, len, nch - 1, lane);
  for (int k = nch - 1; k >= 0; --k) {
    const uint2 w = nxt;
    nxt = load_chunk(code, len, k - 1, lane);
    const bool valid = 32u * (uint32_t)k + lane < len;
    const uint32_t h = TSI_W0_H(w.x), d = TSI_W0_DST(w.x), a = TSI_W0_A(w.x), b = w.y & 255u;
    const bool mmx = valid && TSI_H_IS_MINMAX(h);
    const uint32_t mmb = __ballot_sync(FULL_MASK, mmx);
    m -= __popc(mmb);
    uint2 out = w;
    uint32_t hk = h;
    bool use_a = h != H_CONST, use_b = TSI_H_IS_II(h);
    if (mmx) {
      const uint32_t deps_a = TSI_W0_WITH_DEPS(TSI_W0_DEPS(w.x));
      const uint32_t deps_b = TSI_H_IS_II(h) ? TSI_W0_WITH_DEPS(TSI_W1_DEPS(w.y)) : 0u;
      const uint2 dd = dg[m + __popc(mmb & ((1u << lane) - 1u))];
      const uint32_t ga = (dd.x >> (g * 8u)) & 0xffu, gb = (dd.y >> (g * 8u)) & 0xffu;
      if ((ga & E) == E) {
        out = make_uint2(copy_word(w.x, true, d, a) | deps_b, 0u);
        hk = H_COPY;
        use_b = false;
      } else if ((gb & E) == E) {
        use_a = false;
        if (TSI_H_IS_II(h)) {
          out = make_uint2(copy_word(w.x, false, d, b) | deps_a, 0u);
          hk = H_COPY;
        } else {
          out = make_uint2(TSI_W0(H_CONST, 0u, 0u, d, 0u) | deps_a, w.y);
          hk = H_CONST;
        }
      }
    }
    // registers written and read, as 64-bit masks
    unsigned long long def = valid ? 1ull << d : 0ull, src = 0ull;
    if (use_a) src |= 1ull << a;
    if (use_b) src |= 1ull << b;
    __syncwarp();
    prog_st(R, lane, make_uint4((uint32_t)def, (uint32_t)(def >> 32), (uint32_t)src, (uint32_t)(src >> 32)));
    __syncwarp();
    uint32_t keep = 0;
#pragma unroll 8
    for (int j = 31; j >= 0; --j) {
      const uint4 q = prog_ld(R, (uint32_t)j);
      const bool on = ((live_lo & q.x) | (live_hi & q.y)) != 0u;
      live_lo = (live_lo & ~q.x) | (on ? q.z : 0u);
      live_hi = (live_hi & ~q.y) | (on ? q.w : 0u);
      keep |= on ? 1u << j : 0u;
    }
    // a copy of a register to itself does nothing, forward or reverse, but
    // carry a directed reverse pass's test and clamp an argument
    if (!D) keep &= ~__ballot_sync(FULL_MASK, hk == H_COPY && TSI_W0_A(out.x) == d && !(out.x & TSI_W0_RAW_A));
    if ((keep >> lane) & 1u) {
      tmp[cnt + __popc(keep & ~((2u << lane) - 1u))] = out;
      kept_mm += TSI_H_IS_MINMAX(hk) ? 1u : 0u;
      fc += c_cost_fwd[hk] + TSI_FIX_COST;
      rc += c_cost_rr[hk] + TSI_REV_OPERAND_COST * TSI_H_NREG(hk);
    }
    cnt += __popc(keep);
  }
  mm_kept = __reduce_add_sync(FULL_MASK, kept_mm);
  fwd_cost = __reduce_add_sync(FULL_MASK, fc);
  rev_cost = __reduce_add_sync(FULL_MASK, rc);
  __syncwarp();  // tmp is read by other lanes
  return cnt;
}

// mallocV (compute.wgsl:3437-3450) for a whole brick of 8 siblings.
__device__ uint32_t alloc_brick(const SceneLaunch &S, uint32_t *error) {
  SceneCounters *c = S.ctr;
  int32_t fc = atomicSub(&c->free_count, 1);
  uint32_t b;
  if (fc > 0) {
    b = S.pool.free_list[fc - 1];
  } else {
    b = atomicAdd(&c->bump, 1u);
    if (b >= S.pool.cap_bricks) {
      atomicOr(error, EB_OOM);
      return TSI_NONE;
    }
  }
  return b * 8u;
}

// The wide threshold for children at `level`: deep levels may have one of
// their own.
__device__ __forceinline__ uint32_t wide_min_len(const WideDev &W, uint32_t level) {
  return level >= W.deep_level ? W.deep_min_len : W.min_len;
}
__device__ __forceinline__ StepIdx step_idx(uint32_t step) {
  StepIdx si;
  si.cur = step & TSI_STEP_MASK;
  si.next = (step + 1u) & TSI_STEP_MASK;
  si.buf = step & 1u;
  si.nbuf = (step + 1u) & 1u;
  return si;
}

// Log entries of a cell on a tape of this length, at most.
__device__ __forceinline__ uint32_t log_bound(const WideDev &W, uint32_t len) { return min(len, W.log_len); }
// Whether the log of an item of n parents fits its warp's slice.
__device__ __forceinline__ bool slice_holds(const LaunchParams &P, uint32_t n, uint32_t entries) {
  return (n == 1u ? 9u : n == 2u ? 17u : 32u) * entries <= 32u * P.slice_len;
}
// Whether an item that the length alone sends wide may be a narrow one.
__device__ __forceinline__ bool may_go_narrow(const LaunchParams &P, const WideDev &W, uint32_t level, uint32_t len) {
  return !W.by_length && len >= wide_min_len(W, level) && slice_holds(P, 1u, log_bound(W, len));
}

// Whether children of this step's groups with a tape of this length take the
// wide path: from the threshold on (where a block per cell and a warp per item
// take equally long), but for levels with more long items than blocks.  There
// the threshold is multiplied by the waves of blocks that this step's long
// items need for their eight cells each; the next step seldom has fewer.  A
// step of long items finishes a wide item of 8 cells in 8/296 of a cell's time
// on a B200's 296 blocks, but 2368 narrow items at once: by length alone,
// levels of thousands of long items ran one block per cell.  Rotating swept
// scene (64 primitives, localsubdiv 9) 8.0 to 2.7 ms an inversion, 1024
// primitives (localsubdiv 9) 3.7 to 3.3 ms, 256 primitives unchanged; half and
// twice the multiplier measured 3.1 and 2.7 ms, 3.6 and 3.2 ms.
//
// An item that the length alone would send wide costs neither the log arena
// nor the narrow list anything that others may need:
//  - its log fits its warp's slice (the arena, 16 bytes per instruction and
//    column, is what items below the threshold share), with fewer parents if
//    need be, and where it has to run on a longer tape of its scene it takes
//    the cells in turns (own_slice_passes);
//  - half of the narrow list stays free of such items, and what finds it full
//    goes wide after all (push_children).
//
// by_length: a tape whose log fits no slice, and outward rounding, where a
// one-warp item costs two to four times as much an instruction (no packed
// form, and its sines no short one): rotating swept scenes of 44 and 64
// primitives, localsubdiv 8, three inversions 10.6 and 19.8 ms so, 15.3 and
// 23.0 with the waves.
__device__ __forceinline__ bool goes_wide(const LaunchParams &P, const WideDev &W, uint32_t step, uint32_t level,
                                          uint32_t len) {
  const uint32_t from = wide_min_len(W, level);
  if (!may_go_narrow(P, W, level, len)) return len >= from;
  const uint32_t waves = max(1u, 8u * P.long_count[step & TSI_STEP_MASK] / gridDim.x);
  const uint32_t next = step_idx(step).next;
  return len >= (unsigned long long)from * waves || *(const volatile uint32_t *)&P.item_count[next] > P.item_cap / 2u;
}
// The same for a warp that goes on together: lane 0's answer, for the list may
// grow between the reads of two lanes.
__device__ __forceinline__ bool warp_goes_wide(const LaunchParams &P, const WideDev &W, uint32_t step, uint32_t level,
                                               uint32_t len) {
  return __shfl_sync(FULL_MASK, goes_wide(P, W, step, level, len) ? 1u : 0u, 0) != 0u;
}

// Reserves n words of the code arena (a ring of code_cap words, a power of
// two); returns the word offset, or ~0 when the ring has no room left above
// the low-water mark (the tape then stays unpruned).  A tape never wraps
// around the ring's end.
__device__ __forceinline__ unsigned long long code_alloc(const LaunchParams &P, uint32_t n) {
  const unsigned long long c = atomicAdd(P.code_count, (unsigned long long)n);
  if (c + n > *P.code_low + P.code_cap) return ~0ull;
  const unsigned long long off = c & (P.code_cap - 1ull);
  return off + n <= P.code_cap ? off : ~0ull;
}

// Takes a tape record from the ring [rec_base, rec_cap) (a power-of-two
// size); TSI_NONE when the ring has no room left above the low-water mark.
__device__ __forceinline__ uint32_t rec_alloc(const LaunchParams &P) {
  const unsigned long long r = atomicAdd(P.rec_count, 1ull);
  const uint32_t ring = P.rec_cap - P.rec_base;
  if (r >= *P.rec_low + ring) return TSI_NONE;
  return P.rec_base + ((uint32_t)r & (ring - 1u));
}

__device__ __forceinline__ void find_valid(const LaunchParams &P, uint32_t &rec, TapeRec &TR, float tl, float th) {
  TR = P.recs[rec];
  while (TR.parent != TSI_NONE && !(TR.t_lo <= tl && th <= TR.t_hi)) {
    rec = TR.parent;
    TR = P.recs[rec];
  }
}

// Wide items for the children `rest` (cells[0..7] of one parent), one per
// child, its own children's brick allocated here; returns those that the wide
// list has no room for.  One thread.
__device__ __forceinline__ uint32_t push_wide(const LaunchParams &P, const SceneLaunch &S, uint32_t scene, uint32_t rec,
                                           uint32_t step, uint32_t plevel, uint32_t rest, const uint32_t *cells,
                                           unsigned long long *ws) {
  const StepIdx si = step_idx(step);
  const uint32_t n = __popc(rest);
  const uint32_t pos = atomicAdd(&P.witem_count[si.next], n);
  uint32_t j = 0;
  while (rest && pos + j < P.witem_cap) {
    const uint32_t bit = __ffs(rest) - 1u;
    rest &= rest - 1u;
    const uint32_t c = cells[bit];
    uint32_t b = S.pool.child[c], fresh = 0;
    if (b == TSI_NONE) {
      b = alloc_brick(S, P.error + scene);
      if (b != TSI_NONE) {
        S.pool.child[c] = b;
        fresh = 1;
        atomicAdd(&ws[ST_BRICK_ALLOC], 1ull);
      }
    }
    WorkItem wi;
    wi.scene = scene;
    wi.rec = rec;
    wi.n = 1;
    wi.level = plevel + 1;
    wi.parent[0] = c;
    wi.parent[1] = b;
    wi.parent[2] = fresh;
    wi.parent[3] = 0;
    P.witems[si.nbuf][pos + j++] = wi;
  }
  return rest;
}

// Next-level work for the enqueued children (mask E) of one parent, whose
// cells are cells[0..7]; one thread.  `wide`: wide items; children beyond the
// wide list's capacity, or all of them when not `wide`, go to the narrow list
// in items of up to four.  Every reserved list slot below the capacity is
// written (readers take min(count, capacity) entries).  What the narrow list
// has no room for goes wide if it may, else it is dropped and reported.
// `either`: the log entries of a cell that may go either way, else 0.
__device__ void push_children(const LaunchParams &P, const SceneLaunch &S, uint32_t scene, uint32_t rec,
                              uint32_t step, uint32_t plevel, uint32_t E, const uint32_t *cells, bool wide, uint32_t either,
                              unsigned long long *ws) {
  const StepIdx si = step_idx(step);
  // a scene's items end at its last level: the launch steps of its frame
  // stop there, and in the continuous form later steps belong to others
  if (plevel + 1u >= S.levels) return;
  uint32_t rest = wide ? push_wide(P, S, scene, rec, step, plevel, E, cells, ws) : E;
  if (rest == 0) return;
  // a narrow item takes up to 4 parents (32 cells, one per lane) at the leaf
  // level, where many short evaluations make throughput count, and fewer
  // above it, where more items in flight hide the interpreter's latency
  uint32_t per = (plevel + 2u >= S.levels) ? 4u : max(1u, min(4u, S.narrow_parents));
  while (either && per > 1u && !slice_holds(P, per, either)) per >>= 1;
  const uint32_t nitems = (__popc(rest) + per - 1u) / per;
  const uint32_t pos = atomicAdd(&P.item_count[si.next], nitems);
  WorkItem *dst = P.items[si.nbuf];
  for (uint32_t j = 0; j < nitems && pos + j < P.item_cap; ++j) {
    WorkItem wi;
    wi.scene = scene;
    wi.rec = rec;
    wi.level = plevel + 1;
    uint32_t c = 0;
    while (rest && c < per) {
      const uint32_t bit = __ffs(rest) - 1u;
      rest &= rest - 1u;
      wi.parent[c++] = cells[bit];
    }
    wi.n = c;
    for (uint32_t q = c; q < 4u; ++q) wi.parent[q] = wi.parent[0];
    dst[pos + j] = wi;
  }
  if (rest && either) rest = push_wide(P, S, scene, rec, step, plevel, rest, cells, ws);
  if (rest) atomicOr(P.error + scene, EB_QUEUE_FULL);
}

// push_children for the eight children of one wide item (cells base..base+7),
// by one warp: lanes 0-7 take a child each, so the wide list's entries and
// the brick allocations proceed in parallel; the first wide-list slots go
// to the lowest enqueued octants, as in push_children.  `fresh`: the cells'
// brick is new this step (no cell has children yet), so their child fields
// are not read: they are known to be empty.
__device__ __forceinline__ void push_children_warp(const LaunchParams &P, const SceneLaunch &S, uint32_t scene,
                                                   uint32_t rec, uint32_t step, uint32_t plevel, uint32_t E,
                                                   uint32_t base, bool fresh, bool wide, uint32_t either,
                                                   unsigned long long *ws, uint32_t lane) {
  const StepIdx si = step_idx(step);
  if (plevel + 1u >= S.levels) return;  // the scene's last level (push_children)
  uint32_t rest = E;
  if (wide && E) {
    // the enqueued children's bricks are read before the list reservation
    // (the two round trips overlap)
    const bool cand = lane < 8u && ((E >> lane) & 1u);
    const uint32_t b0 = (cand && !fresh) ? S.pool.child[base + lane] : TSI_NONE;
    uint32_t pos = 0;
    if (lane == 0) pos = atomicAdd(&P.witem_count[si.next], (uint32_t)__popc(E));
    pos = __shfl_sync(FULL_MASK, pos, 0);
    const uint32_t avail = pos < P.witem_cap ? P.witem_cap - pos : 0u;
    const uint32_t j = __popc(E & ((1u << lane) - 1u));
    const bool take = cand && j < avail;
    if (take) {
      const uint32_t c = base + lane;
      uint32_t b = b0, fresh = 0;
      if (b == TSI_NONE) {
        b = alloc_brick(S, P.error + scene);
        if (b != TSI_NONE) {
          S.pool.child[c] = b;
          fresh = 1;
          atomicAdd(&ws[ST_BRICK_ALLOC], 1ull);
        }
      }
      WorkItem wi;
      wi.scene = scene;
      wi.rec = rec;
      wi.n = 1;
      wi.level = plevel + 1;
      wi.parent[0] = c;
      wi.parent[1] = b;
      wi.parent[2] = fresh;
      wi.parent[3] = 0;
      P.witems[si.nbuf][pos + j] = wi;
    }
    rest = E & ~__ballot_sync(FULL_MASK, take);
  }
  if (lane == 0 && rest) {
    uint32_t cells[8];
    for (int q = 0; q < 8; ++q) cells[q] = base + q;
    push_children(P, S, scene, rec, step, plevel, rest, cells, false, wide ? 0u : either, ws);
  }
}

__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(FULL_MASK, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(FULL_MASK, v, o));
  return v;
}

// scratch for one item: operand log + decisions, in the warp's slice or the
// shared overflow arena (long tapes)
__device__ __forceinline__ bool item_scratch(const LaunchParams &P, uint32_t step, uint32_t scene, uint32_t len,
                                             uint32_t lane, float4 *slice_log, uint2 *slice_dec, float4 *&lg,
                                             uint2 *&dg) {
  const StepIdx si = step_idx(step);
  if (len <= P.slice_len) {
    lg = slice_log;
    dg = slice_dec;
    return true;
  }
  const unsigned long long need = (unsigned long long)len * 32ull + ((unsigned long long)len + 1ull) / 2ull;
  unsigned long long off = 0;
  if (lane == 0) off = atomicAdd(P.log_overflow_used + si.cur, need);
  off = __shfl_sync(FULL_MASK, off, 0);
  if (off + need > P.log_overflow_cap) {
    if (lane == 0) atomicOr(P.error + scene, EB_LOG_OOM);
    return false;
  }
  lg = P.log_overflow + off;
  dg = reinterpret_cast<uint2 *>(P.log_overflow + off + (unsigned long long)len * 32ull);
  return true;
}

// The sensitivities of an item's cells (to nearest) on a tape whose log is too
// long for 32 columns of the warp's slice: some columns at a time, at least
// one cell and the lanes' shared column, one forward and one reverse pass
// each.  `log_len`: a bound of the tape's log entries.
struct OwnSlice {
  const uint2 *code;
  uint32_t len, nregs, out_reg, log_len, slice_len, cells;
  Iv x, y, z, t;
  float4 *slice;
  bool take;
  Iv sens[4];  // out
};
static __device__ __noinline__ bool own_slice_passes(OwnSlice &a, NarrowRows R, uint32_t lane) {
  const uint32_t cells = a.cells, per = min(cells, min(31u, 32u * a.slice_len / max(a.log_len, 1u) - 1u));
  R.rf -= min(lane, cells) * 8u;
  R.stride = (per + 1u) * 8u;
  R.log_step = per + 1u;
  bool bad = false;
  for (uint32_t first = 0; first < cells; first += per) {
    const uint32_t c = lane - first, col = min(c, per);  // lanes below `first` wrap around
    NarrowRows Q = R;
    Q.rf += col * 8u;
    uint32_t n = 0;
    Iv s[4];
    bool b = false;
    __syncwarp();  // the lanes' columns change
    (void)narrow_forward<false>(a.code, a.len, a.out_reg, Q, lane, a.x, a.y, a.z, a.t, a.slice + col, nullptr, n);
    narrow_reverse<false>(a.code, a.len, a.nregs, a.out_reg, Q, lane, a.slice + col, n, a.take && c < per, true, s, b);
    if (c < per) {
      for (int q = 0; q < 4; ++q) a.sens[q] = s[q];
      bad = b;
    }
  }
  __syncwarp();
  return bad;
}
// Whether an item of n parents can prune this tape within its warp's slices:
// the decisions and the kept instructions of a group per parent.
__device__ __forceinline__ bool slice_prunes(const LaunchParams &P, const TapeRec &TR, uint32_t n) {
  return TR.n_minmax <= P.slice_len && (unsigned long long)n * TR.len <= 64ull * P.slice_len;
}

template <bool D>
__device__ __noinline__ void process_item(const LaunchParams &P, const WorkItem &it, uint32_t step,
                                          uint32_t rcap, float4 *slice_log, uint2 *slice_dec,
                                          unsigned long long *ws) {
  const StepIdx si = step_idx(step);
  using A = IA<D>;
  const uint32_t lane = threadIdx.x & 31u;
  // this warp's register file and chunk buffer
  const NarrowRows R = narrow_rows(tsi_dyn_smem + (threadIdx.x >> 5) * (rcap * 256u + kNarrowChunkBytes), rcap, lane,
                                   it.n);
  const uint32_t g = lane >> 3, k = lane & 7u;
  const SceneLaunch &S = P.scenes[it.scene];
  const VoxelPoolDev &pool = S.pool;
  const uint32_t flags = S.flags;
  const bool swept = (flags & SF_SWEPT) != 0;

  bool active = g < it.n;
  const uint32_t Pv = it.parent[active ? g : 0];
  const float4 pxy = pool.box_xy[Pv];
  const float2 pz = pool.box_z[Pv];
  const uint32_t pchild = pool.child[Pv];
  const float pfast = pool.fast[Pv];
  const bool new_voxel = (pchild == TSI_NONE);

  // ---- allocate or reuse the 8 children (3564-3580)
  uint32_t base = pchild;
  if (active && new_voxel && k == 0) {
    base = alloc_brick(S, P.error + it.scene);
    if (base != TSI_NONE) atomicAdd(&ws[ST_BRICK_ALLOC], 1ull);
  }
  base = __shfl_sync(FULL_MASK, base, lane & ~7u);
  if (base == TSI_NONE) active = false;
  const uint32_t C = active ? base + k : 0u;
  float c_t = 0.0f, c_f = 1.0f, c_te = 0.0f, c_fast = 0.0f;
  uint32_t c_child = TSI_NONE;
  if (active) {
    if (new_voxel) {
      pool.child[C] = TSI_NONE;
      pool.normal[C] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (k == 0) pool.child[Pv] = base;
    } else {
      c_t = pool.t[C];
      c_f = pool.f[C];
      c_te = pool.time_err[C];
      c_fast = pool.fast[C];
      c_child = pool.child[C];
    }
  }

  // ---- cell setup (3582-3626)
  const float dx = __fdiv_rn(__fsub_rn(pxy.y, pxy.x), 2.0f);
  const float dy = __fdiv_rn(__fsub_rn(pxy.w, pxy.z), 2.0f);
  const float dz = __fdiv_rn(__fsub_rn(pz.y, pz.x), 2.0f);
  float width = fm_max(dx, fm_max(dy, dz));
  const float kx = (float)(k & 1u), ky = (float)((k >> 1) & 1u), kz = (float)(k >> 2);
  Iv cx = Iv{__fadd_rn(pxy.x, __fmul_rn(dx, kx)), __fadd_rn(pxy.x, __fmul_rn(dx, 1.0f + kx))};
  Iv cy = Iv{__fadd_rn(pxy.z, __fmul_rn(dy, ky)), __fadd_rn(pxy.z, __fmul_rn(dy, 1.0f + ky))};
  Iv cz = Iv{__fadd_rn(pz.x, __fmul_rn(dz, kz)), __fadd_rn(pz.x, __fmul_rn(dz, 1.0f + kz))};
  // half extent of this cell's children, as they will compute it
  const float child_width =
      fm_max(__fdiv_rn(__fsub_rn(cx.hi, cx.lo), 2.0f),
             fm_max(__fdiv_rn(__fsub_rn(cy.hi, cy.lo), 2.0f), __fdiv_rn(__fsub_rn(cz.hi, cz.lo), 2.0f)));
  const bool point_branch = new_voxel || pfast == 1.0f || width <= S.eps;
  Iv cur_t;
  if (point_branch) {
    cur_t = swept ? Iv{S.t0, S.time} : iv(S.time);
    c_fast = 0.0f;
  } else {
    cur_t = Iv{c_t, S.time};
  }
  if (active) {
    pool.box_xy[C] = make_float4(cx.lo, cx.hi, cy.lo, cy.hi);
    pool.box_z[C] = make_float2(cz.lo, cz.hi);
    pool.t[C] = S.time;
  }
  if ((flags & SF_POINTSAMPLE) && width <= S.eps) {
    cx = iv(__fdiv_rn(__fadd_rn(cx.lo, cx.hi), 2.0f));
    cy = iv(__fdiv_rn(__fadd_rn(cy.lo, cy.hi), 2.0f));
    cz = iv(__fdiv_rn(__fadd_rn(cz.lo, cz.hi), 2.0f));
    width = 0.0f;
  }
  const Iv targ = Iv{fm_min(cur_t.lo, cur_t.hi), fm_max(cur_t.lo, cur_t.hi)};
  const bool evaluate = active && (new_voxel || c_f >= 0.0f || c_child == TSI_NONE);
  const bool take_deriv = evaluate && ((cur_t.lo != cur_t.hi) || (flags & SF_ALWAYS_DERIV));

  Iv field = iv(0.0f);
  Iv sens[4] = {iv(0.0f), iv(0.0f), iv(0.0f), iv(0.0f)};
  uint32_t rec = it.rec;
  TapeRec TR;
  const uint32_t b_eval = __ballot_sync(FULL_MASK, evaluate);
  const uint32_t b_rev = __ballot_sync(FULL_MASK, take_deriv);
  const bool any_deriv = b_rev != 0;
  bool want_prune = false;
  float4 *lg = nullptr;
  uint2 *dg = nullptr;
  // whether a full level turned the item away from the wide path (or it found
  // the wide list full): it then leaves the log arena alone
  auto leaves_arena = [&]() { return !D && may_go_narrow(P, S.wide, it.level, P.recs[it.rec].len); };

  if (b_eval) {
    // ---- the most pruned tape valid for every evaluated cell
    const float tl = warp_min(evaluate ? targ.lo : fm_inf());
    const float th = warp_max(evaluate ? targ.hi : -fm_inf());
    TR = P.recs[rec];
    if (!(TR.c_level == it.level && TR.c_lo <= tl && th <= TR.c_hi)) find_valid(P, rec, TR, tl, th);
    for (int attempt = 0; attempt < 2; ++attempt) {
      const bool own_slice = leaves_arena(), in_turns = own_slice && !slice_holds(P, it.n, log_bound(S.wide, TR.len));
      want_prune = (flags & SF_PRUNING) && TR.len >= TSI_PRUNE_MIN_LEN && TR.nregs <= TSI_PRUNE_MAX_REGS &&
                   (!own_slice || slice_prunes(P, TR, it.n));
      if (lane == 0 && attempt == 0) {
        if (TR.len >= S.wide.min_len) ws[ST_NARROW_LONG] += 1;
        ws[ST_NARROW_LEN_MAX] = max(ws[ST_NARROW_LEN_MAX], (unsigned long long)TR.len);
      }
      lg = nullptr;
      dg = nullptr;
      if (any_deriv || want_prune) {
        float4 *lgs = slice_log;
        uint2 *dgs = want_prune ? slice_dec : nullptr;
        if (!own_slice && !item_scratch(P, step, it.scene, TR.len, lane, slice_log, slice_dec, lgs, dgs)) return;
        lg = lgs;
        dg = dgs;
      }
      const long long q0 = clock64();
      uint32_t nlog = 0;
      bool bad = false;
      float4 *opl = any_deriv ? lg + min(lane, narrow_cells(it.n)) : nullptr;  // this lane's column of the log
      field = narrow_forward<D>(TR.code, TR.len, TR.out_reg, R, lane, cx, cy, cz, targ, in_turns ? nullptr : opl, dg, nlog);
      const long long q1 = clock64();
      if (any_deriv && in_turns) {
        OwnSlice o{TR.code, TR.len, TR.nregs, TR.out_reg, log_bound(S.wide, TR.len), P.slice_len, narrow_cells(it.n),
                   cx, cy, cz, targ, lg, take_deriv, {sens[0], sens[1], sens[2], sens[3]}};
        bad = own_slice_passes(o, R, lane);
        for (int q = 0; q < 4; ++q) sens[q] = o.sens[q];
      } else if (any_deriv)
        narrow_reverse<D>(TR.code, TR.len, TR.nregs, TR.out_reg, R, lane, opl, nlog, take_deriv, (flags & SF_STRICT) != 0, sens,
                          bad);
      if (lane == 0 && attempt == 0) {
        ws[ST_CYC_N_FWD] += (unsigned long long)(q1 - q0);
        ws[ST_N_FWD_INSTR] += TR.len;
        ws[ST_CYC_N_REV] += (unsigned long long)(clock64() - q1);
      }
      // a pruned tape whose sensitivities overflowed: redo on the full tape
      const bool redo = __any_sync(FULL_MASK, bad) && TR.parent != TSI_NONE;
      if (!redo) break;
      rec = S.root_rec;
      TR = P.recs[rec];
      if (lane == 0) ws[ST_PRUNE_FALLBACK]++;
    }
    if (lane == 0) {
      const uint32_t ne = __popc(b_eval), nr = __popc(b_rev);
      ws[ST_INSTR_FWD] += (unsigned long long)TR.len * ne;
      ws[ST_INSTR_REV] += (unsigned long long)TR.len * nr;
      ws[ST_INSTR_FULL] += (unsigned long long)S.full_len * ne;
      ws[ST_FP32] += (unsigned long long)TR.fwd_cost * ne + (unsigned long long)TR.rev_cost * nr;
    }
  }

  // ---- temporal error bound (3966-3997)
  Iv df = iv(0.0f), df_dt = iv(0.0f);
  const float delta = S.delta;
  if (take_deriv) {
    const float nx = __fdiv_rn(__fadd_rn(sens[0].lo, sens[0].hi), 2.0f);
    const float ny = __fdiv_rn(__fadd_rn(sens[1].lo, sens[1].hi), 2.0f);
    const float nz = __fdiv_rn(__fadd_rn(sens[2].lo, sens[2].hi), 2.0f);
    pool.normal[C] = make_float4(nx, ny, nz, 0.0f);
    df_dt = sens[3];
    const float dt = __fsub_rn(targ.hi, targ.lo);
    df = A::mul_f(df_dt, dt);
    const Iv W = A::mul_f(Iv{-1.0f, 1.0f}, __fsub_rn(field.hi, field.lo));
    df = A::cap(df, W);
    if ((flags & SF_LIPSCHITZ) && A::abs_(df).hi != 0.0f) {
      const float lb =
          A::abs_(A::sqrt_(A::add(A::sqr(sens[0]), A::add(A::sqr(sens[1]), A::sqr(sens[2]))))).lo;
      if (!is_nan_f(lb)) df = A::div(df, iv(lb));
    }
    if (df.lo == -fm_inf() || df.hi == fm_inf() || is_nan_f(df.lo) || is_nan_f(df.hi)) df = iv(delta);
    c_te = __fadd_rn(c_te, fm_min(fm_max(A::abs_(df).hi, 0.0f), delta));
  }
  // ---- fast flag (4003-4009)
  if (evaluate && !swept && (flags & SF_FASTENABLED)) c_fast = (A::abs_(df).hi >= S.fast_thresh) ? 1.0f : 0.0f;

  // ---- classification (4011-4045)
  bool enq = false, dealloc = false, reused = false;
  int cls = 3;
  uint32_t dealloc_brick = 0;
  if (evaluate) {
    if (field.lo <= 0.0f && 0.0f <= field.hi) {
      c_f = 0.0f;
      cls = 0;
      if (width > S.eps) {
        if (new_voxel || is_nan_f(df_dt.lo) || is_nan_f(df_dt.hi) || fabsf(df_dt.lo) == fm_inf() ||
            fabsf(df_dt.hi) == fm_inf() || pfast == 1.0f || cur_t.lo == cur_t.hi || c_te >= delta ||
            c_child == TSI_NONE) {
          c_te = 0.0f;
          enq = true;
        } else {
          reused = true;
        }
      }
    } else {
      if (field.hi <= 0.0f) {
        c_f = -1.0f;
        cls = 2;
      } else {
        cls = 1;
        if (!swept) c_f = 1.0f;
      }
      if (!swept && c_child != TSI_NONE) {
        dealloc = true;
        dealloc_brick = c_child >> 3;
      }
    }
  }
  const uint32_t old_child = c_child;
  if (dealloc) c_child = TSI_NONE;
  if (active) {
    pool.f[C] = c_f;
    pool.time_err[C] = c_te;
    pool.fast[C] = c_fast;
    if (dealloc || new_voxel) pool.child[C] = c_child;
  }

  // ---- deallocation of dropped subtrees (4036-4044)
  {
    const uint32_t m = __ballot_sync(FULL_MASK, dealloc);
    if (m) {
      uint32_t basei = 0;
      if (lane == 0) basei = atomicAdd(&P.dealloc_count[si.next], (uint32_t)__popc(m));
      basei = __shfl_sync(FULL_MASK, basei, 0);
      if (dealloc) {
        const uint32_t pos = basei + __popc(m & ((1u << lane) - 1u));
        if (pos < P.dealloc_cap) P.dealloc[si.nbuf][pos] = make_uint2(it.scene, dealloc_brick);
        else atomicOr(P.error + it.scene, EB_QUEUE_FULL);
      }
    }
  }

  // ---- re-enqueue: one sibling group per parent, pruned tape per group
  const uint32_t em = __ballot_sync(FULL_MASK, enq);
  const uint32_t E = (em >> (g * 8u)) & 0xffu;
  uint32_t new_rec = rec;
  if (em) {
    // time range the children will be evaluated over: [child.t, time], or
    // the point branch's range for children at most eps wide or of a fast
    // cell
    const bool child_point = child_width <= S.eps || c_fast == 1.0f;
    float nl = targ.lo, nh = targ.hi;
    if (enq && old_child != TSI_NONE && !child_point) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float ct = pool.t[old_child + q];
        nl = fm_min(nl, fm_min(ct, S.time));
        nh = fm_max(nh, fm_max(ct, S.time));
      }
    }
    if (enq && swept) {  // swept children start their point-branch interval at t0
      nl = fm_min(nl, fm_min(S.t0, S.time));
      nh = fm_max(nh, fm_max(S.t0, S.time));
    }
    if (!enq) {
      nl = fm_inf();
      nh = -fm_inf();
    }
    const bool widen = enq && (nl < targ.lo || nh > targ.hi);
    const uint32_t wb = __ballot_sync(FULL_MASK, widen);
    uint32_t prec = rec;  // record the group tapes are pruned from
    TapeRec PR = TR;
    bool handed = false;  // the group's children go to the wide path unpruned
    if (want_prune && wb) {
      // decisions over the widened interval, from a tape valid there
      const float wl = warp_min(nl), wh = warp_max(nh);
      uint32_t wrec = rec;
      TapeRec WR;
      find_valid(P, wrec, WR, wl, wh);
      const bool long_tape = warp_goes_wide(P, S.wide, step, it.level + 1u, WR.len), own_slice = leaves_arena();
      if (long_tape) {
        // A long tape: no pass over it on one warp.  A group with a widened
        // child hands its children, with that tape's record, to the wide
        // path; the other groups prune from the first pass's decisions.
        if ((wb >> (g * 8u)) & 0xffu) {
          prec = wrec;
          PR = WR;
          handed = true;
        }
      } else {
        prec = wrec;
        PR = WR;
        want_prune = (flags & SF_PRUNING) && PR.len >= TSI_PRUNE_MIN_LEN && PR.nregs <= TSI_PRUNE_MAX_REGS &&
                     (!own_slice || slice_prunes(P, PR, it.n));
      }
      if (want_prune && !long_tape) {
        float4 *lgs = slice_log;
        uint2 *dgs = slice_dec;
        if (!own_slice && !item_scratch(P, step, it.scene, PR.len, lane, slice_log, slice_dec, lgs, dgs)) return;
        lg = lgs;
        dg = dgs;
        const Iv tw = enq ? Iv{nl, nh} : targ;
        uint32_t nlog = 0;
        (void)narrow_forward<D>(PR.code, PR.len, PR.out_reg, R, lane, cx, cy, cz, tw, nullptr, dg, nlog);
        if (lane == 0) ws[ST_FP32] += (unsigned long long)PR.fwd_cost * __popc(em);
      }
    }
    // validity of the group's pruned tape: intersection of the enqueued
    // siblings' decision intervals (any cell), and their hull (the group's
    // own children, each covered by its parent's decisions)
    float gl = enq ? nl : -fm_inf();
    float gh = enq ? nh : fm_inf();
    float hl = enq ? nl : fm_inf();
    float hh = enq ? nh : -fm_inf();
    for (int o = 1; o < 8; o <<= 1) {
      gl = fmaxf(gl, __shfl_xor_sync(FULL_MASK, gl, o));
      gh = fminf(gh, __shfl_xor_sync(FULL_MASK, gh, o));
      hl = fminf(hl, __shfl_xor_sync(FULL_MASK, hl, o));
      hh = fmaxf(hh, __shfl_xor_sync(FULL_MASK, hh, o));
    }
    uint32_t cnt = 0, mmk = 0, fcost = 0, rcost = 0;
    bool pruned = false;
    uint2 *tmp =
        (want_prune && !handed && lg != nullptr) ? reinterpret_cast<uint2 *>(lg) + (size_t)g * PR.len : nullptr;
    const uint32_t actm = __ballot_sync(FULL_MASK, k == 0 && E != 0 && tmp != nullptr);
    if (actm) {
      const long long q0 = clock64();
      __syncwarp();  // the ballots (lane 0) and the log's last readers
      // every pruning group scans the same tape, one group after another by
      // the whole warp (a group handed to the wide path holds another record)
      for (uint32_t rest = actm; rest; rest &= rest - 1u) {
        const int src = __ffs(rest) - 1;
        const uint2 *pcode = reinterpret_cast<const uint2 *>(
            __shfl_sync(FULL_MASK, reinterpret_cast<unsigned long long>(PR.code), src));
        const uint32_t plen = __shfl_sync(FULL_MASK, PR.len, src);
        const uint32_t pmm = __shfl_sync(FULL_MASK, PR.n_minmax, src);
        const uint32_t pout = __shfl_sync(FULL_MASK, PR.out_reg, src);
        const uint32_t pE = __shfl_sync(FULL_MASK, E, src);
        uint2 *ptmp = reinterpret_cast<uint2 *>(__shfl_sync(FULL_MASK, reinterpret_cast<unsigned long long>(tmp), src));
        uint32_t mk, fc, rc;
        const uint32_t n = prune_group<D>(pcode, plen, pmm, pout, dg, (uint32_t)src >> 3, pE, ptmp, R, lane, mk, fc, rc);
        if ((int)lane == src) {
          cnt = n;
          mmk = mk;
          fcost = fc;
          rcost = rc;
          pruned = n < PR.len;
        }
      }
      if (lane == 0) ws[ST_CYC_N_PRUNE] += (unsigned long long)(clock64() - q0);
    }
    // reserve arena space and a record (lane 8g), then copy with the group
    unsigned long long off = 0;
    uint32_t ri = TSI_NONE;
    if (k == 0 && pruned) {
      off = code_alloc(P, cnt);
      if (off != ~0ull) ri = rec_alloc(P);
    }
    const uint32_t gl0 = lane & ~7u;
    cnt = __shfl_sync(FULL_MASK, cnt, gl0);
    off = __shfl_sync(FULL_MASK, off, gl0);
    ri = __shfl_sync(FULL_MASK, ri, gl0);
    {  // the pruned tapes in program order, one group after another by the whole warp
      uint32_t cm = __ballot_sync(FULL_MASK, k == 0 && ri != TSI_NONE);
      for (; cm; cm &= cm - 1u) {
        const int src = __ffs(cm) - 1;
        const uint32_t n = __shfl_sync(FULL_MASK, cnt, src);
        uint2 *dst = P.code_arena + __shfl_sync(FULL_MASK, off, src);
        const uint2 *ptmp = reinterpret_cast<const uint2 *>(
            __shfl_sync(FULL_MASK, reinterpret_cast<unsigned long long>(tmp), src));
        for (uint32_t j = lane; j < n; j += 32u) dst[j] = ptmp[n - 1u - j];
      }
    }
    if (ri != TSI_NONE) {
      if (k == 0) {
        TapeRec nr;
        nr.code = P.code_arena + off;
        nr.len = cnt;
        nr.nregs = PR.nregs;
        nr.out_reg = PR.out_reg;
        nr.n_minmax = mmk;
        nr.t_lo = gl;
        nr.t_hi = gh;
        nr.parent = prec;
        nr.fwd_cost = fcost;
        nr.rev_cost = rcost;
        nr.c_lo = hl;
        nr.c_hi = hh;
        nr.c_level = it.level + 1u;
        P.recs[ri] = nr;
        atomicAdd(&ws[ST_TAPE_WORDS], (unsigned long long)cnt);
      }
      new_rec = ri;
    } else if (E != 0 && want_prune) {
      new_rec = prec;  // not pruned (or no arena room): the widened-valid tape
    }
    // next-level work: wide items for a long tape, else narrow items
    uint32_t cb[8];
#pragma unroll
    for (int b2 = 0; b2 < 8; ++b2) cb[b2] = __shfl_sync(FULL_MASK, C, gl0 + b2);
    const uint32_t next_len = (new_rec == prec) ? PR.len : ((new_rec == rec) ? TR.len : cnt);
    if (k == 0 && E != 0) {
      if (next_len >= wide_min_len(S.wide, it.level + 1u)) atomicAdd(&P.long_count[si.next], (uint32_t)__popc(E));
      const bool wide = goes_wide(P, S.wide, step, it.level + 1u, next_len);
      const bool either = !wide && may_go_narrow(P, S.wide, it.level + 1u, next_len);
      push_children(P, S, it.scene, new_rec, step, it.level, E, cb, wide, either ? log_bound(S.wide, next_len) : 0u, ws);
    }
  }

  // ---- counters
  const uint32_t b_skip = __ballot_sync(FULL_MASK, active && !evaluate);
  const uint32_t b_amb = __ballot_sync(FULL_MASK, cls == 0);
  const uint32_t b_emp = __ballot_sync(FULL_MASK, cls == 1);
  const uint32_t b_full = __ballot_sync(FULL_MASK, cls == 2);
  const uint32_t b_reu = __ballot_sync(FULL_MASK, reused);
  if (lane == 0) {
    ws[ST_PARENTS] += it.n;
    ws[ST_EVAL] += __popc(b_eval);
    ws[ST_REVERSE] += __popc(b_rev);
    ws[ST_SKIPPED] += __popc(b_skip);
    ws[ST_AMBIG] += __popc(b_amb);
    ws[ST_EMPTY] += __popc(b_emp);
    ws[ST_FULL] += __popc(b_full);
    ws[ST_ENQUEUED] += __popc(em);
    ws[ST_REUSED] += __popc(b_reu);
  }
}

// Recursive free of a dropped subtree (compute.wgsl:3533-3543, freeV
// 3452-3460): 8 lanes per brick; children bricks go to the next level's list.
__device__ void dealloc_brick(const LaunchParams &P, uint2 item, uint32_t step, bool valid) {
  const StepIdx si = step_idx(step);
  const uint32_t lane = threadIdx.x & 31u, k = lane & 7u;
  const SceneLaunch &S = P.scenes[valid ? item.x : 0];
  const VoxelPoolDev &pool = S.pool;
  const uint32_t v = item.y * 8u + k;
  uint32_t ch = TSI_NONE;
  if (valid) {
    ch = pool.child[v];
    pool.child[v] = TSI_NONE;
    pool.f[v] = 0.0f;
    pool.t[v] = 0.0f;
    pool.time_err[v] = 0.0f;
    pool.fast[v] = 0.0f;
  }
  const bool push = valid && ch != TSI_NONE;
  const uint32_t m = __ballot_sync(FULL_MASK, push);
  if (m) {
    uint32_t basei = 0;
    if (lane == 0) basei = atomicAdd(&P.dealloc_count[si.next], (uint32_t)__popc(m));
    basei = __shfl_sync(FULL_MASK, basei, 0);
    if (push) {
      const uint32_t pos = basei + __popc(m & ((1u << lane) - 1u));
      if (pos < P.dealloc_cap) P.dealloc[si.nbuf][pos] = make_uint2(item.x, ch >> 3);
      else atomicOr(P.error + item.x, EB_QUEUE_FULL);
    }
  }
  if (valid && k == 0) {
    const uint32_t pos = atomicAdd(&S.ctr->pending_count, 1u);
    if (pos < pool.cap_bricks) pool.pending[pos] = item.y;
    atomicAdd(&P.stats[(size_t)item.x * ST_COUNT + ST_BRICK_FREE], 1ull);  // the brick's own scene
    if (P.level_stats) atomicAdd(&P.level_stats[(size_t)si.cur * ST_COUNT + ST_BRICK_FREE], 1ull);
  }
}

// ======================================================================
// Wide path: one block per child cell of a wide item, one thread per
// instruction of a bundle (tape_compile.h WideTape).  Long tapes at the top
// of the octree leave the narrow path latency bound (few items, thousands of
// dependent instructions each); here a cell takes one block-wide step per
// bundle.  Every SSA value has its own slot in the cell's working set, so
// the reverse pass reads operands where the forward pass left them; values
// with several users sum per-use contribution records in the sequential
// order, so the results are those of the narrow path bit for bit.  The eight
// cells of an item run on eight blocks; the last to finish prunes the
// group's tape and enqueues its children.

// Byte offsets of a cell's working set (values; sensitivities and, behind
// them, the contribution records; a decision byte per min/max; liveness
// flags) and its size; the host sizes it the same way.
struct CellLayout {
  uint32_t sens, dec, flags, size;
};
__device__ __forceinline__ CellLayout cell_layout(const WideDev &W, uint32_t bm_words) {
  CellLayout L;
  const uint32_t nv = W.nvalues + 2u;
  L.sens = nv * 8u;
  L.dec = (L.sens + (W.global ? nv + W.ncontrib : max(nv, W.gslots)) * 8u + 15u) & ~15u;
  L.flags = L.dec + (bm_words + 1u) * 16u;  // one more for the padding lanes
  L.size = L.flags + ((nv + 15u) & ~15u);
  return L;
}
// Sixteen decision bytes as a word of two bits each (bytes past the tape's
// last min/max hold anything).
__device__ __forceinline__ uint32_t pack_decisions(const uint8_t *dec, uint32_t w) {
  const uint4 b = *reinterpret_cast<const uint4 *>(dec + 16u * w);
  auto four = [](uint32_t x) {
    x &= 0x03030303u;
    return (x | (x >> 6) | (x >> 12) | (x >> 18)) & 255u;
  };
  return four(b.x) | (four(b.y) << 8) | (four(b.z) << 16) | (four(b.w) << 24);
}

// Base of the block's cell working set: dynamic shared memory, or for tapes
// too large for it the block's slice of the global scratch (each block of
// the persistent grid owns one slice; L2 keeps the active slices).
template <bool GM>
__device__ __forceinline__ unsigned char *cell_base(const LaunchParams &P) {
  if constexpr (GM) return P.wscratch + (size_t)blockIdx.x * P.wscratch_stride;
  else return tsi_dyn_smem;
}

// (The kernel's static shared memory is what the largest register files
// leave: eight of 108 registers with their buffers take 227328 of the 232448
// bytes a block may have.)
struct WideShared {
  uint32_t last, E, cnt, mmk, fcost, rcost, ri;
  unsigned long long off;
  float gl, gh, hl, hh;
  uint32_t scan[kWarps];
  float2 sens[4];
  uint2 cost[H_COUNT];  // (finish_group) a handler's forward and reverse cost
};

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *scratch, uint32_t &total) {
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL_MASK, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) scratch[wib] = x;
  __syncthreads();
  uint32_t base = 0, tot = 0;
  for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) {
    if (w < wib) base += scratch[w];
    tot += scratch[w];
  }
  __syncthreads();
  total = tot;
  return base + x - v;
}



// The last cell of a wide item to finish: prunes the full tape with the
// branch decisions shared by all enqueued siblings and enqueues them.  One
// block runs it while the launch's end waits for it, bound by latency: loads
// under a test waited for one after another, a branch per operand, a barrier
// per compaction step and constant tables read at 32 indices made it 34k
// cycles on a 4697-instruction tape and 59k on a 3240-instruction one; as
// written 24k and 35k.
template <bool GM>
__device__ __forceinline__ void finish_group(const LaunchParams &P, const WorkItem &it, uint32_t step,
                                             uint32_t unit0, WideShared &sh, unsigned long long *ws) {
  const StepIdx si = step_idx(step);
  unsigned char *cell = cell_base<GM>(P);
  const uint32_t tid = threadIdx.x;
  const SceneLaunch &S = P.scenes[it.scene];
  const WideDev &W = S.wide;
  const TapeRec root = P.recs[S.root_rec];
  const uint32_t n_narrow = root.len;
  const CellInfo *info = P.cell_info[si.buf] + unit0;
  const long long f0 = clock64();
  // groups above the tape's prune level skip the liveness pass: their
  // children go to the wide path, which evaluates the full tape anyway
  const bool want_prune = (S.flags & SF_PRUNING) && root.nregs <= TSI_PRUNE_MAX_REGS && it.level >= W.prune_level;
  if (tid == 0) {
    ws[ST_PARENTS] += 1;
    ws[ST_WIDE_FIN] += 1;
    // sh.E: the enqueued siblings, from the count-in
    float gl = -fm_inf(), gh = fm_inf(), hl = fm_inf(), hh = -fm_inf();
    if (want_prune) {
      CellInfo ci[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) ci[q] = info[q];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        gl = fmaxf(gl, ci[q].nl);
        gh = fminf(gh, ci[q].nh);
        if (ci[q].enq) {
          hl = fminf(hl, ci[q].nl);
          hh = fmaxf(hh, ci[q].nh);
        }
      }
    }
    sh.gl = gl;
    sh.gh = gh;
    sh.hl = hl;
    sh.hh = hh;
  }
  __syncthreads();
  const uint32_t E = sh.E;
  if (E == 0) return;
  uint32_t new_rec = S.root_rec;
  if (want_prune) {
    const CellLayout L = cell_layout(W, P.bm_words);
    const uint32_t words = (root.n_minmax + 15u) >> 4;
    uint32_t *cb = reinterpret_cast<uint32_t *>(cell + L.dec);  // decisions shared by the enqueued cells
    uint8_t *flags = cell + L.flags;
    if constexpr (GM) {
      // the liveness flags and the decisions of a cell in the global scratch
      // go to shared memory all the same when they fit: the pass below is a
      // chain of them (1024-primitive tape: 65k -> 25k cycles)
      const uint32_t fb = (W.nvalues + 2u + 15u) & ~15u;
      if (fb + (words + 1u) * 4u <= P.dyn_smem) {
        flags = tsi_dyn_smem;
        cb = reinterpret_cast<uint32_t *>(tsi_dyn_smem + fb);
      }
    }
    const uint32_t *gbits = P.cell_bits[si.buf] + (size_t)unit0 * P.bm_words;
    for (uint32_t w = tid; w < words; w += blockDim.x) {
      uint32_t v[8], acc = 0xffffffffu;
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = gbits[(size_t)q * P.bm_words + w];  // (all at once; some unused)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc &= v[q] | (((E >> q) & 1u) ? 0u : 0xffffffffu);
      cb[w] = acc;
    }
    if (tid == 0) cb[words] = 0;  // (of a value that is no min/max)
    if (tid < H_COUNT)
      sh.cost[tid] = make_uint2(c_cost_fwd[tid] + TSI_FIX_COST, c_cost_rr[tid] + TSI_REV_OPERAND_COST * TSI_H_NREG(tid));
    for (uint32_t i = tid; i < W.nvalues + 2u; i += blockDim.x) flags[i] = 0;
    // the values are done with: their place holds the bundle descriptors (a
    // bundle has at least one value, of the same eight bytes)
    uint2 *bt = reinterpret_cast<uint2 *>(cell);
    for (uint32_t i = tid; i < W.nbundles; i += blockDim.x) bt[i] = W.bundles[i];
    __syncthreads();
    // Liveness from the field backwards, bundle by bundle; a step is bound by
    // the latency of its slots, which are on their way four bundles ahead.
    // Threads past a bundle's end repeat its last slot, and the steps past
    // the first bundle repeat that: setting a flag twice changes nothing, and
    // a load under a test or select would be waited for at once.
    {
      const uint4 *__restrict__ slots = W.live;
      const bool same = !(S.flags & SF_DIRECTED);  // (prune_group's rule)
      auto fetch = [&](int kk) -> uint4 {
        const uint2 b = bt[max(kk, 0)];
        return slots[b.x + min(tid, b.y - 1u)];
      };
      if (tid == 0) flags[W.nvalues - 1u] = 1;
      uint4 q[4];
      const int kb0 = (int)W.nbundles - 1;
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = fetch(kb0 - i);
      __syncthreads();
#pragma unroll 1
      for (int kb = kb0; kb >= 0; kb -= 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 s1 = q[i];
          q[i] = fetch(kb - i - 4);
          // a min/max has an ordinal: the decision may rule an operand out
          const bool mm = s1.y != TSI_NONE, live = flags[s1.x] != 0;
          const uint32_t ord = s1.y & ~(WL_SAME_A | WL_SAME_B);
          const uint32_t d = (cb[mm ? ord >> 4 : words] >> (2u * (ord & 15u))) & 3u;
          if (live && s1.z != TSI_NONE && d != 2u) flags[s1.z] = 1;
          if (live && s1.w != TSI_NONE && !(d & 1u)) flags[s1.w] = 1;
          // a copy of a register to itself is not kept (nothing reads this
          // flag again but a thread that repeats the slot)
          if (same && live && mm && ((d & 1u) ? s1.y & WL_SAME_A : d != 0u ? s1.y & WL_SAME_B : 0u)) flags[s1.x] = 0;
          __syncthreads();
        }
      }
    }
    const long long f1 = clock64();
    if (tid == 0) ws[ST_CYC_FIN_LIVE] += (unsigned long long)(f1 - f0);
    // Compaction of the narrow full tape in program order, a warp's 32
    // consecutive instructions at a time: the groups' live counts, their
    // prefix sums, and then every group by itself, without a barrier and with
    // its instructions read four groups ahead.
    const uint32_t lane = tid & 31u, wib = tid >> 5, nw = blockDim.x >> 5;
    const uint32_t groups = (n_narrow + 31u) >> 5;
    uint32_t *first = reinterpret_cast<uint32_t *>(cell);  // (the descriptors are done with)
    for (uint32_t g = wib; g < groups; g += nw) {
      const uint32_t i = g * 32u + lane;
      const uint32_t bal = __ballot_sync(FULL_MASK, i < n_narrow && flags[i + 4u]);
      if (lane == 0) first[g] = __popc(bal);
    }
    __syncthreads();
    uint32_t total = 0;
    for (uint32_t g0 = 0; g0 < groups; g0 += blockDim.x) {
      const uint32_t g = g0 + tid;
      uint32_t sum = 0;
      const uint32_t ex = block_exclusive_scan(g < groups ? first[g] : 0u, sh.scan, sum);
      if (g < groups) first[g] = total + ex;
      total += sum;
    }
    if (tid == 0) {
      sh.ri = TSI_NONE;
      sh.off = 0;
      sh.cnt = total;
      sh.mmk = 0;
      sh.fcost = 0;
      sh.rcost = 0;
      // a pruned record only for children that go to the narrow path (the
      // wide path evaluates the full tape), or may: children the full wide
      // list turns away run narrow on this record
      const bool wide_room = *(const volatile uint32_t *)&P.witem_count[si.next] + 8u <= P.witem_cap;
      if (total < n_narrow && (!goes_wide(P, W, step, it.level + 1u, total) || !wide_room)) {
        const unsigned long long off = code_alloc(P, total);
        if (off != ~0ull) {
          const uint32_t ri = rec_alloc(P);
          if (ri != TSI_NONE) {
            sh.ri = ri;
            sh.off = off;
          }
        }
      }
    }
    __syncthreads();
    if (sh.ri != TSI_NONE) {
      const unsigned long long off = sh.off;
      uint32_t mmk = 0, fc = 0, rc = 0;
      // a group's instructions (past the tape's end: its last)
      auto fetch = [&](uint32_t g, uint2 &w, uint32_t &mm) {
        const uint32_t i = min(g * 32u + lane, n_narrow - 1u);
        w = root.code[i];
        mm = W.narrow_mm[i];
      };
      uint2 wq[4];
      uint32_t mq[4];
#pragma unroll
      for (uint32_t u = 0; u < 4u; ++u) fetch(wib + u * nw, wq[u], mq[u]);
#pragma unroll 1
      for (uint32_t g0 = wib; g0 < groups; g0 += 4u * nw) {
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
          const uint32_t g = g0 + u * nw;
          const uint2 w = wq[u];
          const uint32_t mm = mq[u];
          fetch(g + 4u * nw, wq[u], mq[u]);
          const uint32_t i = g * 32u + lane;
          const bool live = i < n_narrow && flags[i + 4u];
          const uint32_t bal = __ballot_sync(FULL_MASK, live);
          if (live) {
            const uint32_t p = first[g] + __popc(bal & ((1u << lane) - 1u));
            const uint32_t h = TSI_W0_H(w.x);
            uint2 out = w;
            uint32_t hk = h;
            if (TSI_H_IS_MINMAX(h)) {
              const uint32_t d = (cb[mm >> 4] >> (2u * (mm & 15u))) & 3u;
              const uint32_t dd = TSI_W0_DST(w.x);
              const uint32_t deps_a = TSI_W0_WITH_DEPS(TSI_W0_DEPS(w.x));
              const uint32_t deps_b = TSI_H_IS_II(h) ? TSI_W0_WITH_DEPS(TSI_W1_DEPS(w.y)) : 0u;
              if (d & 1u) {
                out = make_uint2(copy_word(w.x, true, dd, TSI_W0_A(w.x)) | deps_b, 0u);
                hk = H_COPY;
              } else if (d & 2u) {
                if (TSI_H_IS_II(h)) {
                  out = make_uint2(copy_word(w.x, false, dd, w.y & 255u) | deps_a, 0u);
                  hk = H_COPY;
                } else {
                  out = make_uint2(TSI_W0(H_CONST, 0u, 0u, dd, 0u) | deps_a, w.y);
                  hk = H_CONST;
                }
              } else {
                ++mmk;
              }
            }
            const uint2 cost = sh.cost[hk];
            fc += cost.x;
            rc += cost.y;
            P.code_arena[off + p] = out;
          }
        }
      }
      atomicAdd(&sh.mmk, mmk);
      atomicAdd(&sh.fcost, fc);
      atomicAdd(&sh.rcost, rc);
    }
    __syncthreads();
    if (sh.ri != TSI_NONE) {
      if (tid == 0) {
        TapeRec nr;
        nr.code = P.code_arena + sh.off;
        nr.len = sh.cnt;
        nr.nregs = root.nregs;
        nr.out_reg = root.out_reg;
        nr.n_minmax = sh.mmk;
        nr.t_lo = sh.gl;
        nr.t_hi = sh.gh;
        nr.parent = S.root_rec;
        nr.fwd_cost = sh.fcost;
        nr.rev_cost = sh.rcost;
        nr.c_lo = sh.hl;
        nr.c_hi = sh.hh;
        nr.c_level = it.level + 1u;
        P.recs[sh.ri] = nr;
        ws[ST_TAPE_WORDS] += sh.cnt;
      }
      new_rec = sh.ri;
    }
  }
  const long long f2 = clock64();
  if (tid < 32u) {
    const uint32_t len = (new_rec == S.root_rec) ? root.len : sh.cnt;
    if (tid == 0 && len >= wide_min_len(W, it.level + 1u)) atomicAdd(&P.long_count[si.next], (uint32_t)__popc(E));
    push_children_warp(P, S, it.scene, new_rec, step, it.level, E, it.parent[1], it.parent[2] != 0u,
                       warp_goes_wide(P, W, step, it.level + 1u, len),
                       may_go_narrow(P, W, it.level + 1u, len) ? log_bound(W, len) : 0u, ws, tid);
  }
  if (tid == 0) {
    const long long f3 = clock64();
    ws[ST_CYC_FIN_COMPACT] += (unsigned long long)(f2 - f0);
    ws[ST_CYC_FIN_PUSH] += (unsigned long long)(f3 - f2);
  }
}

// One child cell (octant k) of a wide item.  unit = item * 8 + k.
template <bool D, bool GM>
__device__ __noinline__ void process_cell(const LaunchParams &P, WorkItem *itp, uint32_t k, uint32_t unit,
                                          uint32_t step, WideShared &sh, unsigned long long *ws) {
  const StepIdx si = step_idx(step);
  unsigned char *cell = cell_base<GM>(P);  // the cell's working set
  using A = IA<D>;
  const uint32_t tid = threadIdx.x;
  const WorkItem &it = *itp;
  const SceneLaunch &S = P.scenes[it.scene];
  const VoxelPoolDev &pool = S.pool;
  const WideDev &W = S.wide;
  const uint32_t flg = S.flags;
  const bool swept = (flg & SF_SWEPT) != 0;
  const uint32_t Pv = it.parent[0];
  const uint32_t base = it.parent[1];
  const bool new_voxel = it.parent[2] != 0;
  if (base == TSI_NONE) return;  // pool exhausted when the item was enqueued (error bit set)
  const TapeRec root = P.recs[S.root_rec];
  const uint32_t n_narrow = root.len;
  const uint32_t C = base + k;
  const CellLayout L = cell_layout(W, P.bm_words);
  if constexpr (!GM) {  // the host sized the launch for this cell; never write past it
    if (L.size > P.dyn_smem) {
      if (tid == 0) atomicOr(P.error + it.scene, EB_SMEM);
      return;
    }
  }
  const CellArray<GM> V(cell), G(cell + L.sens);
  const bool slots = GM && W.fwd_slots && W.fslots * 16u <= P.dyn_smem;  // forward values in shared memory
  uint8_t *dec = cell + L.dec, *dec2 = cell + L.flags;
  const float4 pxy = pool.box_xy[Pv];
  const float2 pz = pool.box_z[Pv];
  const float pfast = pool.fast[Pv];
  float c_t = 0.0f, c_f = 1.0f, c_te = 0.0f, c_fast = 0.0f;
  uint32_t c_child = TSI_NONE;
  if (!new_voxel) {
    c_t = pool.t[C];
    c_f = pool.f[C];
    c_te = pool.time_err[C];
    c_fast = pool.fast[C];
    c_child = pool.child[C];
  }
  __syncthreads();  // every thread has read the cell before thread 0 writes it

  // ---- cell setup (compute.wgsl:3582-3626), uniform across the block
  const float dx = __fdiv_rn(__fsub_rn(pxy.y, pxy.x), 2.0f);
  const float dy = __fdiv_rn(__fsub_rn(pxy.w, pxy.z), 2.0f);
  const float dz = __fdiv_rn(__fsub_rn(pz.y, pz.x), 2.0f);
  float width = fm_max(dx, fm_max(dy, dz));
  const float kx = (float)(k & 1u), ky = (float)((k >> 1) & 1u), kz = (float)(k >> 2);
  Iv cx = Iv{__fadd_rn(pxy.x, __fmul_rn(dx, kx)), __fadd_rn(pxy.x, __fmul_rn(dx, 1.0f + kx))};
  Iv cy = Iv{__fadd_rn(pxy.z, __fmul_rn(dy, ky)), __fadd_rn(pxy.z, __fmul_rn(dy, 1.0f + ky))};
  Iv cz = Iv{__fadd_rn(pz.x, __fmul_rn(dz, kz)), __fadd_rn(pz.x, __fmul_rn(dz, 1.0f + kz))};
  // half extent of this cell's children, as they will compute it
  const float child_width =
      fm_max(__fdiv_rn(__fsub_rn(cx.hi, cx.lo), 2.0f),
             fm_max(__fdiv_rn(__fsub_rn(cy.hi, cy.lo), 2.0f), __fdiv_rn(__fsub_rn(cz.hi, cz.lo), 2.0f)));
  const bool point_branch = new_voxel || pfast == 1.0f || width <= S.eps;
  Iv cur_t;
  if (point_branch) {
    cur_t = swept ? Iv{S.t0, S.time} : iv(S.time);
    c_fast = 0.0f;
  } else {
    cur_t = Iv{c_t, S.time};
  }
  if ((flg & SF_POINTSAMPLE) && width <= S.eps) {
    const Iv ox = cx, oy = cy, oz = cz;
    cx = iv(__fdiv_rn(__fadd_rn(ox.lo, ox.hi), 2.0f));
    cy = iv(__fdiv_rn(__fadd_rn(oy.lo, oy.hi), 2.0f));
    cz = iv(__fdiv_rn(__fadd_rn(oz.lo, oz.hi), 2.0f));
    width = 0.0f;
    if (tid == 0) {
      pool.box_xy[C] = make_float4(ox.lo, ox.hi, oy.lo, oy.hi);
      pool.box_z[C] = make_float2(oz.lo, oz.hi);
    }
  } else if (tid == 0) {
    pool.box_xy[C] = make_float4(cx.lo, cx.hi, cy.lo, cy.hi);
    pool.box_z[C] = make_float2(cz.lo, cz.hi);
  }
  if (tid == 0) {
    pool.t[C] = S.time;
    if (new_voxel) {
      pool.child[C] = TSI_NONE;
      pool.normal[C] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  const Iv targ = Iv{fm_min(cur_t.lo, cur_t.hi), fm_max(cur_t.lo, cur_t.hi)};
  const bool evaluate = new_voxel || c_f >= 0.0f || c_child == TSI_NONE;
  const bool take_deriv = evaluate && ((cur_t.lo != cur_t.hi) || (flg & SF_ALWAYS_DERIV));
  const bool want_prune = (flg & SF_PRUNING) && root.nregs <= TSI_PRUNE_MAX_REGS
                          && it.level >= W.prune_level;  // finish_group's rule
  const uint32_t words = (root.n_minmax + 15u) >> 4;

  // The time range this cell's children would be evaluated over if it is
  // re-enqueued and they do not take the point branch: when it is wider
  // than the cell's own, the decisions for pruning are taken over it in the
  // same forward pass (values over it in the sensitivity array, unused until
  // the reverse pass; decision bits in the liveness flags, unused until the
  // group finishes).  The range is the one computed after classification
  // below, step for step.
  float wl = targ.lo, wh = targ.hi;
  if (evaluate && want_prune) {
    if (c_child != TSI_NONE && !(child_width <= S.eps)) {
      for (int q = 0; q < 8; ++q) {
        const float ct = pool.t[c_child + q];
        wl = fm_min(wl, fm_min(ct, S.time));
        wh = fm_max(wh, fm_max(ct, S.time));
      }
    }
    if (swept) {
      wl = fm_min(wl, fm_min(S.t0, S.time));
      wh = fm_max(wh, fm_max(S.t0, S.time));
    }
  }
  const bool dual = evaluate && want_prune && (wl < targ.lo || wh > targ.hi);

  // ---- forward and reverse over the full tape, bundle by bundle
  Iv field = iv(0.0f);
  Iv sens[4] = {iv(0.0f), iv(0.0f), iv(0.0f), iv(0.0f)};
  if (evaluate) {
    const long long c0 = clock64();
    if constexpr (GM) {
      if (slots)
        field = cell_forward_slots<D>(W, tsi_dyn_smem, V, take_deriv, dual, want_prune ? dec : nullptr, dec2, cx, cy, cz,
                                      targ, Iv{wl, wh});
      else field = cell_forward<D, GM>(W, V, G, dual, want_prune ? dec : nullptr, dec2, cx, cy, cz, targ, Iv{wl, wh});
    } else {
      field = cell_forward<D, GM>(W, V, G, dual, want_prune ? dec : nullptr, dec2, cx, cy, cz, targ, Iv{wl, wh});
    }
    const long long c1 = clock64();
    if (take_deriv) {
      if constexpr (GM) {
        if (W.rev16 && W.gslots * 8u <= P.dyn_smem) cell_reverse16<D>(W, V, CellArray<false>(tsi_dyn_smem), sh.sens);
        else cell_reverse<D>(W, V, G, sh.sens);
      } else {
        cell_reverse16<D>(W, V, G, sh.sens);
      }
      for (int q = 0; q < 4; ++q) sens[q] = Iv{sh.sens[q].x, sh.sens[q].y};
    }
    if (tid == 0) {
      ws[ST_CYC_WIDE_FWD] += (unsigned long long)(c1 - c0);
      ws[ST_CYC_WIDE_REV] += (unsigned long long)(clock64() - c1);
    }
  }

  // ---- temporal error bound, fast flag, classification (3966-4045)
  Iv df = iv(0.0f), df_dt = iv(0.0f);
  const float delta = S.delta;
  if (take_deriv) {
    const float nx = __fdiv_rn(__fadd_rn(sens[0].lo, sens[0].hi), 2.0f);
    const float ny = __fdiv_rn(__fadd_rn(sens[1].lo, sens[1].hi), 2.0f);
    const float nz = __fdiv_rn(__fadd_rn(sens[2].lo, sens[2].hi), 2.0f);
    if (tid == 0) pool.normal[C] = make_float4(nx, ny, nz, 0.0f);
    df_dt = sens[3];
    const float dt = __fsub_rn(targ.hi, targ.lo);
    df = A::mul_f(df_dt, dt);
    const Iv Wd = A::mul_f(Iv{-1.0f, 1.0f}, __fsub_rn(field.hi, field.lo));
    df = A::cap(df, Wd);
    if ((flg & SF_LIPSCHITZ) && A::abs_(df).hi != 0.0f) {
      const float lb =
          A::abs_(A::sqrt_(A::add(A::sqr(sens[0]), A::add(A::sqr(sens[1]), A::sqr(sens[2]))))).lo;
      if (!is_nan_f(lb)) df = A::div(df, iv(lb));
    }
    if (df.lo == -fm_inf() || df.hi == fm_inf() || is_nan_f(df.lo) || is_nan_f(df.hi)) df = iv(delta);
    c_te = __fadd_rn(c_te, fm_min(fm_max(A::abs_(df).hi, 0.0f), delta));
  }
  if (evaluate && !swept && (flg & SF_FASTENABLED)) c_fast = (A::abs_(df).hi >= S.fast_thresh) ? 1.0f : 0.0f;
  bool enq = false, dealloc = false, reused = false;
  int cls = 3;
  if (evaluate) {
    if (field.lo <= 0.0f && 0.0f <= field.hi) {
      c_f = 0.0f;
      cls = 0;
      if (width > S.eps) {
        if (new_voxel || is_nan_f(df_dt.lo) || is_nan_f(df_dt.hi) || fabsf(df_dt.lo) == fm_inf() ||
            fabsf(df_dt.hi) == fm_inf() || pfast == 1.0f || cur_t.lo == cur_t.hi || c_te >= delta ||
            c_child == TSI_NONE) {
          c_te = 0.0f;
          enq = true;
        } else {
          reused = true;
        }
      }
    } else {
      if (field.hi <= 0.0f) {
        c_f = -1.0f;
        cls = 2;
      } else {
        cls = 1;
        if (!swept) c_f = 1.0f;
      }
      if (!swept && c_child != TSI_NONE) dealloc = true;
    }
  }
  const uint32_t old_child = c_child;
  if (dealloc) c_child = TSI_NONE;
  if (tid == 0) {
    pool.f[C] = c_f;
    pool.time_err[C] = c_te;
    pool.fast[C] = c_fast;
    if (dealloc || new_voxel) pool.child[C] = c_child;
    if (dealloc) {
      const uint32_t pos = atomicAdd(&P.dealloc_count[si.next], 1u);
      if (pos < P.dealloc_cap) P.dealloc[si.nbuf][pos] = make_uint2(it.scene, old_child >> 3);
      else atomicOr(P.error + it.scene, EB_QUEUE_FULL);
    }
    ws[ST_EVAL] += evaluate ? 1ull : 0ull;
    ws[ST_REVERSE] += take_deriv ? 1ull : 0ull;
    ws[ST_SKIPPED] += evaluate ? 0ull : 1ull;
    if (cls == 0) ws[ST_AMBIG] += 1ull;
    if (cls == 1) ws[ST_EMPTY] += 1ull;
    if (cls == 2) ws[ST_FULL] += 1ull;
    if (enq) ws[ST_ENQUEUED] += 1ull;
    if (reused) ws[ST_REUSED] += 1ull;
    if (evaluate) {
      ws[ST_INSTR_FWD] += (unsigned long long)n_narrow;
      ws[ST_INSTR_FULL] += (unsigned long long)S.full_len;
      ws[ST_FP32] += (unsigned long long)root.fwd_cost + (take_deriv ? root.rev_cost : 0u);
    }
    if (take_deriv) ws[ST_INSTR_REV] += (unsigned long long)n_narrow;
  }
  // time range the children will be evaluated over: [child.t, time], or
  // the point branch's range for children at most eps wide or of a fast cell
  const bool child_point = child_width <= S.eps || c_fast == 1.0f;
  float nl = targ.lo, nh = targ.hi;
  if (want_prune && enq && old_child != TSI_NONE && !child_point) {
    for (int q = 0; q < 8; ++q) {
      const float ct = pool.t[old_child + q];
      nl = fm_min(nl, fm_min(ct, S.time));
      nh = fm_max(nh, fm_max(ct, S.time));
    }
  }
  if (want_prune && enq && swept) {
    nl = fm_min(nl, fm_min(S.t0, S.time));
    nh = fm_max(nh, fm_max(S.t0, S.time));
  }
  if (want_prune && enq && (nl < targ.lo || nh > targ.hi)) {
    // decisions over the children's (wider) time range
    __syncthreads();
    if (tid == 0) ws[ST_FP32] += (unsigned long long)root.fwd_cost;
    if (dual && nl == wl && nh == wh) {  // taken in the forward pass
      dec = dec2;
    } else {
      const long long r0 = clock64();
      if constexpr (GM) {
        if (slots)
          (void)cell_forward_slots<D>(W, tsi_dyn_smem, V, false, false, dec, nullptr, cx, cy, cz, Iv{nl, nh}, targ);
        else (void)cell_forward<D, GM>(W, V, G, false, dec, nullptr, cx, cy, cz, Iv{nl, nh}, targ);
      } else {
        (void)cell_forward<D, GM>(W, V, G, false, dec, nullptr, cx, cy, cz, Iv{nl, nh}, targ);
      }
      if (tid == 0) {
        ws[ST_WIDE_REFWD] += 1ull;
        ws[ST_CYC_WIDE_REFWD] += (unsigned long long)(clock64() - r0);
      }
    }
  }
  // ---- hand over to the group: decision bits and time range, then count in
  __syncthreads();
  if (want_prune && enq) {
    uint32_t *dst = P.cell_bits[si.buf] + (size_t)unit * P.bm_words;
    for (uint32_t w = tid; w < words; w += blockDim.x) dst[w] = pack_decisions(dec, w);
  }
  if (tid == 0 && want_prune) {  // the time ranges matter only to a pruning finish
    CellInfo ci;
    ci.nl = enq ? nl : -fm_inf();
    ci.nh = enq ? nh : fm_inf();
    ci.enq = enq ? 1u : 0u;
    ci.pad = 0;
    P.cell_info[si.buf][unit] = ci;
  }
  // A pruning finish reads the decision bits and time ranges written above.
  // In a fresh brick this block wrote its cell's child field (empty), which
  // the finish overwrites with a brick for an enqueued cell: that write must
  // be ordered before the finish's.  Otherwise the finish reads nothing this
  // step's blocks wrote (the enqueued siblings come with the count; an
  // enqueued cell of an older brick keeps its child field) and writes
  // nothing they wrote, so no fence is needed.
  const bool fence = want_prune || new_voxel;  // new_voxel: the item's brick is fresh (all 8 cells)
  if (fence) __threadfence();
  __syncthreads();
  // the count (low byte) and the enqueued siblings (bits 8-15) in one atomic
  if (tid == 0) {
    const uint32_t mine = enq ? (1u << k) : 0u;
    const uint32_t old = atomicAdd(&itp->parent[3], 1u + (mine << 8));
    sh.last = (old & 255u) == 7u ? 1u : 0u;
    sh.E = ((old >> 8) | mine) & 255u;
  }
  __syncthreads();
  if (!sh.last) return;
  if (fence) __threadfence();
  finish_group<GM>(P, it, step, unit & ~7u, sh, ws);
}

// Clears the lists and counters of ring entry c.
__device__ __forceinline__ void clear_step(const LaunchParams &P, uint32_t c) {
  P.item_count[c] = 0;
  P.item_cursor[c] = 0;
  P.witem_count[c] = 0;
  P.witem_cursor[c] = 0;
  P.dealloc_count[c] = 0;
  P.dealloc_cursor[c] = 0;
  P.log_overflow_used[c] = 0;
  P.long_count[c] = 0;
}

// A warp's counters belong to the scene whose items it counted: they are
// added to that scene's stats row (and the launch's level row) when the warp
// moves on to another scene's item and at the end of the launch.
__device__ __forceinline__ void flush_stats(const LaunchParams &P, unsigned long long *ws, uint32_t scene,
                                            uint32_t cur, uint32_t lane) {
  __syncwarp();
  unsigned long long *row = P.stats + (size_t)scene * ST_COUNT;
  unsigned long long *lv = P.level_stats ? P.level_stats + (size_t)cur * ST_COUNT : nullptr;
  for (uint32_t i = lane; i < ST_COUNT; i += 32u) {
    const unsigned long long v = ws[i];
    if (!v) continue;
    ws[i] = 0;
    if (i == ST_CYC_WIDE_MAX || i == ST_CYC_NARROW_MAX || i == ST_NARROW_LEN_MAX) {
      atomicMax(row + i, v);
      if (lv) atomicMax(lv + i, v);
    } else {
      atomicAdd(row + i, v);
      if (lv) atomicAdd(lv + i, v);
    }
  }
  __syncwarp();
}

// One launch step over every scene of the launch: the wide items, the narrow
// items and the deallocation items of the step's lists.
__global__ void __launch_bounds__(256) refine_kernel(const __grid_constant__ LaunchParams P, uint32_t step,
                                                     uint32_t rcap) {
  StepIdx si;
  si.cur = step & TSI_STEP_MASK;
  si.next = (step + 1u) & TSI_STEP_MASK;
  si.buf = step & 1u;
  si.nbuf = (step + 1u) & 1u;
  __shared__ unsigned long long s_stats[kWarps][ST_COUNT];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  // Launched as a programmatic dependent of the previous step, the blocks
  // may be resident before that step has ended: nothing of it is read
  // before it has completed.  Then the next step's launch may begin (its
  // blocks take the SMs this launch's blocks leave).
  grid_dependency_wait();
  grid_dependents_launch();
  // the lists of the step after next start empty (no launch of this step
  // touches them; the next step fills them)
  if (blockIdx.x == 0 && threadIdx.x == 0) clear_step(P, (step + 2u) & TSI_STEP_MASK);
  const uint32_t gw = blockIdx.x * (blockDim.x >> 5) + wib;
  float4 *slice_log = P.log_slices + (size_t)gw * P.slice_len * 32u;
  uint2 *slice_dec = P.dec_slices + (size_t)gw * P.slice_len;
  unsigned long long *ws = s_stats[wib];
  for (uint32_t i = lane; i < ST_COUNT; i += 32u) ws[i] = 0;
  __syncwarp();
  uint32_t wscene = TSI_NONE;  // the scene whose counters ws holds (warp uniform)
  auto take = [&](uint32_t sc) {
    if (sc != wscene) {
      if (wscene != TSI_NONE) flush_stats(P, ws, wscene, si.cur, lane);
      wscene = sc;
    }
  };

  __shared__ WideShared sh;
  __shared__ uint32_t s_idx;
  // wide items: one block per child cell (thread 0 and warp 0 count into
  // s_stats[0], warp 0's counters)
  auto wide_phase = [&]() {
    const uint32_t n_units = min(P.witem_count[si.cur], P.witem_cap) * 8u;
    while (true) {
      if (threadIdx.x == 0) s_idx = atomicAdd(&P.witem_cursor[si.cur], 1u);
      __syncthreads();
      const uint32_t u = s_idx;
      __syncthreads();
      if (u >= n_units) break;
      WorkItem *itp = P.witems[si.buf] + (u >> 3);
      const uint32_t sc = itp->scene;
      if (wib == 0) take(sc);
      const long long c0 = clock64();
      const SceneLaunch &S = P.scenes[sc];
      const bool directed = (S.flags & SF_DIRECTED) != 0;
      if (S.wide.global) {
        if (directed) process_cell<true, true>(P, itp, u & 7u, u, step, sh, s_stats[0]);
        else process_cell<false, true>(P, itp, u & 7u, u, step, sh, s_stats[0]);
      } else {
        if (directed) process_cell<true, false>(P, itp, u & 7u, u, step, sh, s_stats[0]);
        else process_cell<false, false>(P, itp, u & 7u, u, step, sh, s_stats[0]);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        const unsigned long long c = (unsigned long long)(clock64() - c0);
        s_stats[0][ST_WIDE_ITEMS] += 1;
        s_stats[0][ST_CYC_WIDE] += c;
        s_stats[0][ST_CYC_WIDE_MAX] = max(s_stats[0][ST_CYC_WIDE_MAX], c);
      }
    }
  };
  // narrow items: one warp per item
  auto narrow_phase = [&]() {
    const uint32_t n_items = min(P.item_count[si.cur], P.item_cap);
    const WorkItem *items = P.items[si.buf];
    while (true) {
      uint32_t idx = 0;
      if (lane == 0) idx = atomicAdd(&P.item_cursor[si.cur], 1u);
      idx = __shfl_sync(FULL_MASK, idx, 0);
      if (idx >= n_items) break;
      const WorkItem &it = items[idx];
      take(it.scene);
      const long long c0 = clock64();
      if (P.scenes[it.scene].flags & SF_DIRECTED) process_item<true>(P, it, step, rcap, slice_log, slice_dec, ws);
      else process_item<false>(P, it, step, rcap, slice_log, slice_dec, ws);
      __syncwarp();
      if (lane == 0) {
        const unsigned long long c = (unsigned long long)(clock64() - c0);
        ws[ST_CYC_NARROW] += c;
        ws[ST_CYC_NARROW_MAX] = max(ws[ST_CYC_NARROW_MAX], c);
      }
    }
  };
  // three blocks in four drain the narrow list first, so both lists start
  // draining at once (half of them measured 0.8% slower, all wide first 6%)
  if ((blockIdx.x & 3u) != 0u) {
    narrow_phase();
    wide_phase();
  } else {
    wide_phase();
    narrow_phase();
  }
  // deallocation items: 4 bricks per warp
  const uint32_t n_dealloc = min(P.dealloc_count[si.cur], P.dealloc_cap);
  const uint2 *dl = P.dealloc[si.buf];
  while (true) {
    uint32_t idx = 0;
    if (lane == 0) idx = atomicAdd(&P.dealloc_cursor[si.cur], 4u);
    idx = __shfl_sync(FULL_MASK, idx, 0);
    if (idx >= n_dealloc) break;
    const uint32_t j = idx + (lane >> 3);
    const bool valid = j < n_dealloc;
    const uint2 item = valid ? dl[j] : make_uint2(0u, 0u);
    dealloc_brick(P, item, step, valid);
  }
  if (wscene != TSI_NONE) flush_stats(P, ws, wscene, si.cur, lane);
}

// buf_main's enqueue(0) (compute.wgsl:4706) for scene s: its root as a work
// item of the step (a wide item, with the root's children brick, when the
// root tape is long enough).
__device__ void seed_root(const LaunchParams &P, uint32_t s, uint32_t step) {
  const StepIdx si = step_idx(step);
  WorkItem w;
  w.scene = s;
  w.rec = P.scenes[s].root_rec;
  w.n = 1;
  w.level = 0;
  w.parent[0] = w.parent[1] = w.parent[2] = w.parent[3] = 0u;
  const SceneLaunch &S = P.scenes[s];
  const uint32_t len = P.recs[S.root_rec].len;
  if (len >= S.wide.min_len) {
    const uint32_t pos = atomicAdd(&P.witem_count[si.cur], 1u);
    if (pos < P.witem_cap) {
      uint32_t b = S.pool.child[0], fresh = 0;
      if (b == TSI_NONE) {
        b = alloc_brick(S, P.error + s);
        if (b != TSI_NONE) {
          S.pool.child[0] = b;
          fresh = 1;
          atomicAdd(&P.stats[(size_t)s * ST_COUNT + ST_BRICK_ALLOC], 1ull);
          if (P.level_stats) atomicAdd(&P.level_stats[(size_t)si.cur * ST_COUNT + ST_BRICK_ALLOC], 1ull);
        }
      }
      w.parent[1] = b;
      w.parent[2] = fresh;
      w.parent[3] = 0;
      P.witems[si.buf][pos] = w;
      return;
    }
  }
  const uint32_t pos = atomicAdd(&P.item_count[si.cur], 1u);
  if (pos < P.item_cap) P.items[si.buf][pos] = w;
  else atomicOr(P.error + s, EB_QUEUE_FULL);
}


// Per frame of the plain and batched forms (steps 0, 1, ... are the levels):
// clear every step's lists, the tape arenas and the scenes' error words and
// counters (a memset each cost a frame 2 us more), seed the root of every
// scene at step 0.  With n_scenes = 0 it only clears (the continuous form's
// start).
__global__ void frame_begin_kernel(const __grid_constant__ LaunchParams P) {
  const uint32_t t = threadIdx.x;
  grid_dependents_launch();  // the first level's launch may begin
  for (uint32_t l = t; l < TSI_STEP_RING; l += blockDim.x) clear_step(P, l);
  if (t == 0) {
    *P.rec_count = 0;
    *P.code_count = 0;
    *P.rec_low = 0;
    *P.code_low = 0;
  }
  for (uint32_t i = t; i < P.n_scenes; i += blockDim.x) P.error[i] = 0;
  for (uint32_t i = t; i < P.n_scenes * ST_COUNT; i += blockDim.x) P.stats[i] = 0;
  if (P.level_stats)
    for (uint32_t i = t; i < TSI_STEP_RING * ST_COUNT; i += blockDim.x) P.level_stats[i] = 0;
  __syncthreads();
  for (uint32_t s = t; s < P.n_scenes; s += blockDim.x) seed_root(P, s, 0u);
}

// An empty octree (main.rs:749-766): root voxel 0 = root box, t 0, no
// children, f 0; no brick but the root's in use.
__global__ void scene_reset_kernel(VoxelPoolDev pool, SceneCounters *ctr, float4 xy, float2 z) {
  pool.box_xy[0] = xy;
  pool.box_z[0] = z;
  pool.t[0] = 0.0f;
  pool.time_err[0] = 0.0f;
  pool.f[0] = 0.0f;
  pool.fast[0] = 0.0f;
  pool.child[0] = TSI_NONE;
  pool.normal[0] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  *ctr = SceneCounters{0, 1u, 0u, 1u};
}

// Start of a step of the continuous form at which slots join: record the
// arena counters at the step's start, move the low-water marks to the oldest
// running slot's first step (always a step at which slots joined), clear
// the stats rows and error words of the joining slots and seed their roots.
// (Each refinement launch clears the lists of the step after its next.)
__global__ void step_begin_kernel(const __grid_constant__ LaunchParams P, uint32_t step,
                                  const __grid_constant__ StepSeeds sd) {
  StepIdx si;
  si.cur = step & TSI_STEP_MASK;
  si.next = (step + 1u) & TSI_STEP_MASK;
  si.buf = step & 1u;
  si.nbuf = (step + 1u) & 1u;
  const uint32_t t = threadIdx.x;
  if (t == 0) {
    P.step_code_start[si.cur] = *P.code_count;
    P.step_rec_start[si.cur] = *P.rec_count;
    *P.code_low = P.step_code_start[sd.oldest & TSI_STEP_MASK];
    *P.rec_low = P.step_rec_start[sd.oldest & TSI_STEP_MASK];
    clear_step(P, si.next);
  }
  const uint32_t n = min(sd.n, (uint32_t)TSI_SEEDS_MAX);
  for (uint32_t i = t; i < n * ST_COUNT; i += blockDim.x) P.stats[(size_t)sd.slot[i / ST_COUNT] * ST_COUNT + i % ST_COUNT] = 0;
  for (uint32_t i = t; i < n; i += blockDim.x) P.error[sd.slot[i]] = 0;
  __syncthreads();
  for (uint32_t i = t; i < n; i += blockDim.x) seed_root(P, sd.slot[i], step);
}

// Per frame end of scenes first .. first + gridDim.x - 1: bricks freed during
// the frame become allocatable; the scene's error word is or-ed into the
// sticky word (asynchronous inversions).
__global__ void frame_end_kernel(const __grid_constant__ LaunchParams P, uint32_t first) {
  grid_dependency_wait();  // the last level has completed
  const uint32_t s = first + blockIdx.x;
  if (s >= P.n_scenes) return;
  const SceneLaunch &S = P.scenes[s];
  SceneCounters *c = S.ctr;
  __shared__ int32_t fc0;
  __shared__ uint32_t np;
  if (threadIdx.x == 0 && P.error_sticky) atomicOr(P.error_sticky, P.error[s]);
  if (threadIdx.x == 0) {
    fc0 = max(c->free_count, 0);
    np = min(c->pending_count, S.pool.cap_bricks);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < np; i += blockDim.x) S.pool.free_list[fc0 + i] = S.pool.pending[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    c->free_count = fc0 + (int32_t)np;
    c->pending_count = 0;
    uint32_t used = min(c->bump, S.pool.cap_bricks);
    c->live_bricks = used - (uint32_t)(fc0 + (int32_t)np);
    // read back with the counters: the host needs no copy of its own for it
    if (P.live) P.live[s] = c->live_bricks;
  }
}

// host-side launch helpers
namespace {
// Launch configuration; `overlap`: a programmatic dependent of the stream's
// previous kernel (its launch overlaps that kernel's last blocks; the
// kernel waits for it to complete before reading what it wrote).
struct LaunchCfg {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  LaunchCfg(int grid, int block, size_t smem, cudaStream_t st, bool overlap) {
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = overlap ? attr : nullptr;
    cfg.numAttrs = overlap ? 1u : 0u;
  }
};
}  // namespace

cudaError_t launch_refine(const LaunchParams &P, uint32_t step, uint32_t rcap, int grid, int block, size_t smem,
                          cudaStream_t st, bool overlap) {
  LaunchCfg lc(grid, block, smem, st, overlap);
  return cudaLaunchKernelEx(&lc.cfg, refine_kernel, P, step, rcap);
}
cudaError_t launch_frame_begin(const LaunchParams &P, cudaStream_t st) {
  frame_begin_kernel<<<1, 256, 0, st>>>(P);
  return cudaGetLastError();
}
cudaError_t launch_scene_reset(const VoxelPoolDev &pool, SceneCounters *ctr, const float lo[3], const float hi[3],
                               cudaStream_t st) {
  scene_reset_kernel<<<1, 1, 0, st>>>(pool, ctr, make_float4(lo[0], hi[0], lo[1], hi[1]), make_float2(lo[2], hi[2]));
  return cudaGetLastError();
}
cudaError_t launch_step_begin(const LaunchParams &P, uint32_t step, const StepSeeds &sd, cudaStream_t st) {
  step_begin_kernel<<<1, 256, 0, st>>>(P, step, sd);
  return cudaGetLastError();
}
cudaError_t launch_frame_end(const LaunchParams &P, uint32_t first, uint32_t count, cudaStream_t st, bool overlap) {
  if (count == 0) return cudaSuccess;
  LaunchCfg lc((int)count, 256, 0, st, overlap);
  return cudaLaunchKernelEx(&lc.cfg, frame_end_kernel, P, first);
}
// The attribute belongs to the kernel on the current device, shared by every
// context of the process: only ever raise it.
cudaError_t refine_set_smem(size_t bytes) {
  static std::mutex mu;
  static size_t set_bytes[64] = {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < 64 && bytes <= set_bytes[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(refine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && dev >= 0 && dev < 64) set_bytes[dev] = bytes;
  return e;
}
cudaError_t refine_occupancy(int block, size_t smem, int *blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, refine_kernel, block, smem);
}
cudaError_t refine_static_smem(size_t *bytes) {
  cudaFuncAttributes fa;
  const cudaError_t e = cudaFuncGetAttributes(&fa, refine_kernel);
  *bytes = e == cudaSuccess ? fa.sharedSizeBytes : 0;
  return e;
}

}  // namespace tsi
