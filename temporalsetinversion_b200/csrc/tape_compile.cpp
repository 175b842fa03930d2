// tape_compile.cpp — handler selection and register allocation.
#include "tape_compile.h"

#include <algorithm>
#include <cmath>
#include <functional>
#include <iterator>
#include <limits>
#include <map>
#include <utility>
#include <cstring>

#include "opcost.h"
#include "wide_tape.h"

namespace tsi {
namespace {

uint32_t op_top_of(const IrInstr &in) {  // ir.rs:146-171
  uint32_t side = 3;
  if (in.larg.is_reg) side -= 2;
  if (in.rarg.is_reg) side -= 1;
  return side;
}

uint32_t handler_of(uint32_t op, uint32_t top) {
  switch (top) {
    case 0:  // compute.wgsl:3710-3749
      switch (op) {
        case TSI_OP_ADD: return H_ADD_II;
        case TSI_OP_SUB: return H_SUB_II;
        case TSI_OP_DIV: return H_DIV_II;
        case TSI_OP_MUL: return H_MUL_II;
        case TSI_OP_MIN: return H_MIN_II;
        case TSI_OP_MAX: return H_MAX_II;
        case TSI_OP_POW: return H_POW_II;
        case TSI_OP_MOD: return H_MOD_II;
        case TSI_OP_ATAN2: return H_ATAN2_II;
        default: return H_BAD_II;
      }
    case 1:  // compute.wgsl:3643-3709
      switch (op) {
        case TSI_OP_SQR: return H_SQR;
        case TSI_OP_SQRT: return H_SQRT;
        case TSI_OP_EXP: return H_EXP;
        case TSI_OP_LOG: return H_LOG;
        case TSI_OP_NEG: return H_NEG;
        case TSI_OP_ABS: return H_ABS;
        case TSI_OP_FLOOR: return H_FLOOR;
        case TSI_OP_SIN: return H_SIN;
        case TSI_OP_COS: return H_COS;
        case TSI_OP_ADD: return H_ADD_IF;
        case TSI_OP_SUB: return H_SUB_IF;
        case TSI_OP_DIV: return H_DIV_IF;
        case TSI_OP_MUL: return H_MUL_IF;
        case TSI_OP_MIN: return H_MIN_IF;
        case TSI_OP_MAX: return H_MAX_IF;
        case TSI_OP_POW: return H_POW_IF;
        case TSI_OP_RET: return H_COPY;
        case TSI_OP_MOD: return H_MOD_IF;
        case TSI_OP_ATAN2: return H_ATAN2_IF;
        default: return H_BAD_I;
      }
    case 2:  // compute.wgsl:3750-3764
      switch (op) {
        case TSI_OP_SUB: return H_SUB_FI;
        case TSI_OP_DIV: return H_DIV_FI;
        default: return H_BAD_FI;
      }
    default:  // compute.wgsl:3765, the value stays I_FROM(0.0)
      return H_CONST;
  }
}

}  // namespace

// Whether the narrow interpreter takes an instruction as linear, to nearest
// (narrow_interp.cuh, decode_forward).
static bool linear_handler(uint32_t h, float lit) {
  switch (h) {
    case H_ADD_II: case H_SUB_II: case H_ADD_IF: case H_SUB_IF: case H_SUB_FI: case H_NEG: case H_COPY: return true;
    case H_MUL_IF: return std::fabs(lit) <= 1000000.0f;
    default: return false;
  }
}

// A bound of log2 |value| from those of the operands; NaN for handlers whose
// value or reverse rule is infinite on ordinary operands.
static double magnitude(uint32_t h, double a, double b, float lit) {
  int e = -150;  // |lit| < 2^e
  if (lit != lit || std::fabs(lit) > 3.4e38f) e = 1000;
  else if (lit != 0.0f) std::frexp(lit, &e);
  const double l = e;
  switch (h) {
    case H_CONST: return l;
    case H_COPY: case H_NEG: case H_ABS: case H_SQRT: return std::max(a, 0.0);
    case H_ADD_II: case H_SUB_II: case H_MIN_II: case H_MAX_II: return std::max(a, b) + 1.0;
    case H_ADD_IF: case H_SUB_IF: case H_SUB_FI: case H_MIN_IF: case H_MAX_IF: return std::max(a, l) + 1.0;
    case H_MUL_II: return std::max(a, 0.0) + std::max(b, 0.0) + 1.0;
    case H_MUL_IF: return a + l + 1.0;
    case H_SQR: return std::max(2.0 * a, 0.0) + 1.0;
    case H_FLOOR: return std::max(a, 0.0) + 1.0;
    case H_SIN: case H_COS: return 1.0;
    default: return std::numeric_limits<double>::quiet_NaN();
  }
}

bool compile_tape(const std::vector<IrInstr> &ins, PackedTape &out, tsi_status &status,
                  std::string &why) {
  const uint32_t n = uint32_t(ins.size());
  if (n < 4) {
    status = TSI_ERR_INVALID_ARGUMENT;
    why = "a tape needs the four ARG slots";
    return false;
  }
  out = PackedTape{};
  out.count = n;
  // last use of every slot; the field (slot n-1) stays live to the end
  std::vector<int64_t> last_use(n, -1);
  std::vector<uint32_t> users(n, 0);  // instructions that read the slot
  for (uint32_t j = 4; j < n; ++j) {
    const IrInstr &in = ins[j];
    uint32_t top = op_top_of(in);
    if (top == 0 || top == 1) last_use[in.larg.reg] = j;
    if (top == 0 || top == 2) last_use[in.rarg.reg] = j;
    if (top == 0 || top == 1) ++users[in.larg.reg];
    if (top == 2 || (top == 0 && in.rarg.reg != in.larg.reg)) ++users[in.rarg.reg];
  }
  last_use[n - 1] = int64_t(n);

  uint8_t used[TSI_MAX_REGS];
  std::memset(used, 0, sizeof(used));
  std::vector<uint32_t> reg(n, 0);
  for (uint32_t a = 0; a < 4; ++a) {
    reg[a] = a;
    used[a] = (last_use[a] >= 0) ? 1 : 0;
  }
  uint32_t maxreg = 3;
  static const uint32_t fwd_cost[H_COUNT] = TSI_OPCOST_FWD_INIT;
  static const uint32_t rr_cost[H_COUNT] = TSI_OPCOST_RR_INIT;
  out.code.reserve(size_t(n - 4) * 2);
  std::vector<double> mag(n, 20.0);  // every slot's bound of log2 |value|
  std::vector<uint8_t> deps(n, 0);   // every slot's arguments
  for (uint32_t a = 0; a < 4 && a < n; ++a) deps[a] = uint8_t(1u << a);
  out.deps.reserve(n - 4);
  for (uint32_t j = 4; j < n; ++j) {
    const IrInstr &in = ins[j];
    const uint32_t top = op_top_of(in);
    const uint32_t h = handler_of(in.op, top);
    uint32_t a_slot = 0, b_slot = 0;
    bool has_a = false, has_b = false;
    uint32_t w1 = 0;
    float lit = 0.0f;
    if (top == 1) lit = in.rarg.lit;
    else if (top == 2 || top == 3) lit = in.larg.is_reg ? 0.0f : in.larg.lit;
    if (top == 3) lit = in.rarg.lit;  // ir.rs:160-168 keeps the rarg literal last
    if (top == 0) {
      a_slot = in.larg.reg; b_slot = in.rarg.reg; has_a = has_b = true;
    } else if (top == 1) {
      a_slot = in.larg.reg; has_a = true;
    } else if (top == 2) {
      a_slot = in.rarg.reg; has_a = true;
    }
    const uint32_t ra = has_a ? reg[a_slot] : 0;
    const uint32_t rb = has_b ? reg[b_slot] : 0;
    const uint32_t fa = has_a ? (((ins[a_slot].uses & 0xFFFFu) == 1u) ? 1u : 0u) : 0u;
    const uint32_t fb = has_b ? (((ins[b_slot].uses & 0xFFFFu) == 1u) ? 1u : 0u) : 0u;
    if (top == 0) {
      w1 = rb;
    } else {
      float v = (h == H_CONST) ? 0.0f : lit;  // op_top 3 evaluates to [0,0]
      std::memcpy(&w1, &v, 4);
    }
    // free operands at their last use (before allocating the destination)
    if (has_a && last_use[a_slot] == int64_t(j)) used[ra] = 0;
    if (has_b && last_use[b_slot] == int64_t(j)) used[rb] = 0;
    uint32_t d = 0;
    while (d < TSI_MAX_REGS && used[d]) ++d;
    if (d >= TSI_MAX_REGS) {
      status = TSI_ERR_TAPE_TOO_WIDE;
      why = "more than 256 interval values live at slot " + std::to_string(j);
      return false;
    }
    reg[j] = d;
    used[d] = (last_use[j] >= 0) ? 1 : 0;  // a never-read value frees at once
    if (d > maxreg) maxreg = d;
    const bool odd = (fa && users[a_slot] > 1u) || (fb && users[b_slot] > 1u);
    out.code.push_back(TSI_W0(h, fa, fb, d, ra) | (odd ? TSI_W0_ODD : 0u) |
                       (has_a && a_slot < 4u ? TSI_W0_RAW_A : 0u) | (has_b && b_slot < 4u ? TSI_W0_RAW_B : 0u));
    out.code.push_back(w1);
    if (TSI_H_IS_MINMAX(h)) out.n_minmax++;
    if (odd || !linear_handler(h, lit)) out.log_len++;
    const uint32_t da = has_a ? deps[a_slot] : 0u, db = has_b ? deps[b_slot] : 0u;
    deps[j] = uint8_t(da | db);
    out.deps.push_back(uint8_t(da | (db << 4)));
    mag[j] = magnitude(h, has_a ? mag[a_slot] : 0.0, has_b ? mag[b_slot] : 0.0, lit);
    if (odd || !(mag[j] < 120.0) || (h == H_SQRT && !fa)) out.strict = true;
    out.fwd_cost += fwd_cost[h] + TSI_FIX_COST;
    out.rev_cost += rr_cost[h] + TSI_REV_OPERAND_COST * TSI_H_NREG(h);
  }
  out.nregs = maxreg + 1;
  out.out_reg = reg[n - 1];
  out.slot_reg = reg;
  return true;
}

bool compile_wide(const std::vector<IrInstr> &ins, const PackedTape &narrow, WideTape &out, tsi_status &status,
                  std::string &why) {
  const uint32_t n = uint32_t(ins.size());
  out = WideTape{};
  if (n <= 4) return true;
  if (n >= (1u << 24)) {
    status = TSI_ERR_TAPE_TOO_WIDE;
    why = "bundled tape limited to 2^24 slots";
    return false;
  }
  // operands of every slot
  std::vector<uint32_t> opa(n, TSI_NONE), opb(n, TSI_NONE);
  for (uint32_t j = 4; j < n; ++j) {
    const uint32_t top = op_top_of(ins[j]);
    if (top == 0) {
      opa[j] = ins[j].larg.reg;
      opb[j] = ins[j].rarg.reg;
    } else if (top == 1) {
      opa[j] = ins[j].larg.reg;
    } else if (top == 2) {
      opa[j] = ins[j].rarg.reg;
    }
  }
  auto handler = [&](uint32_t j) { return TSI_W0_H(narrow.code[2 * (j - 4)]); };
  // users of every value, in program order (an instruction reading one value
  // through both operands is one user)
  std::vector<uint32_t> first_user(size_t(n) + 1, 0), user;  // value v's: user[first_user[v] .. first_user[v + 1])
  for (uint32_t j = 4; j < n; ++j) {
    if (opa[j] != TSI_NONE) ++first_user[opa[j] + 1];
    if (opb[j] != TSI_NONE && opb[j] != opa[j]) ++first_user[opb[j] + 1];
  }
  for (uint32_t v = 0; v < n; ++v) first_user[v + 1] += first_user[v];
  user.resize(first_user[n]);
  {
    std::vector<uint32_t> at(first_user.begin(), first_user.end() - 1);
    for (uint32_t j = 4; j < n; ++j) {
      if (opa[j] != TSI_NONE) user[at[opa[j]]++] = j;
      if (opb[j] != TSI_NONE && opb[j] != opa[j]) user[at[opb[j]]++] = j;
    }
  }
  auto users = [&](uint32_t v) { return first_user[v + 1] - first_user[v]; };
  // The reverse pass accumulates a value's sensitivity user by user, in
  // reverse program order, and that order fixes the rounding.  A value with
  // one user receives it directly; a value with several gets one
  // contribution record per user, which the value sums in that order when
  // the reverse pass reaches it.  The skip rule (zero sensitivity of a
  // single-use operand) relies on the ir.rs use count agreeing with the
  // users found here.
  for (uint32_t j = 4; j < n; ++j) {
    const uint32_t w0 = narrow.code[2 * (j - 4)];
    if ((TSI_W0_FA(w0) && opa[j] != TSI_NONE && users(opa[j]) != 1) ||
        (TSI_W0_FB(w0) && opb[j] != TSI_NONE && users(opb[j]) != 1)) {
      status = TSI_ERR_INVALID_ARGUMENT;
      why = "single-use flag on a value with several users";
      return false;
    }
  }
  std::vector<uint32_t> gbase(n, TSI_NONE), rec_a(n, TSI_NONE), rec_b(n, TSI_NONE);
  uint32_t ncontrib = 0;
  for (uint32_t v = 0; v < n; ++v) {
    if (users(v) < 2) continue;
    gbase[v] = ncontrib;
    for (uint32_t u = first_user[v + 1]; u-- > first_user[v];) {  // last user first
      const uint32_t j = user[u];
      if (opa[j] == v) rec_a[j] = ncontrib;
      if (opb[j] == v) rec_b[j] = ncontrib;
      ++ncontrib;
    }
  }
  // List scheduling into bundles of warp groups: a bundle is one block step,
  // at most 8 groups of at most 32 mutually independent instructions, each
  // group of one handler (so a warp runs its group without divergence and
  // groups of different handlers share a step).  Priority is the longest
  // chain from the instruction to the field; a step repeatedly takes the 32
  // highest-priority ready instructions of the handler whose best ready
  // instruction has the highest priority (the oldest instruction on a tie).
  // Users of a step's instructions become ready at the next step.
  const uint32_t groups_per_bundle = WideTape::kWidth / 32u;
  // the handlers the device evaluates inline (interp.cuh op_forward
  // and constants); the others run out of line
  auto inline_handler = [](uint32_t h) {
    switch (h) {
      case H_CONST: case H_COPY: case H_ADD_II: case H_SUB_II: case H_MUL_II: case H_MIN_II: case H_MAX_II:
      case H_ADD_IF: case H_SUB_IF: case H_MUL_IF: case H_MIN_IF: case H_MAX_IF: case H_SQR: case H_SQRT:
      case H_NEG: case H_ABS: case H_SUB_FI:
        return true;
      default:
        return false;
    }
  };
  std::vector<uint32_t> prio(n, 0);
  for (uint32_t j = n; j-- > 4;) {
    uint32_t p = 0;
    for (uint32_t u = first_user[j]; u < first_user[j + 1]; ++u) p = std::max(p, prio[user[u]]);
    prio[j] = p + 1u;
  }
  std::vector<uint32_t> indeg(n, 0);
  for (uint32_t j = 4; j < n; ++j) {
    if (opa[j] != TSI_NONE && opa[j] >= 4) ++indeg[j];
    if (opb[j] != TSI_NONE && opb[j] >= 4 && opb[j] != opa[j]) ++indeg[j];
  }
  // heaps of ~priority << 32 | instruction: the least, with the highest
  // priority and then the oldest, in front
  std::vector<std::vector<uint64_t>> ready(64);
  auto insert = [&](uint32_t j) {
    std::vector<uint64_t> &r = ready[handler(j)];
    r.push_back(uint64_t(~prio[j]) << 32 | j);
    std::push_heap(r.begin(), r.end(), std::greater<uint64_t>());
  };
  for (uint32_t j = 4; j < n; ++j)
    if (indeg[j] == 0) insert(j);
  std::vector<std::vector<std::vector<uint32_t>>> bundles;  // bundle -> groups -> instructions
  uint32_t scheduled = 0;
  std::vector<uint32_t> next;
  while (scheduled < n - 4) {
    std::vector<std::vector<uint32_t>> groups;
    // an out-of-line handler waits while it has slack (its best ready
    // instruction is off the step's critical path) and inline work is ready,
    // so that its instructions gather into few steps
    uint32_t cp = 0;
    bool inline_ready = false;
    for (uint32_t h = 0; h < 64; ++h)
      if (!ready[h].empty()) {
        cp = std::max(cp, ~uint32_t(ready[h].front() >> 32));
        inline_ready = inline_ready || inline_handler(h);
      }
    auto eligible = [&](uint32_t h) {
      return inline_handler(h) || !inline_ready || ~uint32_t(ready[h].front() >> 32) >= cp;
    };
    while (groups.size() < groups_per_bundle) {
      uint32_t hb = 64;
      for (uint32_t h = 0; h < 64; ++h)
        if (!ready[h].empty() && eligible(h) && (hb == 64 || ready[h].front() < ready[hb].front())) hb = h;
      if (hb == 64) break;
      // a group of an out-of-line handler (elementary functions, divisions:
      // a step of them costs several steps of the others) takes every ready
      // instruction of its handler into this step, so that such handlers
      // occupy as few steps as possible
      do {
        std::vector<uint32_t> g;
        while (g.size() < 32u && !ready[hb].empty()) {
          g.push_back(uint32_t(ready[hb].front()));
          std::pop_heap(ready[hb].begin(), ready[hb].end(), std::greater<uint64_t>());
          ready[hb].pop_back();
        }
        groups.push_back(std::move(g));
      } while (!inline_handler(hb) && !ready[hb].empty() && groups.size() < groups_per_bundle);
    }
    if (groups.empty()) {
      status = TSI_ERR_INVALID_ARGUMENT;
      why = "bundle scheduling made no progress";
      return false;
    }
    next.clear();
    for (const auto &g : groups)
      for (uint32_t j : g) {
        ++scheduled;
        for (uint32_t u = first_user[j]; u < first_user[j + 1]; ++u)
          if (--indeg[user[u]] == 0) next.push_back(user[u]);
      }
    for (uint32_t u : next) insert(u);
    bundles.push_back(std::move(groups));
  }
  const uint32_t nb = uint32_t(bundles.size());
  // slots: a bundle's groups at 32-slot strides (lane = slot - first - 32 x
  // group); the lanes a group leaves free are padding slots (handler
  // TSI_H_PAD, no operands, no records)
  uint32_t nslots = 0;
  for (const auto &bg : bundles) nslots += 32u * uint32_t(bg.size() - 1) + uint32_t(bg.back().size());
  out.slots.assign(size_t(nslots) * 12, 0);
  out.bundles.assign(size_t(nb) * 2, 0);
  out.narrow_mm.assign(n - 4, TSI_NONE);
  {
    uint32_t mm = 0;
    for (uint32_t j = 4; j < n; ++j) {
      const uint32_t h = TSI_W0_H(narrow.code[2 * (j - 4)]);
      if (TSI_H_IS_MINMAX(h)) out.narrow_mm[j - 4] = mm++;
    }
  }
  uint32_t off = 0;
  for (uint32_t k = 0; k < nb; ++k) {
    const auto &bg = bundles[k];
    const uint32_t count = 32u * uint32_t(bg.size() - 1) + uint32_t(bg.back().size());
    for (uint32_t s = 0; s < count; ++s) {
      uint32_t *S = &out.slots[size_t(off + s) * 12];
      const auto &g = bg[s / 32u];
      if (s % 32u >= g.size()) {  // padding
        S[0] = TSI_H_PAD;
        S[5] = S[6] = S[7] = S[8] = S[9] = S[10] = TSI_NONE;
        continue;
      }
      const uint32_t j = g[s % 32u];
      const uint32_t w0 = narrow.code[2 * (j - 4)], w1 = narrow.code[2 * (j - 4) + 1];
      const uint32_t h = TSI_W0_H(w0);
      S[0] = h | (TSI_W0_FA(w0) << 6) | (TSI_W0_FB(w0) << 7) | (j << 8);
      // the min/max ordinal sits in the word the handler does not use: the
      // literal's for two registers, B's for a register and a literal
      const uint32_t mmo = TSI_H_IS_MINMAX(h) ? out.narrow_mm[j - 4] : 0u;
      S[1] = opa[j] != TSI_NONE ? opa[j] : 0u;
      S[2] = opb[j] != TSI_NONE ? opb[j] : (TSI_H_IS_II(h) ? 0u : mmo);
      S[3] = TSI_H_IS_II(h) ? mmo : w1;  // literal bits
      S[4] = j;
      S[5] = out.narrow_mm[j - 4];
      S[6] = opa[j];
      S[7] = opb[j];
      S[8] = rec_a[j];
      S[9] = rec_b[j];
      S[10] = gbase[j];
      S[11] = gbase[j] == TSI_NONE ? 0u : users(j);
    }
    out.bundles[2 * k] = off;
    out.bundles[2 * k + 1] = count;
    off += count;
  }
  for (uint32_t a = 0; a < 4; ++a) {
    out.arg_gbase[a] = gbase[a];
    out.arg_gcount[a] = gbase[a] == TSI_NONE ? 0u : users(a);
  }
  out.ncontrib = ncontrib;
  out.nvalues = n;
  out.nbundles = nb;
  return true;
}

// Slots of the sensitivities in the order of the reverse pass (wide_tape.h):
// first fit, but for single slots, which are taken again last in, first out.
struct SlotPool {
  std::map<uint32_t, uint32_t> gaps;  // first slot, length
  std::vector<uint32_t> ones;
  uint32_t tail = 0, top = 0;  // from tail on nothing is taken, from top on nothing ever was
  uint32_t take(uint32_t n) {
    if (n == 1u && !ones.empty()) {
      const uint32_t at = ones.back();
      ones.pop_back();
      return at;
    }
    for (auto it = gaps.begin(); it != gaps.end(); ++it) {
      if (it->second < n) continue;
      const uint32_t at = it->first, left = it->second - n;
      gaps.erase(it);
      if (left) gaps.emplace(at + n, left);
      return at;
    }
    tail += n;
    top = std::max(top, tail);
    return tail - n;
  }
  void give(uint32_t at, uint32_t n) {
    if (n == 1u) {
      ones.push_back(at);
      return;
    }
    auto next = gaps.lower_bound(at);
    if (next != gaps.end() && next->first == at + n) {
      n += next->second;
      next = gaps.erase(next);
    }
    if (next != gaps.begin()) {
      auto prev = std::prev(next);
      if (prev->first + prev->second == at) {
        at = prev->first;
        n += prev->second;
        gaps.erase(prev);
      }
    }
    if (at + n == tail) tail = at;
    else gaps.emplace(at, n);
  }
};

void decode_wide(const WideTape &wt, const PackedTape &pt, WideTapeDev &out) {
  const uint32_t nv = wt.nvalues, zero = nv, dummy = nv + 1u, nv2 = nv + 2u;
  out = WideTapeDev{};
  std::vector<uint8_t> used(nv, 0);  // values some instruction reads
  uint32_t n_minmax = 0;             // a padding lane's ordinal is one past the last
  for (size_t i = 0; i < wt.slots.size(); i += 12) {
    const uint32_t *S = &wt.slots[i];
    if ((S[0] & 63u) == TSI_H_PAD) continue;
    if (S[6] != TSI_NONE) used[S[6]] = 1;
    if (S[7] != TSI_NONE) used[S[7]] = 1;
    if (S[5] != TSI_NONE) n_minmax = std::max(n_minmax, S[5] + 1u);
  }
  // value v is the narrow tape's instruction v - 4
  auto same = [&](uint32_t v) -> uint32_t {
    const uint32_t w0 = pt.code[2 * size_t(v - 4u)], w1 = pt.code[2 * size_t(v - 4u) + 1];
    const bool a = TSI_W0_DST(w0) == TSI_W0_A(w0) && !(w0 & TSI_W0_RAW_A);
    const bool b = TSI_H_IS_II(TSI_W0_H(w0)) && TSI_W0_DST(w0) == (w1 & 255u) && !(w0 & TSI_W0_RAW_B);
    return (a ? WL_SAME_A : 0u) | (b ? WL_SAME_B : 0u);
  };
  std::vector<uint32_t> targets;
  auto push4 = [](std::vector<uint32_t> &v, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t q[4] = {a, b, c, d};
    v.insert(v.end(), q, q + 4);
  };
  const uint32_t minus0 = 0x80000000u;
  // ---- the sensitivities' slots: per value its place or its records' first
  std::vector<uint32_t> place(nv, TSI_NONE), count(nv, 0u), first_rec(nv, 0u);
  {
    SlotPool pool;
    pool.take(2);  // the zero, the dummy
    for (uint32_t q = 0; q < 4u; ++q) {
      count[q] = wt.arg_gcount[q];
      first_rec[q] = count[q] ? wt.arg_gbase[q] : 0u;
      out.g_arg[q] = place[q] = pool.take(std::max(1u, count[q]));
    }
    for (size_t i = 0; i < wt.slots.size(); i += 12) {
      const uint32_t *S = &wt.slots[i];
      if ((S[0] & 63u) == TSI_H_PAD || !S[11]) continue;
      count[S[4]] = S[11];
      first_rec[S[4]] = S[10];
    }
    if (place[nv - 1u] == TSI_NONE) place[nv - 1u] = pool.take(1);
    out.g_field = place[nv - 1u];
    for (uint32_t k = wt.nbundles; k-- > 0u;) {
      const uint32_t first = wt.bundles[2 * k], last = first + wt.bundles[2 * k + 1];
      for (uint32_t s = first; s < last; ++s) {
        const uint32_t *S = &wt.slots[size_t(s) * 12];
        if ((S[0] & 63u) == TSI_H_PAD) continue;
        for (int q = 6; q < 8; ++q)
          if (S[q] != TSI_NONE && place[S[q]] == TSI_NONE) place[S[q]] = pool.take(std::max(1u, count[S[q]]));
      }
      for (uint32_t s = first; s < last; ++s) {  // read in this step: free from the next on
        const uint32_t *S = &wt.slots[size_t(s) * 12];
        if ((S[0] & 63u) != TSI_H_PAD && place[S[4]] != TSI_NONE) pool.give(place[S[4]], std::max(1u, count[S[4]]));
      }
    }
    out.gslots = pool.top;
  }
  // ---- the forward values' slots
  std::vector<uint32_t> fplace;  // (of the zero and the dummy too)
  if (nv >= kForwardSlotsMin) {
    fplace.assign(nv2, 0u);
    fplace[dummy] = 1u;
    std::vector<uint32_t> last_use(nv, 0u);
    for (uint32_t k = 0; k < wt.nbundles; ++k)
      for (uint32_t s = wt.bundles[2 * k], e = s + wt.bundles[2 * k + 1]; s < e; ++s) {
        const uint32_t *S = &wt.slots[size_t(s) * 12];
        if ((S[0] & 63u) == TSI_H_PAD) continue;
        if (S[6] != TSI_NONE) last_use[S[6]] = k;
        if (S[7] != TSI_NONE) last_use[S[7]] = k;
      }
    SlotPool pool;
    pool.take(2);
    for (uint32_t q = 0; q < 4u; ++q) fplace[q] = pool.take(1);
    std::vector<std::vector<uint32_t>> ends(wt.nbundles);  // the values read for the last time in a bundle
    for (uint32_t v = 4; v + 1u < nv; ++v)
      if (used[v]) ends[last_use[v]].push_back(v);
    for (uint32_t k = 0; k < wt.nbundles; ++k) {
      std::vector<uint32_t> unread;
      for (uint32_t s = wt.bundles[2 * k], e = s + wt.bundles[2 * k + 1]; s < e; ++s) {
        const uint32_t *S = &wt.slots[size_t(s) * 12];
        if ((S[0] & 63u) == TSI_H_PAD) continue;
        fplace[S[4]] = pool.take(1);
        if (!used[S[4]] && S[4] != nv - 1u) unread.push_back(S[4]);
      }
      for (uint32_t v : ends[k]) pool.give(fplace[v], 1);
      for (uint32_t v : unread) pool.give(fplace[v], 1);
    }
    out.fslots = pool.top;
    out.f_field = fplace[nv - 1u];
    if (out.fslots > 65536u) fplace.clear();
  }
  const bool small = nv2 <= 65536u && out.gslots <= 65536u;  // (a value's records are as many as its users)
  {  // the arrays' final sizes, or a little more
    size_t padded = 32;  // and a slot past a warp's last group
    for (uint32_t k = 0; k < wt.nbundles; ++k) padded += (wt.bundles[2 * k + 1] + 31u) & ~31u;
    out.fwd.reserve(padded * 4u);
    if (!fplace.empty()) out.fwd_slots.reserve(padded * 4u);
    out.rev.reserve(padded * 8u);
    targets.reserve(padded * 4u);
    if (small) out.rev16.reserve(padded * 4u);
    out.live.reserve(padded * 4u);
  }
  // One group (warp g of bundle k) of the forward or reverse streams; its
  // kind.
  auto emit = [&](uint32_t k, uint32_t g, bool reverse) -> uint32_t {
    const uint32_t first = wt.bundles[2 * k] + 32u * g, left = wt.bundles[2 * k + 1] - 32u * g;
    const uint32_t h = wt.slots[size_t(first) * 12] & 63u;  // the group's handler
    const bool ii = TSI_H_IS_II(h);
    if (reverse && h == H_CONST) return WK_NONE;  // nothing to propagate
    uint32_t kind = WK_OTHER, base = ii ? WC_II : 0u;
    bool gather = false;
    switch (h) {
      case H_ADD_II: case H_ADD_IF: case H_SUB_IF: case H_COPY: case H_SUB_II: case H_SUB_FI: case H_NEG:
        kind = WK_LIN;
        break;
      case H_MUL_IF: kind = WK_SCALE; break;
      case H_MUL_II: kind = WK_MUL; break;
      case H_SQR: kind = WK_SQR; break;
      case H_ABS: kind = WK_ABS; break;
      case H_SQRT: kind = WK_SQRT; break;
      case H_SIN: kind = WK_SIN; break;
      case H_MAX_II: case H_MAX_IF: base |= WC_MAX; kind = WK_MM; break;
      case H_MIN_II: case H_MIN_IF: kind = WK_MM; break;
      default: break;
    }
    const bool has_a = h != H_CONST;  // (B: ii)
    // 32 more slots at an array's end
    auto grow = [](std::vector<uint32_t> &v) {
      v.resize(v.size() + 128u);
      return &v[v.size() - 128u];
    };
    auto put = [](uint32_t *&at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
      at[0] = a;
      at[1] = b;
      at[2] = c;
      at[3] = d;
      at += 4;
    };
    if (!reverse) {
      uint32_t c = base, flip = 0u;
      switch (h) {
        case H_ADD_II: case H_COPY: c |= WC_ZERO; break;
        case H_SUB_II: c |= WC_ZERO | WC_NEG | WC_SWAP; break;
        case H_SUB_IF: flip = minus0; break;
        case H_SUB_FI: c |= WC_NEG | WC_SWAP; break;
        case H_NEG: c |= WC_NEG | WC_SWAP | WC_ZERO; break;
        default: break;
      }
      uint32_t *f = grow(out.fwd), *fs = fplace.empty() ? nullptr : grow(out.fwd_slots);
      for (uint32_t s = 0; s < 32u; ++s) {
        const uint32_t *S = s < left ? &wt.slots[size_t(first + s) * 12] : nullptr;
        const bool pad = !S || (S[0] & 63u) == TSI_H_PAD;
        uint32_t x = pad || !has_a ? zero : S[6], y = pad || !ii ? zero : S[7], w = pad || ii ? 0u : S[3];
        const uint32_t d = pad ? dummy : S[4];
        // the ordinal or the handler travels where the literal or B does not
        if (kind == WK_MM || kind == WK_OTHER) (ii ? w : y) = kind == WK_OTHER ? h : pad ? n_minmax : S[5];
        if (h == H_SUB_II) std::swap(x, y);
        w = (c & WC_ZERO) ? minus0 : w ^ flip;
        put(f, c | (d << WC_DST_SHIFT), x, y, w);
        if (fs) put(fs, c | (d << WC_DST_SHIFT), fplace[x] | (fplace[d] << 16), ii ? fplace[y] : y, w);
      }
      return kind;
    }
    uint32_t *r = grow(out.rev), *t = grow(targets), *r16 = small ? grow(out.rev16) : nullptr;
    for (uint32_t s = 0; s < 32u; ++s) {
      const uint32_t *S = s < left ? &wt.slots[size_t(first + s) * 12] : nullptr;
      const bool pad = !S || (S[0] & 63u) == TSI_H_PAD;
      const uint32_t x = pad || !has_a ? zero : S[6], y = pad || !ii ? zero : S[7], w = pad || ii ? 0u : S[3];
      uint32_t c = base;
      if (h == H_SUB_II) c |= WC_NEG2;
      if (h == H_SUB_FI || h == H_NEG) c |= WC_NEG;
      uint32_t ta = dummy, tb = dummy, src = zero, n = 0;
      uint32_t ga = 1u, gb = 1u, gs = 0u;  // the same in the 16-bit form's slots
      if (!pad) {
        const uint32_t fa = (S[0] >> 6) & 1u, fb = (S[0] >> 7) & 1u;
        if (fa && (!ii || fb)) c |= WC_SKIP;
        auto target = [&](uint32_t v, uint32_t rec, uint32_t &to, uint32_t &place16) {
          const bool one = rec == TSI_NONE;
          to = one ? v : nv2 + rec;
          place16 = place[v] + (one ? 0u : rec - first_rec[v]);
        };
        if (has_a) target(S[6], S[8], ta, ga);
        if (ii) target(S[7], S[9], tb, gb);
        // a value nobody reads has sensitivity zero, the field one
        n = S[11];
        src = n ? nv2 + S[10] : (used[S[4]] || S[4] == nv - 1u ? S[4] : zero);
        if (src != zero) gs = place[S[4]];
        gather = gather || n != 0u;
      }
      put(r, c | (h << 8), x, y, w);
      put(t, ta, tb, src, n);
      if (r16) put(r16, x | (gs << 16), ga | (gb << 16), ii ? y : w, c | (h << 8) | (n << 16));
    }
    return kind | (gather ? WK_GATHER : 0u);
  };
  for (uint32_t dir = 0; dir < 2u; ++dir) {
    const bool reverse = dir == 1u;
    for (uint32_t g = 0; g < kWideWarps; ++g) {
      out.streams.push_back(uint32_t((reverse ? out.rev : out.fwd).size() / 4));
      out.streams.push_back(uint32_t(out.ctl.size()));
      std::vector<uint8_t> bytes;
      for (uint32_t q = 0; q < wt.nbundles; ++q) {
        const uint32_t k = reverse ? wt.nbundles - 1u - q : q;
        bytes.push_back(uint8_t(32u * g < wt.bundles[2 * k + 1] ? emit(k, g, reverse) : WK_NONE));
      }
      while (bytes.size() % kWideAhead) bytes.push_back(uint8_t(WK_NONE));
      for (uint32_t q = 0; q < kWideAhead + 4u; ++q) bytes.push_back(uint8_t(WK_NONE));
      for (size_t i = 0; i < bytes.size(); i += 4)
        out.ctl.push_back(bytes[i] | (uint32_t(bytes[i + 1]) << 8) | (uint32_t(bytes[i + 2]) << 16) |
                          (uint32_t(bytes[i + 3]) << 24));
    }
  }
  // a warp reads one slot past its last group's
  for (uint32_t s = 0; s < 32u; ++s) {
    push4(out.fwd, dummy << WC_DST_SHIFT, zero, zero, 0u);
    if (!fplace.empty()) push4(out.fwd_slots, dummy << WC_DST_SHIFT, 1u << 16, zero, 0u);
    push4(out.rev, 0u, zero, zero, 0u);
    push4(targets, dummy, dummy, zero, 0u);
    if (small) push4(out.rev16, zero, 1u | (1u << 16), 0u, 0u);
  }
  out.rev_slots = uint32_t(out.rev.size() / 4);
  out.rev.insert(out.rev.end(), targets.begin(), targets.end());
  uint32_t nslots = 0;
  for (uint32_t k = 0; k < wt.nbundles; ++k) {
    const uint32_t first = wt.bundles[2 * k], count = wt.bundles[2 * k + 1];
    const uint32_t padded = (count + 31u) & ~31u;
    out.bundles.push_back(nslots);
    out.bundles.push_back(padded);
    nslots += padded;
    for (uint32_t s = 0; s < padded; ++s) {
      const uint32_t *S = s < count ? &wt.slots[size_t(first + s) * 12] : nullptr;
      if (!S || (S[0] & 63u) == TSI_H_PAD) push4(out.live, dummy, TSI_NONE, TSI_NONE, TSI_NONE);
      else push4(out.live, S[4], S[5] == TSI_NONE ? TSI_NONE : S[5] | same(S[4]), S[6], S[7]);
    }
  }
}

}  // namespace tsi
