// wide_tape.h — device form of the bundled tape: the slots of tape_compile.h's
// WideTape decoded for wide_interp.cuh, written once per tape by the host.
//
// The passes read the tape as eight streams, one per warp of the block: a
// warp's groups of 32 slots one after another, in the order of their bundles
// (the reverse pass's streams in the reverse order), so that the next slot's
// address is the last one's plus 512 bytes.  Beside them runs a byte per step
// (bundle) and warp, four to a word: the kind of the warp's group, or that it
// has none.
// A padding lane has its group's kind, reads the zero value and writes the
// dummy.  Value indices: the SSA values 0 .. nvalues-1, then the zero (the
// one an addition leaves unchanged) and the dummy.  Sensitivity targets index
// the values' places and, after the dummy's, the contribution records.
//   forward  x: flags, destination << 8   y: operand A   z: operand B
//            w: literal or factor; the min/max ordinal sits in w (two
//            registers) or z (register and literal), the handler of WK_OTHER
//            likewise
//   reverse  x: flags, handler << 8   y: A   z: B   w: literal or factor
//            second array: targets of A's and of B's share, the slot's own
//            sensitivity: its place, or its first record and their count
//   reverse, when every index has 16 bits, one array:
//            x: A, own sensitivity << 16   y: targets of A's, B's << 16
//            z: B (two registers) or the literal   w: flags, handler << 8,
//            record count << 16
// In that form the sensitivities have slots of their own, taken when the first
// share is written and given back after the step that reads their value's, a
// value's records next to one another: slot 0 holds the zero, slot 1 is the
// dummy, then come the four arguments (or their records).
// For cells whose values are in the global scratch (long tapes), the forward
// slots once more with the values in slots of shared memory, taken at their
// definition and given back after the step of their last use (0 the zero, 1
// the dummy, 2 to 5 the arguments):
//            x: as above (the destination for the reverse pass)   y: A's slot,
//            the result's << 16   z: B's slot, or as above   w: as above
// The liveness pass walks bundles, whose slots are padded to whole warps.
#pragma once
#include <stdint.h>

#include <vector>

namespace tsi {

constexpr uint32_t WK_LIN = 0, WK_SQR = 1, WK_MM = 2, WK_MUL = 3, WK_ABS = 4, WK_SQRT = 5, WK_SIN = 6, WK_OTHER = 7;
constexpr uint32_t WK_SCALE = 8;  // a literal's multiple (linear to nearest, a product directed)
constexpr uint32_t WK_NONE = 9;   // no group
constexpr uint32_t WK_GATHER = 16;  // (reverse) some slot of the group sums contribution records: + kind
constexpr uint32_t WC_II = 1u << 0;     // two register operands
constexpr uint32_t WC_SWAP = 1u << 1;   // (forward linear) A's bounds change places
constexpr uint32_t WC_NEG = 1u << 2;    // (linear) factor -1 on A
constexpr uint32_t WC_ZERO = 1u << 3;   // (forward linear) the literal is the zero that changes no sum
constexpr uint32_t WC_NEG2 = 1u << 4;   // (reverse linear) factor -1 on B
constexpr uint32_t WC_MAX = 1u << 5;    // (min/max) max
constexpr uint32_t WC_SKIP = 1u << 6;   // (reverse) every operand is flagged single-use
constexpr uint32_t WC_DST_SHIFT = 8;
constexpr uint32_t kWideAhead = 4;  // steps whose slots a warp has on their way (a multiple of 4)
constexpr uint32_t kWideWarps = 8;

struct WideTape;
struct PackedTape;

// Of a min/max in the liveness slots: its register is the operand's, which is
// no argument, so the copy that it becomes when that operand is always chosen
// does nothing.
constexpr uint32_t WL_SAME_A = 1u << 30, WL_SAME_B = 1u << 31;

struct WideTapeDev {
  std::vector<uint32_t> fwd;      // 4 words per slot, stream after stream
  std::vector<uint32_t> rev;      // 4 words per slot of the first array, then the second array
  std::vector<uint32_t> rev16;    // 4 words per slot (empty: some index needs more than 16 bits)
  std::vector<uint32_t> ctl;      // step bytes, four to a word: the forward streams, then the reverse ones,
                                  // each with kWideAhead steps and a word more at its end
  std::vector<uint32_t> streams;  // 2 words per stream (8 forward, 8 reverse): first slot, first ctl word
  std::vector<uint32_t> live;     // 4 words per slot: destination, min/max ordinal and WL bits, A, B (TSI_NONE: absent)
  std::vector<uint32_t> bundles;  // of `live`: first slot, slot count (a multiple of 32)
  uint32_t rev_slots = 0;         // slots of the reverse streams
  std::vector<uint32_t> fwd_slots;  // the forward slots with shared-memory slots (empty: none)
  uint32_t fslots = 0, f_field = 0;  // of fwd_slots: the values' slots, the field's
  // of rev16: the sensitivities' slots, the arguments' (first) ones, the field's
  uint32_t gslots = 0, g_arg[4] = {0, 0, 0, 0}, g_field = 0;
};
// Tapes of at least this many values get fwd_slots: with 17 bytes a value and
// what its decisions take, cells of some 6500 values and more leave the 111 KB
// that a cell has in shared memory with two blocks an SM, and shorter tapes
// would carry the slots, a fifth more bytes, for nothing.  Where a
// smaller budget or wider register files send a shorter tape's cells to the
// global scratch, they take the form that reads its operands there.
constexpr uint32_t kForwardSlotsMin = 6144;
void decode_wide(const WideTape &wt, const PackedTape &pt, WideTapeDev &out);
}  // namespace tsi
