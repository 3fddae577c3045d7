// msd.cuh — interface of the MSD record sort (msd.cu).
#pragma once

#include "common.cuh"

namespace capssa {
namespace msd {

// The leading digits a sort of n records distributes by before the pieces fit
// one block's shared memory; level 0's digit counts are the caller's job (the
// kernel that makes the records sees each of them anyway).
struct Plan {
    int levels;     // planned distribution levels: 0 (one block's worth), 1 or 2
    int bits[2];    // bits of each level's digit, from the top of the key
};

constexpr uint32_t kOneBlock = 2560;  // records one block sorts on its own
constexpr int kMaxDigit = 12;  // bits of a planned digit

// n records with nbits key bits, of which the leading top_bits number equally
// sized or `longest`-bounded pieces (a segment or bucket index; longest = n
// without one); eff: bits of entropy per key bit.
Plan plan(uint64_t n, int nbits, int top_bits, uint64_t longest, double eff);

// Sorts n records by key bits [low, low + nbits), records with equal keys by
// position.  vals null: each u64 record carries its position in the low bits
// (the whole record is the order).  Otherwise u64 keys with u32 positions.
// Records in (ka, va), scratch (kb, vb); sorted into (ka, va).  counts: the
// 2^bits[0] digit counts of level 0 (device; overwritten).  pos_order false:
// the order of equal keys is left open (it is then whatever is cheapest).
// gen_vals: the input values are not read, value i is i.  levels_out: levels over the whole array (the planned ones).
capssa_status sort(Ctx &c, const Plan &pl, uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb,
                   uint32_t n, int low, int nbits, int pos_bits, bool pos_order,
                   bool gen_vals, uint32_t *counts, int *levels_out);

// Records a thread handles in a distribution tile (stats.radix_items).
constexpr uint32_t records_per_thread(bool pairs) { return pairs ? 12u : 16u; }

// Device buffer for level 0's digit counts (2^kMaxDigit words), zeroed.
uint32_t *count_buffer(Ctx &c);

}  // namespace msd
}  // namespace capssa
