// msd.cuh — interface of the MSD record sort (msd.cu).
#pragma once

#include <functional>

#include "common.cuh"

namespace capssa {
namespace msd {

// The leading digits a sort of n records distributes by before the pieces fit
// one block's shared memory; level 0's digit counts are the caller's job (the
// kernel that makes the records sees each of them anyway).
struct Plan {
    int levels;     // planned distribution levels: 0, 1 or 2
    int bits[2];    // bits of each level's digit, from the top of the key
    int given;      // leading key bits the records already lie in order of (see plan)
};

constexpr uint32_t kOneBlock = 2560;  // records one block sorts on its own
constexpr int kMaxDigit = 12;  // bits of a planned digit
constexpr int kMaxGiven = 14;  // ... of a given one (a chunk holds 15 bits of digit)

// n records with nbits key bits, of which the leading top_bits number equally
// sized or `longest`-bounded pieces (a segment or bucket index; longest = n
// without one); eff: bits of entropy per key bit.  in_pieces: the records are
// laid out piece by piece, in the order of those bits.  Up to kMaxGiven such
// bits are then given: no level distributes by them, the pieces' ends are read
// instead (2,048 genomes of 47,000 symbols: 2.83 ms for 3.40 with two levels
// over both, whose first moved every tile's records to the same few digits).
Plan plan(uint64_t n, int nbits, int top_bits, uint64_t longest, double eff, bool in_pieces);
// Digit bits of a level past the first over `ranges` ranges of n records, at
// most `want`.  Its bins, a word for each digit value of each range, stay
// within 64 MB or a byte a record, whichever is more.  A range holds over
// kOneBlock / 2 records, so 8 bits always fit; what a wider digit leaves is up to
// the levels past the planned ones.
constexpr uint64_t kFreeBins = 1ull << 24;
inline int level_bits(uint64_t n, uint64_t ranges, int want) {
    const uint64_t most = n / 4 > kFreeBins ? n / 4 : kFreeBins;
    while (want > 1 && ranges << want > most) want--;
    return want;
}
// The pieces of a plan with given bits: piece i ends at record ends[i]
// (device), and the last at n.
struct Pieces {
    const uint64_t *ends;
    uint32_t n;
};

// A chunk of the distributed records, at most kOneBlock of them, holding whole
// runs of equal keys: (start, length | kInB, first digit value, key), the key
// packing the digit's values span, shift and width (chunk_key).  Every record
// of a chunk agrees above that digit.
constexpr uint32_t kInB = 0x80000000u;  // the records are in the b buffers
struct Chunks {
    const uint4 *list;       // device
    const uint32_t *count;   // device
    uint4 single;            // length > 0: this chunk alone
    uint4 *spare;            // device, room for as many entries again
    uint32_t *n_spare;       // device, zero
};
// Entries of a run of equal keys longer than a chunk, when the order of equal
// keys is left open (see distribute): pieces (start, length | kInB, the run's
// first index, kRunPiece) and one (start, kInB or 0, run length, kRunWhole).
constexpr uint32_t kRunPiece = 0x80000000u, kRunWhole = 0xC0000000u;

// Pieces of at most `per` in n (up to the largest n: n + per - 1 would wrap).
__host__ __device__ __forceinline__ uint32_t pieces_of(uint32_t n, uint32_t per) {
    return n / per + (n % per ? 1u : 0u);
}

struct Digit {  // `bits` bits at `shift` of the key, or of the position
    int shift, bits, from_val;
};
// span digit values: a chunk's keys are first .. first + span - 1 of digit d
__host__ __device__ __forceinline__ uint32_t chunk_key(uint32_t span, const Digit &d) {
    return span | (uint32_t)d.shift << 16 | (uint32_t)d.bits << 24 | (uint32_t)d.from_val << 31;
}
// Bin of a chunk's record among at most 2^log2_bins: its digit less the first,
// and the bits below down to bit `low`; or the digit without its lowest bits
// where more digit values than bins lie between the first and the last (few
// records over a wide digit: a thin range of a sort with two 12-bit levels).
// Bins grow with the key.
struct ChunkBins {
    int sh;
    uint32_t mask, base;
    __device__ __forceinline__ ChunkBins(const uint4 &ch, int log2_bins, int low) {
        const uint32_t span = ch.w & 0xFFFFu, last = ch.z + span - 1;
        const int shift = (int)(ch.w >> 16) & 63, bits = (int)(ch.w >> 24) & 15;
        int g = log2_bins - (31 - __clz((int)span));  // span << g <= 2^log2_bins
        if ((span & (span - 1)) != 0) g--;
        if (g > shift - low) g = shift - low;
        if (g < 0) {
            g = 0;
            while ((last >> -g) - (ch.z >> -g) >= 1u << log2_bins) g--;
        }
        sh = shift - g;
        mask = (1u << (bits + g)) - 1u;
        base = g < 0 ? ch.z >> -g : ch.z << g;
    }
    __device__ __forceinline__ uint32_t of(uint64_t key) const {
        return ((uint32_t)(key >> sh) & mask) - base;
    }
};

// Distributes packed records (u64, position in the low bits, distinct) by key
// bits [low, low + nbits) until every chunk fits one block, and calls finish
// for each batch of chunks (it must leave the records it is given where they
// are until it has read them; the b buffer is scratch).  synced: set when the
// host has waited for the last batch.  Equal keys stay
// together; a run of more than a chunk comes as kRunPiece / kRunWhole entries.
capssa_status distribute(Ctx &c, const Plan &pl, uint64_t *ka, uint64_t *kb, uint32_t n, int low,
                         int nbits, uint32_t *counts, const Pieces &given, int *levels_out,
                         const std::function<capssa_status(const Chunks &)> &finish,
                         bool *synced);

// Sorts n records by key bits [low, low + nbits), records with equal keys by
// position.  vals null: each u64 record carries its position in the low bits
// (the whole record is the order).  Otherwise u64 keys with u32 positions.
// Records in (ka, va), scratch (kb, vb); sorted into (ka, va).  counts: the
// 2^bits[0] digit counts of level 0 (device; overwritten).  gen_vals: the input
// values are not read, value i is i.  levels_out: planned levels run.
capssa_status sort(Ctx &c, const Plan &pl, uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb,
                   uint32_t n, int low, int nbits, int pos_bits, bool gen_vals,
                   uint32_t *counts, const Pieces &given, int *levels_out);

// Records a thread handles in a distribution tile (stats.radix_items).
constexpr uint32_t records_per_thread(bool pairs) { return pairs ? 12u : 16u; }

// Device buffer for level 0's digit counts (2^kMaxDigit words, zeroed), or the
// ends of given pieces.
uint32_t *count_buffer(Ctx &c);

}  // namespace msd
}  // namespace capssa
