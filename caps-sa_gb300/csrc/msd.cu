// msd.cu — MSD distribution sort of suffix records.
//
// The records of the initial suffix sort are distinct (key, position) words,
// so their order needs no stable passes: each level distributes the records
// of every piece by the next digit from the top, and a piece that fits shared
// memory is finished by one block.  Compared with the stable 8-bit LSD passes
// (radix.cu) that sorted them before, ranking costs one shared-memory atomic
// a record instead of eight ballots, a tile reserves its place in every
// bucket with one global atomic a digit instead of a look-back over the tiles
// before it, and the number of levels follows log2(n), not the key's width:
// two for up to 2^30 DNA suffixes, then one local sort.
//
// The scheme (distribution by leading digits with piecewise local sorts and
// small pieces joined) is that of Stehle and Jacobsen's hybrid radix sort
// (SIGMOD 2017); the kernels are this project's.
//
// Pieces longer than kPiece records become the next level's ranges; the
// shorter neighbours are joined into chunks of at most kChunk records
// for the local sort.  Skewed keys (runs, few symbols in use) leave long
// pieces after the planned levels: those alone go through further levels of 8
// bits until nothing is left.
#include <algorithm>
#include <cmath>

#include "msd.cuh"

namespace capssa {
namespace msd {

namespace {

// Shapes measured on 2^28 random records (GB300): distribution tiles of 8,192
// records (512 threads, two blocks an SM) 1.00 ms a level, 4,096 or 6,144
// records 1.3 to 1.6 ms, 1,024 threads 1.2 ms; local sorts of up to 2,560
// records with 2,048 bins, three blocks an SM, 2.1 ms, larger or smaller
// chunks and 4,096 bins 2.2 to 3.5 ms.
constexpr int kThreads = 512;              // of a distribution tile
constexpr int kItKeys = (int)records_per_thread(false), kItPairs = (int)records_per_thread(true);
constexpr int kHistUnroll = 4;
constexpr int kLocalThreads = 512, kLocalIt = 5;
constexpr int kLocalBlocks = 3;            // resident blocks per SM
constexpr uint32_t kChunk = kLocalThreads * kLocalIt;  // records a local sort holds
static_assert(kChunk == kOneBlock, "one block's worth");
constexpr uint32_t kPiece = kChunk / 2;    // longest piece joined into a chunk
constexpr int kLogLocalBins = 11;
constexpr uint32_t kLocalBins = 1u << kLogLocalBins;
constexpr uint32_t kBinMax = 48;           // records of one bin ordered by counting
constexpr int kExtraBits = 8;              // digit of the levels past the planned ones

struct Range {
    uint32_t start, len;
};
struct Tile {
    uint32_t start, len, range;
};
struct Counters {
    uint32_t ranges, tiles, chunks, unused;
};
template <bool PAIRS>
__device__ __forceinline__ uint32_t digit_of(uint64_t key, uint32_t val, const Digit &d) {
    if (PAIRS && d.from_val) return (val >> d.shift) & ((1u << d.bits) - 1u);
    return (uint32_t)(key >> d.shift) & ((1u << d.bits) - 1u);
}

// Digit counts of every range (bins[range << bits | digit]), a tile at a time.
template <bool PAIRS>
__global__ void __launch_bounds__(kThreads)
    hist_kernel(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ vals, Digit dg,
                const Tile *__restrict__ tiles, const Counters *__restrict__ ctr,
                uint32_t *__restrict__ bins) {
    extern __shared__ uint32_t s_cnt[];
    const uint32_t R = 1u << dg.bits, nt = ctr->tiles;
    for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
        const Tile tl = tiles[t];
        for (uint32_t i = threadIdx.x; i < R; i += kThreads) s_cnt[i] = 0;
        __syncthreads();
        for (uint32_t i0 = 0; i0 < tl.len; i0 += kHistUnroll * kThreads) {
            uint64_t k[kHistUnroll];
            uint32_t v[kHistUnroll];
#pragma unroll
            for (int j = 0; j < kHistUnroll; j++) {
                const uint32_t i = i0 + j * kThreads + threadIdx.x;
                k[j] = 0;
                v[j] = 0;
                if (i < tl.len) {
                    if (PAIRS && dg.from_val)
                        v[j] = vals[tl.start + i];
                    else
                        k[j] = keys[tl.start + i];
                }
            }
#pragma unroll
            for (int j = 0; j < kHistUnroll; j++)
                if (i0 + j * kThreads + threadIdx.x < tl.len)
                    atomicAdd(&s_cnt[digit_of<PAIRS>(k[j], v[j], dg)], 1u);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < R; i += kThreads)
            if (s_cnt[i]) atomicAdd(&bins[((uint64_t)tl.range << dg.bits) + i], s_cnt[i]);
        __syncthreads();
    }
}

// Counts -> the position of each bin's first record (a block per range;
// whole > 0: one range of that many records).
__global__ void __launch_bounds__(256)
    offsets_kernel(const Range *__restrict__ ranges, const Counters *__restrict__ ctr, int bits,
                   uint32_t whole, uint32_t *__restrict__ bins) {
    __shared__ uint32_t s_w[8];
    const uint32_t R = 1u << bits, nr = whole ? 1u : ctr->ranges;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t r = blockIdx.x; r < nr; r += gridDim.x) {
        uint32_t *b = bins + ((uint64_t)r << bits);
        uint32_t before = whole ? 0u : ranges[r].start;
        for (uint32_t d0 = 0; d0 < R; d0 += 256) {
            const uint32_t d = d0 + threadIdx.x;
            const uint32_t v = d < R ? b[d] : 0u;
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_w[warp] = x;
            __syncthreads();
            uint32_t pre = 0, total = 0;
            for (int w = 0; w < 8; w++) {
                if (w < warp) pre += s_w[w];
                total += s_w[w];
            }
            if (d < R) b[d] = before + pre + x - v;
            before += total;
            __syncthreads();
        }
    }
}

// The bins of given pieces, as a level that distributed by their index would
// leave them: piece i's end, and n past the last piece.
__global__ void __launch_bounds__(256)
    given_kernel(Pieces given, uint32_t n, uint32_t R, uint32_t *__restrict__ bins) {
    for (uint32_t d = blockIdx.x * 256 + threadIdx.x; d < R; d += gridDim.x * 256)
        bins[d] = d + 1 < given.n ? (uint32_t)given.ends[d] : n;
}

__global__ void __launch_bounds__(256) iota_kernel(uint32_t *__restrict__ out, uint32_t n) {
    for (uint64_t i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull)
        out[i] = (uint32_t)i;
}

// One tile of a range at a time: ranks by digit in shared memory, a place in
// every bin from one global atomic per digit present, records staged in digit
// order and written as runs.  bins: each bin's next free position (its end,
// once every tile is done).  Bound by HBM plus about 25 instructions a
// record; a tile of 8,192 records (6,144 pairs) keeps the runs of a 512-way
// digit at 128 bytes, and 64 registers two blocks an SM.
template <bool PAIRS>
__global__ void __launch_bounds__(kThreads, 2)
    scatter_kernel(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ vals,
                   uint64_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out, uint32_t n,
                   int gen_vals, Digit dg, const Tile *__restrict__ tiles,
                   const Counters *__restrict__ ctr,
                   uint32_t *__restrict__ bins) {
    constexpr int IT = PAIRS ? kItPairs : kItKeys;
    constexpr uint32_t T = kThreads * IT;
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *s_key = reinterpret_cast<uint64_t *>(smem);
    uint32_t *s_val = reinterpret_cast<uint32_t *>(s_key + T);
    uint32_t *s_cnt = s_val + (PAIRS ? T : 0);       // counts, then starts in the tile
    uint32_t *s_base = s_cnt + (1u << dg.bits);      // global position less tile position
    __shared__ uint32_t s_w[kThreads / 32];
    const uint32_t R = 1u << dg.bits;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nt = tiles ? ctr->tiles : pieces_of(n, T);
    for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
        Tile tl;
        if (tiles) {
            tl = tiles[t];
        } else {  // one range: the whole array
            tl.start = t * T;
            tl.len = n - tl.start < T ? n - tl.start : T;
            tl.range = 0;
        }
        for (uint32_t i = tid; i < R; i += kThreads) s_cnt[i] = 0;
        uint64_t k[IT];
        uint32_t v[PAIRS ? IT : 1];
        uint16_t rk[IT];
#pragma unroll
        for (int j = 0; j < IT; j++) {
            const uint32_t i = j * kThreads + tid;
            if (i < tl.len) {
                k[j] = keys[tl.start + i];
                if (PAIRS) v[j] = gen_vals ? tl.start + i : vals[tl.start + i];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IT; j++) {
            if (j * kThreads + tid < tl.len)
                rk[j] = (uint16_t)atomicAdd(
                    &s_cnt[digit_of<PAIRS>(k[j], PAIRS ? v[PAIRS ? j : 0] : 0u, dg)], 1u);
        }
        __syncthreads();
        // starts in the tile (exclusive prefix of the counts) and in the bins
        uint32_t before = 0;
        for (uint32_t d0 = 0; d0 < R; d0 += kThreads) {
            const uint32_t d = d0 + tid;
            const uint32_t cv = d < R ? s_cnt[d] : 0u;
            uint32_t g = 0;
            if (cv) g = atomicAdd(&bins[((uint64_t)tl.range << dg.bits) + d], cv);
            uint32_t x = cv;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)lane >= o) x += y;
            }
            if (lane == 31) s_w[warp] = x;
            __syncthreads();
            uint32_t pre = before;
#pragma unroll
            for (uint32_t w = 0; w < kThreads / 32; w++) {
                const uint32_t sw = s_w[w];
                if (w < warp) pre += sw;
                before += sw;
            }
            if (d < R) {
                const uint32_t start = pre + x - cv;
                s_cnt[d] = start;
                s_base[d] = g - start;
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < IT; j++) {
            if (j * kThreads + tid < tl.len) {
                const uint32_t d = digit_of<PAIRS>(k[j], PAIRS ? v[PAIRS ? j : 0] : 0u, dg);
                const uint32_t p = s_cnt[d] + rk[j];
                s_key[p] = k[j];
                if (PAIRS) s_val[p] = v[j];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IT; j++) {
            const uint32_t i = j * kThreads + tid;
            if (i < tl.len) {
                const uint64_t key = s_key[i];
                const uint32_t val = PAIRS ? s_val[i] : 0u;
                const uint32_t out = s_base[digit_of<PAIRS>(key, val, dg)] + i;
                if (out < n) {
                    keys_out[out] = key;
                    if (PAIRS) vals_out[out] = val;
                }
            }
        }
        __syncthreads();
    }
}

// The pieces of a finished level: a thread per bin.  A piece longer than
// kPiece becomes a range of the next level with its tiles (or, when no digit
// is left to order by, chunks of kChunk records); the others are joined: bins
// whose starts lie in the same kPiece-sized stretch of their range form one
// chunk, written by the bin that starts it.
__global__ void __launch_bounds__(256)
    pieces_kernel(const Range *__restrict__ ranges, const Counters *__restrict__ ctr,
                  uint32_t whole, Digit dg,
                  const uint32_t *__restrict__ bins, uint32_t tile_recs, int last, int runs,
                  uint32_t in_b, Range *__restrict__ next_ranges, Tile *__restrict__ next_tiles,
                  Counters *__restrict__ next, uint4 *__restrict__ chunks,
                  uint32_t *__restrict__ n_chunks) {
    const int bits = dg.bits;
    const uint64_t total = (uint64_t)(whole ? 1u : ctr->ranges) << bits;
    const uint32_t R = 1u << bits;
    for (uint64_t idx = blockIdx.x * 256ull + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * 256) {
        const uint32_t r = (uint32_t)(idx >> bits), d = (uint32_t)idx & (R - 1);
        const uint32_t *e = bins + ((uint64_t)r << bits);  // ends of the range's bins
        const Range rg = whole ? Range{0u, whole} : ranges[r];
        const uint32_t s0 = rg.start;
        const uint32_t start = d ? e[d - 1] : s0, end = e[d];
        if (end == start) continue;
        if (end - start > kPiece) {
            const uint32_t len = end - start;
            if (last) {
                // one key: a run entry and its pieces, or pieces to sort alone
                const uint32_t nc = pieces_of(len, kChunk);
                uint32_t at = atomicAdd(n_chunks, nc + (runs ? 1 : 0));
                if (runs) chunks[at++] = make_uint4(start, in_b, len, kRunWhole);
                for (uint32_t q = 0; q < nc; q++)
                    chunks[at + q] =
                        make_uint4(start + q * kChunk, min(kChunk, len - q * kChunk) | in_b,
                                   runs ? start : d, runs ? kRunPiece : chunk_key(1, dg));
            } else {
                const uint32_t nt = pieces_of(len, tile_recs);
                const uint32_t id = atomicAdd(&next->ranges, 1u);
                const uint32_t at = atomicAdd(&next->tiles, nt);
                next_ranges[id] = Range{start, len};
                for (uint32_t q = 0; q < nt; q++)
                    next_tiles[at + q] = Tile{start + q * tile_recs,
                                              min(tile_recs, len - q * tile_recs), id};
            }
            continue;
        }
        // first end at or past x among the range's bins
        auto first_end = [&](uint32_t x) {
            uint32_t lo = 0, hi = R - 1;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (e[mid] < x)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            return lo;
        };
        const uint32_t q = (start - s0) / kPiece;
        if (start != (q ? e[first_end(s0 + q * kPiece)] : s0)) continue;  // not the chunk's first bin
        // the chunk's last bin holds the stretch's end; a long one is left out
        const uint64_t stop = (uint64_t)s0 + (uint64_t)(q + 1) * kPiece;
        const uint32_t z = stop >= (uint64_t)s0 + rg.len ? R - 1 : first_end((uint32_t)stop);
        uint32_t last_start = z ? e[z - 1] : s0;
        uint32_t stop_at = e[z];
        if (stop_at - last_start > kPiece) stop_at = last_start;
        const uint32_t zz = stop_at == last_start && z ? z - 1 : z;  // digits d .. zz
        chunks[atomicAdd(n_chunks, 1u)] =
            make_uint4(start, (stop_at - start) | in_b, d, chunk_key(zz - d + 1, dg));
    }
}

template <bool PAIRS>
__device__ __forceinline__ bool rec_less(uint64_t ka, uint32_t va, uint64_t kb, uint32_t vb) {
    return ka < kb || (PAIRS && ka == kb && va < vb);
}

// One chunk at a time, sorted in shared memory: the bits from the chunk's
// digits on, kLocalBins of them in value, place a record at its bin's start
// plus an atomic rank, which leaves bins of one or two records on spread
// keys; each record then counts the smaller ones in its bin.  A chunk with a
// bin over kBinMax records (many equal keys) is left to crowd_kernel.
template <bool PAIRS>
__global__ void __launch_bounds__(kLocalThreads, kLocalBlocks)
    local_kernel(uint64_t *ka, uint32_t *va, const uint64_t *kb, const uint32_t *vb, uint4 single,
                 int gen_vals, const uint4 *__restrict__ chunks,
                 const uint32_t *__restrict__ n_chunks, uint4 *__restrict__ crowded,
                 uint32_t *__restrict__ n_crowded) {
    constexpr int IT = kLocalIt;
    constexpr uint32_t kPer = kLocalBins / kLocalThreads;
    static_assert(kPer % 4 == 0 || kPer == 2 || kPer == 1, "bins per thread");
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *s_key = reinterpret_cast<uint64_t *>(smem);
    uint32_t *s_bin = reinterpret_cast<uint32_t *>(s_key + kChunk);  // counts, then starts
    uint32_t *s_val = s_bin + kLocalBins + 4;
    __shared__ uint32_t s_w[kLocalThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nc = single.y ? 1u : *n_chunks;
    for (uint32_t ci = blockIdx.x; ci < nc; ci += gridDim.x) {
        const uint4 ch = single.y ? single : chunks[ci];
        const uint32_t m = ch.y & ~kInB, at = ch.x;
        const uint64_t *ks = (ch.y & kInB) ? kb : ka;
        const uint32_t *vs = (ch.y & kInB) ? vb : va;
        uint64_t k[IT];
        uint32_t v[PAIRS ? IT : 1];
#pragma unroll
        for (int j = 0; j < IT; j++) {
            const uint32_t i = j * kLocalThreads + tid;
            if (i < m) {
                k[j] = ks[at + i];
                if (PAIRS) v[j] = gen_vals ? at + i : vs[at + i];
            }
        }
        const ChunkBins bins(ch, kLogLocalBins, 0);
        const bool fv = PAIRS && (ch.w >> 31);
        auto bin_of = [&](uint64_t key, uint32_t val) { return bins.of(fv ? (uint64_t)val : key); };
        for (uint32_t i = tid; i <= kLocalBins / 4; i += kLocalThreads)
            reinterpret_cast<uint4 *>(s_bin)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        uint32_t rk[IT];
        bool crowd = false;
#pragma unroll
        for (int j = 0; j < IT; j++) {
            if (j * kLocalThreads + tid < m) {
                rk[j] = atomicAdd(&s_bin[bin_of(k[j], PAIRS ? v[PAIRS ? j : 0] : 0u)], 1u);
                crowd |= rk[j] >= kBinMax;
            }
        }
        if (__syncthreads_or(crowd ? 1 : 0)) {
            if (tid == 0) crowded[atomicAdd(n_crowded, 1u)] = ch;
            __syncthreads();
            continue;
        }
        // exclusive prefix of the bins
        uint32_t c[kPer], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            c[q] = s_bin[tid * kPer + q];
            sum += c[q];
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)lane >= o) x += y;
        }
        if (lane == 31) s_w[warp] = x;
        __syncthreads();
        uint32_t run = x - sum;
#pragma unroll
        for (uint32_t w = 0; w < kLocalThreads / 32; w++) run += w < warp ? s_w[w] : 0u;
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            s_bin[tid * kPer + q] = run;
            run += c[q];
        }
        if (tid == kLocalThreads - 1) s_bin[kLocalBins] = m;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IT; j++) {
            if (j * kLocalThreads + tid < m) {
                const uint32_t p = s_bin[bin_of(k[j], PAIRS ? v[PAIRS ? j : 0] : 0u)] + rk[j];
                s_key[p] = k[j];
                if (PAIRS) s_val[p] = v[j];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IT; j++) {
            const uint32_t i = j * kLocalThreads + tid;
            if (i < m) {
                const uint64_t key = s_key[i];
                const uint32_t val = PAIRS ? s_val[i] : 0u;
                const uint32_t b = bin_of(key, val);
                const uint32_t s = s_bin[b], e = s_bin[b + 1];
                uint32_t p = s;
                if (e - s > 1)
                    for (uint32_t u = s; u < e; u++)
                        p += rec_less<PAIRS>(s_key[u], PAIRS ? s_val[u] : 0u, key, val) ? 1u : 0u;
                ka[at + p] = key;
                if (PAIRS) va[at + p] = val;
            }
        }
        __syncthreads();
    }
}

// The chunks local_kernel left: a merge sort in shared memory, by counting
// inside 32 slots, then runs of doubling length by binary search.
template <bool PAIRS>
__global__ void __launch_bounds__(kLocalThreads)
    crowd_kernel(uint64_t *ka, uint32_t *va, const uint64_t *kb, const uint32_t *vb, int gen_vals,
                 const uint4 *__restrict__ chunks, const uint32_t *__restrict__ n_chunks) {
    constexpr int IT = kLocalIt;
    __shared__ uint64_t s_key[kChunk];
    __shared__ uint32_t s_val[PAIRS ? kChunk : 1];
    const uint32_t tid = threadIdx.x;
    const uint32_t nc = *n_chunks;
    for (uint32_t ci = blockIdx.x; ci < nc; ci += gridDim.x) {
        const uint4 ch = chunks[ci];
        const uint32_t m = ch.y & ~kInB, at = ch.x;
        const uint64_t *ks = (ch.y & kInB) ? kb : ka;
        const uint32_t *vs = (ch.y & kInB) ? vb : va;
        uint64_t k[IT];
        uint32_t v[IT];
#pragma unroll
        for (int j = 0; j < IT; j++) {
            const uint32_t i = j * kLocalThreads + tid;
            if (i < m) {
                s_key[i] = ks[at + i];
                if (PAIRS) s_val[i] = gen_vals ? at + i : vs[at + i];
            }
        }
        __syncthreads();
        for (uint32_t run = 0; run < m; run = run ? run * 2 : 32) {
            uint32_t to[IT];
#pragma unroll
            for (int j = 0; j < IT; j++) {
                const uint32_t i = j * kLocalThreads + tid;
                if (i < m) {
                    k[j] = s_key[i];
                    v[j] = PAIRS ? s_val[PAIRS ? i : 0] : 0u;
                    auto before = [&](uint32_t u) {
                        return rec_less<PAIRS>(s_key[u], PAIRS ? s_val[PAIRS ? u : 0] : 0u, k[j],
                                               v[j]);
                    };
                    if (run == 0) {
                        const uint32_t b0 = i & ~31u, b1 = min(m, b0 + 32);
                        uint32_t p = b0;
                        for (uint32_t u = b0; u < b1; u++) p += before(u) ? 1u : 0u;
                        to[j] = p;
                    } else {
                        const uint32_t p0 = i & ~(2 * run - 1), mid = p0 + run;
                        const bool left = i < mid;
                        const uint32_t a0 = left ? min(mid, m) : p0;
                        const uint32_t a1 = left ? min(mid + run, m) : mid;
                        uint32_t l = a0, h = a1;
                        while (l < h) {
                            const uint32_t mm = (l + h) >> 1;
                            if (before(mm))
                                l = mm + 1;
                            else
                                h = mm;
                        }
                        to[j] = left ? i + (l - a0) : i - (a1 - l);
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < IT; j++) {
                if (j * kLocalThreads + tid < m) {
                    s_key[to[j]] = k[j];
                    if (PAIRS) s_val[to[j]] = v[j];
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < IT; j++) {
            const uint32_t i = j * kLocalThreads + tid;
            if (i < m) {
                ka[at + i] = s_key[i];
                if (PAIRS) va[at + i] = s_val[i];
            }
        }
        __syncthreads();
    }
}

template <bool PAIRS>
size_t scatter_smem(int bits) {
    const size_t T = (size_t)kThreads * (PAIRS ? kItPairs : kItKeys);
    return T * (PAIRS ? 12 : 8) + ((size_t)8 << bits);
}

template <bool PAIRS>
capssa_status run(Ctx &c, const Plan &pl, uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb,
                  uint32_t n, int low, int nbits, int pos_bits, bool pos_order, bool gen_vals,
                  uint32_t *counts, const Pieces &given, int *levels_out,
                  const std::function<capssa_status(const Chunks &)> &finish,
                  bool *synced = nullptr) {
    constexpr uint32_t T = (uint32_t)kThreads * (PAIRS ? kItPairs : kItKeys);
    const size_t local_smem =
        (size_t)kChunk * (PAIRS ? 12 : 8) + ((size_t)kLocalBins + 4) * 4 + 16;
    const unsigned blocks = (unsigned)c.sm_count;
    cudaFuncSetAttribute(local_kernel<PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)local_smem);
    *levels_out = 0;
    cudaFuncSetAttribute(scatter_kernel<PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)scatter_smem<PAIRS>(kMaxDigit));
    // workspace: the chunks of three levels (each level: one per stretch of its
    // ranges, which number at most n / kPiece, and the cut-up long pieces of a
    // last level), two range and tile lists, the counters
    const uint64_t max_ranges = (uint64_t)n / kPiece + 2;
    const uint64_t max_tiles = (uint64_t)n / T + max_ranges + 2;
    const uint64_t max_chunks = 8 * ((uint64_t)n / kPiece + 4) + 64;
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t bytes = 2 * up(max_chunks * 16) + 2 * up(max_ranges * sizeof(Range)) +
                         2 * up(max_tiles * sizeof(Tile)) + 4096;
    char *w = (char *)ws_get(c, WS_MSD, bytes);
    if (!w) return set_err(c, CAPSSA_ENOMEM, "record sort workspace");
    Counters *ctr[2] = {(Counters *)w, (Counters *)(w + 64)};
    uint32_t *n_chunks = (uint32_t *)(w + 128), *n_crowded = (uint32_t *)(w + 132);
    CAPSSA_CUDA(c, cudaMemsetAsync(w, 0, 256, c.stream));
    char *q = w + 256;
    uint4 *chunks = (uint4 *)q;
    q += up(max_chunks * 16);
    uint4 *crowded = (uint4 *)q;
    q += up(max_chunks * 16);
    Range *ranges[2];
    Tile *tiles[2];
    for (int i = 0; i < 2; i++) {
        ranges[i] = (Range *)q;
        q += up(max_ranges * sizeof(Range));
    }
    for (int i = 0; i < 2; i++) {
        tiles[i] = (Tile *)q;
        q += up(max_tiles * sizeof(Tile));
    }
    // sorts the listed chunks (or the one given)
    auto local = [&](uint4 single) -> capssa_status {
        if (finish) return finish(Chunks{chunks, n_chunks, single, crowded, n_crowded});
        const unsigned lg = single.y ? 1u : blocks * kLocalBlocks;
        local_kernel<PAIRS><<<lg, kLocalThreads, local_smem, c.stream>>>(
            ka, va, kb, vb, single, single.y && gen_vals ? 1 : 0, chunks, n_chunks, crowded,
            n_crowded);
        CAPSSA_LAUNCHED(c);
        crowd_kernel<PAIRS><<<single.y ? 1u : blocks * 2, kLocalThreads, 0, c.stream>>>(
            ka, va, kb, vb, single.y && gen_vals ? 1 : 0, crowded, n_crowded);
        CAPSSA_LAUNCHED(c);
        return CAPSSA_OK;
    };
    if (n <= kChunk) {
        // one digit value, the key's top bit or (a key that fills the word) two
        const int top = PAIRS ? nbits : low + nbits;
        const Digit all{std::min(top, 63), 1, 0};
        return local(make_uint4(0, n, 0, chunk_key(top > 63 ? 2 : 1, all)));
    }
    int key_left = nbits;                    // key bits below the digits used so far
    int val_left = PAIRS ? pos_bits : low;   // then position bits
    uint32_t nr_bound = 1;
    Counters *hc = (Counters *)c.h_scratch;
    int cur = 0;
    const int first = pl.given ? -1 : 0;  // level -1: the given pieces
    if (pl.given && gen_vals) {  // (their short ones never pass through a scatter)
        iota_kernel<<<std::min<unsigned>(grid_for(n, 256), blocks * 16), 256, 0, c.stream>>>(va, n);
        CAPSSA_LAUNCHED(c);
        gen_vals = false;
    }
    int moved = 0;  // scatters so far: the records lie in the b buffers after an odd number
    for (int level = first;; level++) {
        // this level's digit
        Digit dg;
        int want = level < 0 ? pl.given : level < pl.levels ? pl.bits[level] : kExtraBits;
        if (level > first && (uint64_t)nr_bound << want > kFreeBins) {
            // the ranges there can be, times the digit's values, is a lot of
            // bins (10,000 texts, one of them of 250 M symbols: up to 9 GB), and
            // mostly few ranges are left: read their number
            CAPSSA_CUDA(c, cudaMemcpyAsync(hc, ctr[cur], sizeof(Counters), cudaMemcpyDeviceToHost,
                                           c.stream));
            CAPSSA_CUDA(c, cudaStreamSynchronize(c.stream));
            nr_bound = std::max(1u, std::min(nr_bound, hc->ranges));
            want = level_bits(n, nr_bound, want);
        }
        if (key_left > 0) {
            dg.bits = std::min(want, key_left);
            key_left -= dg.bits;
            dg.shift = key_left + (PAIRS ? 0 : low);
            dg.from_val = 0;
        } else {
            dg.bits = std::min(want, val_left);
            val_left -= dg.bits;
            dg.shift = val_left;
            dg.from_val = PAIRS ? 1 : 0;
        }
        const uint32_t whole = level == first ? n : 0u;  // one range: the whole array
        const bool last = key_left == 0 && (!pos_order || val_left == 0);
        const uint64_t n_bins = (uint64_t)nr_bound << dg.bits;
        uint32_t *bins = counts;
        if (level != first) {
            bins = (uint32_t *)ws_get(c, WS_MSD_BINS, n_bins * 4);
            if (!bins) return set_err(c, CAPSSA_ENOMEM, "record sort bins");
        }
        if (level < 0) {
            given_kernel<<<grid_for(n_bins, 256), 256, 0, c.stream>>>(given, n, (uint32_t)n_bins,
                                                                      bins);
            CAPSSA_LAUNCHED(c);
        } else {
            const bool in_b = moved & 1;  // this level reads the b buffers
            const uint64_t *ki = in_b ? kb : ka;
            const uint32_t *vi = in_b ? vb : va;
            uint64_t *ko = in_b ? ka : kb;
            uint32_t *vo = in_b ? va : vb;
            const unsigned tile_grid =
                (unsigned)std::min<uint64_t>((uint64_t)n / T + nr_bound + 1, (uint64_t)blocks * 4);
            if (!whole) {
                CAPSSA_CUDA(c, cudaMemsetAsync(bins, 0, n_bins * 4, c.stream));
                hist_kernel<PAIRS><<<tile_grid, kThreads, (size_t)4 << dg.bits, c.stream>>>(
                    ki, vi, dg, tiles[cur], ctr[cur], bins);
                CAPSSA_LAUNCHED(c);
            }
            offsets_kernel<<<std::min<unsigned>(nr_bound, blocks * 8), 256, 0, c.stream>>>(
                ranges[cur], ctr[cur], dg.bits, whole, bins);
            CAPSSA_LAUNCHED(c);
            const size_t sm = scatter_smem<PAIRS>(dg.bits);
            if (level < 16) cudaEventRecord(c.kev[2 * level], c.stream);
            scatter_kernel<PAIRS>
                <<<std::min<unsigned>(tile_grid, blocks * 2), kThreads, sm, c.stream>>>(
                    ki, vi, ko, vo, n, gen_vals && whole ? 1 : 0, dg,
                    whole ? nullptr : tiles[cur], ctr[cur], bins);
            CAPSSA_LAUNCHED(c);
            if (level < 16) cudaEventRecord(c.kev[2 * level + 1], c.stream);
            moved++;
            if (level < pl.levels) (*levels_out)++;
        }
        const int nxt = cur ^ 1;
        CAPSSA_CUDA(c, cudaMemsetAsync(ctr[nxt], 0, sizeof(Counters), c.stream));
        pieces_kernel<<<(unsigned)std::min<uint64_t>((n_bins + 255) / 256, (uint64_t)blocks * 16),
                        256, 0, c.stream>>>(ranges[cur], ctr[cur], whole, dg, bins, T, last ? 1 : 0,
                                            finish ? 1 : 0, (moved & 1) ? kInB : 0u, ranges[nxt],
                                            tiles[nxt], ctr[nxt], chunks, n_chunks);
        CAPSSA_LAUNCHED(c);
        nr_bound = (uint32_t)std::min<uint64_t>(n_bins, max_ranges);
        cur = nxt;
        if (level + 1 < pl.levels && !last) continue;
        // the planned levels are done: sort what fits, see whether long
        // pieces are left
        const capssa_status ls = local(make_uint4(0, 0, 0, 0));
        if (ls != CAPSSA_OK) return ls;
        if (last) break;
        CAPSSA_CUDA(c, cudaMemcpyAsync(hc, ctr[cur], sizeof(Counters), cudaMemcpyDeviceToHost,
                                       c.stream));
        CAPSSA_CUDA(c, cudaMemsetAsync(n_chunks, 0, 8, c.stream));
        CAPSSA_CUDA(c, cudaStreamSynchronize(c.stream));
        if (hc->ranges == 0) {
            if (synced) *synced = true;
            break;
        }
        nr_bound = hc->ranges;
    }
    return CAPSSA_OK;
}

}  // namespace

Plan plan(uint64_t n, int nbits, int top_bits, uint64_t longest, double eff, bool in_pieces) {
    Plan p{0, {0, 0}, 0};
    if (n <= kChunk) return p;
    // pieces of at most 0.8 kPiece records on average, which spread keys stay
    // below kPiece with
    const double half = 0.8 * kPiece;
    double need = 0;  // effective bits below the top ones
    if (top_bits) {
        need = (double)longest > half ? std::log2((double)longest / half) : 0.0;
    } else {
        need = std::log2((double)n / half);
    }
    const double e = std::min(1.0, std::max(eff, 0.25));
    if (in_pieces && top_bits > 0 && top_bits <= kMaxGiven) {
        p.given = top_bits;
        nbits -= top_bits;
        top_bits = 0;
    }
    int bits = top_bits + (int)std::ceil(need / e);
    bits = std::max(1, std::min(bits, nbits));
    if (p.given && need == 0) return p;  // every piece fits a block
    // one level keeps runs of 8 records a digit up to 2^10 of them in use
    if (bits <= kMaxDigit && top_bits + need <= 10.0) {
        p.levels = 1;
        p.bits[0] = bits;
        return p;
    }
    bits = std::min(bits, 2 * kMaxDigit);
    p.levels = 2;
    p.bits[0] = (bits + 1) / 2;
    p.bits[1] = bits - p.bits[0];
    return p;
}

uint32_t *count_buffer(Ctx &c) {
    static_assert(kMaxGiven >= kMaxDigit, "room for either");
    uint32_t *b = (uint32_t *)ws_get(c, WS_MSD_COUNTS, ((size_t)1 << kMaxGiven) * 4);
    if (b && cudaMemsetAsync(b, 0, ((size_t)1 << kMaxDigit) * 4, c.stream) != cudaSuccess)
        return nullptr;
    return b;
}

capssa_status sort(Ctx &c, const Plan &pl, uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb,
                   uint32_t n, int low, int nbits, int pos_bits, bool gen_vals,
                   uint32_t *counts, const Pieces &given, int *levels_out) {
    if (n == 0) {
        *levels_out = 0;
        return CAPSSA_OK;
    }
    return va ? run<true>(c, pl, ka, va, kb, vb, n, low, nbits, pos_bits, /*pos_order=*/true,
                          gen_vals, counts, given, levels_out, nullptr)
              : run<false>(c, pl, ka, nullptr, kb, nullptr, n, low, nbits, pos_bits,
                           /*pos_order=*/true, false, counts, given, levels_out, nullptr);
}

capssa_status distribute(Ctx &c, const Plan &pl, uint64_t *ka, uint64_t *kb, uint32_t n, int low,
                         int nbits, uint32_t *counts, const Pieces &given, int *levels_out,
                         const std::function<capssa_status(const Chunks &)> &finish,
                         bool *synced) {
    return run<false>(c, pl, ka, nullptr, kb, nullptr, n, low, nbits, 0, false, false, counts,
                      given, levels_out, finish, synced);
}

}  // namespace msd
}  // namespace capssa
