// dyc_bins.cuh -- the repeated keys of a batch, found bin by bin in shared
// memory (inserts, erases and mixed batches of a table, and batches of a set).
//
// A chunk's ops are split by a hash of their key into bins of about 1024
// (k_bin_scatter), and one block per bin finds the keys that occur more than
// once with a key table in shared memory (k_bin_group). Every other op keeps
// its bit in a bitmap and is resolved by the probe kernels in op order, with
// coalesced batch reads and results. The open-addressing table in global
// memory that this replaces took one random L2 or DRAM atomic per op over 64
// MB of cells (99-113 us for 2^22 ops), a pass over the cells (23-28 us) and,
// for mixed batches, a second random read per op (56 us). The split is bound
// by its 8-byte stores to random sectors (47 us, of which 5 us is the bytes),
// the grouping by the latency of its steps (19 us for inserts and erases, 27
// us for mixed ops). 2^24 mixed ops on 2^27 keys: 3.64 -> 2.31 ms a pair of
// batches.
//
// Splitting by the region of a key's first bucket instead, so that a bin's
// probes fall close together, and probing from the bins in the same kernel,
// both measured slower: neighbouring lines gained 4 %, and the values, result
// words and bits at random places cost more than that (312 us against 47 + 39
// + 187 for 2^22 mixed ops).
//
// A small batch runs as one kernel (k_bin_small): every block reads the whole
// batch, keeps its bin's ops and resolves them itself, and the last block writes
// the counters to the host. A mixed batch of 4096 ops took ten kernels, four
// memsets and two copies: 97 -> 46 us a call on a table of 2^24 keys.
//
// A bin with more ops than its capacity (few keys, each repeated hundreds of
// times, or a skewed batch's most popular ones) gets a second, exact set of
// records, which its block streams (group_hot); in a small batch its block reads
// the batch again.
#pragma once

#include "dyc_apply.cuh"

namespace dyc {

constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallR = kSmallCap / kSmallThreads;  // records per thread (k_bin_small)
constexpr int kSmallTab = 2 * kSmallCap;            // cells of a bin's key table
constexpr int kSplitThreads = 512;
constexpr uint32_t kSplitBins = 4096;               // bins counted in shared memory (k_bin_scatter)
constexpr int kGroupThreads = 512;
constexpr int kGroupR = kBinCap / kGroupThreads;    // records per thread (k_bin_group)
constexpr int kGroupPre = kBinMean / kGroupThreads; // of them, read along with the count
constexpr uint32_t kBinOffs = 64;                   // tables of a set batch's bin told apart in shared memory
constexpr int kGroupTab = 2 * kBinCap;              // cells of a bin's first table, half as many of its second

// An op of a small batch's bin: index << 2 | code (2 bits; any other code reads).
__device__ __forceinline__ uint32_t op_word(uint64_t i, uint8_t op) {
    return ((uint32_t)i << 2) | (op == kOpInsert ? 1u : op == kOpErase ? 2u : 0u);
}

template <int KB>
__device__ __forceinline__ uint32_t bin_of(typename SlotT<KB>::K k, uint32_t nbins) {
    return __umulhi(cell_hash((uint64_t)k), nbins);
}

// What a record keeps of its key: a 4-byte key itself, or 32 mixed bits of an
// 8-byte key (records with the same tag compare their keys in the batch).
__device__ __forceinline__ uint32_t bin_tag(uint32_t k) { return k; }
__device__ __forceinline__ uint32_t bin_tag(uint64_t k) {
    return (uint32_t)k ^ ((uint32_t)(k >> 32) * 0x85EBCA6Bu);
}

// First cell of a tag in a bin's key table of 2^BITS cells.
template <int BITS> __device__ __forceinline__ uint32_t bin_cell(uint32_t tag) {
    return ((tag ^ (tag >> 15)) * 0x9E3779B1u) >> (32 - BITS);
}

// Start of a small batch: the call counters and the result bits zeroed.
template <int KB>
__global__ void __launch_bounds__(256) k_small_clear(unsigned long long *zero, uint32_t nzero,
                                                     uint32_t *bits, uint64_t words) {
    after_previous();
    const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id < nzero) zero[id] = 0ull;
    for (uint64_t w = id; w < words; w += (uint64_t)gridDim.x * blockDim.x) bits[w] = 0u;
}

// A record's op word: index << 2 | code, or (batches of 2^30 ops and more,
// A.wide) index << 1 | insert. The segments of listed keys hold the former, or
// plain indexes.
__device__ __forceinline__ uint32_t rec_word(const ApplyScratch &A, uint32_t i, uint32_t code) {
    return A.wide ? i << 1 | (code & 1u) : i << 2 | code;
}
__device__ __forceinline__ uint32_t rec_index(const ApplyScratch &A, uint32_t w) {
    return A.wide ? w >> 1 : w >> 2;
}
__device__ __forceinline__ uint32_t seg_word(const ApplyScratch &A, uint32_t w) {
    return A.wide ? w >> 1 : w;
}

__device__ __forceinline__ void clear_single(const BinScratch &B, uint32_t i) {
    atomicAnd(&B.single[i >> 5], ~(1u << (i & 31)));
}

// The bin of a set batch's op: its table's ops are [o0, o1), its key's hash names
// a place among them, and a bin holds the ops of kSetBinMean places (tables with
// few ops share one, and no bin belongs to a table without any). So a bin gets
// kSetBinMean ops of distinct keys on average, whatever the tables are, and its
// ops belong to the tables that have ops at its places. Offsets are clamped to
// n, so device offsets that are out of order (reported by the call) stay inside
// the scratch. (With bins of its own every table took 16 KB of records: 1.6 GB
// of scratch for a 1000-op batch over 100000 tables.)
static_assert(kSetBinMean % kTidxStep == 0, "the table of a bin's first place is in tidx");
__device__ __forceinline__ uint32_t set_bin(const uint32_t *off, uint32_t t, uint32_t hash, uint64_t n) {
    const uint64_t a = __ldg(off + t), b = __ldg(off + t + 1);
    const uint32_t o0 = (uint32_t)(a < n ? a : n - 1), o1 = (uint32_t)(b < n ? b : n);
    return (o0 + (o1 > o0 ? __umulhi(hash, o1 - o0) : 0u)) / kSetBinMean;
}

// A record's tag in a set batch: the same key in different tables of a bin has
// different tags.
__device__ __forceinline__ uint32_t table_mix(uint32_t t) { return t * 0x9E3779B1u; }

// Where the records of the bins that went over start in `hot`: their counts
// summed in bin order. Every block of the pass that needs the starts computes
// them all (the same values, so the writes agree).
template <int KB> __device__ __noinline__ void plan_hot(const BinScratch &B, uint32_t nbins) {
    __shared__ uint32_t s_w[kSplitThreads / 32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t per = (nbins + kSplitThreads - 1) / kSplitThreads;
    const uint32_t b0 = threadIdx.x * per, b1 = min(b0 + per, nbins);
    uint32_t sum = 0u;
    for (uint32_t b = b0; b < b1; ++b) {
        const uint32_t c = B.count[b];
        if (c > (uint32_t)kBinCap) sum += c;
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_w[w] = x;
    __syncthreads();
    uint32_t at = x - sum;
    for (uint32_t v = 0; v < w; ++v) at += s_w[v];
    for (uint32_t b = b0; b < b1; ++b) {
        const uint32_t c = B.count[b];
        if (c <= (uint32_t)kBinCap) continue;
        B.start[b] = at;
        at += c;
    }
    __syncthreads();
}

// Split a chunk into its bins: a block takes PER * 512 consecutive ops, counts
// them per bin in shared memory (each op's place among the block's ops of its
// bin comes back from the count), takes a range of every bin it has ops for,
// and writes the ops' records there. Records of one bin come in no order; the
// op index in the record orders the ops of a key. Key-0 ops belong to no bin.
// Ops beyond a bin's capacity are not written, which raises B.state[kBinOver]:
// the pass HOT then gives all ops of such bins a record in `hot` (an insert or
// erase batch: k_bin_hot).
// SET: the ops of table t are [off[t], off[t + 1]) and go to bins of its range;
// a block's ops then fall into a short range of bins (its records land in long
// runs), and ops outside a range of kSplitBins take their places one by one.
// tile_ops (at most PER * 512, a multiple of 512): the ops a block takes, so
// that the blocks come to whole waves. Loads go out kLoad ops at a time: in a
// set's split the records it may write kept the compiler from grouping them,
// and with three blocks an SM a 2^25-op round's split took 189 us, not 297 (a
// single table's waits for its stores either way: two blocks, 47 us for 2^22).
// A single table's chunk starts here: the call counters (ctr), A.ctr and the
// result bits are zeroed and the single bits set (k_set_prep does so for a
// set). The bin counts, cursors and state are zero on entry: k_bin_group
// leaves them so.
template <int KB, int PER, bool SET, bool HOT>
__global__ void __launch_bounds__(kSplitThreads, SET ? 3 : 2) k_bin_scatter(
    const __grid_constant__ BinScratch B, const __grid_constant__ ApplyScratch A,
    const uint32_t *__restrict__ off, const uint8_t *__restrict__ ops,
    const void *__restrict__ keys, uint64_t n, unsigned long long *ctr, uint32_t *bits,
    uint32_t tile_ops) {
    after_previous();
    using K = typename SlotT<KB>::K;
    static_assert(PER * kSplitThreads <= 1 << 13 && kSplitBins <= 1 << 13, "a place and a bin take 13 bits each");
    __shared__ uint32_t s_cnt[kSplitBins];
    if (HOT && B.state[kBinOver] == 0u) return;
    uint32_t *cursor = HOT ? B.cursor : B.count;
    const uint64_t gid = (uint64_t)blockIdx.x * kSplitThreads + threadIdx.x;
    if (SET) n = set_op_count(A, off);
    if (SET && !HOT) {
        // offsets that disagree with the host's, or are out of order, are
        // reported (every access below stays inside the scratch either way)
        if (gid == 0 && ((uint64_t)off[A.ntables] != A.ctr[kCtrHostN] || off[0] != 0u))
            note_bad(A, kCtrBadOffsets);
        for (uint64_t t = gid; t < A.ntables; t += (uint64_t)gridDim.x * kSplitThreads)
            if (off[t] > off[t + 1]) note_bad(A, kCtrBadOffsets);
    }
    if (!SET && !HOT) {
        if (gid < sizeof(Counters) / 8 - 1) ctr[gid] = 0ull;
        if (A.ctr != nullptr && gid < (uint64_t)kCtrSlots) A.ctr[gid] = 0ull;
    }
    bool went_over = false, planned = false;
    auto put = [&](uint32_t b, uint32_t p, uint32_t tag, uint32_t word) {
        const unsigned long long r = (unsigned long long)tag | ((unsigned long long)word << 32);
        if (HOT) {
            B.hot[(uint64_t)B.start[b] + p] = r;
            return;
        }
        if (p < (uint32_t)kBinCap) B.rec[(uint64_t)b * kBinCap + p] = r;
        else went_over = true;
    };
    for (uint64_t tile = (uint64_t)blockIdx.x * tile_ops; tile < n; tile += (uint64_t)gridDim.x * tile_ops) {
        uint32_t lo = 0u, nb = B.nbins;
        if (SET) {
            const uint64_t last = (tile + tile_ops < n ? tile + tile_ops : n) - 1;
            const uint32_t t0 = table_at(A.tidx, off, (uint32_t)tile, (uint32_t)tile);
            const uint32_t t1 = table_at(A.tidx, off, (uint32_t)last, (uint32_t)last);
            const uint32_t hi = set_bin(off, t1, 0xffffffffu, n);
            lo = set_bin(off, t0, 0u, n);
            nb = hi >= lo ? hi - lo + 1u : 0u;
            const bool all = nb <= kSplitBins;
            if (!all) nb = kSplitBins;
            if (HOT && all) {  // no bin of the tile's tables went over
                bool any = false;
                for (uint32_t b2 = threadIdx.x; b2 < nb; b2 += kSplitThreads)
                    any |= B.count[lo + b2] > (uint32_t)kBinCap;
                if (!__syncthreads_or(any)) continue;
            }
        }
        if (HOT && !planned) {
            planned = true;
            plan_hot<KB>(B, SET ? (uint32_t)set_nbins(n) : B.nbins);
        }
        if (!SET && !HOT) {
            const uint64_t words = ((tile + tile_ops < n ? tile + tile_ops : n) + 31) / 32;
            for (uint64_t w = tile / 32 + threadIdx.x; w < words; w += kSplitThreads) {
                B.single[w] = 0xffffffffu;
                if (bits != nullptr) bits[w] = 0u;
            }
        }
        for (uint32_t b = threadIdx.x; b < nb; b += kSplitThreads) s_cnt[b] = 0u;
        __syncthreads();
        // at: place | bin - lo << 13 | op code << 26; ~0: key 0, or done
        uint32_t tag[PER], at[PER];
        constexpr int kLoad = 8;
        K key[kLoad];
        uint8_t op[kLoad];
        const uint64_t end = tile + tile_ops < n ? tile + tile_ops : n;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (j % kLoad == 0) {  // loads in flight together
#pragma unroll
                for (int x = 0; x < kLoad; ++x) {
                    const uint64_t i = tile + (uint64_t)(j + x) * kSplitThreads + threadIdx.x;
                    key[x] = i < end ? load_key<KB>(keys, i) : (K)0;
                    op[x] = (ops != nullptr && i < end) ? ops[i] : (uint8_t)kOpFind;
                }
            }
            const uint64_t i = tile + (uint64_t)j * kSplitThreads + threadIdx.x;
            const K k = key[j % kLoad];
            const uint32_t code = op_word(0, op[j % kLoad]);
            tag[j] = bin_tag(k);
            at[j] = 0xffffffffu;
            if (k == 0) continue;
            uint32_t b;
            if (SET) {
                const uint32_t t = table_at(A.tidx, off, (uint32_t)i, (uint32_t)i);
                b = set_bin(off, t, cell_hash((uint64_t)k), n);
                tag[j] ^= table_mix(t);
            } else {
                b = bin_of<KB>(k, nb);
            }
            if (HOT && B.count[b] <= (uint32_t)kBinCap) continue;
            if (!SET || b - lo < nb) at[j] = (b - lo) << 13 | code << 26;
            else put(b, atomicAdd(&cursor[b], 1u), tag[j], rec_word(A, (uint32_t)i, code));
        }
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (at[j] != 0xffffffffu) at[j] |= atomicAdd(&s_cnt[(at[j] >> 13) & 0x1fffu], 1u);
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < nb; b += kSplitThreads) {
            const uint32_t c = s_cnt[b];
            if (c) s_cnt[b] = atomicAdd(&cursor[lo + b], c);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (at[j] == 0xffffffffu) continue;
            const uint32_t b = (at[j] >> 13) & 0x1fffu, p = s_cnt[b] + (at[j] & 0x1fffu);
            const uint32_t i = (uint32_t)tile + (uint32_t)j * kSplitThreads + threadIdx.x;
            put(lo + b, p, tag[j], rec_word(A, i, at[j] >> 26));
        }
        __syncthreads();  // the counts are reused by the next tile
    }
    if (!HOT && went_over) B.state[kBinOver] = 1u;
}

// The pass HOT of an insert or erase batch. Of a key's ops in a tile only one
// can count in the batch (the last of an insert's, the first of an erase's): the
// others lose their single bit here and get no record, so the block of a bin
// that went over streams a record per key and tile, not one per op. Each op
// leaves its place in its key's cell by a plain store; where another key stays
// there, its ops all get records. With a record per op that block took nearly
// all of a call: 2^22 inserts of 8-byte keys, one key 12.7 ms (now 0.15), Zipf
// 1.2 2.49 (0.21), a tenth of the ops on one key 1.62 (0.28), distinct keys 0.25.
// Losing bits are cleared a word a warp; by an atomic per op, 1500 keys took 282
// us for 251.
template <int KB, int MODE>
__global__ void __launch_bounds__(kSplitThreads, 2) k_bin_hot(
    const __grid_constant__ BinScratch B, const __grid_constant__ ApplyScratch A,
    const void *__restrict__ keys, uint64_t n) {
    after_previous();
    using K = typename SlotT<KB>::K;
    static_assert(MODE == kBinModeInsert || MODE == kBinModeErase, "one op of a key counts");
    constexpr int kPer = 8;
    constexpr uint32_t kTile = kPer * kSplitThreads, kNone = 0xffffffffu;
    static_assert(kTile == 1u << 12, "a cell per op of the tile, 12 bits");
    __shared__ uint16_t s_first[kTile];
    __shared__ uint32_t s_best[kTile];
    __shared__ uint32_t s_cnt[kSplitBins];  // records per bin, then where they go
    if (B.state[kBinOver] == 0u) return;
    plan_hot<KB>(B, B.nbins);
    for (uint64_t tile = (uint64_t)blockIdx.x * kTile; tile < n; tile += (uint64_t)gridDim.x * kTile) {
        for (uint32_t c = threadIdx.x; c < kTile; c += kSplitThreads)
            s_best[c] = MODE == kBinModeInsert ? 0u : kNone;
        for (uint32_t b = threadIdx.x; b < B.nbins; b += kSplitThreads) s_cnt[b] = 0u;
        K key[kPer];
        uint32_t cell[kPer];  // kNone: not an op of a bin that went over
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint64_t i = tile + (uint64_t)j * kSplitThreads + threadIdx.x;
            key[j] = i < n ? load_key<KB>(keys, i) : (K)0;
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            cell[j] = kNone;
            if (key[j] == 0 || B.count[bin_of<KB>(key[j], B.nbins)] <= (uint32_t)kBinCap) continue;
            cell[j] = bin_cell<12>(bin_tag(key[j]));
            s_first[cell[j]] = (uint16_t)(j * kSplitThreads + threadIdx.x);
        }
        __syncthreads();
        bool same[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (cell[j] == kNone) continue;
            const uint32_t at = j * kSplitThreads + threadIdx.x, lead = s_first[cell[j]];
            same[j] = lead == at || load_key<KB>(keys, tile + lead) == key[j];
            if (!same[j]) continue;
            if (MODE == kBinModeInsert) atomicMax(&s_best[cell[j]], at);
            else atomicMin(&s_best[cell[j]], at);
        }
        __syncthreads();
        uint32_t at[kPer];  // place among the tile's records of the bin
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint32_t x = j * kSplitThreads + threadIdx.x;
            const bool out = cell[j] != kNone && same[j] && s_best[cell[j]] != x;
            if (out) cell[j] = kNone;
            // a warp's ops share a bitmap word, so far all ones
            const unsigned outs = __ballot_sync(kFull, out);
            if (outs && (threadIdx.x & 31) == 0) B.single[((uint32_t)tile + x) >> 5] = ~outs;
            if (cell[j] != kNone) at[j] = atomicAdd(&s_cnt[bin_of<KB>(key[j], B.nbins)], 1u);
        }
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < B.nbins; b += kSplitThreads)
            if (s_cnt[b]) s_cnt[b] = B.start[b] + atomicAdd(&B.cursor[b], s_cnt[b]);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (cell[j] == kNone) continue;
            const uint32_t i = (uint32_t)tile + j * kSplitThreads + threadIdx.x;
            B.hot[(uint64_t)s_cnt[bin_of<KB>(key[j], B.nbins)] + at[j]] =
                (unsigned long long)bin_tag(key[j]) | ((unsigned long long)rec_word(A, i, 0u) << 32);
        }
        __syncthreads();  // the cells are reused by the next tile
    }
}

// A bin that went over (few keys, each repeated many times, or a skewed
// batch's most popular ones): the block streams the bin's records twice, first
// to count each key in a table in shared memory, then to give every op its
// place. The table takes kHotMax keys; a bin with more is taken in parts by
// further mixed bits of the key, split again until they fit, so every bin is
// resolved whatever its keys.
// kHotMax is above a bin's ordinary keys (kBinMean and some), or a bin with one
// popular key more would be split in two half of the time.
constexpr uint32_t kHotTab = 2048, kHotMax = 1472;

struct HotSmem {
    uint32_t first[kHotTab];  // index + 1 of an op with the cell's key
    uint32_t cnt[kHotTab];    // ops of the key; insert / erase: the op that counts
    uint32_t off[kHotTab];    // next place in seg (~0: the key has one op)
    uint16_t id[kHotTab];
    uint64_t part_mask[72], part[72];  // parts to do (each split adds one)
    uint32_t top, nkey, nseg, nwarp, nmid, ndist, over, ok;
    unsigned long long bkey, bseg, bwarp, bmid;
};

// 64 mixed bits of a key, different for different keys (splitmix64's finalizer).
__device__ __forceinline__ uint64_t part_bits(uint64_t k) {
    k = (k ^ (k >> 30)) * 0xBF58476D1CE4E5B9ull;
    k = (k ^ (k >> 27)) * 0x94D049BB133111EBull;
    return k ^ (k >> 31);
}

// List key d (its segment at `at`) by its number of ops, for k_repeat.
__device__ __forceinline__ void list_long(const ApplyScratch &A, uint32_t d, uint32_t c,
                                          uint32_t *nwarp, uint32_t *nmid,
                                          unsigned long long bwarp, unsigned long long bmid) {
    if (c > kWarpSeg) A.mid[bmid + atomicAdd(nmid, 1u)] = d;
    else if (c > kShortSeg) A.wseg[bwarp + atomicAdd(nwarp, 1u)] = d;
}

// A block's ranges of the listed keys, their ops and the long-segment lists;
// false when they would not fit (counts this batch cannot have produced).
__device__ __forceinline__ bool take_ranges(const ApplyScratch &A, uint32_t nkey, uint32_t nseg,
                                            uint32_t nwarp, uint32_t nmid, unsigned long long &bkey,
                                            unsigned long long &bseg, unsigned long long &bwarp,
                                            unsigned long long &bmid) {
    bkey = atomicAdd(&A.ctr[kCtrDistinct], (unsigned long long)nkey);
    bseg = atomicAdd(&A.ctr[kCtrPlaced], (unsigned long long)nseg);
    bwarp = nwarp ? atomicAdd(&A.ctr[kCtrWarp], (unsigned long long)nwarp) : 0ull;
    bmid = nmid ? atomicAdd(&A.ctr[kCtrMid], (unsigned long long)nmid) : 0ull;
    const bool ok = bkey + nkey <= A.cap_ops && bseg + nseg <= A.cap_ops &&
                    bwarp + nwarp <= A.cap_ops && bmid + nmid <= A.cap_ops;
    if (!ok) note_bad(A);
    return ok;
}

// The table of op i of a set batch's bin (bin_tables: its first table, and 1
// when that is the only one).
__device__ __forceinline__ uint32_t bin_table(const ApplyScratch &A, const uint32_t *off, uint2 tables,
                                              uint32_t i) {
    return tables.y ? tables.x : table_at(A.tidx, off, i, i);
}

template <int KB, int MODE, bool SET>
__device__ __noinline__ void group_hot(const BinScratch &B, const ApplyScratch &A, const void *keys,
                                       uint32_t bin, uint32_t m, const uint32_t *off, HotSmem &M) {
    using K = typename SlotT<KB>::K;
    const uint32_t tid = threadIdx.x, lane = tid & 31, nt = kGroupThreads;
    const unsigned long long *rec = B.hot + B.start[bin];
    const uint2 tables = SET ? B.tables[bin] : make_uint2(0u, 1u);
    auto table_of_op = [&](uint32_t i) { return bin_table(A, off, tables, i); };
    // record r, of a key of the part: its key, table, tag, op index and word. (A
    // bin's tables are at most kSetBinMean, so that many of its keys share one
    // of these sums at most, and a part of one sum fits.)
    static_assert(kSetBinMean <= kHotMax, "a part that cannot be split further fits");
    uint64_t mask = 0ull, part = 0ull;
    auto op_at = [&](uint32_t r, K &k, uint32_t &t, uint32_t &tag, uint32_t &i, uint32_t &w) -> bool {
        if (r >= m) return false;
        tag = (uint32_t)rec[r];
        w = (uint32_t)(rec[r] >> 32);
        i = rec_index(A, w);
        k = load_key<KB>(keys, i);
        t = SET ? table_of_op(i) : 0u;
        return (part_bits((uint64_t)k + (uint64_t)t * 0x9E3779B97F4A7C15ull) & mask) == part;
    };
    // the cell of key k of table t; claimed for op i when it has none yet (claim)
    auto cell_of = [&](K k, uint32_t t, uint32_t tag, uint32_t i, bool claim) -> uint32_t {
        uint32_t h = bin_cell<11>(tag);
        static_assert(kHotTab == 1u << 11, "bin_cell takes 11 bits");
        // claims stop at kHotMax keys, plus one per thread on the way: cells
        // stay free and the probe ends
        static_assert(kHotMax + kGroupThreads < kHotTab, "a free cell remains");
        while (true) {
            uint32_t f = *(volatile uint32_t *)&M.first[h];
            if (f == 0u) {
                if (!claim || *(volatile uint32_t *)&M.over) return h;
                f = atomicCAS(&M.first[h], 0u, i + 1u);
                if (f == 0u) {
                    if (atomicAdd(&M.ndist, 1u) >= kHotMax) *(volatile uint32_t *)&M.over = 1u;
                    return h;
                }
            }
            if (load_key<KB>(keys, f - 1u) == k && (!SET || tables.y || table_of_op(f - 1u) == t)) return h;
            h = (h + 1u) & (kHotTab - 1u);
        }
    };
    __syncthreads();
    if (tid == 0) {
        M.top = 1u;
        M.part_mask[0] = M.part[0] = 0ull;
    }
    __syncthreads();
    while (M.top != 0u) {
        const uint32_t top = M.top;
        mask = M.part_mask[top - 1];
        part = M.part[top - 1];
        for (uint32_t c = tid; c < kHotTab; c += nt) {
            M.first[c] = 0u;
            M.cnt[c] = MODE == kBinModeErase ? 0xffffffffu : 0u;
            M.off[c] = 0xffffffffu;
        }
        if (tid == 0) M.nkey = M.nseg = M.nwarp = M.nmid = M.ndist = M.over = 0u;
        __syncthreads();
        for (uint32_t r0 = 0; r0 < m; r0 += nt) {
            if (__any_sync(kFull, *(volatile uint32_t *)&M.over != 0u)) break;
            K k = 0;
            uint32_t t = 0u, tag = 0u, i = 0u, w = 0u;
            const bool sel = op_at(r0 + tid, k, t, tag, i, w);
            const uint32_t h = sel ? cell_of(k, t, tag, i, true) : 0u;
            __syncwarp();
            const unsigned peers = __match_any_sync(kFull, sel ? h : 0x80000000u | lane);
            if (MODE == kBinModeMixed) {
                if (sel && __ffs(peers) - 1 == (int)lane) atomicAdd(&M.cnt[h], __popc(peers));
            } else if (sel) {
                const uint32_t v = MODE == kBinModeInsert ? __reduce_max_sync(peers, i)
                                                          : __reduce_min_sync(peers, i);
                if (__ffs(peers) - 1 == (int)lane) {
                    if (MODE == kBinModeInsert) atomicMax(&M.cnt[h], v);
                    else atomicMin(&M.cnt[h], v);
                }
            }
        }
        __syncthreads();
        const bool over = M.over != 0u;
        __syncthreads();
        if (tid == 0) {
            if (over && mask == ~0ull) {  // only with offsets that are out of order
                note_bad(A);
                M.top = top - 1u;
            } else if (over) {  // two parts by one more bit; nothing has been written for this one
                M.part_mask[top - 1] = M.part_mask[top] = 2ull * mask + 1ull;
                M.part[top] = part | (mask + 1ull);
                M.top = top + 1u;
            } else {
                M.top = top - 1u;
            }
        }
        __syncthreads();
        if (over) continue;
        if constexpr (MODE == kBinModeMixed) {
            for (uint32_t c = tid; c < kHotTab; c += nt) {
                const uint32_t k = M.cnt[c];
                if (M.first[c] == 0u || k <= 1u) continue;
                M.off[c] = atomicAdd(&M.nseg, k);
                M.id[c] = (uint16_t)atomicAdd(&M.nkey, 1u);
                if (k > kShortSeg) atomicAdd(k > kWarpSeg ? &M.nmid : &M.nwarp, 1u);
            }
            __syncthreads();
            if (tid == 0) {
                M.ok = take_ranges(A, M.nkey, M.nseg, M.nwarp, M.nmid, M.bkey, M.bseg, M.bwarp, M.bmid);
                M.nwarp = M.nmid = 0u;
            }
            __syncthreads();
            if (!M.ok) continue;
            for (uint32_t c = tid; c < kHotTab; c += nt) {
                if (M.off[c] == 0xffffffffu) continue;
                const uint32_t d = (uint32_t)M.bkey + M.id[c], at = (uint32_t)M.bseg + M.off[c];
                ((K *)A.dkey)[d] = load_key<KB>(keys, M.first[c] - 1u);
                A.dcnt[d] = M.cnt[c];
                A.dseg[d] = (unsigned long long)at << 32;
                if (SET) A.dtid[d] = table_of_op(M.first[c] - 1u);
                list_long(A, d, M.cnt[c], &M.nwarp, &M.nmid, M.bwarp, M.bmid);
                M.off[c] = at;
            }
            __syncthreads();
        }
        uint32_t ins = 0u;
        for (uint32_t r0 = 0; r0 < m; r0 += nt) {
            K k = 0;
            uint32_t t = 0u, tag = 0u, i = 0u, w = 0u;
            const bool sel = op_at(r0 + tid, k, t, tag, i, w);
            const uint32_t h = sel ? cell_of(k, t, tag, i, false) : 0u;
            if constexpr (MODE == kBinModeMixed) {
                const bool several = sel && M.cnt[h] > 1u;
                if (SET && sel && !several && (w & 1u)) {
                    if (tables.y) ++ins;
                    else atomicAdd(&A.tup[t], 1u);
                }
                __syncwarp();
                const unsigned peers = __match_any_sync(kFull, several ? h : 0x80000000u | lane);
                const int lead = __ffs(peers) - 1;
                uint32_t at = 0u;
                if (several && lead == (int)lane) at = atomicAdd(&M.off[h], __popc(peers));
                at = __shfl_sync(kFull, at, lead) + __popc(peers & ((1u << lane) - 1u));
                if (several) {
                    A.seg[at] = seg_word(A, w);
                    clear_single(B, i);
                }
            } else if (sel && M.cnt[h] != i) {
                clear_single(B, i);
            }
        }
        if (SET && MODE == kBinModeMixed) {
            ins = __reduce_add_sync(kFull, ins);
            if (lane == 0 && ins) atomicAdd(&A.tup[tables.x], ins);
        }
        __syncthreads();
    }
}

template <bool SET> struct GroupSmem {
    uint32_t tag[kBinCap], word[kBinCap], cnt[kBinCap], tab[kBinCap];
    uint16_t first[kGroupTab];
    // in a bin of several tables: a record's table (its id from the first
    // one's on; kBinOffs: looked up by op), where the tables end, and the
    // inserts that count for each
    uint8_t table[SET ? kBinCap : 1];
    uint32_t off[SET ? kBinOffs : 1], ins[SET ? kBinOffs : 1];
};
template <bool SET> constexpr size_t kGroupSmem = sizeof(GroupSmem<SET>);

// One block per bin: its ops grouped by key in shared memory. Insert batches
// keep the single bit of a key's last op, erase batches of its first. In a
// mixed batch the ops of keys with several ops lose theirs and the keys are
// listed: id d gets dkey, dcnt, dseg and (SET) dtid, and its op indexes a
// range of seg; ids with more than kShortSeg ops go to wseg or mid as well.
// SET: the inserts among the other ops are counted as upserts of their tables
// (the upsize policy's insert batch); sized: the grid is the batch's bins.
// A record leaves its number in its key's cell with a plain store; the record
// that stays leads the key's group, and most records find themselves there.
// Only records whose cell another key has claim one in a second table by
// compare-and-swap, and only a group's further records count themselves in:
// with one swap and one count for every record 2^22 erases took 26 us (now 19)
// and 2^22 mixed ops 42 (now 27, of which 7 from fewer barriers and segments
// written without a stop in shared memory).
template <int KB, int MODE, bool SET>
__global__ void __launch_bounds__(kGroupThreads, 4) k_bin_group(
    const __grid_constant__ BinScratch B, const __grid_constant__ ApplyScratch A,
    const uint32_t *__restrict__ off, const void *__restrict__ keys, bool sized) {
    after_previous();
    using K = typename SlotT<KB>::K;
    using Smem = GroupSmem<SET>;
    __shared__ __align__(16) unsigned char s_raw[sizeof(Smem)];
    static_assert(sizeof(HotSmem) <= sizeof(Smem), "one block of shared memory for both");
    Smem &M = *reinterpret_cast<Smem *>(s_raw);
    __shared__ uint32_t s_place, s_nwarp, s_nmid, s_ok, s_ins;  // place: ops | keys << 16
    __shared__ unsigned long long s_bseg, s_bkey, s_bwarp, s_bmid;
    const uint32_t tid = threadIdx.x, bin = blockIdx.x;
    // nothing there, and no counts to zero
    if (SET && !sized && bin >= set_nbins(set_op_count(A, off))) return;
    const uint2 tables = SET ? B.tables[bin] : make_uint2(0u, 1u);
    const bool one = tables.y != 0u;
    // the first kGroupPre rounds of records are read along with their count
    unsigned long long x[kGroupR];
#pragma unroll
    for (int q = 0; q < kGroupPre; ++q) x[q] = B.rec[(uint64_t)bin * kBinCap + q * kGroupThreads + tid];
    const uint32_t count = B.count[bin];
    if (count == 0u) {
        if (bin == 0 && tid < (uint32_t)kBinStates) B.state[tid] = 0u;
        return;
    }
    // the records written to `hot`: all of the bin's ops, except those that
    // cannot count (k_bin_hot), and where device offsets that are out of order
    // put ops in bins outside their tile's range
    const uint32_t nhot = count > (uint32_t)kBinCap ? B.cursor[bin] : 0u;
    // with one record a key and tile most bins that went over fit after all
    // (32768 inserts, a tenth of them on one key: 61 us by group_hot, 47 here)
    const bool again = MODE != kBinModeMixed && count > (uint32_t)kBinCap && nhot <= (uint32_t)kBinCap;
    const uint32_t m = again ? nhot : count;
    for (uint32_t c = tid; c < (uint32_t)kBinCap; c += kGroupThreads) M.tab[c] = 0u;
    if (tid == 0) s_place = s_nwarp = s_nmid = s_ins = 0u;
    if (m <= (uint32_t)kBinCap) {
        const unsigned long long *rec = again ? B.hot + B.start[bin] : B.rec + (uint64_t)bin * kBinCap;
#pragma unroll
        for (int q = 0; q < kGroupR; ++q) {
            const uint32_t r = q * kGroupThreads + tid;
            if (r < m && (q >= kGroupPre || again)) x[q] = rec[r];
        }
#pragma unroll
        for (int q = 0; q < kGroupR; ++q) {
            const uint32_t r = q * kGroupThreads + tid;
            if (r < m) {
                const uint32_t tag = (uint32_t)x[q], w = (uint32_t)(x[q] >> 32);
                M.tag[r] = tag;
                M.word[r] = w;
                M.cnt[r] = MODE == kBinModeMixed ? 0u : w;
                M.first[bin_cell<12>(tag)] = (uint16_t)r;  // one of the cell's records stays
            }
        }
        if (SET && !one && tid < kBinOffs) {
            const uint32_t t = tables.x + 1u + tid;
            M.off[tid] = off[t < A.ntables ? t : A.ntables];
            M.ins[tid] = 0u;
        }
    }
    __syncthreads();
    // every thread has read the counts: the next batch finds them, and the
    // split's state, zero
    if (tid == 0) B.count[bin] = B.cursor[bin] = 0u;
    if (bin == 0 && tid < (uint32_t)kBinStates) B.state[tid] = 0u;
    if (m > (uint32_t)kBinCap) {
        group_hot<KB, MODE, SET>(B, A, keys, bin, nhot, off, *reinterpret_cast<HotSmem *>(s_raw));
        return;
    }
    if (SET && !one) {
        for (uint32_t r = tid; r < m; r += kGroupThreads) {
            const uint32_t i = rec_index(A, M.word[r]);
            uint32_t t = 0u;  // ends up to and with i
#pragma unroll
            for (uint32_t w = kBinOffs / 2; w; w >>= 1)
                if (M.off[t + w - 1u] <= i) t += w;
            M.table[r] = (uint8_t)(t + (M.off[t] <= i ? 1u : 0u));
        }
        __syncthreads();
    }
    uint32_t lr[kGroupR];  // the key's lead record | the op's rank << 16
    // the table of record r, op i
    auto table_rec = [&](uint32_t r, uint32_t i) -> uint32_t {
        if (!SET || one) return tables.x;
        return M.table[r] == kBinOffs ? table_at(A.tidx, off, i, i) : tables.x + M.table[r];
    };
    static_assert(kGroupTab == 1 << 12 && kBinCap == 1 << 11, "cells of 12 and 11 bits");
#pragma unroll
    for (int q = 0; q < kGroupR; ++q) {
        const uint32_t r = q * kGroupThreads + tid;
        lr[q] = r;
        if (r >= m) continue;
        const uint32_t tag = M.tag[r], w = M.word[r];
        auto same = [&](uint32_t x) {
            if (x == r) return true;
            if (M.tag[x] != tag) return false;
            if (KB == 4 && (!SET || one)) return true;
            const uint32_t i = rec_index(A, w), j = rec_index(A, M.word[x]);
            if (KB != 4 && load_key<KB>(keys, j) != load_key<KB>(keys, i)) return false;
            if (!SET || one || M.table[x] != M.table[r]) return !SET || one;
            // 4-byte keys: tag and table give the key
            return M.table[r] != kBinOffs || table_rec(x, j) == table_rec(r, i);
        };
        uint32_t lead = M.first[bin_cell<12>(tag)];
        if (!same(lead)) {
            // another key has the cell: at most kBinCap - 1 records come here, so
            // a cell of the second table stays free and the probe ends
            uint32_t h = bin_cell<23>(tag) & (kBinCap - 1);
            while (true) {
                const uint32_t old = atomicCAS(&M.tab[h], 0u, r + 1u);
                lead = old == 0u ? r : old - 1u;
                if (old == 0u || same(lead)) break;
                h = (h + 1u) & (kBinCap - 1);
            }
        }
        if (lead == r) continue;
        if (MODE == kBinModeInsert) atomicMax(&M.cnt[lead], w);
        else if (MODE == kBinModeErase) atomicMin(&M.cnt[lead], w);
        else lr[q] = lead | (atomicAdd(&M.cnt[lead], 1u) + 1u) << 16;
        if (MODE != kBinModeMixed) lr[q] = lead;
    }
    __syncthreads();
    if constexpr (MODE != kBinModeMixed) {
#pragma unroll
        for (int q = 0; q < kGroupR; ++q) {
            const uint32_t r = q * kGroupThreads + tid;
            if (r < m && M.cnt[lr[q]] != M.word[r]) clear_single(B, rec_index(A, M.word[r]));
        }
    } else {
        // the second table's cells now hold each key's place in its block's ranges
        uint32_t ins = 0u;
#pragma unroll
        for (int q = 0; q < kGroupR; ++q) {
            const uint32_t r = q * kGroupThreads + tid, lead = lr[q] & 0xffffu;
            if (r >= m) continue;
            const uint32_t c = M.cnt[lead] + 1u;
            if (c == 1u) {
                if (SET && (M.word[r] & 1u)) {
                    if (one) ++ins;
                    else if (M.table[r] != kBinOffs) atomicAdd(&M.ins[M.table[r]], 1u);
                    else atomicAdd(&A.tup[table_rec(r, rec_index(A, M.word[r]))], 1u);
                }
            } else if (lead == r) {
                M.tab[r] = atomicAdd(&s_place, c | 1u << 16);
                if (c > kShortSeg) atomicAdd(c > kWarpSeg ? &s_nmid : &s_nwarp, 1u);
            }
        }
        if (SET) {
            ins = __reduce_add_sync(kFull, ins);
            if ((tid & 31) == 0 && ins) atomicAdd(&s_ins, ins);
        }
        __syncthreads();
        if (SET && tid == 0 && s_ins) atomicAdd(&A.tup[tables.x], s_ins);
        if (SET && !one && tid < kBinOffs && M.ins[tid]) atomicAdd(&A.tup[tables.x + tid], M.ins[tid]);
        if (s_place == 0u) return;
        if (tid == 0) {
            s_ok = take_ranges(A, s_place >> 16, s_place & 0xffffu, s_nwarp, s_nmid, s_bkey, s_bseg,
                               s_bwarp, s_bmid);
            s_nwarp = s_nmid = 0u;
        }
        __syncthreads();
        if (!s_ok) return;
#pragma unroll
        for (int q = 0; q < kGroupR; ++q) {
            const uint32_t r = q * kGroupThreads + tid, lead = lr[q] & 0xffffu;
            if (r >= m) continue;
            const uint32_t c = M.cnt[lead] + 1u;
            if (c == 1u) continue;
            const uint32_t w = M.word[r], i = rec_index(A, w);
            const uint32_t place = (uint32_t)s_bseg + (M.tab[lead] & 0xffffu);
            A.seg[place + (lr[q] >> 16)] = seg_word(A, w);
            clear_single(B, i);
            if (lead == r) {
                const uint32_t d = (uint32_t)s_bkey + (M.tab[lead] >> 16);
                const uint32_t t = table_rec(r, i);
                ((K *)A.dkey)[d] = KB == 4 ? (K)(M.tag[r] ^ table_mix(t)) : load_key<KB>(keys, i);
                A.dcnt[d] = c;
                A.dseg[d] = (unsigned long long)place << 32;
                if (SET) A.dtid[d] = t;
                list_long(A, d, c, &s_nwarp, &s_nmid, s_bwarp, s_bmid);
            }
        }
    }
}

// A lane's key and what the probes of its two buckets found.
template <int KB> struct RepKey {
    typename SlotT<KB>::K k;
    uint32_t tb, hk;
    char *p1, *p2;
    KvOut r1, r2;
    bool found1, found2, pre;
    uint64_t pre_value;
};

// Key k of every lane with act in table D (warp-collective).
template <int KB, int SB>
__device__ __forceinline__ RepKey<KB> probe_key(const Desc &D, typename SlotT<KB>::K k, bool act,
                                                unsigned char *stage) {
    using Gm = Geo<KB, SB>;
    RepKey<KB> x;
    x.k = k;
    x.tb = 0u;
    x.hk = fold(k);
    const Pair p = pair_of(x.hk, D.d);
    x.p1 = bucket_ptr<KB, SB>(D, p.first, bucket_index(D, p.first, x.hk));
    x.p2 = bucket_ptr<KB, SB>(D, p.second, bucket_index(D, p.second, x.hk));
    x.r1 = place_probe<KB, SB, false>(x.p1, k, act, p.first, D.d, stage);
    x.found1 = act && x.r1.match >= 0;
    // the second bucket: where the key or an empty slot may be there
    const bool check2 = act && !x.found1 && ((!Gm::kMeta || x.r1.overflow) || x.r1.empty == 0u);
    x.r2 = KvOut{-1, 0ull, false, 0u};
    if (__any_sync(kFull, check2))
        x.r2 = place_probe<KB, SB, false>(x.p2, k, check2, p.second, D.d, stage);
    x.found2 = check2 && x.r2.match >= 0;
    x.pre = x.found1 || x.found2;
    x.pre_value = x.found1 ? x.r1.value : (x.found2 ? x.r2.value : 0ull);
    return x;
}

// An op word of a segment (SegOps::wide: a plain index).
struct SegOps {
    const uint8_t *ops;
    uint32_t wide;
    __device__ __forceinline__ uint32_t index(uint32_t w) const { return wide ? w : w >> 2; }
    __device__ __forceinline__ uint8_t code(uint32_t w) const {
        return wide ? ops[w] : (uint8_t)(w & 3u);  // 1 insert, 2 erase; others read
    }
};
static_assert(kOpInsert == 1 && kOpErase == 2, "a segment's op codes are the ops'");

// Replay of the op words idx[0..cnt) (op indices in increasing order) by the
// whole block, an op a thread at a time: an op's state comes from the latest
// mutation before it in its warp (a ballot), else in the warps before, else
// from the state carried in; present / value carry the key's state in every
// thread. (By one warp, 32 ops a step, a batch of 2^22 ops on 5000 keys took 764
// us, the other warps idle; by all 663.)
template <int THREADS, bool WRITE>
__device__ __forceinline__ void block_replay(const uint32_t *idx, uint32_t cnt, bool &present,
                                             uint64_t &value, const SegOps &ops,
                                             const void *__restrict__ vals, uint32_t vb,
                                             void *__restrict__ vals_out,
                                             uint32_t *__restrict__ bits_out) {
    // a warp's latest mutation: 0 none, 1 erase, 2 insert, and its value
    constexpr uint32_t kWarps = THREADS / 32;
    __shared__ uint32_t s_kind[2][kWarps];
    __shared__ uint64_t s_val[2][kWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t buf = 0u;
    for (uint32_t c0 = 0; c0 < cnt; c0 += THREADS, buf ^= 1u) {
        const bool v = c0 + threadIdx.x < cnt;
        const uint32_t w = v ? idx[c0 + threadIdx.x] : 0u, i = ops.index(w);
        const uint8_t op = v ? ops.code(w) : (uint8_t)kOpFind;
        const bool mut = op == kOpInsert || op == kOpErase;  // other codes read
        const uint64_t myval = op == kOpInsert ? load_val(vals, vb, i) : 0ull;
        const unsigned mm = __ballot_sync(kFull, mut);
        const unsigned before = mm & ((1u << lane) - 1u);
        const int src = before ? 31 - __clz(before) : (int)lane;
        const uint32_t kind = mut ? (op == kOpInsert ? 2u : 1u) : 0u;
        const uint64_t srcval = shfl64(myval, src);
        const uint32_t srckind = __shfl_sync(kFull, kind, src);
        if ((int)lane == (mm ? 31 - __clz(mm) : 0)) {
            s_kind[buf][warp] = kind;
            s_val[buf][warp] = myval;
        }
        __syncthreads();  // the other buffer is written in the next step
        bool st = present;
        uint64_t sval = value;
#pragma unroll
        for (uint32_t x = 0; x < kWarps; ++x) {
            if (x == warp) {
                st = present;
                sval = value;
            }
            const uint32_t k = s_kind[buf][x];
            if (k == 0u) continue;
            present = k == 2u;
            value = s_val[buf][x];  // 0 of an erase
        }
        if (before) {
            st = srckind == 2u;
            sval = srcval;
        }
        if (WRITE && v) {
            if (vals_out) store_val(vals_out, vb, i, st ? sval : 0ull);
            if (st && bits_out) atomicOr(&bits_out[i >> 5], 1u << (i & 31));
        }
    }
}

struct RepCounts {
    uint32_t ins = 0, upd = 0, del = 0;
};

// The final state of a lane's key (act) to the table; entries without a slot
// go to list_a. Warp-collective.
template <int KB, int SB>
__device__ __forceinline__ void mutate_listed(const RepKey<KB> &x, bool up, bool er, uint64_t value,
                                              void *list_a, uint64_t list_cap, Counters *gctr,
                                              RepCounts &n) {
    using T = SlotT<KB>;
    typename T::S e = T::empty();
    bool pend = false;
    if (up) {
        e = T::make(x.k, value);
        if (x.found1) {
            T::store(slot_ptr<KB, SB>(x.p1, x.r1.match), e);
            ++n.upd;
        } else if (x.found2) {
            T::store(slot_ptr<KB, SB>(x.p2, x.r2.match), e);
            ++n.upd;
        } else {
            bool ok = claim_empty<KB, SB>(x.p1, x.r1.empty, e);
            if (!ok && x.r2.empty) {
                mark_overflow<KB, SB>(x.p1, x.hk);
                ok = claim_empty<KB, SB>(x.p2, x.r2.empty, e);
            }
            if (ok) ++n.ins;
            else pend = true;
        }
    } else if (er) {
        T::store(x.found1 ? slot_ptr<KB, SB>(x.p1, x.r1.match) : slot_ptr<KB, SB>(x.p2, x.r2.match),
                 T::empty());
        ++n.del;
    }
    __syncwarp();
    const unsigned long long at = agg_inc(&gctr->pending, pend);
    if (pend) {
        if (at < list_cap) ((typename T::S *)list_a)[at] = e;
        else atomicAdd(&gctr->spill, 1ull);
    }
}

// Ascending sort of s[0..c) by one warp (mirrored bitonic merges: every
// compare is ascending, so the places past c, read as larger than any word,
// need no storage).
__device__ __forceinline__ void warp_sort_words(uint32_t *s, uint32_t c) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t P = 2;
    while (P < c) P <<= 1;
    for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t q = lane; q < P / 2; q += 32) {
                // pair q of the stage: t below, u above
                const uint32_t t = (q / j) * 2 * j + (q % j);
                const uint32_t u = j == k >> 1 ? (t ^ (k - 1)) : t + j;
                if (u < c) {
                    const uint32_t a = s[t], b = s[u];
                    if (a > b) {
                        s[t] = b;
                        s[u] = a;
                    }
                }
            }
            __syncwarp();
        }
    }
}

// Results of the sorted op words w[0..c) of one key by one warp, 32 ops a step
// (as block_replay): present / value carry the key's state.
template <bool WRITE>
__device__ __forceinline__ void warp_replay_words(const uint32_t *w, uint32_t c, bool &present,
                                                  uint64_t &value, const void *__restrict__ vals,
                                                  uint32_t vb, void *__restrict__ vals_out,
                                                  uint32_t *__restrict__ bits_out) {
    const int lane = threadIdx.x & 31;
    for (uint32_t c0 = 0; c0 < c; c0 += 32) {
        const bool v = c0 + lane < c;
        const uint32_t x = v ? w[c0 + lane] : 0u, i = x >> 2, op = x & 3u;
        const uint64_t myval = (v && op == 1u) ? load_val(vals, vb, i) : 0ull;
        const unsigned mm = __ballot_sync(kFull, v && op != 0u);
        const unsigned ins = __ballot_sync(kFull, v && op == 1u);
        const unsigned before = mm & ((1u << lane) - 1u);
        const int src = before ? 31 - __clz(before) : -1;
        const uint64_t srcval = shfl64(myval, src < 0 ? lane : src);
        bool st_present = present;
        uint64_t st_value = value;
        if (src >= 0) {
            st_present = (ins >> src) & 1u;
            st_value = st_present ? srcval : 0ull;
        }
        if (WRITE && v) {
            if (vals_out) store_val(vals_out, vb, i, st_present ? st_value : 0ull);
            if (st_present && bits_out) atomicOr(&bits_out[i >> 5], 1u << (i & 31));
        }
        if (mm) {
            const int last = 31 - __clz(mm);
            present = (ins >> last) & 1u;
            const uint64_t lv = shfl64(myval, last);
            value = present ? lv : 0ull;
        }
    }
}

constexpr uint32_t kBinShort = 8;   // ops of one key replayed by one lane
constexpr uint32_t kSmallLong = 512;  // most ops of one key replayed by one warp (k_bin_small)
constexpr uint32_t kTailWalk = 64;  // pending entries the last block places itself

template <int KB, int SB> struct BinSmem {
    alignas(128) unsigned char stage[kSmallWarps][32 * SB];  // between the probes: tables, bitmaps
    typename SlotT<KB>::K key[kSmallCap];
    uint32_t word[kSmallCap];
    // per first op of a key: the word that counts; mixed: its ops | place in seg << 16
    uint32_t cnt[kSmallCap];
    uint16_t multi[kSmallCap];  // keys with several ops, and those of more than kSmallLong
    uint16_t longs[kBinSmallOps / kSmallLong];  // each has more ops than that
    uint64_t part_mask[72], part[72];  // parts of a bin that went over (each split adds one)
    uint32_t m, nseg, nmulti, nlong, ndist, over, top, last;
    uint32_t warp_sum[kSmallWarps];
    unsigned long long sum[6];
    uint32_t seg[kSmallCap];  // the last member: mixed batches of more ops get a word for each
};

// Bytes of a small batch's BinSmem.
template <int KB, int SB> constexpr size_t bin_smem(int mode, uint64_t n) {
    return sizeof(BinSmem<KB, SB>) +
           (mode >= kBinModeMixed && n > (uint64_t)kSmallCap ? (n - kSmallCap) * sizeof(uint32_t) : 0);
}

// Key k's cell among the cells `cell` (index + 1 of an op of the cell's key);
// claimed for op i when it has none yet (claim). A probe of kSmallProbe cells
// (in a table half full they are one or two) gives its part up (M.over), so
// the cells never run out.
constexpr uint32_t kSmallProbe = 256;
template <int KB, int SB>
__device__ __forceinline__ uint32_t small_cell(BinSmem<KB, SB> &M, uint32_t *cell, const void *keys,
                                               typename SlotT<KB>::K k, uint32_t i, bool claim) {
    static_assert(kSmallTab == 1 << 11, "bin_cell takes 11 bits");
    uint32_t h = bin_cell<11>(bin_tag(k));
    for (uint32_t p = 0; p < kSmallProbe; ++p) {
        uint32_t f = *(volatile uint32_t *)&cell[h];
        if (f == 0u) {
            if (!claim) return h;
            f = atomicCAS(&cell[h], 0u, i + 1u);
            if (f == 0u) return h;
        }
        if (load_key<KB>(keys, f - 1u) == k) return h;
        h = (h + 1u) & (kSmallTab - 1);
    }
    *(volatile uint32_t *)&M.over = 1u;
    return h;
}

// f(key, index, bin's own) for the ops of a batch, 32 to a warp, until stop();
// down: from the last op to the first.
template <int KB, int kLoad, class F, class Stop>
__device__ __forceinline__ void stream_batch(const void *keys, uint32_t n, bool down, Stop &&stop, F &&f) {
    using K = typename SlotT<KB>::K;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t base = threadIdx.x & ~31u; base < n; base += kLoad * kSmallThreads) {
        if (stop()) break;
        K k[kLoad];
#pragma unroll
        for (int x = 0; x < kLoad; ++x) {
            const uint32_t i = base + x * kSmallThreads + lane;
            k[x] = i < n ? load_key<KB>(keys, down ? n - 1u - i : i) : (K)0;
        }
#pragma unroll
        for (int x = 0; x < kLoad; ++x) {
            const uint32_t i = base + x * kSmallThreads + lane;
            f(k[x], down ? n - 1u - i : i, i < n);
        }
    }
}

// After the ops of the next part (top of M.part) of a bin have their cells: the
// places of a thread's used cells among the part's keys. False, and the part
// split in two by one more bit of its keys, when they are more than kSmallCap.
constexpr int kSmallCells = kSmallTab / kSmallThreads;
template <int KB, int SB>
__device__ __forceinline__ bool end_part(BinSmem<KB, SB> &M, const uint32_t *cell, uint32_t (&d)[kSmallCells]) {
    const uint32_t lane = threadIdx.x & 31;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kSmallCells; ++q) {
        const unsigned m = __ballot_sync(kFull, cell[q * kSmallThreads + threadIdx.x] != 0u);
        uint32_t at = 0u;
        if (lane == 0 && m) at = atomicAdd(&M.ndist, (uint32_t)__popc(m));
        d[q] = __shfl_sync(kFull, at, 0) + __popc(m & ((1u << lane) - 1u));
    }
    __syncthreads();
    const bool over = M.over != 0u || M.ndist > (uint32_t)kSmallCap;
    if (threadIdx.x == 0) {
        const uint32_t top = M.top;
        if (over) {
            const uint64_t mask = M.part_mask[top - 1];
            M.part[top] = M.part[top - 1] | (mask + 1ull);
            M.part_mask[top - 1] = M.part_mask[top] = 2ull * mask + 1ull;
            M.top = top + 1u;
        } else {
            M.top = top - 1u;
        }
    }
    return !over;
}

// An insert or erase batch's bin of more than kSmallCap ops (a popular key, or a
// few): the keys of its next part to M.key, streamed from the batch again, and
// the op of each that counts to M.word. Returns their number (0: the part was
// split). An insert reads the batch from its end: the op met first is then
// mostly the one that counts, and the others of a popular key only read its
// cell. n_sup: ops that do not count; n_rej: key-0 ops in [own0, own1), an
// empty range once they are counted.
template <int KB, int SB, int MODE>
__device__ __noinline__ uint32_t gather_keys(BinSmem<KB, SB> &M, const void *keys, uint32_t n,
                                                uint32_t own0, uint32_t &own1, uint32_t &n_sup,
                                                uint32_t &n_rej) {
    using K = typename SlotT<KB>::K;
    const uint32_t tid = threadIdx.x, bin = blockIdx.x, nbins = gridDim.x;
    uint32_t *cell = reinterpret_cast<uint32_t *>(M.stage);  // index + 1 of the op that counts so far
    const uint64_t mask = M.part_mask[M.top - 1], part = M.part[M.top - 1];
    for (uint32_t c = tid; c < (uint32_t)kSmallTab; c += kSmallThreads) cell[c] = 0u;
    if (tid == 0) M.ndist = M.over = 0u;
    __syncthreads();
    uint32_t seen = 0u, rej = 0u;
    stream_batch<KB, 4>(
        keys, n, MODE == kBinModeInsert, [&] { return *(volatile uint32_t *)&M.over != 0u; },
        [&](K k, uint32_t i, bool here) {
            if (k == 0) {
                if (here && i >= own0 && i < own1) ++rej;
                return;
            }
            if (bin_of<KB>(k, nbins) != bin) return;
            if (mask && (part_bits((uint64_t)k) & mask) != part) return;
            ++seen;
            const uint32_t h = small_cell<KB, SB>(M, cell, keys, k, i, true);
            const uint32_t f = *(volatile uint32_t *)&cell[h];
            if (MODE == kBinModeInsert && f < i + 1u) atomicMax(&cell[h], i + 1u);
            if (MODE == kBinModeErase && f > i + 1u) atomicMin(&cell[h], i + 1u);
        });
    uint32_t d[kSmallCells];
    const bool done = end_part<KB, SB>(M, cell, d);
    if (done) {
        n_sup += seen;
        n_rej += rej;
        own1 = own0;
#pragma unroll
        for (int q = 0; q < kSmallCells; ++q) {
            const uint32_t f = cell[q * kSmallThreads + tid];
            if (f == 0u) continue;
            M.key[d[q]] = load_key<KB>(keys, f - 1u);
            M.word[d[q]] = (f - 1u) << 2;
            --n_sup;
        }
    }
    const uint32_t m = done ? M.ndist : 0u;
    __syncthreads();
    return m;
}

// The same of a mixed batch: the keys of the next part to M.key with their ops,
// M.cnt the ops | place in seg << 16, M.word the only op of a key with one; the
// op words of the others in seg, in no order. Returns the number of keys (0:
// the part was split).
template <int KB, int SB>
__device__ __noinline__ uint32_t gather_part(BinSmem<KB, SB> &M, const void *keys, const uint8_t *ops,
                                             uint32_t n) {
    using K = typename SlotT<KB>::K;
    const uint32_t tid = threadIdx.x, lane = tid & 31, bin = blockIdx.x, nbins = gridDim.x;
    // a cell's ops; then the next place in seg (kNone: its key has one op)
    constexpr uint32_t kNone = 0xffffffffu;
    uint32_t *cell = reinterpret_cast<uint32_t *>(M.stage), *cnt = cell + kSmallTab;
    static_assert(sizeof(M.stage) >= 2 * kSmallTab * sizeof(uint32_t), "two tables fit the stage");
    const uint64_t mask = M.part_mask[M.top - 1], part = M.part[M.top - 1];
    for (uint32_t c = tid; c < (uint32_t)kSmallTab; c += kSmallThreads) cell[c] = cnt[c] = 0u;
    if (tid == 0) M.nseg = M.nmulti = M.nlong = M.ndist = M.over = 0u;
    __syncthreads();
    auto mine = [&](K k) {
        return k != 0 && bin_of<KB>(k, nbins) == bin && (!mask || (part_bits((uint64_t)k) & mask) == part);
    };
    stream_batch<KB, 4>(
        keys, n, false, [&] { return __any_sync(kFull, *(volatile uint32_t *)&M.over != 0u) != 0; },
        [&](K k, uint32_t i, bool) {
            const bool own = mine(k);
            if (!__any_sync(kFull, own)) return;
            const uint32_t h = own ? small_cell<KB, SB>(M, cell, keys, k, i, true) : kNone;
            __syncwarp();
            const unsigned peers = __match_any_sync(kFull, h);
            if (own && __ffs(peers) - 1 == (int)lane) atomicAdd(&cnt[h], (uint32_t)__popc(peers));
        });
    uint32_t d[kSmallCells];
    const bool done = end_part<KB, SB>(M, cell, d);
    if (done) {
#pragma unroll
        for (int q = 0; q < kSmallCells; ++q) {
            const uint32_t c = q * kSmallThreads + tid, k = cnt[c];
            if (cell[c] == 0u) continue;
            const uint32_t i = cell[c] - 1u;
            M.key[d[q]] = load_key<KB>(keys, i);
            uint32_t at = 0u;
            if (k == 1u) {
                M.word[d[q]] = op_word(i, ops[i]);
                cnt[c] = kNone;
            } else {
                at = atomicAdd(&M.nseg, k);
                if (k > kSmallLong) M.longs[atomicAdd(&M.nlong, 1u)] = (uint16_t)d[q];
                else M.multi[atomicAdd(&M.nmulti, 1u)] = (uint16_t)d[q];
                cnt[c] = at;
            }
            M.cnt[d[q]] = k | at << 16;
        }
    }
    const uint32_t m = done ? M.ndist : 0u;
    __syncthreads();
    if (M.nseg != 0u)
        stream_batch<KB, 4>(
            keys, n, false, [] { return false; },
            [&](K k, uint32_t i, bool) {
                const bool own = mine(k);
                if (!__any_sync(kFull, own)) return;
                const uint32_t h = own ? small_cell<KB, SB>(M, cell, keys, k, i, false) : 0u;
                const bool put = own && *(volatile uint32_t *)&cnt[h] != kNone;
                const uint32_t w = put ? op_word(i, ops[i]) : 0u;
                __syncwarp();
                const unsigned peers = __match_any_sync(kFull, put ? h : kNone);
                const int lead = __ffs(peers) - 1;
                uint32_t at = 0u;
                if (put && lead == (int)lane) at = atomicAdd(&cnt[h], (uint32_t)__popc(peers));
                at = __shfl_sync(kFull, at, lead) + __popc(peers & ((1u << lane) - 1u));
                if (put) M.seg[at] = w;
            });
    __syncthreads();
    return m;
}

// The c op words of one key at M.seg[off] into index order by the whole block: a bit per op and two for its code, then the words
// again from the bits. (Bitonic networks of that length take 100 barriers.)
template <int KB, int SB>
__device__ __noinline__ void sort_long(BinSmem<KB, SB> &M, uint32_t off, uint32_t c) {
    constexpr uint32_t kPer = 2, kWords = kPer * kSmallThreads;
    static_assert(kWords * 32u >= kBinSmallOps, "a bit for every op");
    static_assert(sizeof(M.stage) >= 3 * kWords * sizeof(uint32_t), "three bitmaps fit the stage");
    uint32_t *bits = reinterpret_cast<uint32_t *>(M.stage);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    for (uint32_t w = tid; w < 3u * kWords; w += kSmallThreads) bits[w] = 0u;
    __syncthreads();
    for (uint32_t j = tid; j < c; j += kSmallThreads) {
        const uint32_t w = M.seg[off + j], i = w >> 2, b = 1u << (i & 31u);
        atomicOr(&bits[i >> 5], b);
        if (w & 1u) atomicOr(&bits[kWords + (i >> 5)], b);
        if (w & 2u) atomicOr(&bits[2u * kWords + (i >> 5)], b);
    }
    __syncthreads();
    uint32_t own = 0u;
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q) own += __popc(bits[tid * kPer + q]);
    uint32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) M.warp_sum[warp] = incl;
    __syncthreads();
    uint32_t at = off + incl - own;
    for (uint32_t w = 0; w < warp; ++w) at += M.warp_sum[w];
    for (uint32_t q = 0; q < kPer; ++q) {
        const uint32_t x = tid * kPer + q, one = bits[kWords + x], two = bits[2u * kWords + x];
        for (uint32_t b = bits[x]; b; b &= b - 1u) {
            const uint32_t p = __ffs(b) - 1;
            M.seg[at++] = (x * 32u + p) << 2 | ((one >> p) & 1u) | ((two >> p) & 1u) << 1;
        }
    }
    __syncthreads();
}

// Place the pending entries of list_a (a few) by eviction walks, from the last
// block of a small batch's kernel.
template <int KB, int SB>
__device__ __forceinline__ void tail_walk(const Desc &D, const Scratch &S, Counters *ctr, uint64_t np) {
    using Sl = typename SlotT<KB>::S;
    for (uint64_t i = threadIdx.x >> 5; i < np; i += kSmallWarps) {
        // written by other blocks of this kernel: read past the L1
        const unsigned long long *src = (const unsigned long long *)((const Sl *)S.list_a + i);
        Sl e;
        if constexpr (KB == 4) e = __ldcg(src);
        else e = Sl{__ldcg(src), __ldcg(src + 1)};
        const WalkOut<KB> w = walk_lookahead<KB, SB>(D, e, D.max_evict);
        if ((threadIdx.x & 31) != 0) continue;
        if (w.steps) atomicAdd(&ctr->evict_steps, (unsigned long long)w.steps);
        if (w.ok) {
            atomicAdd(&ctr->inserted, 1ull);
            atomicAdd(&ctr->size, 1ull);
        } else {
            const unsigned long long at = atomicAdd(&ctr->overflow, 1ull);
            if (at < S.list_cap) ((Sl *)S.list_b)[at] = w.left;
            else atomicAdd(&ctr->spill, 1ull);
        }
    }
}

// A small batch in one kernel: every block reads the whole batch, keeps the ops
// of its bin, finds the repeated keys among them in shared memory and probes
// the table; the last block to finish places the few entries left without a
// slot and writes the counters to the host. A bin of more than kSmallCap ops is
// taken by its block as well, in parts of up to kSmallCap keys (gather_keys,
// gather_part). It used to leave the batch to the split kernels, after a wait:
// 8000 inserts on 7 keys 72 -> 41 us, 16000 mixed ops on 7 keys 236 -> 91.
template <int KB, int SB, int MODE>
__global__ void __launch_bounds__(kSmallThreads, 1) k_bin_small(
    const __grid_constant__ Desc D, const __grid_constant__ Scratch S,
    const uint8_t *__restrict__ ops, const void *__restrict__ keys, const void *__restrict__ vals,
    uint32_t vb, void *__restrict__ vals_out, uint32_t *__restrict__ bits_out, uint64_t n,
    uint32_t flags, Counters *ctr, Counters *h_ctr) {
    using T = SlotT<KB>;
    using K = typename T::K;
    using Sl = typename T::S;
    using Gm = Geo<KB, SB>;
    extern __shared__ __align__(128) unsigned char s_raw[];
    BinSmem<KB, SB> &M = *reinterpret_cast<BinSmem<KB, SB> *>(s_raw);
    uint32_t *tab = reinterpret_cast<uint32_t *>(M.stage);
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    unsigned char *stage = M.stage[tid >> 5];
    const uint32_t bin = blockIdx.x;
    uint32_t n_ins = 0, n_upd = 0, n_del = 0, n_sup = 0, n_rej = 0;

    const uint32_t own0 = (uint32_t)(((uint64_t)bin * n) / gridDim.x);
    uint32_t own1 = (uint32_t)(((uint64_t)(bin + 1) * n) / gridDim.x);
    if (tid == 0) {
        M.m = M.nseg = M.nmulti = M.nlong = 0u;
        M.top = 1u;
        M.part_mask[0] = M.part[0] = 0ull;
    }
    if (tid < 6) M.sum[tid] = 0ull;
    // the bin's ops listed, as long as they are at most kSmallCap
    for (uint32_t c = tid; c < (uint32_t)kSmallTab; c += kSmallThreads) tab[c] = 0u;
    for (uint32_t c = tid; c < (uint32_t)kSmallCap; c += kSmallThreads)
        M.cnt[c] = MODE == kBinModeErase ? 0xffffffffu : 0u;
    __syncthreads();
    stream_batch<KB, 8>(
        keys, (uint32_t)n, false,
        [&] { return MODE < kBinModeMixed && *(volatile uint32_t *)&M.m > (uint32_t)kSmallCap; },
        [&](K k, uint32_t i, bool here) {
            if (k == 0) {  // belongs to no bin: one block answers it
                if (!here || i < own0 || i >= own1) return;
                ++n_rej;
                if (MODE == kBinModeMixed && vals_out) store_val(vals_out, vb, i, 0ull);
                return;
            }
            // a popular key's ops stop counting here once the bin is full
            if (bin_of<KB>(k, gridDim.x) != bin || *(volatile uint32_t *)&M.m > (uint32_t)kSmallCap) return;
            const uint32_t r = atomicAdd(&M.m, 1u);
            if (r < (uint32_t)kSmallCap) {
                M.key[r] = k;
                M.word[r] = i << 2;
            }
        });
    __syncthreads();
    const bool fits = M.m <= (uint32_t)kSmallCap;
    uint32_t m = fits ? M.m : 0u;  // keys or ops listed
    if constexpr (MODE >= kBinModeMixed) {
        for (uint32_t r = tid; r < m; r += kSmallThreads)
            M.word[r] = op_word(M.word[r] >> 2, ops[M.word[r] >> 2]);
    } else if (!fits) {
        n_rej = 0u;  // counted by gather_keys
    }
    __syncthreads();
    // so far the batch was read and key-0 results written, which the clear
    // before this kernel does not touch; its grid waited for the ones before it
    after_previous();

    while (true) {
        K key[kSmallR];
        uint32_t word[kSmallR];
        bool mine[kSmallR];  // the op resolves its key alone
        if (fits) {
            // group: each record finds its key's first record (lead)
            uint32_t lead[kSmallR], rank[kSmallR];
#pragma unroll
            for (int q = 0; q < kSmallR; ++q) {
                const uint32_t r = q * kSmallThreads + tid;
                lead[q] = rank[q] = 0u;
                word[q] = 0u;
                key[q] = 0;
                if (r >= m) continue;
                key[q] = M.key[r];
                word[q] = M.word[r];
                uint32_t h = bin_cell<11>(bin_tag(key[q]));
                // at most kSmallCap of the kSmallTab cells are taken: the probe ends
                while (true) {
                    const uint32_t old = atomicCAS(&tab[h], 0u, r + 1u);
                    if (old == 0u) {
                        lead[q] = r;
                        break;
                    }
                    if (M.key[old - 1u] == key[q]) {
                        lead[q] = old - 1u;
                        break;
                    }
                    h = (h + 1u) & (kSmallTab - 1);
                }
                if (MODE == kBinModeInsert) atomicMax(&M.cnt[lead[q]], word[q]);
                else if (MODE == kBinModeErase) atomicMin(&M.cnt[lead[q]], word[q]);
                else rank[q] = atomicAdd(&M.cnt[lead[q]], 1u);
            }
            __syncthreads();  // the key table is done: the stage may be used

            // keys with several ops: a range of seg each, their op words listed there
            if constexpr (MODE >= kBinModeMixed) {
                bool any = false;
#pragma unroll
                for (int q = 0; q < kSmallR; ++q) {
                    const uint32_t r = q * kSmallThreads + tid;
                    const uint32_t c = r < m ? M.cnt[lead[q]] : 0u;
                    mine[q] = c == 1u;
                    any |= c > 1u;
                }
                if (__syncthreads_or(any)) {
#pragma unroll
                    for (int q = 0; q < kSmallR; ++q) {
                        const uint32_t r = q * kSmallThreads + tid;
                        if (r < m && !mine[q] && lead[q] == r) {
                            const uint32_t c = M.cnt[r];
                            M.cnt[r] = c | (atomicAdd(&M.nseg, c) << 16);
                            if (c > kSmallLong) M.longs[atomicAdd(&M.nlong, 1u)] = (uint16_t)r;
                            else M.multi[atomicAdd(&M.nmulti, 1u)] = (uint16_t)r;
                        }
                    }
                    __syncthreads();
#pragma unroll
                    for (int q = 0; q < kSmallR; ++q) {
                        const uint32_t r = q * kSmallThreads + tid;
                        if (r < m && !mine[q]) M.seg[(M.cnt[lead[q]] >> 16) + rank[q]] = word[q];
                    }
                    __syncthreads();
                }
            } else {
#pragma unroll
                for (int q = 0; q < kSmallR; ++q) {
                    const uint32_t r = q * kSmallThreads + tid;
                    mine[q] = r < m && M.cnt[lead[q]] == word[q];  // op indexes are distinct
                    if (r < m && !mine[q]) ++n_sup;
                }
            }
        } else {
            if constexpr (MODE >= kBinModeMixed)
                m = gather_part<KB, SB>(M, keys, ops, (uint32_t)n);
            else
                m = gather_keys<KB, SB, MODE>(M, keys, (uint32_t)n, own0, own1, n_sup, n_rej);
#pragma unroll
            for (int q = 0; q < kSmallR; ++q) {
                const uint32_t r = q * kSmallThreads + tid;
                mine[q] = r < m && (MODE < kBinModeMixed || (M.cnt[r] & 0xffffu) == 1u);
                key[q] = r < m ? M.key[r] : (K)0;
                word[q] = mine[q] ? M.word[r] : 0u;
            }
        }

        // keys with one op (the winning op of an insert or erase batch): one probe
#pragma unroll
        for (int q = 0; q < kSmallR; ++q) {
            if ((uint32_t)(q * kSmallThreads) + (tid & ~31u) >= m) break;  // warp-uniform
            const bool act = mine[q];
            const uint32_t i = word[q] >> 2;
            const uint32_t op = MODE == kBinModeInsert ? 1u : MODE == kBinModeErase ? 2u : (word[q] & 3u);
            const bool ins = act && op == 1u, del = act && op == 2u;
            Sl e = T::empty();
            if (ins) e = T::make(key[q], load_val(vals, vb, i));
            const uint32_t hk = fold(key[q]);
            const Pair p = pair_of(hk, D.d);
            char *p1 = bucket_ptr<KB, SB>(D, p.first, bucket_index(D, p.first, hk));
            char *p2 = bucket_ptr<KB, SB>(D, p.second, bucket_index(D, p.second, hk));
            const KvOut r1 = place_probe<KB, SB, false>(p1, key[q], act, p.first, D.d, stage);
            const bool found1 = act && r1.match >= 0;
            const bool want_slot = MODE != kBinModeCount && ins && r1.empty == 0u;
            const bool may2 = !Gm::kMeta || r1.overflow;
            const bool check2 =
                act && !found1 && ((may2 && !(MODE == kBinModeInsert && (flags & kBinNewKeys))) || want_slot);
            KvOut r2{-1, 0ull, false, 0u};
            if (__any_sync(kFull, check2))
                r2 = place_probe<KB, SB, false>(p2, key[q], check2, p.second, D.d, stage);
            const bool found2 = check2 && r2.match >= 0;
            const bool present = found1 || found2;
            const uint64_t before = found1 ? r1.value : (found2 ? r2.value : 0ull);
            if constexpr (MODE == kBinModeCount) {
                if (ins && (!present || before != T::val(e))) ++n_ins;
                if (del && present) ++n_del;
                continue;
            }
            bool pend = false;
            if (ins) {
                if (present) {
                    if (!(MODE == kBinModeMixed && (flags & kBinSkipEqual) && before == T::val(e))) {
                        T::store(found1 ? slot_ptr<KB, SB>(p1, r1.match) : slot_ptr<KB, SB>(p2, r2.match), e);
                        ++n_upd;
                    }
                } else {
                    bool ok = claim_empty<KB, SB>(p1, r1.empty, e);
                    if (!ok && check2 && r2.empty) {
                        mark_overflow<KB, SB>(p1, hk);
                        ok = claim_empty<KB, SB>(p2, r2.empty, e);
                    }
                    if (ok) ++n_ins;
                    else pend = true;
                }
            } else if (del && present) {
                T::store(found1 ? slot_ptr<KB, SB>(p1, r1.match) : slot_ptr<KB, SB>(p2, r2.match),
                         T::empty());
                ++n_del;
            }
            // a mixed op's result; the value an erased key had
            if ((MODE == kBinModeMixed && act || MODE == kBinModeErase && present) && vals_out != nullptr)
                store_val(vals_out, vb, i, before);
            if (MODE != kBinModeInsert && act && present && bits_out != nullptr)
                atomicOr(&bits_out[i >> 5], 1u << (i & 31));
            if constexpr (MODE != kBinModeErase) {
                __syncwarp();
                const unsigned long long at = agg_inc(&ctr->pending, pend);
                if (pend) {
                    if (at < S.list_cap) ((Sl *)S.list_a)[at] = e;
                    else atomicAdd(&ctr->spill, 1ull);
                }
            }
        }

        // keys with several ops: probe, replay the ops in index order, apply the
        // final state
        if constexpr (MODE >= kBinModeMixed) {
            RepCounts rc;
            auto finish = [&](const RepKey<KB> &x, bool act, bool present, uint64_t value) {
                const bool up = act && present && (!x.pre || value != x.pre_value);
                const bool er = act && !present && x.pre;
                if constexpr (MODE == kBinModeCount) {
                    rc.ins += up ? 1u : 0u;
                    rc.del += er ? 1u : 0u;
                } else {
                    mutate_listed<KB, SB>(x, up, er, value, S.list_a, S.list_cap, ctr, rc);
                }
            };
            // Key x of the list goes to lane x / 16 of warp x % 16, so a few long
            // segments spread over the warps.
            const uint32_t nm = M.nmulti;
            for (uint32_t x0 = 0; x0 < nm; x0 += kSmallThreads) {
                const uint32_t y = x0 + lane * kSmallWarps + (tid >> 5);
                const bool act = y < nm;
                if (!__any_sync(kFull, act)) continue;
                const uint32_t r = act ? M.multi[y] : 0u;
                const uint32_t c = act ? M.cnt[r] & 0xffffu : 0u, off = act ? M.cnt[r] >> 16 : 0u;
                const RepKey<KB> x = probe_key<KB, SB>(D, act ? M.key[r] : (K)0, act, stage);
                bool present = x.pre;
                uint64_t value = x.pre_value;
                if (act && c <= kBinShort) {
                    uint32_t w[kBinShort];
#pragma unroll
                    for (uint32_t a = 0; a < kBinShort; ++a) w[a] = a < c ? M.seg[off + a] : 0xffffffffu;
#pragma unroll
                    for (uint32_t t = 0; t < kBinShort; ++t) {
#pragma unroll
                        for (uint32_t a = t & 1u; a + 1 < kBinShort; a += 2) {
                            const uint32_t lo = min(w[a], w[a + 1]), hi = max(w[a], w[a + 1]);
                            w[a] = lo;
                            w[a + 1] = hi;
                        }
                    }
#pragma unroll
                    for (uint32_t a = 0; a < kBinShort; ++a) {
                        if (a >= c) break;
                        const uint32_t i = w[a] >> 2, op = w[a] & 3u;
                        const uint64_t in = op == 1u ? load_val(vals, vb, i) : 0ull;
                        if (MODE == kBinModeMixed) {
                            if (vals_out) store_val(vals_out, vb, i, present ? value : 0ull);
                            if (present && bits_out) atomicOr(&bits_out[i >> 5], 1u << (i & 31));
                        }
                        replay_op((uint8_t)op, in, present, value);
                    }
                }
                for (unsigned big = __ballot_sync(kFull, c > kBinShort); big; big &= big - 1u) {
                    const int j = __ffs(big) - 1;
                    const uint32_t cj = __shfl_sync(kFull, c, j), oj = __shfl_sync(kFull, off, j);
                    bool pj = __shfl_sync(kFull, present, j);
                    uint64_t vj = shfl64(value, j);
                    __syncwarp();
                    warp_sort_words(M.seg + oj, cj);
                    warp_replay_words<MODE == kBinModeMixed>(M.seg + oj, cj, pj, vj, vals, vb, vals_out,
                                                             bits_out);
                    if ((int)lane == j) {
                        present = pj;
                        value = vj;
                    }
                }
                finish(x, act, present, value);
            }
            // keys with more than kSmallLong ops: the whole block each
            const uint32_t nl = M.nlong;
            for (uint32_t y = 0; y < nl; ++y) {
                const uint32_t r = M.longs[y], c = M.cnt[r] & 0xffffu, off = M.cnt[r] >> 16;
                sort_long<KB, SB>(M, off, c);
                __shared__ uint64_t s_before;
                __shared__ uint32_t s_present;
                RepKey<KB> x;
                if (tid < 32) {
                    x = probe_key<KB, SB>(D, M.key[r], lane == 0, stage);
                    if (tid == 0) {
                        s_present = x.pre ? 1u : 0u;
                        s_before = x.pre_value;
                    }
                }
                __syncthreads();
                bool present = s_present != 0u;
                uint64_t value = s_before;
                block_replay<kSmallThreads, MODE == kBinModeMixed>(M.seg + off, c, present, value,
                                                                   SegOps{ops, 0u}, vals, vb, vals_out,
                                                                   bits_out);
                if (tid < 32) finish(x, lane == 0, present, value);
                __syncthreads();
            }
            n_ins += rc.ins;
            n_upd += rc.upd;
            n_del += rc.del;
        }
        if (fits || M.top == 0u) break;
        __syncthreads();  // the lists are reused by the next part
    }

    // one atomic per counter per block
    n_ins = __reduce_add_sync(kFull, n_ins);
    n_upd = __reduce_add_sync(kFull, n_upd);
    n_del = __reduce_add_sync(kFull, n_del);
    n_sup = __reduce_add_sync(kFull, n_sup);
    n_rej = __reduce_add_sync(kFull, n_rej);
    if (lane == 0) {
        if (n_ins) atomicAdd(&M.sum[0], (unsigned long long)n_ins);
        if (n_upd) atomicAdd(&M.sum[1], (unsigned long long)n_upd);
        if (n_del) atomicAdd(&M.sum[2], (unsigned long long)n_del);
        if (n_sup) atomicAdd(&M.sum[3], (unsigned long long)(long long)(int32_t)n_sup);  // may be below 0
        if (n_rej) atomicAdd(&M.sum[4], (unsigned long long)n_rej);
    }
    __syncthreads();
    if (tid == 0) {
        const unsigned long long ins = M.sum[0], upd = M.sum[1], del = M.sum[2];
        if constexpr (MODE == kBinModeCount) {
            if (ins) atomicAdd(&ctr->nins, ins);
            if (del) atomicAdd(&ctr->erased, del);
        } else {
            if (ins) atomicAdd(&ctr->inserted, ins);
            if (upd) atomicAdd(&ctr->updated, upd);
            if (del) atomicAdd(&ctr->erased, del);
            const long long net = (long long)ins - (long long)del;
            if (net) atomicAdd(&ctr->size, (unsigned long long)net);
        }
        if (MODE <= kBinModeErase && M.sum[3]) atomicAdd(&ctr->superseded, M.sum[3]);
        if (MODE == kBinModeInsert && M.sum[4]) atomicAdd(&ctr->rejected, M.sum[4]);
    }
    {
        // the last block sees every other block's lists and counters
        __threadfence();
        __syncthreads();
        if (tid == 0) M.last = atomicAdd(&ctr->ticket, 1ull) == gridDim.x - 1;
        __syncthreads();
        if (!M.last) return;
        __threadfence();
        if constexpr (MODE != kBinModeErase && MODE != kBinModeCount) {
            const uint64_t np = *(volatile unsigned long long *)&ctr->pending;
            if (np && np <= kTailWalk) {
                tail_walk<KB, SB>(D, S, ctr, np);
                __threadfence();
                __syncthreads();
                if (tid == 0) *(volatile unsigned long long *)&ctr->pending = 0ull;
                __syncthreads();
            }
        }
        if (tid < sizeof(Counters) / 8)
            ((volatile unsigned long long *)h_ctr)[tid] = ((volatile unsigned long long *)ctr)[tid];
        __threadfence_system();
    }
}

}  // namespace dyc
