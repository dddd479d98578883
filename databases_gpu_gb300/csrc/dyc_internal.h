// dyc_internal.h -- shared between the kernels and the host side of the
// C ABI: the device-side table descriptor, the per-table counters and the
// kernel launchers.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace dyc {

// Every device and pinned-host allocation the library makes goes through
// these (counted for dyc_debug_alloc_count).
extern std::atomic<unsigned long long> g_lib_allocs;
template <class T> cudaError_t lib_malloc(T **p, size_t bytes) {
    g_lib_allocs.fetch_add(1, std::memory_order_relaxed);
    return cudaMalloc((void **)p, bytes);
}
template <class T> cudaError_t lib_malloc_host(T **p, size_t bytes) {
    g_lib_allocs.fetch_add(1, std::memory_order_relaxed);
    return cudaMallocHost((void **)p, bytes);
}

// The reference's modulus before the bucket modulo, written as in
// GPU/dyhash/dy_hash.h:24 (294967291, not the prime 4294967291).
constexpr uint32_t kPrime = 294967291u;
constexpr int kMaxSub = 6;
// Polls of a bounded device wait (mbarrier try_wait): far beyond any copy's
// completion; a wait that runs out records a timeout instead of hanging.
constexpr uint32_t kWaitTries = 1u << 22;

// Table descriptor passed by value to every kernel (the reference keeps one
// in __constant__ memory, cuckoo.cu:16, which limits a process to one table).
struct Desc {
    void *sub[kMaxSub];       // subtable base addresses
    uint64_t magic[kMaxSub];  // fastmod reciprocals of nb[]
    uint32_t nb[kMaxSub];     // buckets per subtable
    uint32_t d;               // subtable count
    uint32_t max_evict;       // eviction bound of this table (read by the set kernels)
    uint32_t l2_keep;         // 1: the table fits the L2; its bucket reads ask to stay there
    uint32_t pad;
};

// Per-table device counters (one 128-byte block). `size` persists; the rest
// are per-call and reset before each insert / erase / resize.
struct Counters {
    unsigned long long size;
    unsigned long long inserted, updated, erased, rejected, superseded;
    unsigned long long pending, overflow, evict_steps;
    unsigned long long spill;  // pending entries a list could not hold (must stay 0)
    unsigned long long pad[2];      // scratch words of dyc_export and dyc_snapshot
    unsigned long long timeouts;    // bounded device waits that gave up (must stay 0)
    // scratch word: insert ops of a dyc_apply batch (its upserts, from the
    // counting pass of a batch resolved by bins)
    unsigned long long nins;
    unsigned long long ticket;      // blocks of a call's last kernel that have finished
    unsigned long long pad2;
};
static_assert(sizeof(Counters) == 128, "Counters is one 128-byte block");

// Where a call's last kernel writes its counters for the host (pinned memory),
// instead of a copy behind it; null: nowhere.
struct Publish {
    Counters *h_ctr = nullptr;
    const unsigned long long *actr = nullptr;  // a mixed batch's ApplyScratch::ctr
    unsigned long long *h_actr = nullptr;
};

// A chunk's ops split by key into bins (dyc_bins.cuh): bin b's records are
// [b * kBinCap, b * kBinCap + count[b]), a bin holding kBinMean ops of distinct
// random keys on average. The ops of a bin with more than kBinCap (few keys,
// each repeated many times) get records in `hot` instead. kBinMean * 2 =
// kBinCap, so the records of n ops take 2n words. Batches of up to
// kBinSmallOps mixed ops, or kBinSmallUpserts inserts or erases, are split by
// the kernel that resolves them (k_bin_small), into bins of kBinSmallMean ops.
// The lines lie where the split kernels get as fast, in us of a call on a table
// of 2^24 4-byte keys, one kernel / split:
//   mixed ops       8000       16000       24000       32768
//     distinct     47 / 49     50 / 52     54 / 53     56 / 54
//     7 keys       70 / 86     91 / 106   112 / 118   134 / 152
//     100 keys     55 / 80     65 / 122   116 / 130   134 / 84
//   inserts         8000       12000       16000       32768
//     distinct     37 / 38     39 / 38     40 / 39     45 / 40
//     7 keys       41 / 44     44 / 45     47 / 45     60 / 47
constexpr int kBinCap = 2048;
constexpr int kBinMean = 1024;
constexpr int kSmallCap = 1024;
constexpr int kBinSmallMean = 384;
constexpr uint64_t kBinSmallOps = 24576, kBinSmallUpserts = 8192;
enum : int {
    kBinOver = 0,  // nonzero: some bin went over
    kBinStates = 1
};
struct BinScratch {
    unsigned long long *rec;  // key tag | op word << 32 (rec_word)
    unsigned long long *hot;  // records of the bins that went over (one per op of the batch)
    uint32_t *count;          // per bin: ops
    uint32_t *start, *cursor; // per bin that went over: its records in hot; ops written
    uint32_t *state;          // kBinOver
    uint2 *tables;            // set batches: a bin's first table; 1: its only one
    uint32_t nbins;
    // one bit per op: cleared for the ops of keys with several ops (an insert
    // or erase batch: all but the op that counts)
    uint32_t *single;
};

// Scratch lists used by one insert / erase / resize chunk.
struct Scratch {
    // dyc_erase_noalloc: an open-addressing table of (key, op index), cleared
    // by the caller; other batches name the op of a key that counts in winbits
    void *dedup;
    uint32_t *dedup_idx;    // op index array for 8-byte keys
    uint64_t dedup_cap;     // power of two
    void *list_a;           // pending entries (slots)
    void *list_b;           // overflow entries (slots)
    uint64_t list_cap;      // entries per list
    // one bit per op of the chunk, set for the op of its key that counts
    uint32_t *winbits;
    unsigned long long *rec;  // records of the chunk's bins (BinScratch)
    uint32_t *bin_words;      // the bins' state, counts, starts and cursors
};

enum : int {
    kBinModeInsert = 0,  // the last op of a key wins (dyc_insert)
    kBinModeErase = 1,   // the first op wins (dyc_erase)
    kBinModeMixed = 2,   // the ops take effect in index order (dyc_apply)
    kBinModeCount = 3    // as kBinModeMixed, but only counts the upserts and erases
};
enum : uint32_t {
    kBinNewKeys = 1,   // the caller promises absent keys (DYC_FLAG_NEW_KEYS)
    kBinSkipEqual = 2  // an insert that finds its own value writes and counts nothing
};

// Scratch of one mixed batch of at most `cap_ops` ops. The multi-table
// fields are null for a single table.
struct ApplyScratch {
    void *dkey;                // keys with several ops in the batch
    uint32_t *dcnt;            // per such key: ops
    unsigned long long *dseg;  // per such key: segment start << 32
    uint32_t *seg;             // ops grouped by key: index << 2 | code, plain indices if wide
    uint32_t wide;             // batches of 2^30 ops and more
    void *up_key, *up_val;     // upserts to apply
    void *er_key;              // erases to apply
    unsigned long long *ctr;   // see kCtr*
    uint32_t *wseg;            // ids of segments replayed by a warp
    uint32_t *mid;             // ids of segments replayed by a block
    uint32_t *sort_tmp;        // merge scratch of long segments (same offsets as seg)
    uint64_t cap_ops;
    // bit i set when op i is its key's only op, or a key-0 op: left to the
    // one-pass kernels
    uint32_t *single;
    // multi-table batches
    uint32_t *dtid;            // table of a listed key
    uint32_t *up_tid, *er_tid; // table of each upsert / erase
    uint32_t *tup;             // per table: upserts listed (the upsize policy's insert batch)
    uint32_t *ter;             // per table: erases listed (keys present before the batch)
    uint32_t *tidx;            // table of every kTidxStep-th op (cap_ops / kTidxStep + 1)
    uint32_t ntables;
    unsigned long long *rec;   // records of the batch's bins (BinScratch); the other bin
    uint32_t *bin_words;       // arrays; records of bins that went over
    unsigned long long *hot;
    uint2 *bin_tables;
};

constexpr uint32_t kTidxStep = 64;  // ops per entry of ApplyScratch::tidx

// Places a bin of a set batch takes (set_bin in dyc_bins.cuh). (A round of 2^25
// ops over 4096 tables: 301 us of grouping, 313 with 960 places, 321 with 896.)
constexpr uint32_t kSetBinMean = 1024;
__host__ __device__ inline uint64_t set_nbins(uint64_t n) { return (n + kSetBinMean - 1) / kSetBinMean; }

// ApplyScratch::ctr slots. Every count and id the batch kernels read from
// device memory is checked against the scratch capacity (and table ids
// against the table count) before it indexes anything; a value out of range
// is clamped or its item skipped, and counted in kCtrBad (an internal count
// out of range) or kCtrBadOffsets (the device offsets of a set batch
// disagree with the op count the host declared, kCtrHostN). The host turns
// either count into an error.
enum : int {
    kCtrDistinct = 0,    // listed keys (several ops each)
    kCtrPlaced = 1,      // ops given a segment slot
    kCtrUp = 2,          // upserts listed
    kCtrEr = 3,          // erases listed
    kCtrMid = 4,         // block segments
    kCtrWarp = 5,        // warp segments
    kCtrBad = 6,         // device-read counts or ids out of range (must stay 0)
    kCtrBadOffsets = 7,  // set batch: offsets[ntables] != kCtrHostN, or an op outside its table
    kCtrHostN = 8,       // set batch: op count from the host's offsets (copied before the kernels)
    kCtrSlots = 16
};


// Upsizes of many subtables (of different tables) in one launch: job j
// doubles old_sub (old_nb buckets, subtable index t of its table) into
// new_sub; its blocks are [block0, next job's block0). Passed by value as the
// kernel's parameter block, so at most kMaxResizeJobs per launch.
struct ResizeJob {
    const void *old_sub;
    void *new_sub;
    uint64_t magic;  // fastmod reciprocal of 2 * old_nb
    uint32_t old_nb, t, block0;
    uint32_t table;  // member of a table set (jobs the set's upsize policy lists on the device)
};
constexpr uint32_t kMaxResizeJobs = 768;
constexpr uint32_t kResizeChunksPerBlock = 2048;  // 32-byte chunks a block moves
struct ResizeJobs {
    uint32_t n, blocks;
    ResizeJob j[kMaxResizeJobs];
};
static_assert(sizeof(ResizeJobs) <= 32000, "kernel parameter block limit");

// The subtable an upsize doubles (api.cpp:115-122): the first one after a
// subtable twice its size, else subtable 0 (subtables grow in index order).
__host__ __device__ inline uint32_t pick_up_index(const uint32_t *nb, uint32_t d) {
    for (uint32_t i = 0; i + 1 < d; ++i)
        if (nb[i] == 2u * nb[i + 1]) return i + 1;
    return 0;
}

// A table-set member's next upsize target, allocated by the host ahead of
// the round that needs it: new_sub holds 2 * old_nb buckets for subtable ti.
// It fits only while subtable ti is the one pick_up_index names and still
// has old_nb buckets.
struct Spare {
    void *new_sub;  // null: none
    uint32_t ti, old_nb;
};
// What the device half of a set round's upsize policy did: jobs listed for
// k_resize_up_list (tasks of kResizeChunksPerBlock chunks), and whether a
// member needs more than its one device upsize (phase B then waits for the
// host to apply the rest of the policy).
struct SetPolicyOut {
    uint32_t njobs, ntasks, host, pad;
};

// Launch parameters picked once per kernel from the occupancy calculator.
struct LaunchCtx {
    int sms;
    cudaStream_t stream;
    int max_blocks_per_sm = 0;  // 0: as many as fit (else a cap, chosen by a tuner)
};

// What a set call's last kernel writes to the host (pinned memory): one launch
// instead of a copy for each. pout and what follows may be null (no device
// policy in the sequence).
struct SetReport {
    const Counters *gctr;
    Counters *h_gctr;
    const unsigned long long *actr;
    unsigned long long *h_actr;
    const Counters *tctr;           // per table: its size goes to h_size
    unsigned long long *h_size;
    uint32_t ntables;
    const SetPolicyOut *pout;
    SetPolicyOut *h_pout;
    const uint8_t *grew;            // written when the policy listed upsizes
    uint8_t *h_grew;
    const uint32_t *tup, *ter;      // written when the host must finish the policy
    uint32_t *h_tup, *h_ter;
};

// Launch a kernel that begins with after_previous() (programmatic dependent
// launch on the kernel before it in the stream).
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                         cudaStream_t stream, A &&...args) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// Launchers of the bin kernels that probe buckets of SB bytes (dyc_bins_sb.cuh),
// behind Ops::repeat and Ops::bin_small.
template <int KB, int SB> struct BinsSb {
    static cudaError_t repeat(const LaunchCtx &L, const ApplyScratch &A, const Desc *descs,
                              uint32_t ntables, bool set, const uint8_t *ops, const void *vals,
                              uint32_t vb, void *vals_out, uint32_t *bits_out, uint64_t n, void *list_a,
                              uint64_t list_cap, Counters *gctr);
    static cudaError_t small(const LaunchCtx &L, const Desc &D, const Scratch &S, int mode,
                             const uint8_t *ops, const void *keys, const void *vals, uint32_t vb,
                             void *vals_out, uint32_t *bits_out, uint64_t n, uint32_t flags,
                             Counters *ctr, Counters *h_ctr);
};

// Kernel launchers, one set per key width; `sb` = bucket bytes (32/64/128).
// All return cudaGetLastError() of their launches.
template <int KB> struct Ops {
    static cudaError_t find(const LaunchCtx &L, const Desc &D, int sb, const void *keys,
                            void *vals, uint32_t vb, uint32_t *hits, uint64_t n);
    // erase_noalloc's batch dedup into S.dedup (cleared by the caller): each
    // key's first op
    static cudaError_t dedup(const LaunchCtx &L, const Scratch &S, const void *keys, uint64_t n);
    // insert: place or update every op; ops whose two buckets are full go to
    // list_a (counted in pending). new_keys = caller promises absent keys.
    static cudaError_t place(const LaunchCtx &L, const Desc &D, int sb, const Scratch &S,
                             bool use_dedup, bool new_keys, const void *keys, const void *vals,
                             uint32_t vb, uint64_t n, Counters *ctr);
    // eviction walks for the entries of `src` (count at *src_count); entries
    // that reach the bound go to `dst` (count at *dst_count). count_new adds
    // successes to ctr->inserted and ctr->size.
    static cudaError_t walk(const LaunchCtx &L, const Desc &D, int sb, const void *src,
                            const unsigned long long *src_count, void *dst,
                            unsigned long long *dst_count, uint64_t dst_cap, uint32_t max_evict,
                            bool count_new, Counters *ctr, uint64_t max_entries,
                            const Publish &pub = Publish());
    // old (may be null): the value each removed key had (vb bytes each; other
    // ops' words are not written)
    static cudaError_t erase(const LaunchCtx &L, const Desc &D, int sb, const Scratch &S,
                             bool use_dedup, const void *keys, uint64_t n, uint32_t *bits,
                             Counters *ctr, void *old = nullptr, uint32_t vb = 0u,
                             const Publish &pub = Publish());
    static cudaError_t resize_up(const LaunchCtx &L, int sb, uint32_t t, const void *old_sub,
                                 uint32_t old_nb, void *new_sub);
    // J.n jobs in one launch of J.blocks blocks (job block ranges filled in)
    static cudaError_t resize_up_many(const LaunchCtx &L, int sb, const ResizeJobs &J);
    // the jobs a set's device policy listed (out->njobs of them, at most
    // max_jobs, out->ntasks tasks), on a grid fixed at launch
    static cudaError_t resize_up_list(const LaunchCtx &L, int sb, const ResizeJob *jobs,
                                      const SetPolicyOut *out, uint32_t max_jobs);
    // device half of a set round's upsize policy (one block): members whose
    // upserts take them above upper x capacity switch to their spare subtable
    // (descriptor rewritten, move listed in jobs, grew[t] = 1)
    static cudaError_t set_policy(const LaunchCtx &L, Desc *descs, uint32_t ntables,
                                  const Counters *tctr, const uint32_t *tup, const uint32_t *ter,
                                  const Spare *spares, double upper, uint32_t slots, int sb,
                                  ResizeJob *jobs, uint8_t *grew, SetPolicyOut *out);
    // halve an even subtable: merged buckets to new_sub, leftovers to list;
    // a tile-copy wait gives up after tile_wait_tries polls (counted in
    // *timeouts; old_sub is only read)
    static cudaError_t resize_down(const LaunchCtx &L, int sb, const void *old_sub,
                                   uint32_t old_nb, void *new_sub, void *list,
                                   unsigned long long *list_count, uint64_t list_cap,
                                   unsigned long long *spill, unsigned long long *timeouts,
                                   uint32_t tile_wait_tries);
    // every live slot of one subtable to list (general rehash)
    static cudaError_t collect(const LaunchCtx &L, int sb, const void *sub, uint32_t nb,
                               void *list, unsigned long long *list_count, uint64_t list_cap,
                               unsigned long long *spill);
    // a mixed batch whose keys are all distinct, in one probe pass (ops left
    // without a slot go to S.list_a, counted in ctr->pending). With a single
    // bitmap, only the ops whose bit is set, and their hit bits are ORed in.
    // flags: kBinSkipEqual.
    static cudaError_t apply_unique(const LaunchCtx &L, const Desc &D, int sb, const Scratch &S,
                                    const uint8_t *ops, const void *keys, const void *vals,
                                    uint32_t vb, void *vals_out, uint32_t *bits_out, uint64_t n,
                                    Counters *ctr, const uint32_t *single = nullptr,
                                    uint32_t flags = 0u);
    // *count += the INSERT ops among ops[0..n)
    static cudaError_t count_inserts(const LaunchCtx &L, const uint8_t *ops, uint64_t n,
                                     unsigned long long *count);
    // the listed keys (dyc_repeat.cuh): state before the batch, replay,
    // results. list_a set (one table, counters in gctr): the final states go
    // to the table, entries without a slot to list_a; else to A's upsert and
    // erase lists. n bounds the op count. set: keys carry their table (A.dtid).
    static cudaError_t repeat(const LaunchCtx &L, const ApplyScratch &A, const Desc *descs,
                              uint32_t ntables, int sb, bool set, const uint8_t *ops,
                              const void *vals, uint32_t vb, void *vals_out, uint32_t *bits_out,
                              uint64_t n, void *list_a = nullptr, uint64_t list_cap = 0,
                              Counters *gctr = nullptr);
    // a set batch's prep (counters, gctr, result bits) and the split into bins
    // and grouping (bin_group, per table); sized: n is the op count, not a bound
    static cudaError_t set_group(const LaunchCtx &L, const ApplyScratch &A, const BinScratch &B,
                                 const uint32_t *off, const uint8_t *ops, const void *keys,
                                 uint64_t n, bool sized, uint32_t *bits, Counters *gctr);
    // The set kernels below read their item counts from device memory and
    // clamp them to max_n / max_entries (the capacity of the lists behind
    // them); a table id at or above ntables skips its item. Either event is
    // counted in *bad. hint: the members keep their lines in the L2 (their
    // probes carry L2 eviction-priority hints; plain loads otherwise).
    // erases and upserts of a set batch in one launch (max_n: both lists'
    // bound); nothing when *hold is nonzero (the host finishes the policy first)
    static cudaError_t set_mutate(const LaunchCtx &L, const Desc *descs, uint32_t ntables,
                                  Counters *tctr, int sb, const void *er_keys,
                                  const uint32_t *er_tids, const unsigned long long *ne_ptr,
                                  const void *up_keys, const void *up_vals, uint32_t vb,
                                  const uint32_t *up_tids, const unsigned long long *nu_ptr,
                                  uint64_t max_n, void *list_a, uint32_t *list_a_tid,
                                  uint64_t list_cap, Counters *gctr, unsigned long long *bad,
                                  const uint32_t *hold = nullptr, bool hint = false);
    // the ops of a set batch whose key has no other op in it
    // (and key-0 ops), one probe each (k_set_unique); max_n bounds the grid,
    // the op count is read on the device; nothing when *hold is nonzero
    static cudaError_t set_unique(const LaunchCtx &L, const ApplyScratch &A, const uint32_t *off,
                                  const Desc *descs, uint32_t ntables, Counters *tctr, int sb,
                                  const uint8_t *ops, const void *keys, const void *vals,
                                  uint32_t vb, void *vals_out, uint32_t *bits_out,
                                  uint64_t max_n, void *list_a, uint32_t *list_a_tid,
                                  uint64_t list_cap, Counters *gctr, const uint32_t *hold,
                                  bool hint);
    static cudaError_t set_walk(const LaunchCtx &L, const Desc *descs, uint32_t ntables,
                                Counters *tctr, int sb, const void *src, const uint32_t *src_tid,
                                const unsigned long long *src_count, void *dst, uint32_t *dst_tid,
                                unsigned long long *dst_count, uint64_t dst_cap,
                                uint32_t max_evict, Counters *gctr, uint64_t max_entries,
                                unsigned long long *bad, const Publish &pub = Publish());
    // A chunk's repeated keys (dyc_bins.cuh): the bin counts, the call counters
    // (ctr), A.ctr and the result bits zeroed, the single bits set, the ops
    // split into bins, and the ops of repeated keys found: their single bits
    // cleared and, for a mixed batch (mode kBinModeMixed), their keys and
    // segments listed in A. ops is null for the insert and erase modes.
    static cudaError_t bin_group(const LaunchCtx &L, const BinScratch &B, const ApplyScratch &A,
                                 int mode, const uint8_t *ops, const void *keys, uint32_t *bits_out,
                                 uint64_t n, Counters *ctr);
    // a batch of up to kBinSmallOps ops in one kernel, in one of the kBinMode*
    // modes; the
    // counters go to h_ctr
    static cudaError_t bin_small(const LaunchCtx &L, const Desc &D, int sb, const Scratch &S,
                                 int mode, const uint8_t *ops, const void *keys, const void *vals,
                                 uint32_t vb, void *vals_out, uint32_t *bits_out, uint64_t n,
                                 uint32_t flags, Counters *ctr, Counters *h_ctr);
    // ctr->nins / ctr->erased += the upserts and erases that apply_unique
    // would make for the ops whose single bit is set
    static cudaError_t apply_count(const LaunchCtx &L, const Desc &D, int sb, const uint8_t *ops,
                                   const void *keys, const void *vals, uint32_t vb, uint64_t n,
                                   const uint32_t *single, Counters *ctr);
    static cudaError_t set_report(const LaunchCtx &L, const SetReport &R);
    // set every fingerprint bit of every bucket of a subtable
    static cudaError_t mark_all(const LaunchCtx &L, int sb, void *sub, uint32_t nb);
    static cudaError_t export_all(const LaunchCtx &L, const Desc &D, int sb, void *keys,
                                  void *vals, uint32_t vb, uint64_t cap,
                                  unsigned long long *count);
};

}  // namespace dyc
