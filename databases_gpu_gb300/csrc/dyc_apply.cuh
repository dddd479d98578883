// dyc_apply.cuh -- kernels of a mixed batch (finds, inserts and erases in
// one call) with batch-order semantics: ops on the same key take effect in
// index order, a find sees the latest earlier insert/erase of its key in the
// batch (else the table as it was before the batch), and the table ends up
// as if the ops had run one by one.
//
// Steps (stream-ordered kernels):
//   group   : the keys with several ops in the batch are found bin by bin
//             (dyc_bins.cuh) and listed, each with a segment of the op index
//             array; every other op keeps its bit in a bitmap
//   repeat  : each listed key's state before the batch, then its ops replayed
//             in index order (dyc_repeat.cuh): by a lane, a warp (more than
//             kShortSeg ops) or a block (more than kWarpSeg). Every op's
//             result is written; the final states go to the table, or to the
//             lists of upserts and erases
//   unique  : the ops in the bitmap, one probe of their key's buckets each
//   (the erase + upsert and eviction-walk kernels of dyc_set.cuh follow)
// Each key is written by one kernel, at most once, so the usual insert/erase
// phases keep their guarantees. Counts the
// kernels need are read from ApplyScratch::ctr on the device, so the sequence
// has no host reads. Every such count, key id and segment range is checked
// against the scratch capacity before it indexes anything (values out of range
// are clamped or their item skipped and counted in ctr[kCtrBad]); a set batch's
// op count is the smaller of its device offsets' total and the count the
// host declared (ctr[kCtrHostN]), a disagreement counted in
// ctr[kCtrBadOffsets].
#pragma once

#include "dyc_kernels.cuh"

namespace dyc {

enum : uint8_t { kOpFind = 0, kOpInsert = 1, kOpErase = 2 };

constexpr uint32_t kShortSeg = 8;    // segments replayed by one thread
constexpr uint32_t kWarpSeg = 256;   // segments sorted and replayed by one warp
constexpr uint32_t kMidSeg = 4096;   // longest segment sorted in shared memory alone
// Warp segments a warp takes in a row; lane j probes segment j's key and keeps
// its state, so a task costs one round of probes and one warp-aggregated
// atomic per list. Few segments per task keep more warps busy.
constexpr uint32_t kWarpTask = 8;

// Hash of a key for the bins (independent of the subtable hashes).
__device__ __forceinline__ uint32_t cell_hash(uint64_t k) {
    return mix32(fold(k) ^ (uint32_t)(k >> 32));
}

__device__ __forceinline__ void note_bad(const ApplyScratch &A, int slot = kCtrBad) {
    atomicAdd(&A.ctr[slot], 1ull);
}

// Op count of a set batch: offsets[ntables], bounded by the count the host
// declared for this batch and by the scratch.
__device__ __forceinline__ uint64_t set_op_count(const ApplyScratch &A,
                                                 const uint32_t *__restrict__ off) {
    uint64_t n = off[A.ntables];
    const uint64_t h = A.ctr[kCtrHostN];
    if (n > h) n = h;
    return n < A.cap_ops ? n : A.cap_ops;
}

// A device counter of listed items, clamped to the scratch's op capacity.
__device__ __forceinline__ uint64_t ctr_count(const ApplyScratch &A, int slot) {
    const uint64_t n = A.ctr[slot];
    return n < A.cap_ops ? n : A.cap_ops;
}

// Segment [off, off + cnt) of a distinct key lies inside the op scratch.
__device__ __forceinline__ bool seg_ok(const ApplyScratch &A, uint32_t off, uint32_t cnt) {
    return (uint64_t)off + cnt <= A.cap_ops;
}

// Largest t < ntables with off[t] <= i.
__device__ __forceinline__ uint32_t table_of(const uint32_t *__restrict__ off, uint32_t ntables,
                                             uint32_t i) {
    uint32_t lo = 0, hi = ntables;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Table of op i through the coarse index tidx (the table of every
// kTidxStep-th op, filled by k_set_prep): a lower bound, then a forward scan
// over the offsets. Replaces a binary search of log2(ntables) dependent loads
// per lookup.
__device__ __forceinline__ uint32_t table_at(const uint32_t *__restrict__ tidx,
                                             const uint32_t *__restrict__ bound, uint32_t i,
                                             uint32_t op) {
    uint32_t t = __ldg(tidx + (op / kTidxStep));
    while (__ldg(bound + t + 1) <= i) ++t;
    return t;
}

// Start of a set batch of off[ntables] ops, in one launch: zero the batch
// counters (all but kCtrHostN, copied in before this kernel), the probe
// phase's counters (gctr, gctr_words words), the result bits and the per-
// table new-key counts; set the single bits; fill the op index and the bins'
// tables.
template <int KB>
__global__ void __launch_bounds__(256) k_set_prep(const __grid_constant__ ApplyScratch A,
                                                  const uint32_t *__restrict__ off,
                                                  uint32_t *__restrict__ bits,
                                                  unsigned long long *__restrict__ gctr,
                                                  uint32_t gctr_words) {
    after_previous();
    const uint64_t n = set_op_count(A, off);
    const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    if (id < (uint64_t)kCtrSlots && id != (uint64_t)kCtrHostN) A.ctr[id] = 0ull;
    if (gctr != nullptr && id < gctr_words) gctr[id] = 0ull;
    for (uint64_t t = id; t < A.ntables; t += stride) A.tup[t] = A.ter[t] = 0u;
    for (uint64_t b = id; b * kTidxStep < n; b += stride) {
        const uint32_t i = (uint32_t)(b * kTidxStep), t = table_of(off, A.ntables, i);
        A.tidx[b] = t;
        if (i % kSetBinMean != 0u) continue;
        // a bin starts here: its first table, and whether it is the only one
        const uint32_t end = (uint32_t)(n - i < kSetBinMean ? n : i + kSetBinMean);
        A.bin_tables[i / kSetBinMean] = make_uint2(t, off[t + 1] >= end ? 1u : 0u);
    }
    for (uint64_t w = id; w < (n + 31) / 32; w += stride) {
        if (bits != nullptr) bits[w] = 0u;
        A.single[w] = 0xffffffffu;
    }
}

// Block-wide exclusive allocation of F counters at once: x packs F fields of
// B bits (no field's block total may exceed B bits); one scan, one atomic per
// nonzero field total, out[f] = that counter's base + the field's sum over
// the threads before this one. Every thread of the block must call it at the
// same point.
template <int F, int B>
__device__ __forceinline__ void block_alloc(unsigned long long *ctr, const int (&slot)[F],
                                            unsigned long long x, uint32_t (&out)[F]) {
    __shared__ unsigned long long wsum[32];
    __shared__ unsigned long long bbase[F];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned long long mask = B == 64 ? ~0ull : ((1ull << B) - 1ull);
    unsigned long long incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
        const unsigned long long v = lane < nw ? wsum[lane] : 0ull;
        unsigned long long vi = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, vi, o);
            if (lane >= o) vi += y;
        }
        if (lane < nw) wsum[lane] = vi - v;
        if (lane == 31) {
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const unsigned long long tot = (vi >> (f * B)) & mask;
                bbase[f] = tot ? atomicAdd(&ctr[slot[f]], tot) : 0ull;
            }
        }
    }
    __syncthreads();
    const unsigned long long ex = wsum[w] + incl - x;
#pragma unroll
    for (int f = 0; f < F; ++f) out[f] = (uint32_t)(bbase[f] + ((ex >> (f * B)) & mask));
    __syncthreads();  // wsum / bbase are reused by the next call
}

// Add 1 to cnt[t] for every lane with pred, one atomic per distinct t in the
// warp. All 32 lanes must call.
__device__ __forceinline__ void warp_count_by(uint32_t *cnt, uint32_t t, bool pred) {
    const unsigned peers = __match_any_sync(kFull, pred ? t : 0xffffffffu);
    const int lane = threadIdx.x & 31;
    if (pred && (__ffs(peers) - 1) == lane) atomicAdd(&cnt[t], (uint32_t)__popc(peers));
}

__device__ __forceinline__ uint32_t seg_off(const ApplyScratch &A, uint32_t d) {
    return (uint32_t)(A.dseg[d] >> 32);
}

// State after one op (an insert stores inval, an erase removes, any other
// code reads).
__device__ __forceinline__ void replay_op(uint8_t op, uint64_t inval, bool &present,
                                          uint64_t &value) {
    if (op == kOpInsert) {
        present = true;
        value = inval;
    } else if (op == kOpErase) {
        present = false;
        value = 0ull;
    }
}

// ----------------------------------------------------------------------------
// The ops of a mixed batch that are their keys' only ones: the whole batch
// when the caller promises distinct keys (DYC_FLAG_UNIQUE), else those whose
// bit the grouping left set in `single` (key-0 ops too). With one op per key
// no op depends on another, so each is resolved and applied in a single pass.
// An op probes its key's first bucket, and the second one where the key or
// (for an insert) an empty slot may be there; it reports the key's state
// before it. Then an insert updates the key's own slot or claims an empty one
// (ops left without a slot go to list_a for the eviction walks that follow
// the pass), and an erase clears the key's slot. Ops on different keys run
// side by side: nothing in the pass moves an entry, so a find never misses a
// key that is present, and a key's own slot is written only by its own op.
// Bound by its random lines; five blocks an SM keep more of them in flight than
// the registers would allow by themselves (2^22 ops: 4-byte keys 185 -> 176 us,
// 8-byte keys, three blocks, 207 -> 183; six spill: 197 and 198).
// ----------------------------------------------------------------------------
template <int KB, int SB, bool HINT>
__global__ void __launch_bounds__(256, 5) k_apply_unique(
    const __grid_constant__ Desc D, const __grid_constant__ Scratch S,
    const uint8_t *__restrict__ ops, const void *__restrict__ keys,
    const void *__restrict__ vals, uint32_t vb, void *__restrict__ vals_out,
    uint32_t *__restrict__ bits_out, uint64_t n, Counters *ctr, const uint32_t *single,
    uint32_t flags) {
    after_previous();
    using T = SlotT<KB>;
    using Sl = typename T::S;
    using Gm = Geo<KB, SB>;
    const bool all_ops = single == nullptr;
    __shared__ __align__(128) unsigned char s_stage[SB >= 64 ? kWarpsPerBlock : 1][32 * SB];
    unsigned char *stage = s_stage[SB >= 64 ? (threadIdx.x >> 5) : 0];
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t step = warp_stride();
    const unsigned long long tpol = HINT ? l2_policies(true).table : 0ull;
    uint32_t n_ins = 0, n_upd = 0, n_del = 0;
    for (uint64_t base = warp_base(); base < n; base += step) {
        const uint64_t i = base + lane;
        typename T::K k = 0;
        uint8_t op = kOpFind;
        Sl e = T::empty();
        bool mine = i < n;  // this kernel resolves op i
        if (mine && !all_ops) mine = (single[i >> 5] >> (i & 31)) & 1u;  // one op, or key 0
        if (mine) {
            k = load_key<KB>(keys, i);
            op = ops[i];
        }
        const bool act = k != 0;  // ops on key 0 miss and change nothing
        const bool ins = act && op == kOpInsert, del = act && op == kOpErase;
        if (ins) e = T::make(k, load_val(vals, vb, i));
        const uint32_t hk = fold(k);
        const Pair p = pair_of(hk, D.d);
        char *p1 = bucket_ptr<KB, SB>(D, p.first, bucket_index(D, p.first, hk));
        char *p2 = bucket_ptr<KB, SB>(D, p.second, bucket_index(D, p.second, hk));
        const KvOut r1 = place_probe<KB, SB, HINT>(p1, k, act, p.first, D.d, stage, tpol);
        const bool found1 = act && r1.match >= 0;
        // the second bucket holds the key only if the first one's fingerprint
        // bit allows it (always without metadata); an insert also looks there
        // for an empty slot when the first bucket is full
        const bool check2 =
            act && !found1 && ((!Gm::kMeta || r1.overflow) || (ins && r1.empty == 0u));
        KvOut r2{-1, 0ull, false, 0u};
        if (__any_sync(kFull, check2))
            r2 = place_probe<KB, SB, HINT>(p2, k, check2, p.second, D.d, stage, tpol);
        const bool found2 = check2 && r2.match >= 0;
        const bool present = found1 || found2;
        const uint64_t before = found1 ? r1.value : (found2 ? r2.value : 0ull);
        bool pend = false;
        if (ins) {
            if (present && (flags & kBinSkipEqual) && before == T::val(e)) {
                // the key's value stays: neither written nor counted
            } else if (found1) {
                T::store(slot_ptr<KB, SB>(p1, r1.match), e);
                ++n_upd;
            } else if (found2) {
                T::store(slot_ptr<KB, SB>(p2, r2.match), e);
                ++n_upd;
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
        if (vals_out != nullptr && mine) store_val(vals_out, vb, i, before);
        const unsigned m = __ballot_sync(kFull, present);
        if (bits_out != nullptr && lane == 0) {
            if (all_ops) bits_out[base >> 5] = m;
            else if (m) atomicOr(&bits_out[base >> 5], m);  // the replays own the other bits
        }
        __syncwarp();
        const unsigned long long at = agg_inc(&ctr->pending, pend);
        if (pend) {
            if (at < S.list_cap) ((Sl *)S.list_a)[at] = e;
            else atomicAdd(&ctr->spill, 1ull);
        }
    }
    // one atomic per counter per block
    __shared__ unsigned long long s_sum[3];
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0ull;
    __syncthreads();
    const uint32_t w_ins = __reduce_add_sync(kFull, n_ins), w_upd = __reduce_add_sync(kFull, n_upd);
    const uint32_t w_del = __reduce_add_sync(kFull, n_del);
    if (lane == 0) {
        if (w_ins) atomicAdd(&s_sum[0], (unsigned long long)w_ins);
        if (w_upd) atomicAdd(&s_sum[1], (unsigned long long)w_upd);
        if (w_del) atomicAdd(&s_sum[2], (unsigned long long)w_del);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_sum[0]) atomicAdd(&ctr->inserted, s_sum[0]);
        if (s_sum[1]) atomicAdd(&ctr->updated, s_sum[1]);
        if (s_sum[2]) atomicAdd(&ctr->erased, s_sum[2]);
        const long long net = (long long)s_sum[0] - (long long)s_sum[2];
        if (net) atomicAdd(&ctr->size, (unsigned long long)net);  // size += inserted - erased
    }
}

// The upserts and erases k_apply_unique would make (with kBinSkipEqual) for
// the ops whose single bit is set: a batch whose upsize policy needs the counts
// first. Finds are not probed. (Five blocks an SM: 8-byte keys 149 -> 121 us.)
template <int KB, int SB>
__global__ void __launch_bounds__(256, 5) k_apply_count(
    const __grid_constant__ Desc D, const uint8_t *__restrict__ ops, const void *__restrict__ keys,
    const void *__restrict__ vals, uint32_t vb, uint64_t n, const uint32_t *__restrict__ single,
    Counters *ctr) {
    after_previous();
    using T = SlotT<KB>;
    using Gm = Geo<KB, SB>;
    __shared__ __align__(128) unsigned char s_stage[kWarpsPerBlock][32 * SB];
    unsigned char *stage = s_stage[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t step = warp_stride();
    uint32_t n_up = 0, n_er = 0;
    for (uint64_t base = warp_base(); base < n; base += step) {
        const uint64_t i = base + lane;
        typename T::K k = 0;
        uint8_t op = kOpFind;
        if (i < n && ((single[i >> 5] >> lane) & 1u)) {
            op = ops[i];
            if (op == kOpInsert || op == kOpErase) k = load_key<KB>(keys, i);
        }
        const bool act = k != 0;
        const uint64_t v = act && op == kOpInsert ? load_val(vals, vb, i) : 0ull;
        const uint32_t hk = fold(k);
        const Pair p = pair_of(hk, D.d);
        const char *p1 = bucket_ptr<KB, SB>(D, p.first, bucket_index(D, p.first, hk));
        const KvOut r1 = kv_probe<KB, SB, 1>(p1, k, act, stage);
        bool hit = act && r1.match >= 0;
        uint64_t before = r1.value;
        const bool need2 = act && !hit && (!Gm::kMeta || r1.overflow);
        if (__any_sync(kFull, need2)) {
            const char *p2 = bucket_ptr<KB, SB>(D, p.second, bucket_index(D, p.second, hk));
            const KvOut r2 = kv_probe<KB, SB, 1>(p2, k, need2, stage);
            if (need2 && r2.match >= 0) {
                hit = true;
                before = r2.value;
            }
        }
        if (act && op == kOpInsert && (!hit || before != v)) ++n_up;
        if (act && op == kOpErase && hit) ++n_er;
    }
    __shared__ unsigned long long s_sum[2];
    if (threadIdx.x < 2) s_sum[threadIdx.x] = 0ull;
    __syncthreads();
    n_up = __reduce_add_sync(kFull, n_up);
    n_er = __reduce_add_sync(kFull, n_er);
    if (lane == 0) {
        if (n_up) atomicAdd(&s_sum[0], (unsigned long long)n_up);
        if (n_er) atomicAdd(&s_sum[1], (unsigned long long)n_er);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_sum[0]) atomicAdd(&ctr->nins, s_sum[0]);
        if (s_sum[1]) atomicAdd(&ctr->erased, s_sum[1]);
    }
}

// *count += the INSERT ops among ops[0..n) (one atomic per block).
template <int KB>
__global__ void __launch_bounds__(256) k_count_inserts(const uint8_t *__restrict__ ops, uint64_t n,
                                                       unsigned long long *count) {
    uint32_t c = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    // 16 ops a load where the array allows it
    const uint64_t n16 = ((uintptr_t)ops & 15u) == 0 ? n / 16 : 0;
    for (uint64_t i = id; i < n16; i += stride) {
        const uint4 v = __ldg((const uint4 *)ops + i);
        const uint32_t one = kOpInsert * 0x01010101u;
        c += (__popc(__vcmpeq4(v.x, one)) + __popc(__vcmpeq4(v.y, one)) + __popc(__vcmpeq4(v.z, one)) +
              __popc(__vcmpeq4(v.w, one))) / 8;
    }
    for (uint64_t i = n16 * 16 + id; i < n; i += stride) c += ops[i] == kOpInsert ? 1u : 0u;
    __shared__ unsigned long long s_c;
    if (threadIdx.x == 0) s_c = 0ull;
    __syncthreads();
    c = __reduce_add_sync(kFull, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_c, (unsigned long long)c);
    __syncthreads();
    if (threadIdx.x == 0 && s_c) atomicAdd(count, s_c);
}

}  // namespace dyc
