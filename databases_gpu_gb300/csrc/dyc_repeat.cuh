// dyc_repeat.cuh -- the keys with several ops in a mixed batch (listed by
// k_bin_group), each resolved once: one probe of its buckets gives its state
// before the batch, its ops are replayed in index order, every op's result is
// written, and the final state goes to the table (MUT) or to the upsert and
// erase lists (where the upsize policy must run in between).
#pragma once

#include "dyc_bins.cuh"

namespace dyc {

// Key d of every lane with act (warp-collective).
template <int KB, int SB, bool SET>
__device__ __forceinline__ RepKey<KB> probe_listed(const ApplyScratch &A, const Desc *__restrict__ descs,
                                                   uint32_t ntables, uint32_t d, bool act,
                                                   unsigned char *stage) {
    RepKey<KB> x;
    x.k = 0;
    x.tb = 0u;
    if (act) {
        x.k = ((const typename SlotT<KB>::K *)A.dkey)[d];
        if (SET) x.tb = A.dtid[d];
        if (x.tb >= ntables) {
            note_bad(A);
            x.tb = 0u;
            x.k = 0;
        }
    }
    const uint32_t tb = x.tb;
    x = probe_key<KB, SB>(descs[tb], x.k, act && x.k != 0, stage);
    x.tb = tb;
    return x;
}

// Ascending sort of a warp's 32 * R words, the word at place lane * R + r in
// s[r]: a bitonic network in registers, across lanes by shuffles.
template <int R> __device__ __forceinline__ void warp_sort(uint32_t (&s)[R]) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= R) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint32_t e = lane * R + r;
                    const uint32_t o = __shfl_xor_sync(kFull, s[r], j / R);
                    const bool low = ((e & j) == 0) == ((e & k) == 0);
                    s[r] = low ? min(s[r], o) : max(s[r], o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r & j) continue;
                    const bool up = ((lane * R + r) & k) == 0;
                    const uint32_t a = min(s[r], s[r | j]), b = max(s[r], s[r | j]);
                    s[r] = up ? a : b;
                    s[r | j] = up ? b : a;
                }
            }
        }
    }
}

// Ops of one key, up to 32 * R of them, by one warp: the op indexes sorted in
// registers (element e in lane e / R; merges across lanes by shuffles), then
// each lane takes its R consecutive ops. The op codes and values of all ops
// are read at once, so a segment costs two dependent memory round trips
// whatever its length. (Sorted in shared memory and replayed 32 ops a step,
// the segments of a 4096-table round took 407 us of a warp kernel of their
// own.)
template <int R>
__device__ __forceinline__ void warp_segment(const uint32_t *__restrict__ seg, uint32_t cnt,
                                             bool &present, uint64_t &value,
                                             const SegOps &ops,
                                             const void *__restrict__ vals, uint32_t vb,
                                             void *__restrict__ vals_out,
                                             uint32_t *__restrict__ bits_out) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t e = lane * R + r;
        s[r] = e < cnt ? seg[e] : 0xffffffffu;
    }
    warp_sort<R>(s);
    uint8_t op[R];
    uint64_t in[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool v = s[r] != 0xffffffffu;  // no op word: indexes end below 2^30 and 2^31
        op[r] = v ? ops.code(s[r]) : (uint8_t)kOpFind;
        if (v) s[r] = ops.index(s[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) in[r] = op[r] == kOpInsert ? load_val(vals, vb, s[r]) : 0ull;
    bool mut = false, last_present = false;
    uint64_t last_value = 0ull;
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (op[r] == kOpInsert || op[r] == kOpErase) {
            mut = true;
            last_present = op[r] == kOpInsert;
            last_value = in[r];
        }
    // the state a lane's ops meet: the last mutation of the lanes before it
    const unsigned mm = __ballot_sync(kFull, mut);
    const unsigned mp = __ballot_sync(kFull, last_present);
    const unsigned before = mm & ((1u << lane) - 1u);
    const int src = before ? 31 - __clz(before) : (int)lane;
    const uint64_t sv = shfl64(last_value, src);
    bool st = before ? (mp >> src) & 1u : present;
    uint64_t sval = before ? (st ? sv : 0ull) : value;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (s[r] == 0xffffffffu) continue;
        if (vals_out) store_val(vals_out, vb, s[r], st ? sval : 0ull);
        if (st && bits_out) atomicOr(&bits_out[s[r] >> 5], 1u << (s[r] & 31));
        replay_op(op[r], in[r], st, sval);
    }
    if (mm) {
        const int last = 31 - __clz(mm);
        const uint64_t lv = shfl64(last_value, last);
        present = (mp >> last) & 1u;
        value = present ? lv : 0ull;
    }
}

// The block's warps sort src[0..cnt) into s in runs of kSortRun words.
constexpr uint32_t kSortRun = 128;
__device__ __forceinline__ void sort_runs(const uint32_t *src, uint32_t cnt, uint32_t *s) {
    constexpr int R = (int)kSortRun / 32;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t first = (threadIdx.x >> 5) * kSortRun; first < cnt; first += kWarpsPerBlock * kSortRun) {
        uint32_t x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t e = first + r * 32u + lane;
            x[r] = e < cnt ? src[e] : 0xffffffffu;
        }
        warp_sort<R>(x);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (first + lane * R + r < cnt) s[first + lane * R + r] = x[r];
    }
    __syncthreads();
}

// Sorted runs of w words (the last one shorter) of src[0..cnt) merged in pairs
// into dst, each word placed by its rank in the other run (op indices are
// distinct, so ranks are exact). By the whole block.
__device__ __forceinline__ void merge_runs(const uint32_t *src, uint32_t *dst, uint32_t cnt, uint32_t w) {
    for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
        const uint32_t r0 = i / (2 * w) * (2 * w);
        const uint32_t mid = r0 + w < cnt ? r0 + w : cnt;
        const uint32_t end = r0 + 2 * w < cnt ? r0 + 2 * w : cnt;
        const uint32_t v = src[i];
        // rank of v in the other run (elements smaller than v)
        uint32_t lo = i < mid ? mid : r0, hi = i < mid ? end : mid;
        const uint32_t base = lo;
        while (lo < hi) {
            const uint32_t m = (lo + hi) >> 1;
            if (src[m] < v) lo = m + 1;
            else hi = m;
        }
        const uint32_t own = i < mid ? i - r0 : i - mid;
        dst[r0 + own + (lo - base)] = v;
    }
    __syncthreads();
}

// Up to kMidSeg words of src sorted by the block in s (2 * kMidSeg words):
// runs by its warps in registers, then rounds of merges. Returns where they
// are. (One bitonic network over all words in shared memory, a barrier a
// stage: 663 us for 2^22 ops on 5000 keys, now 457; on 1500 keys 915, now 590.
// Runs of up to 512 words a warp spilled 200 bytes.)
__device__ __forceinline__ uint32_t *mid_sort(const uint32_t *src, uint32_t cnt, uint32_t *s) {
    sort_runs(src, cnt, s);
    uint32_t *t = s + kMidSeg;
    for (uint32_t w = kSortRun; w < cnt; w *= 2) {
        merge_runs(s, t, cnt, w);
        uint32_t *x = s;
        s = t;
        t = x;
    }
    return s;
}

// Sort the segment of one key with more than kWarpSeg ops by the whole block:
// in shared memory up to kMidSeg ops, beyond that in kMidSeg chunks merged in
// global memory, run widths doubling, ping-ponging between src and dst. Returns
// the sorted indices.
__device__ __forceinline__ const uint32_t *block_sort(uint32_t *src, uint32_t *dst, uint32_t cnt,
                                                      uint32_t *s) {
    if (cnt <= kMidSeg) return mid_sort(src, cnt, s);
    for (uint32_t c0 = 0; c0 < cnt; c0 += kMidSeg) {  // sorted chunks, in place
        const uint32_t m = cnt - c0 < kMidSeg ? cnt - c0 : kMidSeg;
        const uint32_t *r = mid_sort(src + c0, m, s);
        for (uint32_t j = threadIdx.x; j < m; j += blockDim.x) src[c0 + j] = r[j];
        __syncthreads();
    }
    for (uint32_t w = kMidSeg; w < cnt; w *= 2) {  // merge runs of w into runs of 2w
        merge_runs(src, dst, cnt, w);
        uint32_t *t = src;
        src = dst;
        dst = t;
    }
    return src;
}

// A lane's key (act) to the lists of changes, at place u (upserts) or e (erases).
template <int KB>
__device__ __forceinline__ void list_change(const ApplyScratch &A, const RepKey<KB> &x, bool up,
                                            bool er, uint64_t value, uint32_t vb,
                                            unsigned long long u, unsigned long long e) {
    using K = typename SlotT<KB>::K;
    if ((up && u >= A.cap_ops) || (er && e >= A.cap_ops)) {
        note_bad(A);
    } else if (up) {
        ((K *)A.up_key)[u] = x.k;
        store_val(A.up_val, vb, u, value);
        if (A.up_tid) A.up_tid[u] = x.tb;
    } else if (er) {
        ((K *)A.er_key)[e] = x.k;
        if (A.er_tid) A.er_tid[e] = x.tb;
    }
}

// Bound by the latency of its probes and segment reads. A set's rounds have
// many segments for a warp each, and a fourth block an SM hides more of them:
// 2^25 ops over 4096 tables 495 -> 430 us; with five the spilled registers cost
// as much, and a single table's short segments are faster with three.
template <int KB, int SB, bool SET, bool MUT>
__global__ void __launch_bounds__(256, SET ? 4 : 3) k_repeat(
    const __grid_constant__ ApplyScratch A, const Desc *__restrict__ descs, uint32_t ntables,
    const uint8_t *__restrict__ ops, const void *__restrict__ vals, uint32_t vb,
    void *__restrict__ vals_out, uint32_t *__restrict__ bits_out, void *list_a, uint64_t list_cap,
    Counters *gctr) {
    after_previous();
    constexpr int kStage = 32 * SB * kWarpsPerBlock;
    constexpr int kSort = (int)(2 * kMidSeg * sizeof(uint32_t));
    __shared__ __align__(128) unsigned char s_raw[kStage > kSort ? kStage : kSort];
    unsigned char *stage = s_raw + (threadIdx.x >> 5) * (32 * SB);
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const SegOps so{ops, A.wide};
    RepCounts n;
    // a lane's final state, outside the block-wide allocation of the short keys
    auto finish = [&](const RepKey<KB> &x, bool act, bool present, uint64_t value) {
        const bool up = act && present && (!x.pre || value != x.pre_value);
        const bool er = act && !present && x.pre;
        if constexpr (MUT) {
            mutate_listed<KB, SB>(x, up, er, value, list_a, list_cap, gctr, n);
        } else {
            const unsigned long long u = agg_inc(&A.ctr[kCtrUp], up);
            const unsigned long long e = agg_inc(&A.ctr[kCtrEr], er);
            if (A.tup) {
                warp_count_by(A.tup, x.tb, up);
                warp_count_by(A.ter, x.tb, er);
            }
            list_change<KB>(A, x, up, er, value, vb, u, e);
        }
    };
    // keys with more than kWarpSeg ops: a block each
    const uint64_t nmid = ctr_count(A, kCtrMid);
    for (uint64_t y = blockIdx.x; y < nmid; y += gridDim.x) {
        const uint32_t d = A.mid[y];  // d, cnt and off are the same for the whole block
        if (d >= A.cap_ops) {
            if (tid == 0) note_bad(A);
            continue;
        }
        const uint32_t cnt = A.dcnt[d], off = seg_off(A, d);
        if (cnt <= kWarpSeg || !seg_ok(A, off, cnt)) {
            if (tid == 0) note_bad(A);
            continue;
        }
        const uint32_t *sorted = block_sort(A.seg + off, A.sort_tmp + off, cnt, (uint32_t *)s_raw);
        __syncthreads();
        // the sorted indices fill the other warps' stages
        __shared__ __align__(128) unsigned char s_one[SB >= 64 ? 32 * SB : 16];
        __shared__ uint64_t s_before;
        __shared__ uint32_t s_present;
        RepKey<KB> x;
        if (tid < 32) {
            x = probe_listed<KB, SB, SET>(A, descs, ntables, d, lane == 0, s_one);
            if (tid == 0) {
                s_present = x.pre ? 1u : 0u;
                s_before = x.pre_value;
            }
        }
        __syncthreads();
        bool present = s_present != 0u;
        uint64_t value = s_before;
        block_replay<kBlockThreads, true>(sorted, cnt, present, value, so, vals, vb, vals_out, bits_out);
        if (tid < 32) finish(x, lane == 0 && x.k != 0, present, value);
        __syncthreads();  // the sorted indices are reused by the next segment
    }
    // keys with more than kShortSeg: a warp each, kWarpTask of them probed together
    const uint64_t nw = ctr_count(A, kCtrWarp);
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + tid) >> 5;
    for (uint64_t x0 = gw * kWarpTask; x0 < nw; x0 += warps * kWarpTask) {
        uint32_t d = 0u, cnt = 0u, off = 0u;
        bool act = lane < kWarpTask && x0 + lane < nw;
        if (act) {
            d = A.wseg[x0 + lane];
            act = d < A.cap_ops;
            if (act) {
                cnt = A.dcnt[d];
                off = seg_off(A, d);
                act = cnt <= kWarpSeg && seg_ok(A, off, cnt);
            }
            if (!act) note_bad(A);
        }
        const RepKey<KB> x = probe_listed<KB, SB, SET>(A, descs, ntables, d, act, stage);
        bool present = x.pre;
        uint64_t value = x.pre_value;
        for (unsigned todo = __ballot_sync(kFull, act); todo; todo &= todo - 1u) {
            const int j = __ffs(todo) - 1;
            const uint32_t c = __shfl_sync(kFull, cnt, j);
            const uint32_t *seg = A.seg + __shfl_sync(kFull, off, j);
            bool pj = __shfl_sync(kFull, present, j);
            uint64_t vj = shfl64(value, j);
            if (c <= 32) warp_segment<1>(seg, c, pj, vj, so, vals, vb, vals_out, bits_out);
            else if (c <= 64) warp_segment<2>(seg, c, pj, vj, so, vals, vb, vals_out, bits_out);
            else if (c <= 128) warp_segment<4>(seg, c, pj, vj, so, vals, vb, vals_out, bits_out);
            else warp_segment<8>(seg, c, pj, vj, so, vals, vb, vals_out, bits_out);
            if ((int)lane == j) {
                present = pj;
                value = vj;
            }
        }
        finish(x, act && x.k != 0, present, value);
    }
    // the others: a lane each (whole blocks step, for the block-wide allocation)
    const uint64_t nd = ctr_count(A, kCtrDistinct);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const int slots[2] = {kCtrUp, kCtrEr};
    for (uint64_t d0 = (uint64_t)blockIdx.x * blockDim.x; d0 < nd; d0 += stride) {
        const uint64_t d = d0 + tid;
        const uint32_t cnt = d < nd ? A.dcnt[d] : 0u;
        bool act = cnt > 1u && cnt <= kShortSeg;  // segment inside the scratch: the grouping checked it
        uint32_t s[kShortSeg];
        const uint32_t off = act ? seg_off(A, (uint32_t)d) : 0u;
#pragma unroll
        for (uint32_t a = 0; a < kShortSeg; ++a) s[a] = act && a < cnt ? A.seg[off + a] : 0xffffffffu;
        const RepKey<KB> x = probe_listed<KB, SB, SET>(A, descs, ntables, (uint32_t)d, act, stage);
        act = act && x.k != 0;
        bool present = x.pre;
        uint64_t value = x.pre_value;
        // odd-even transposition network in registers (padding sorts last)
#pragma unroll
        for (uint32_t r = 0; r < kShortSeg; ++r) {
#pragma unroll
            for (uint32_t a = r & 1u; a + 1 < kShortSeg; a += 2) {
                const uint32_t lo = min(s[a], s[a + 1]), hi = max(s[a], s[a + 1]);
                s[a] = lo;
                s[a + 1] = hi;
            }
        }
        if (act) {
#pragma unroll
            for (uint32_t a = 0; a < kShortSeg; ++a) {
                if (a >= cnt) break;
                const uint32_t i = so.index(s[a]);
                const uint8_t op = so.code(s[a]);
                // every op reports the state just before it
                if (vals_out) store_val(vals_out, vb, i, present ? value : 0ull);
                if (present && bits_out) atomicOr(&bits_out[i >> 5], 1u << (i & 31));
                replay_op(op, op == kOpInsert ? load_val(vals, vb, i) : 0ull, present, value);
            }
        }
        if constexpr (MUT) {
            finish(x, act, present, value);
        } else {
            const bool up = act && present && (!x.pre || value != x.pre_value);
            const bool er = act && !present && x.pre;
            uint32_t got[2];
            block_alloc<2, 32>(A.ctr, slots, (unsigned long long)up | ((unsigned long long)er << 32), got);
            if (A.tup) {
                warp_count_by(A.tup, x.tb, up);
                warp_count_by(A.ter, x.tb, er);
            }
            list_change<KB>(A, x, up, er, value, vb, got[0], got[1]);
        }
    }
    if constexpr (MUT) {  // one atomic per counter per block
        __shared__ unsigned long long s_sum[3];
        __syncthreads();
        if (tid < 3) s_sum[tid] = 0ull;
        __syncthreads();
        const uint32_t ins = __reduce_add_sync(kFull, n.ins), upd = __reduce_add_sync(kFull, n.upd);
        const uint32_t del = __reduce_add_sync(kFull, n.del);
        if (lane == 0) {
            if (ins) atomicAdd(&s_sum[0], (unsigned long long)ins);
            if (upd) atomicAdd(&s_sum[1], (unsigned long long)upd);
            if (del) atomicAdd(&s_sum[2], (unsigned long long)del);
        }
        __syncthreads();
        if (tid == 0) {
            if (s_sum[0]) atomicAdd(&gctr->inserted, s_sum[0]);
            if (s_sum[1]) atomicAdd(&gctr->updated, s_sum[1]);
            if (s_sum[2]) atomicAdd(&gctr->erased, s_sum[2]);
            const long long net = (long long)s_sum[0] - (long long)s_sum[2];
            if (net) atomicAdd(&gctr->size, (unsigned long long)net);  // size += inserted - erased
        }
    }
}

}  // namespace dyc
