// dyc_bins_ops.cuh -- host launchers of the bin kernels (dyc_bins.cuh) for one
// key width. Included by dyc_bins4.cu and dyc_bins8.cu, which compile beside
// dyc_ops4.cu and dyc_ops8.cu, and by dyc_bins_sb.cuh.
#pragma once

#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

#include "dyc_bins.cuh"

namespace dyc {

// Raise a kernel's dynamic shared memory limit, once per device.
inline cudaError_t allow_smem(const void *kernel, int bytes) {
    static std::mutex mu;
    static std::set<std::pair<int, const void *>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(mu);
    if (done.count({dev, kernel})) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.insert({dev, kernel});
    return e;
}

// A grid within a tuner's cap on the resident blocks.
inline unsigned capped(const LaunchCtx &L, uint64_t blocks) {
    const uint64_t cap = (uint64_t)std::max(L.max_blocks_per_sm, 0) * (uint64_t)std::max(L.sms, 1);
    return (unsigned)(cap && blocks > cap ? cap : std::max<uint64_t>(blocks, 1));
}

// The same for a kernel with a block for every bin: dynamic shared memory that
// leaves an SM room for no more blocks (`used` bytes each) than the cap.
constexpr size_t kSmemPerSm = 228 << 10;
inline size_t cap_pad(const LaunchCtx &L, size_t used) {
    if (L.max_blocks_per_sm <= 0) return 0;
    const size_t bytes = kSmemPerSm / (size_t)(L.max_blocks_per_sm + 1) + 16;
    return bytes > used ? bytes - used : 0;
}

// The split, the bins that went over, and the grouping (cap_n sizes the grids;
// a set's kernels read the op count on the device, and it is cap_n if sized).
template <int KB, int MODE, bool SET>
cudaError_t bin_passes(const LaunchCtx &L, const BinScratch &B, const ApplyScratch &A,
                       const uint32_t *off, const uint8_t *ops, const void *keys, uint64_t cap_n,
                       unsigned long long *ctr, uint32_t *bits, bool sized = true) {
    // whole waves of the blocks an SM holds, of at most 16 ops a thread (below
    // 2^21 ops, where 8 fill the chip, of 8)
    const uint64_t slots = (SET ? 3u : 2u) * (uint64_t)std::max(L.sms, 1), unit = kSplitThreads;
    const uint64_t per = cap_n >= (1ull << 21) ? 16 : 8;
    const uint64_t waves = (cap_n + slots * per * unit - 1) / (slots * per * unit);
    const uint64_t share = (cap_n + waves * slots - 1) / (waves * slots);
    const uint32_t tile = (uint32_t)((share + unit - 1) / unit * unit);
    const unsigned blocks = capped(L, (cap_n + tile - 1) / tile);
    auto split = per == 16 ? k_bin_scatter<KB, 16, SET, false> : k_bin_scatter<KB, 8, SET, false>;
    launch_after(split, blocks, kSplitThreads, 0, L.stream, B, A, off, ops, keys, cap_n, ctr, bits, tile);
    // nothing to do in most batches: a fixed grid of one wave
    const unsigned some = capped(L, std::min<uint64_t>((cap_n + 8 * unit - 1) / (8 * unit),
                                                       4u * (uint64_t)std::max(L.sms, 1)));
    if constexpr (MODE == kBinModeMixed)
        launch_after(k_bin_scatter<KB, 8, SET, true>, some, kSplitThreads, 0, L.stream, B, A, off, ops, keys,
                     cap_n, ctr, nullptr, 8u * kSplitThreads);
    else
        launch_after(k_bin_hot<KB, MODE>, some, kSplitThreads, 0, L.stream, B, A, keys, cap_n);
    auto group = k_bin_group<KB, MODE, SET>;
    const size_t pad = cap_pad(L, kGroupSmem<SET>);
    if (pad) {
        const cudaError_t e = allow_smem((const void *)group, (int)(kSmemPerSm / 2));
        if (e != cudaSuccess) return e;
    }
    launch_after(group, SET ? (unsigned)set_nbins(cap_n) : B.nbins, kGroupThreads, pad, L.stream, B, A, off,
                 keys, sized);
    return cudaGetLastError();
}

template <int KB>
cudaError_t Ops<KB>::bin_group(const LaunchCtx &L, const BinScratch &B, const ApplyScratch &A,
                               int mode, const uint8_t *ops, const void *keys, uint32_t *bits_out,
                               uint64_t n, Counters *ctr) {
    if (n == 0) return cudaSuccess;
    unsigned long long *c = &ctr->inserted;
    if (mode == kBinModeInsert)
        return bin_passes<KB, kBinModeInsert, false>(L, B, A, nullptr, ops, keys, n, c, bits_out);
    if (mode == kBinModeErase)
        return bin_passes<KB, kBinModeErase, false>(L, B, A, nullptr, ops, keys, n, c, bits_out);
    return bin_passes<KB, kBinModeMixed, false>(L, B, A, nullptr, ops, keys, n, c, bits_out);
}

template <int KB>
cudaError_t Ops<KB>::set_group(const LaunchCtx &L, const ApplyScratch &A, const BinScratch &B,
                               const uint32_t *off, const uint8_t *ops, const void *keys,
                               uint64_t n, bool sized, uint32_t *bits, Counters *gctr) {
    const uint64_t work = std::max<uint64_t>(n / 32 + 1, A.ntables);
    launch_after(k_set_prep<KB>, capped(L, std::min<uint64_t>((work + 255) / 256, 8ull * L.sms)), 256, 0,
                 L.stream, A, off, bits, (unsigned long long *)gctr, (uint32_t)(sizeof(Counters) / 8));
    if (n == 0) return cudaGetLastError();
    return bin_passes<KB, kBinModeMixed, true>(L, B, A, off, ops, keys, n, nullptr, nullptr, sized);
}

// The launchers of a bucket size (BinsSb).
#define DYC_BINS_SB(sb, call) \
    (sb == 32 ? BinsSb<KB, 32>::call : sb == 64 ? BinsSb<KB, 64>::call : BinsSb<KB, 128>::call)

template <int KB>
cudaError_t Ops<KB>::repeat(const LaunchCtx &L, const ApplyScratch &A, const Desc *descs,
                            uint32_t ntables, int sb, bool set, const uint8_t *ops,
                            const void *vals, uint32_t vb, void *vals_out, uint32_t *bits_out,
                            uint64_t n, void *list_a, uint64_t list_cap, Counters *gctr) {
    if (n == 0) return cudaSuccess;
    return DYC_BINS_SB(sb, repeat(L, A, descs, ntables, set, ops, vals, vb, vals_out, bits_out, n, list_a,
                                  list_cap, gctr));
}

template <int KB>
cudaError_t Ops<KB>::bin_small(const LaunchCtx &L, const Desc &D, int sb, const Scratch &S,
                               int mode, const uint8_t *ops, const void *keys, const void *vals,
                               uint32_t vb, void *vals_out, uint32_t *bits_out, uint64_t n,
                               uint32_t flags, Counters *ctr, Counters *h_ctr) {
    if (n == 0) return cudaSuccess;
    const uint64_t words = bits_out ? (n + 31) / 32 : 0;
    launch_after(k_small_clear<KB>, (unsigned)((words + 255) / 256 + 1), 256, 0, L.stream, &ctr->inserted,
                 (uint32_t)(sizeof(Counters) / 8 - 1), bits_out, words);
    return DYC_BINS_SB(sb, small(L, D, S, mode, ops, keys, vals, vb, vals_out, bits_out, n, flags, ctr, h_ctr));
}

}  // namespace dyc
