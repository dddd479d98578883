// dyc_bins_sb.cuh -- host launchers of the bin kernels that probe buckets
// (k_repeat, k_bin_small), for one key width and bucket size. A module each
// (dyc_bins_sb.cu): a process loads those that its calls use, when they first do
// (0.5 ms, and 0.3 for the split and grouping). As one module per key width with
// all bucket sizes, loaded with the first table, they took 1.2 to 1.4 ms of its
// creation, for callers too that only find: a first table 1.58 -> 0.40 ms, the
// first insert 1.18 -> 1.40, the first mixed batch after it 0.45 -> 0.89.
#pragma once

#include "dyc_bins_ops.cuh"
#include "dyc_repeat.cuh"

namespace dyc {

template <int KB, int SB>
cudaError_t BinsSb<KB, SB>::repeat(const LaunchCtx &L, const ApplyScratch &A, const Desc *descs,
                                   uint32_t ntables, bool set, const uint8_t *ops, const void *vals,
                                   uint32_t vb, void *vals_out, uint32_t *bits_out, uint64_t n,
                                   void *list_a, uint64_t list_cap, Counters *gctr) {
    // a listed key has at least two ops; blocks loop over keys and segments
    const uint64_t need = (n / 2 + 255) / 256 + 1, wave = 8ull * (uint64_t)(L.sms > 0 ? L.sms : 1);
    const unsigned grid = capped(L, std::min<uint64_t>(need, 2 * wave));
    auto k = set ? k_repeat<KB, SB, true, false>
                 : list_a ? k_repeat<KB, SB, false, true> : k_repeat<KB, SB, false, false>;
    launch_after(k, grid, 256, 0, L.stream, A, descs, ntables, ops, vals, vb, vals_out, bits_out, list_a,
                 list_cap, gctr);
    return cudaGetLastError();
}

template <int KB, int SB>
cudaError_t BinsSb<KB, SB>::small(const LaunchCtx &L, const Desc &D, const Scratch &S, int mode,
                                  const uint8_t *ops, const void *keys, const void *vals, uint32_t vb,
                                  void *vals_out, uint32_t *bits_out, uint64_t n, uint32_t flags,
                                  Counters *ctr, Counters *h_ctr) {
    auto k = mode == kBinModeInsert  ? k_bin_small<KB, SB, kBinModeInsert>
             : mode == kBinModeErase ? k_bin_small<KB, SB, kBinModeErase>
             : mode == kBinModeMixed ? k_bin_small<KB, SB, kBinModeMixed>
                                     : k_bin_small<KB, SB, kBinModeCount>;
    const cudaError_t e = allow_smem((const void *)k, (int)bin_smem<KB, SB>(mode, kBinSmallOps));
    if (e != cudaSuccess) return e;
    launch_after(k, (unsigned)((n + kBinSmallMean - 1) / kBinSmallMean), kSmallThreads,
                 bin_smem<KB, SB>(mode, n), L.stream, D, S, ops, keys, vals, vb, vals_out, bits_out, n, flags,
                 ctr, h_ctr);
    return cudaGetLastError();
}

}  // namespace dyc
