// dyc_bins_ops.cuh -- host launchers of the bin kernels (dyc_bins.cuh) for one
// key width. Included by dyc_bins4.cu and dyc_bins8.cu, which compile beside
// dyc_ops4.cu and dyc_ops8.cu.
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

template <int KB>
cudaError_t Ops<KB>::bin_group(const LaunchCtx &L, const BinScratch &B, const ApplyScratch &A,
                               int mode, const uint8_t *ops, const void *keys, uint32_t *bits_out,
                               uint64_t n, Counters *ctr) {
    if (n == 0) return cudaSuccess;
    const uint64_t words = (n + 31) / 32;
    k_bin_clear<KB><<<(unsigned)std::min<uint64_t>((words + 255) / 256, 1024), 256, 0, L.stream>>>(
        B, &ctr->inserted, (uint32_t)(sizeof(Counters) / 8 - 1), A.ctr, bits_out, words);
    const int smem = (int)B.nbins * 4;
    // 16 ops a thread where that still fills the chip, else 8
    if (n >= (1ull << 21))
        k_bin_scatter<KB, 16><<<(unsigned)((n + 8191) / 8192), 512, smem, L.stream>>>(B, ops, keys, n);
    else
        k_bin_scatter<KB, 8><<<(unsigned)((n + 4095) / 4096), 512, smem, L.stream>>>(B, ops, keys, n);
    auto k = mode == kBinModeInsert  ? k_bin_group<KB, kBinModeInsert>
             : mode == kBinModeErase ? k_bin_group<KB, kBinModeErase>
                                     : k_bin_group<KB, kBinModeMixed>;
    k<<<B.nbins, kGroupThreads, 0, L.stream>>>(B, A, keys, ctr);
    return cudaGetLastError();
}

using BinFn = void (*)(Desc, Scratch, BinScratch, const uint8_t *, const void *, const void *, uint32_t,
                       void *, uint32_t *, uint64_t, uint32_t, Counters *, Counters *);

template <int KB, int SB> BinFn small_kernel(int mode) {
    if (mode == kBinModeInsert) return k_bin_small<KB, SB, kBinModeInsert>;
    if (mode == kBinModeErase) return k_bin_small<KB, SB, kBinModeErase>;
    if (mode == kBinModeMixed) return k_bin_small<KB, SB, kBinModeMixed>;
    return k_bin_small<KB, SB, kBinModeCount>;
}

template <int KB>
cudaError_t Ops<KB>::bin_small(const LaunchCtx &L, const Desc &D, int sb, const Scratch &S,
                               const BinScratch &B, int mode, const uint8_t *ops, const void *keys,
                               const void *vals, uint32_t vb, void *vals_out, uint32_t *bits_out,
                               uint64_t n, uint32_t flags, Counters *ctr, Counters *h_ctr) {
    if (n == 0) return cudaSuccess;
    const uint64_t words = bits_out ? (n + 31) / 32 : 0;
    k_bin_clear<KB><<<(unsigned)((words + 255) / 256 + 1), 256, 0, L.stream>>>(
        B, &ctr->inserted, (uint32_t)(sizeof(Counters) / 8 - 1), nullptr, bits_out, words);
    const BinFn k = sb == 32   ? small_kernel<KB, 32>(mode)
                    : sb == 64 ? small_kernel<KB, 64>(mode)
                               : small_kernel<KB, 128>(mode);
    const int bytes = (int)(sb == 32   ? sizeof(BinSmem<KB, 32>)
                            : sb == 64 ? sizeof(BinSmem<KB, 64>)
                                       : sizeof(BinSmem<KB, 128>));
    const cudaError_t e = allow_smem((const void *)k, bytes);
    if (e != cudaSuccess) return e;
    k<<<B.nbins, 256, bytes, L.stream>>>(D, S, B, ops, keys, vals, vb, vals_out, bits_out, n, flags,
                                         ctr, h_ctr);
    return cudaGetLastError();
}

}  // namespace dyc
