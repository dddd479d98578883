// Bin kernels and launchers for 4-byte keys.
#include "dyc_bins_ops.cuh"
template cudaError_t dyc::Ops<4>::bin_group(const LaunchCtx &, const BinScratch &,
                                            const ApplyScratch &, int, const uint8_t *,
                                            const void *, uint32_t *, uint64_t, Counters *);
template cudaError_t dyc::Ops<4>::bin_small(const LaunchCtx &, const Desc &, int, const Scratch &,
                                            int, const uint8_t *, const void *,
                                            const void *, uint32_t, void *, uint32_t *, uint64_t,
                                            uint32_t, Counters *, Counters *);
template cudaError_t dyc::Ops<4>::set_group(const LaunchCtx &, const ApplyScratch &,
                                            const BinScratch &, const uint32_t *, const uint8_t *,
                                            const void *, uint64_t, bool, uint32_t *, Counters *);
template cudaError_t dyc::Ops<4>::repeat(const LaunchCtx &, const ApplyScratch &, const Desc *,
                                         uint32_t, int, bool, const uint8_t *, const void *,
                                         uint32_t, void *, uint32_t *, uint64_t, void *, uint64_t,
                                         Counters *);
