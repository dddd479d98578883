// Bin kernels that probe buckets, for keys of DYC_KB bytes and buckets of DYC_SB.
#include "dyc_bins_sb.cuh"
template struct dyc::BinsSb<DYC_KB, DYC_SB>;
