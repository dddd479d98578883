// The launches of a set batch's grouping and replay under a cap on the resident
// blocks (dyc_set_configure), without a GPU: the runtime's launch call is
// defined here, ahead of the library's, and keeps the shapes.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "dyc_internal.h"

static std::vector<cudaLaunchConfig_t> g_launches;

extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) {
    g_launches.push_back(*c);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

// Launches of set_group and repeat for n ops: prints block counts and dynamic
// shared memory, the grouping's last but one.
template <int KB> void run(int cap, uint64_t n) {
    g_launches.clear();
    dyc::LaunchCtx L{152, nullptr, cap};
    dyc::ApplyScratch A{};
    A.ntables = 64;
    dyc::BinScratch B{};
    B.nbins = (uint32_t)dyc::set_nbins(n);
    if (dyc::Ops<KB>::set_group(L, A, B, nullptr, nullptr, nullptr, n, true, nullptr, nullptr) != cudaSuccess ||
        dyc::Ops<KB>::repeat(L, A, nullptr, 64, 128, true, nullptr, nullptr, KB, nullptr, nullptr, n) != cudaSuccess)
        exit(1);
    for (size_t i = 0; i < g_launches.size(); ++i)
        printf("%d %llu %s %u %zu\n", cap, (unsigned long long)n,
               i + 2 == g_launches.size() ? "group" : "loop", g_launches[i].gridDim.x,
               g_launches[i].dynamicSmemBytes);
}

int main() {
    for (int cap = 0; cap <= 8; ++cap)
        for (uint64_t n : {100ull, 100000ull, 1ull << 24}) {
            run<4>(cap, n);
            run<8>(cap, n);
        }
    return 0;
}
