// dyc_left.cuh -- the ops of bins that went over (dyc_bins.cuh: few keys, each
// repeated many times in the chunk), gathered in index order for the general
// path, and the way back of their results.
#pragma once

#include "dyc_bins.cuh"

namespace dyc {

// Whether op i's bin went over.
template <int KB>
__device__ __forceinline__ bool is_left(const BinScratch &B, const void *keys, uint64_t i, uint64_t n) {
    if (i >= n) return false;
    const typename SlotT<KB>::K k = load_key<KB>(keys, i);
    return k != 0 && B.count[bin_of<KB>(k, B.nbins)] > B.cap;
}

// The ops left over, per tile of kLeftTile ops.
template <int KB>
__global__ void __launch_bounds__(256) k_left_count(const __grid_constant__ BinScratch B,
                                                    const __grid_constant__ Scratch S,
                                                    const void *__restrict__ keys, uint64_t n) {
    __shared__ uint32_t s_n;
    if (threadIdx.x == 0) s_n = 0u;
    __syncthreads();
    uint32_t c = 0;
    for (int j = 0; j < kLeftTile / 256; ++j)
        c += is_left<KB>(B, keys, (uint64_t)blockIdx.x * kLeftTile + j * 256 + threadIdx.x, n) ? 1u : 0u;
    c = __reduce_add_sync(kFull, c);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_n, c);
    __syncthreads();
    if (threadIdx.x == 0) S.left_cnt[blockIdx.x] = s_n;
}

// Exclusive scan of the tiles' counts, one block.
template <int KB>
__global__ void __launch_bounds__(1024) k_left_scan(uint32_t *cnt, uint32_t tiles) {
    __shared__ uint32_t s_w[32];
    __shared__ uint32_t s_carry;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_carry = 0u;
    __syncthreads();
    for (uint32_t b = 0; b < tiles; b += 1024) {
        const uint32_t t = b + threadIdx.x;
        const uint32_t v = t < tiles ? cnt[t] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31) s_w[w] = x;
        __syncthreads();
        if (w == 0) {
            const uint32_t a = s_w[lane];
            uint32_t y = a;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t z = __shfl_up_sync(kFull, y, o);
                if (lane >= (uint32_t)o) y += z;
            }
            s_w[lane] = y - a;
        }
        __syncthreads();
        const uint32_t carry = s_carry;
        if (t < tiles) cnt[t] = carry + s_w[w] + x - v;
        __syncthreads();
        if (threadIdx.x == 1023) s_carry = carry + s_w[w] + x;
        __syncthreads();
    }
}

template <int KB>
__global__ void __launch_bounds__(256) k_left_gather(const __grid_constant__ BinScratch B,
                                                     const __grid_constant__ Scratch S,
                                                     const uint8_t *__restrict__ ops,
                                                     const void *__restrict__ keys,
                                                     const void *__restrict__ vals, uint32_t vb,
                                                     uint64_t n, void *__restrict__ keys_left,
                                                     void *__restrict__ vals_left) {
    using K = typename SlotT<KB>::K;
    __shared__ uint32_t s_w[8];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t at = S.left_cnt[blockIdx.x];
    for (int j = 0; j < kLeftTile / 256; ++j) {
        const uint64_t i = (uint64_t)blockIdx.x * kLeftTile + j * 256 + threadIdx.x;
        const bool l = is_left<KB>(B, keys, i, n);
        const unsigned vote = __ballot_sync(kFull, l);
        if (lane == 0) s_w[w] = __popc(vote);
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (uint32_t x = 0; x < 8; ++x) {
            before += x < w ? s_w[x] : 0u;
            total += s_w[x];
        }
        if (l) {
            const uint32_t r = at + before + __popc(vote & ((1u << lane) - 1u));
            S.left_idx[r] = (uint32_t)i;
            ((K *)keys_left)[r] = load_key<KB>(keys, i);
            if (vals != nullptr) store_val(vals_left, vb, r, load_val(vals, vb, i));
            if (ops != nullptr) S.left_ops[r] = ops[i];
        }
        at += total;
        __syncthreads();
    }
}

template <int KB>
__global__ void __launch_bounds__(256) k_left_return(const __grid_constant__ Scratch S, uint64_t m,
                                                     const void *__restrict__ out, uint32_t vb,
                                                     void *__restrict__ vals_out,
                                                     uint32_t *__restrict__ bits_out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += stride) {
        const uint32_t i = S.left_idx[r];
        if (vals_out != nullptr) store_val(vals_out, vb, i, load_val(out, vb, r));
        if (bits_out != nullptr && ((S.left_bits[r >> 5] >> (r & 31)) & 1u))
            atomicOr(&bits_out[i >> 5], 1u << (i & 31));
    }
}

}  // namespace dyc
