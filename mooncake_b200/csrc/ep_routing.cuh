// Reading and counting the index matrix on the device: helpers of the dispatch
// and layout kernels.
//
// Receive order is token order, so the position of a token among the tokens that
// chose an expert is the number of EARLIER tokens that chose it. For small
// batches every block of a dispatch kernel counts them itself (count_tokens: one
// lane per token, shared-memory counters); a warp's 32 counter updates take about
// 21 cycles, so 296 tokens of 8 choices take 0.8 us, 4096 tokens would take 12 us
// in every block - larger batches have a layout kernel count once for all.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ep_device.cuh"
#include "ep_kernels.cuh"

namespace mcep {

// An entry of the index matrix as the elastic calls read it: all 64 bits decide whether it
// names an expert (negative: it does not). The legacy calls look at the low 32 bits.
__device__ __forceinline__ int all_bits(int64_t v) { return (int)(v >> 32) == 0 ? (int)v : -1; }

// The K choices of token t: e[k] = -1 for masked and out-of-range entries (and
// for k >= K). `vec`: K is even and the matrix 16-byte aligned, two choices per load.
// kWide: as all_bits.
template <int KB, bool kWide>
__device__ __forceinline__ void load_choices(const int64_t* __restrict__ topk_idx, int t, int K, int E,
                                             bool vec, int (&e)[KB]) {
    const int64_t* p = topk_idx + (size_t)t * K;
    if (vec) {
#pragma unroll
        for (int k = 0; k < KB; k += 2) {
            longlong2 v = make_longlong2(-1, -1);
            if (k < K) v = ld_ro(reinterpret_cast<const longlong2*>(p + k));
            e[k] = kWide ? all_bits(v.x) : (int)v.x, e[k + 1] = kWide ? all_bits(v.y) : (int)v.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            const int64_t v = k < K ? ld_ro(p + k) : -1;
            e[k] = kWide ? all_bits(v) : (int)v;
        }
    }
#pragma unroll
    for (int k = 0; k < KB; ++k)
        if (e[k] >= E) e[k] = -1;  // (negative already means "no expert")
}

// An expert listed twice by one token counts once: at its first listing, or at
// its last one (the elastic calls: kKeepLast).
template <int KB, bool kKeepLast>
__device__ __forceinline__ void drop_repeats(int (&e)[KB]) {
    if (kKeepLast) {
#pragma unroll
        for (int k = 0; k < KB - 1; ++k) {
            bool dup = false;
#pragma unroll
            for (int kk = k + 1; kk < KB; ++kk) dup |= (e[kk] == e[k]);
            if (dup) e[k] = -1;
        }
    } else {
#pragma unroll
        for (int k = KB - 1; k > 0; --k) {
            bool dup = false;
#pragma unroll
            for (int kk = 0; kk < k; ++kk) dup |= (e[kk] == e[k]);
            if (dup) e[k] = -1;
        }
    }
}

// Adds tokens [from, to) to hist[E] (shared memory); all threads of the block
// share the work, nobody waits. kTokens tokens per lane are requested together.
template <int KB, int kTokens, bool kKeepLast>
__device__ __forceinline__ void count_tokens_of(const int64_t* __restrict__ topk_idx, int from, int to, int K,
                                                int E, bool vec, int* hist) {
    const int nthr = blockDim.x;
    for (int t0 = from + threadIdx.x; t0 < to; t0 += nthr * kTokens) {
        int e[kTokens][KB];
#pragma unroll
        for (int u = 0; u < kTokens; ++u) {
            if (t0 + u * nthr < to) {
                load_choices<KB, kKeepLast>(topk_idx, t0 + u * nthr, K, E, vec, e[u]);
            } else {
#pragma unroll
                for (int k = 0; k < KB; ++k) e[u][k] = -1;
            }
        }
#pragma unroll
        for (int u = 0; u < kTokens; ++u) {
            drop_repeats<KB, kKeepLast>(e[u]);
#pragma unroll
            for (int k = 0; k < KB; ++k)
                if (e[u][k] >= 0) atomicAdd(&hist[e[u][k]], 1);
        }
    }
}

template <int kTokens, bool kKeepLast = false>
__device__ __forceinline__ void count_tokens(const int64_t* __restrict__ topk_idx, int from, int to, int K, int E,
                                             bool vec, int* hist) {
    if (K <= 4)
        count_tokens_of<4, kTokens, kKeepLast>(topk_idx, from, to, K, E, vec, hist);
    else if (K <= 8)
        count_tokens_of<8, kTokens, kKeepLast>(topk_idx, from, to, K, E, vec, hist);
    else
        count_tokens_of<16, 1, kKeepLast>(topk_idx, from, to, K, E, vec, hist);
}

__device__ __forceinline__ bool choices_in_pairs(const int64_t* topk_idx, int K) {
    return K % 2 == 0 && (reinterpret_cast<uintptr_t>(topk_idx) & 15) == 0;
}

// ---- positions from the layout kernel's bits (RouteBits) ------------------------------
// Sum of the first `n` counts of a row of bytes, sixteen per load. kHere: written by other
// blocks of this kernel.
template <bool kHere>
__device__ __forceinline__ int sum_counts(const uint8_t* row, int n) {
    int sum = 0;
    for (int c0 = 0; c0 < n; c0 += 16) {
        const uint4* at = reinterpret_cast<const uint4*>(row + c0);
        const uint4 v = kHere ? ld_l2(at) : ld_ro(at);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int there = n - c0 - 4 * j;  // bytes of this word that count
            const uint32_t keep = there >= 4 ? 0xffffffffu : there > 0 ? (1u << (8 * there)) - 1u : 0u;
            sum = (int)__dp4a(w[j] & keep, 0x01010101u, (unsigned)sum);
        }
    }
    return sum;
}
// Tokens before t that chose expert e.
__device__ __forceinline__ int bits_before(const RouteBits& b, int e, int t) {
    const int chunk = t / kChunkTokens, bit = t % kChunkTokens;  // (the tables lie in 16 MB: 32-bit places)
    const uint4 v = ld_ro(b.words + (chunk * b.experts + e));
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    int n = sum_counts<false>(b.counts + e * b.stride, chunk);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int lower = bit - 32 * j;  // bits of this word that are lower
        n += __popc(w[j] & (lower >= 32 ? 0xffffffffu : lower > 0 ? (1u << lower) - 1u : 0u));
    }
    return n;
}
// Tokens that chose expert e.
template <bool kHere = false>
__device__ __forceinline__ int bits_total(const RouteBits& b, int e) {
    return sum_counts<kHere>(b.counts + (size_t)e * b.stride, b.chunks);
}
// use(expert, tokens that chose it) for every expert; whole block. A lane per sixteen chunks
// of an expert, kAhead loads of a lane requested together (2048 experts of 28 chunks, a thread
// per expert and one load after the other: 13 us of 224 threads).
template <int kAhead, typename Use>
__device__ __forceinline__ void bits_totals(const RouteBits& b, int E, Use use) {
    const int loads = b.stride / 16, lanes = loads <= 1 ? 1 : loads <= 2 ? 2 : loads <= 4 ? 4 : 8;  // per expert
    const int per = blockDim.x / lanes, mine = threadIdx.x / lanes, l = threadIdx.x - mine * lanes;
    for (int x0 = mine; x0 - mine < E; x0 += kAhead * per) {
        uint4 v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int x = x0 + u * per;
            v[u] = make_uint4(0u, 0u, 0u, 0u);
            if (x < E && l < loads) v[u] = ld_ro(reinterpret_cast<const uint4*>(b.counts + (size_t)x * b.stride) + l);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int x = x0 + u * per;
            const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
            unsigned n = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int there = b.chunks - 16 * l - 4 * j;  // bytes of this word that count
                n = __dp4a(w[j] & (there >= 4 ? 0xffffffffu : there > 0 ? (1u << (8 * there)) - 1u : 0u), 0x01010101u, n);
            }
            for (int d = lanes / 2; d > 0; d /= 2) n += __shfl_xor_sync(0xffffffffu, n, d);
            if (x < E && l == 0) use(x, (int)n);
        }
    }
}

}  // namespace mcep
