// Device-side primitives for the EP kernels (sm_100a only).
//
// Counterparts in the reference: the memory-order helpers of
// mooncake-transfer-engine/include/transport/device/cuda/cuda_ops.cuh:14-139
// and the warp utilities of mooncake-ep/include/mooncake_ep_utils.cuh:141-209.
// Differences that matter here: 32-byte (256-bit) vector loads and stores,
// 64-bit flags that carry an epoch, and wall-clock (%globaltimer) timeouts.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mcep {

struct alignas(32) V32 {  // 32 bytes = 16 bf16 = 8 x b32
    uint32_t w[8];
};

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---- flags ------------------------------------------------------------------
__device__ __forceinline__ uint64_t ld_acquire_sys(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t ld_acquire_gpu(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_sys(uint64_t* p, uint64_t v) {
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Flag store without a fence of its own: used where the writer has already
// fenced everything the flag announces (or announces nothing but a count).
__device__ __forceinline__ void st_relaxed_sys(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ int ld_volatile_s32(const int* p) {
    int v;
    asm volatile("ld.volatile.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_volatile_s32(int* p, int v) {
    asm volatile("st.volatile.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// ---- inputs -----------------------------------------------------------------------
// Data that the kernel AHEAD may have written and this one only reads. Not __ldg and
// not ld.global.nc: both promise that the data does not change while the kernel runs,
// and a kernel that was launched early runs already while the one ahead still writes.
// With them a copy kernel read the positions of an earlier call although the loads
// stood behind griddepcontrol.wait; plain volatile loads are ordered by it.
__device__ __forceinline__ int ld_ro(const int32_t* p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ld_ro(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int64_t ld_ro(const int64_t* p) {
    int64_t v;
    asm volatile("ld.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ longlong2 ld_ro(const longlong2* p) {
    longlong2 v;
    asm volatile("ld.global.v2.s64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ld_ro(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
// The same for words that other blocks of this kernel may be writing (L2).
__device__ __forceinline__ int ld_l2(const int32_t* p) {
    int v;
    asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ld_l2(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
// ---- 32-byte vector memory ops ----------------------------------------------
// Inputs that are read once (x, expert outputs): see above, no .nc; not kept in L1.
__device__ __forceinline__ V32 ld32_readonly(const void* p) {
    V32 r;
    asm volatile(
        "ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]),
          "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
        : "l"(p));
    return r;
}
// Staging memory that peers wrote before the flag this kernel acquired: coherent
// path, never through the read-only cache and never allocated in L1.
__device__ __forceinline__ V32 ld32_coherent(const void* p) {
    V32 r;
    asm volatile(
        "ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]),
          "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
        : "l"(p)
        : "memory");
    return r;
}
__device__ __forceinline__ void st32(void* p, const V32& r) {
    asm volatile(
        "st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p),
        "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(r.w[4]), "r"(r.w[5]),
        "r"(r.w[6]), "r"(r.w[7])
        : "memory");
}
// ---- what L2 should give up first -----------------------------------------------
// A layer of a large batch moves more than the 126 MB of L2, and what stays there decides how much
// of it HBM sees. Nobody reads the experts' outputs again once combine has them, nor, where
// input_beyond_l2 says so, finds a dispatch's input there: marked evict-first, they make room for the rows
// that the next kernel wants.
// (Bytes that combine read from memory: 437 of 470 MB of rows handed straight to it, marked 390; 25 of
// the 59 MB of a flat elastic layer, marked 0.)
// us of a program - a kernel that writes the input, dispatch, the experts' kernel, combine, one that
// adds the result to what there was - with no mark | the experts' outputs | the input too: 2000 rows of
// 8 KB to 8 107.3 | 103.4 | 103.0, in FP8 238.5 | 235.1 | 234.3; 4096 of 14 KB to 8 354.4 | 348.2 | 348.1, in FP8
// 834 | 827.5 | 823.5; 4096 of 8 KB to 2 82.6 | 81.7 | 80.2; of 14 KB to 1 104.6 | 101.4 | 99.2.
// Combine's result is not marked: the next kernel reads it (2 us more for the last but one, 1.5 for
// 4096 of 14 KB to 8). The received rows are not either: they are what the next kernel wants.
// The loads above, with that mark where `last`.
__device__ __forceinline__ V32 ld32_readonly(const void* p, bool last) {
    if (!last) return ld32_readonly(p);
    V32 r;
    asm volatile(
        "ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]),
          "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
        : "l"(p));
    return r;
}
__device__ __forceinline__ V32 ld32_coherent(const void* p, bool last) {
    if (!last) return ld32_coherent(p);
    V32 r;
    asm volatile(
        "ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]),
          "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
        : "l"(p)
        : "memory");
    return r;
}
__device__ __forceinline__ uint4 ld16_coherent(const void* p) {
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p)
                 : "memory");
    return r;
}
__device__ __forceinline__ void st16(void* p, const uint4& r) {
    asm volatile("st.global.L1::no_allocate.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(r.x),
                 "r"(r.y), "r"(r.z), "r"(r.w)
                 : "memory");
}
__device__ __forceinline__ float ld_f32_coherent(const void* p) {
    float r;
    asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(r) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ int ld_s32_coherent(const void* p) {
    int r;
    asm volatile("ld.global.L1::no_allocate.s32 %0, [%1];" : "=r"(r) : "l"(p) : "memory");
    return r;
}

// ---- programmatic dependent launch ---------------------------------------------
// No-ops unless the kernel was launched with the programmatic-serialisation
// attribute; then `pdl_wait` blocks until the previous kernel in the stream has
// completed and its writes are visible, and `pdl_launch_dependents` lets the
// next kernel's blocks start their prologue early.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---- thread-block clusters -----------------------------------------------------------
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The word at the same place of block `rank`'s shared memory. (Volatile, but no
// memory clobber: a run of these loads is in flight together.)
__device__ __forceinline__ int ld_cluster_s32(const int* p, int rank) {
    const uint32_t local = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t remote;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(remote));
    return v;
}
// The sums of that word over all `blocks` blocks of the cluster and over those below
// `rank`. One round trip: with the bounds as branches around the loads each of them
// waited for the one before, 4 of the 9 us of a layout kernel.
template <int kMaxBlocks>
__device__ __forceinline__ int cluster_sum(const int* p, int rank, int blocks, int* lower) {
    int v[kMaxBlocks];
#pragma unroll
    for (int r = 0; r < kMaxBlocks; ++r) v[r] = ld_cluster_s32(p, r < blocks ? r : blocks - 1);
    int sum = 0, lo = 0;
#pragma unroll
    for (int r = 0; r < kMaxBlocks; ++r) {
        if (r < blocks) sum += v[r];
        if (r < rank) lo += v[r];
    }
    *lower = lo;
    return sum;
}

// ---- bf16 / fp8 ------------------------------------------------------------------
__device__ __forceinline__ float bf16lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Two fp32 -> two e4m3 bytes, round-to-nearest-even, saturating to +-448:
// the conversion of mooncake-ep/include/mooncake_ep_device.h:98-100.
__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi) {
    return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
}

// 16 bf16 (one V32) -> 16 e4m3 bytes with a per-128-channel scale shared by the
// 8 lanes that hold one group. Arithmetic of
// mooncake-ep/src/mooncake_ep_kernel.cu:184,239-264:
//   amax = max(1e-4f, max|x|); scale = 448.0f / amax (IEEE division);
//   scale_inv = amax * (1.0f / 448.0f); q = e4m3(x * scale).
// All 32 lanes must call it (shuffles); lanes without data pass zeros.
__device__ __forceinline__ uint4 quantize16(const V32& v, float& scale_inv) {
    float f[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        f[2 * i] = bf16lo(v.w[i]);
        f[2 * i + 1] = bf16hi(v.w[i]);
    }
    float amax = 1e-4f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(f[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    const float scale = __fdiv_rn(448.0f, amax);
    scale_inv = __fmul_rn(amax, 1.0f / 448.0f);
    uint32_t q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t a = cvt_e4m3x2(__fmul_rn(f[4 * i], scale), __fmul_rn(f[4 * i + 1], scale));
        uint32_t b = cvt_e4m3x2(__fmul_rn(f[4 * i + 2], scale), __fmul_rn(f[4 * i + 3], scale));
        q[i] = a | (b << 16);
    }
    return make_uint4(q[0], q[1], q[2], q[3]);
}

// 16 fp32 -> 16 bf16, round-to-nearest-even (`__float2bfloat16`,
// mooncake-ep/src/mooncake_ep_kernel.cu:750).
__device__ __forceinline__ V32 pack_bf16x16(const float (&a)[16]) {
    V32 r;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a[2 * i], a[2 * i + 1]);
        r.w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return r;
}

}  // namespace mcep
