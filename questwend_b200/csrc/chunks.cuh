// What the chunked recurrences share: copies into shared memory, and which sequences they take.
#pragma once

#include "common.cuh"

__device__ __forceinline__ float rc_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float4 rc_load4(const float* p, bool ok) { return ok ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f); }
static bool rc_aligned16(const void* p) { return (uintptr_t)p % 16 == 0; }

// 16 bytes from global to shared memory without passing through registers; not ok: zeros
__device__ __forceinline__ void rc_copy16(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0));
}
__device__ __forceinline__ void rc_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void rc_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Which sequences a chunked form takes: those that bring at least `from` tokens (0: all).  A grid has a plane for each that there can
// be, `rc_planes`; plane z is the z-th of them, found by every warp for itself.  -1: there are no so many.
static int rc_planes(int T, int B, int from) { return from > 0 && T / from < B ? T / from : B; }
__device__ __forceinline__ int rc_sequence(const int* __restrict__ cu_seqlens, int B, int from, int z) {
    if (from <= 0) return z;
    const int lane = threadIdx.x & 31;
    for (int first = 0; first < B; first += 32) {
        const int b = first + lane;
        unsigned mine = __ballot_sync(0xffffffffu, b < B && cu_seqlens[b + 1] - cu_seqlens[b] >= from);
        const int n = __popc(mine);
        if (z < n) {
            for (; z > 0; --z) mine &= mine - 1;
            return first + __ffs(mine) - 1;
        }
        z -= n;
    }
    return -1;
}
