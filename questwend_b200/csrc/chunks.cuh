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
// ... and how many places chunks of `tokens` tokens have (below)
static unsigned rc_places(int T, int B, int from, int tokens) { return B == 1 ? (T + tokens - 1) / tokens : T / tokens + rc_planes(T, B, from); }
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

// The chunk in a place of the scratch memory: its first token and its tokens (none or fewer: no sequence fills this place).  The z-th
// sequence that the form takes (rc_sequence) begins at place cu_seqlens / TOKENS + z, so T / TOKENS + rc_planes places hold all
// chunks.  A grid of chunks x sequences, as long as the longest and as wide as all that there can be, was mostly blocks without work where
// one prompt stands beside many short ones, and these cost a block's start with all of its shared memory: a Mamba-2 prompt of 8,192 tokens
// beside 63 single ones 3,900 us, as places 600; the mLSTM's (16 heads of 128 x 128) 2,370, as places 565.  A full warp calls.
template <int TOKENS>
__device__ __forceinline__ int rc_chunk(const int* __restrict__ cu_seqlens, int B, int from, int place, int& t0) {
    const int lane = threadIdx.x & 31;
    if (B == 1) { t0 = cu_seqlens[0] + place * TOKENS; return min(TOKENS, cu_seqlens[1] - t0); }
    int begin = 0, end = 0, start = 0, taken = 0;
    for (int first = 0; first < B; first += 32) {
        const int b = first + lane, lo = b < B ? cu_seqlens[b] : 0, hi = b < B ? cu_seqlens[b + 1] : 0;
        const unsigned mine = __ballot_sync(0xffffffffu, b < B && hi - lo >= from);
        const int at = lo / TOKENS + taken + __popc(mine & ((1u << lane) - 1u));
        const unsigned before = __ballot_sync(0xffffffffu, ((mine >> lane) & 1u) && at <= place);
        if (before) {                                               // the last of them
            const int last = 31 - __clz(before);
            begin = __shfl_sync(0xffffffffu, lo, last);
            end = __shfl_sync(0xffffffffu, hi, last);
            start = __shfl_sync(0xffffffffu, at, last);
        }
        if (before != mine) break;
        taken += __popc(mine);
    }
    t0 = begin + (place - start) * TOKENS;
    return min(TOKENS, end - t0);
}
