// The matrix products of the recurrences whose state is a sum of outer products with one decay a token and head (Mamba-2, the mLSTM), in
// chunks of 128 tokens, on tcgen05 (the delta rule's outputs take ct_products from here too).  With k_j, v_j the keys and values of a chunk's tokens, q_i what reads, w_j the write strengths, G_i the
// sum of the log decays up to token i and S0 the state at the chunk's start,
//     own   = sum_j k_j (e^(G_end - G_j) w_j v_j)^T                                          ct_state
//     out_i = (e^(G_i) q_i) S0 + sum_{j <= i} (e^(G_i - G_j) w_j (q_i . k_j)) v_j            ct_out, the products q_i . k_j from ct_pairs
// before them ct_gates makes what depends on the gates alone, between them ct_carry goes through a sequence's chunks and puts into the place
// of each `own` the state that its chunk starts from.
//
// Every product is 128 x R by R x 64, in stages of 32 of R.  32-bit products: a number is the sum of three bfloat16 ones (each the nearest to
// what the ones before leave: exact), a product of two is six products of parts; the other three are below 2^-26 of it.  The tensor cores
// cut what they add and do not round it, so the largest parts' product is summed over a stage at a time, from 0, and these sums are added up
// by rounded additions; the five small ones are summed on the side, where 2^-8 of a cut is lost.  CT_CUT is what the cut additions of a
// stage take from its sum on average (measured: errors of the outputs against 64 bits 0.95e-7 without, 0.86 with 4e-8, 0.99 with 8e-8).
// A value that is not finite, or within 0.4 % of the largest float, has a part that is not finite and another that is no number, and so makes
// all sums of its row or column no numbers, also those that it enters with a weight of 0.  A thread that ends up with such a sum forms
// its sums again by plain multiply-adds, over the terms that they have (ct_lost).  Of a value below 2^-110 the last part has fewer digits than it
// wants: it is below bfloat16's range.
//
// 256 threads, two blocks an SM.  All of them load a stage's rows (24 values a thread, on their way while the stage before is prepared),
// weigh them, split them and store the parts into one half of the shared memory, in the swizzled rows of 128 bytes that tcgen05 reads, while
// the other half is multiplied; one thread issues the products, and the sums of the stage before are collected behind that.  Products that
// share the left parts are one instruction (right parts side by side), as what bounds them is the reading of shared memory: 30 KB in place
// of 36 for 16 of R.  Tensor memory, 64 columns each: the large sums of two stages, the two small ones.  What was measured on the way, 2,048
// tokens of 64 Mamba-2 heads of 64 x 128, us of the own sums / of the outputs: plain multiply-adds 81 / 107; mma.sync with the parts in
// shared memory 75 / 100 (its products alone leave 63 / 80); tcgen05 in stages of 64 that wait for their products 41 / 75; in stages
// of 32 39 / 60 (the last product as wide as those before it, and a token's own value behind the sums, since: 3 and 3 more in all).
#pragma once

#include "chunks.cuh"
#include "attention_tc.cuh"

#define CT_TOKENS 128
#define CT_THREADS 256
#define CT_R 32
#define CT_A_PART 16384                 // 128 rows of 64 bfloat16, or 64 rows of 2 x 64
#define CT_B_PART 8192
#define CT_SMEM (3 * (CT_A_PART + CT_B_PART) + 1024)      // 1,024: to align
#define CT_CUT 4e-8f
#define CT_TMEM 256

// What depends on the gates of a chunk and head, in scratch memory: sums of log decays (64-bit), e^(G_end - G_j) w_j, e^(G of the token's
// eight - G_j) w_j, e^(G_i); near: e^(G_i - G_j) w_j of the tokens j <= i of i's own eight, 0 behind them
struct CtGates { double G[CT_TOKENS]; float coef[CT_TOKENS], left[CT_TOKENS], fade[CT_TOKENS], near[CT_TOKENS][8]; };
#define CT_GATE_FLOATS (13 * CT_TOKENS)
static_assert(sizeof(CtGates) == CT_GATE_FLOATS * sizeof(float), "laid out without gaps");

// A chunk of a head (or of a group of heads): its n tokens' rows, `ld` floats apart.
struct CtRows { const float *q, *k, *v; int ld, n; };

struct CtBlock {
    unsigned char *a, *b;               // the parts of the stage, 1,024-byte aligned
    uint64_t* bars;                     // of even and odd stages
    uint32_t tmem;
    int* error;
};

__device__ __forceinline__ uint32_t ct_pack(float x, float y) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(y), "f"(x));
    return d;
}
// Eight neighbouring values of row r, the c-th eight of its 64, as parts: the three tiles `stride` bytes apart
__device__ __forceinline__ void ct_put(unsigned char* tile, uint32_t stride, int r, int c, const float (&v)[8]) {
    uint32_t f[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float x = v[2 * i], y = v[2 * i + 1];
        f[0][i] = ct_pack(x, y);
        x -= __uint_as_float(f[0][i] << 16); y -= __uint_as_float(f[0][i] & 0xffff0000u);
        f[1][i] = ct_pack(x, y);
        x -= __uint_as_float(f[1][i] << 16); y -= __uint_as_float(f[1][i] & 0xffff0000u);
        f[2][i] = ct_pack(x, y);
    }
    unsigned char* at = tile + r * 128 + ((c ^ (r & 7)) << 4);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(at + p * stride) = make_uint4(f[p][0], f[p][1], f[p][2], f[p][3]);
}
// values col .. col + 7 of `cols` (a multiple of 4) of a row, 0 where there are none
__device__ __forceinline__ void ct_load(const float* row, int col, int cols, bool ok, float (&v)[8]) {
    const float4 x = rc_load4(row + col, ok && col < cols), y = rc_load4(row + col + 4, ok && col + 4 < cols);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
}
// A matrix in planes of four columns, [columns / 4][rows][4]: what a thread that owns a row leaves and takes without turning
__device__ __forceinline__ void ct_load_planes(const float* m, int rows, int row, int col, int cols, bool ok, float (&v)[8]) {
    const float* at = m + ((size_t)(col / 4) * rows + row) * 4;
    const float4 x = rc_load4(at, ok && col < cols), y = rc_load4(at + (size_t)rows * 4, ok && col + 4 < cols);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
}

// What a step of 16 of R is made of: left part a by `parts` right parts from part b on, side by side, onto the sums from `column` on (the
// large sum of odd stages 64 further).  tcgen05.mma's are ordered against each other when accumulator and shape are the same: products onto
// shared columns must have both.  So the last one makes its second product (2^-27 of the sum) only for its shape.
struct CtProduct { int a, b, parts, column; };
#define CT_PRODUCTS 4
__device__ constexpr CtProduct ct_product[CT_PRODUCTS] = {{0, 0, 1, 0}, {0, 1, 2, 128}, {1, 0, 2, 128}, {2, 0, 2, 128}};
__host__ __device__ constexpr bool ct_ordered() {
    for (int i = 0; i < CT_PRODUCTS; ++i)
        for (int j = 0; j < i; ++j) {
            const CtProduct &x = ct_product[i], &y = ct_product[j];
            const int wide_x = i == 0 ? 128 : 64 * x.parts, wide_y = j == 0 ? 128 : 64 * y.parts;          // the first: both large sums
            if (x.column < y.column + wide_y && y.column < x.column + wide_x && !(x.column == y.column && x.parts == y.parts)) return false;
        }
    return true;
}
static_assert(ct_ordered(), "products onto the same columns in one shape only");

// The block's shared and tensor memory; the whole block calls, ct_end too
__device__ __forceinline__ CtBlock ct_begin(int* error) {
    extern __shared__ unsigned char ct_smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t slot;
    CtBlock c;
    c.a = reinterpret_cast<unsigned char*>(((uintptr_t)ct_smem + 1023) & ~(uintptr_t)1023);
    c.b = c.a + 3 * CT_A_PART;
    c.bars = bars;
    c.error = error;
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&slot)), "r"(CT_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else if (threadIdx.x == 32) {
        at_bar_init(&bars[0], 1);
        at_bar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    at_fence_before();
    __syncthreads();
    at_fence_after();
    c.tmem = slot;
    return c;
}
__device__ __forceinline__ void ct_end(const CtBlock& c) {
    at_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(CT_TMEM) : "memory");
}
__device__ __forceinline__ void ct_ld16(uint32_t taddr, float (&r)[16]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]),
                   "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// sum [32] = this thread's part of the 128 x 64 sums: row 32 (warp % 4) + lane, columns 32 (warp / 4) ...  load(s, rows): stage s's values into
// registers (two eights of the left matrix, one of the right); make(s, rows): weighs them and puts them into half s % 2 of c.a and c.b.  `ready`
// runs behind the first loads' issue and is followed by a barrier.  A_ROWS, B_ROWS: rows of the parts are indices of R (else of the result).
// False: a wait ran out (for the whole block alike).
template <bool A_ROWS, bool B_ROWS, class Load, class Ready, class Make>
__device__ __forceinline__ bool ct_products(const CtBlock& c, int stages, Load load, Ready ready, Make make, float (&sum)[32]) {
    constexpr uint32_t one = at_idesc(128, 64, B_ROWS) | ((A_ROWS ? 1u : 0u) << 15), two = at_idesc(128, 128, B_ROWS) | ((A_ROWS ? 1u : 0u) << 15);
    constexpr uint32_t STEP_A = A_ROWS ? 128 : 2, STEP_B = B_ROWS ? 128 : 2;        // 16 of R, in 16 bytes
    const int warp = threadIdx.x >> 5;
    const uint32_t mine = c.tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 32 * (warp >> 2);
    float rows[3][8];
#pragma unroll
    for (int i = 0; i < 32; ++i) sum[i] = 0.f;
    load(0, rows);
    ready();
    __syncthreads();
    bool ok = true;
    auto collect = [&](int column) {                                // 32 columns of a large sum in tensor memory, 16 at a time
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float r[16];
            ct_ld16(mine + column + 16 * half, r);
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[16 * half + i] += r[i];
        }
    };
    for (int s = 0; s < stages; ++s) {
        make(s, rows);
        if (s + 1 < stages) load(s + 1, rows);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        at_fence_before();
        ok = __syncthreads_and(ok);
        if (!ok) break;
        if (warp == 0 && at_elect()) {
            at_fence_after();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int k = 2 * (s & 1) + i;
                uint64_t a[3], b[2];
#pragma unroll
                for (int p = 0; p < 3; ++p) a[p] = (A_ROWS ? at_desc_mnmajor(c.a + p * CT_A_PART, 8192) : at_desc_kmajor(c.a + p * CT_A_PART)) + STEP_A * k;
#pragma unroll
                for (int p = 0; p < 2; ++p) b[p] = (B_ROWS ? at_desc_mnmajor(c.b + p * CT_B_PART, CT_B_PART) : at_desc_kmajor(c.b + p * CT_B_PART)) + STEP_B * k;
#pragma unroll
                for (int p = 0; p < CT_PRODUCTS; ++p) {
                    const CtProduct& m = ct_product[p];
                    const bool first = i == 0 && (p == 0 || (p == 1 && s == 0));
                    at_mma(c.tmem + m.column + (p == 0 ? 64 * (s & 1) : 0), a[m.a], b[m.b], m.parts == 2 ? two : one, !first);
                }
            }
            at_commit(&c.bars[s & 1]);
        }
        __syncwarp();
        if (s > 0) {
            ok = at_wait(&c.bars[(s - 1) & 1], ((s - 1) >> 1) & 1);
            at_fence_after();
            collect(64 * ((s - 1) & 1));
        }
    }
    if (ok) ok = at_wait(&c.bars[(stages - 1) & 1], ((stages - 1) >> 1) & 1);
    ok = __syncthreads_and(ok);
    if (!ok) {
        if (threadIdx.x == 0) atomicExch(c.error, 3);
        return false;
    }
    at_fence_after();
    collect(64 * ((stages - 1) & 1));
#pragma unroll
    for (int half = 0; half < 2; ++half) {                          // the small sums, and what was cut off
        float x[16], y[16];
        ct_ld16(mine + 128 + 16 * half, x);
        ct_ld16(mine + 192 + 16 * half, y);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[16 * half + i] += fmaf(sum[16 * half + i], CT_CUT, x[i] + y[i]);
    }
    return true;
}

// G[i] = the sum of the first i + 1 tokens' numbers, thread i bringing token i's (from 128 on: anything); synchronises once, the caller does
// before G is read
__device__ __forceinline__ void ct_sums(float own, double* G, double* warps) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double run = (double)own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    if (lane == 31 && warp < 4) warps[warp] = run;
    __syncthreads();
    if (warp >= 4) return;
    for (int w = 0; w < warp; ++w) run += warps[w];
    G[threadIdx.x] = run;
}
// From thread i's token's log decay and write strength (beyond the chunk: 0 and 0); at least 128 threads.  coef, in shared memory, too.
__device__ __forceinline__ void ct_gates(float log_decay, float write, CtGates* out, float* total, float* coef) {
    __shared__ double G[CT_TOKENS], warps[4];
    __shared__ float writes[CT_TOKENS];
    const int i = threadIdx.x;
    ct_sums(log_decay, G, warps);
    __syncthreads();
    if (i < CT_TOKENS) {
        coef[i] = expf((float)(G[CT_TOKENS - 1] - G[i])) * write;
        out->G[i] = G[i];
        out->coef[i] = coef[i];
        out->left[i] = expf((float)(G[i | 7] - G[i])) * write;
        out->fade[i] = expf((float)G[i]);
        if (i == 0) *total = expf((float)G[CT_TOKENS - 1]);
        writes[i] = write;
    }
    __syncthreads();
    if (i < CT_TOKENS) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int j = (i & ~7) + e;
            v[e] = j <= i ? expf((float)(G[i] - G[j])) * writes[j] : 0.f;
        }
        float4* near = reinterpret_cast<float4*>(out->near[i]);
        near[0] = make_float4(v[0], v[1], v[2], v[3]);
        near[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

// Whether a sum is no number.  If so, all of them are 0, for the caller to add its terms up without the tensor cores.
__device__ __forceinline__ bool ct_lost(float (&sum)[32]) {
    bool lost = false;
#pragma unroll
    for (int i = 0; i < 32; ++i) lost |= sum[i] != sum[i];
    if (lost) {
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[i] = 0.f;
    }
    return lost;
}
// sum[i] += x * w * y[i / 4][i % 4], `count` (a multiple of 4) of y, four neighbours at a time, `step` floats apart
__device__ __forceinline__ void ct_add(float (&sum)[32], float x, float w, const float* y, size_t step, int count) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (4 * i >= count) break;
        const float4 v = *reinterpret_cast<const float4*>(y + i * step);
        sum[4 * i] += x * (w * v.x); sum[4 * i + 1] += x * (w * v.y); sum[4 * i + 2] += x * (w * v.z); sum[4 * i + 3] += x * (w * v.w);
    }
}

// Which eight of a stage are a lane's.  Of rows in memory whose neighbouring values are neighbours of R: row 8 warp + ct_row(lane), the
// (lane % 4)-th eight; a quarter of a warp then writes to all banks of shared memory.  Of rows that are indices of R: row 4 warp + lane / 8, the
// (lane % 8)-th eight.  Of a matrix in planes: a row a lane, an eight a warp.
__device__ __forceinline__ int ct_row(int lane) { return (lane >> 3) + (lane & 4); }

// The products q_i . k_j of all the chunk's tokens i with 64 tokens from j0 on, in planes of four tokens j of 128 rows i
__device__ __forceinline__ void ct_pairs(const CtRows& r, int K, int j0, float* pairs, int* error) {
    const CtBlock c = ct_begin(error);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = 8 * warp + ct_row(lane), eight = lane & 3;
    float sum[32];
    const bool ok = ct_products<false, false>(
        c, (K + CT_R - 1) / CT_R,
        [&](int s, float (&v)[3][8]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) ct_load(r.q + (size_t)(64 * i + row) * r.ld, CT_R * s + 8 * eight, K, 64 * i + row < r.n, v[i]);
            ct_load(r.k + (size_t)(j0 + row) * r.ld, CT_R * s + 8 * eight, K, j0 + row < r.n, v[2]);
        },
        [] {},
        [&](int s, float (&v)[3][8]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) ct_put(c.a, CT_A_PART, 64 * i + row, 4 * (s & 1) + eight, v[i]);
            ct_put(c.b, CT_B_PART, row, 4 * (s & 1) + eight, v[2]);
        },
        sum);
    if (ok && ct_lost(sum)) {
        const int token = 32 * (warp & 3) + lane, j = j0 + 32 * (warp >> 2);
#pragma unroll 1
        for (int k = 0; token < r.n && k < K; ++k) {
            const float x = r.q[(size_t)token * r.ld + k];
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (j + i < r.n) sum[i] += x * r.k[(size_t)(j + i) * r.ld + k];
        }
    }
    if (ok) {
        float4* to = reinterpret_cast<float4*>(pairs) + (size_t)(j0 / 4 + 8 * (warp >> 2)) * CT_TOKENS + 32 * (warp & 3) + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i) to[i * CT_TOKENS] = make_float4(sum[4 * i], sum[4 * i + 1], sum[4 * i + 2], sum[4 * i + 3]);
    }
    ct_end(c);
}

// 128 key rows (from k0 of K) x 64 values (from p0 of P) of a chunk's own sum, in planes of four values of K key rows
__device__ __forceinline__ void ct_state(const CtRows& r, const CtGates* gates, int K, int P, int k0, int p0, float* own, int* error) {
    __shared__ float coef[CT_TOKENS];
    const CtBlock c = ct_begin(error);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = 4 * warp + (lane >> 3), eight = lane & 7;
    float sum[32];
    const bool ok = ct_products<true, true>(
        c, (r.n + CT_R - 1) / CT_R,
        [&](int s, float (&v)[3][8]) {
            const int j = CT_R * s + row;
#pragma unroll
            for (int i = 0; i < 2; ++i) ct_load(r.k + (size_t)j * r.ld, k0 + 64 * i + 8 * eight, K, j < r.n, v[i]);
            ct_load(r.v + (size_t)j * r.ld, p0 + 8 * eight, P, j < r.n, v[2]);
        },
        [&] { if (threadIdx.x < CT_TOKENS) coef[threadIdx.x] = gates->coef[threadIdx.x]; },
        [&](int s, float (&v)[3][8]) {
            const int at = CT_R * (s & 1) + row;
            const float w = coef[CT_R * s + row];
#pragma unroll
            for (int i = 0; i < 2; ++i) ct_put(c.a, CT_A_PART, 64 * i + at, eight, v[i]);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[2][e] *= w;
            ct_put(c.b, CT_B_PART, at, eight, v[2]);
        },
        sum);
    const int k = k0 + 32 * (warp & 3) + lane, p = p0 + 32 * (warp >> 2);
    if (ok && ct_lost(sum) && k < K) {
#pragma unroll 1
        for (int j = 0; j < r.n; ++j) ct_add(sum, r.k[(size_t)j * r.ld + k], coef[j], r.v + (size_t)j * r.ld + p, 4, P - p);
    }
    if (ok && k < K) {
        float4* to = reinterpret_cast<float4*>(own) + (size_t)(p / 4) * K + k;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (p + 4 * i < P) to[(size_t)i * K] = make_float4(sum[4 * i], sum[4 * i + 1], sum[4 * i + 2], sum[4 * i + 3]);
    }
    ct_end(c);
}

// Four values of a key row a thread (the at-th of K P / 4), through the `chunks` chunks of a sequence: `own` and `total` are the first chunk's,
// `step` and `heads` floats apart.  state: this head's [P][K], read and (`keep`) written.
__device__ __forceinline__ void ct_carry(float* own, size_t step, const float* total, int heads, int chunks, float* state, int K, int P, int at, bool keep) {
    constexpr int AHEAD = 8;
    if (at >= K * (P / 4)) return;
    float* S = state + (size_t)(at / K * 4) * K + at % K;
    float4 s = make_float4(S[0], S[K], S[2 * K], S[3 * K]);
    float* to = own + (size_t)at * 4;
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 u[AHEAD];
        float d[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < chunks) { u[i] = *reinterpret_cast<const float4*>(to + (c0 + i) * step); d[i] = total[(size_t)(c0 + i) * heads]; }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < chunks) {
                *reinterpret_cast<float4*>(to + (c0 + i) * step) = s;
                s = make_float4(d[i] * s.x + u[i].x, d[i] * s.y + u[i].y, d[i] * s.z + u[i].z, d[i] * s.w + u[i].w);
            }
    }
    if (keep) { S[0] = s.x; S[K] = s.y; S[2 * K] = s.z; S[3 * K] = s.w; }
}

// A chunk's 128 tokens x 64 values (from p0 of P): put(token, value column, four sums, what ahead(token, value column) gave).  starts: the chunk's, in planes.  norm0 (K values) or null: divide(token, n . q) too.
template <class Ahead, class Put, class Divide>
__device__ __forceinline__ void ct_out(const CtRows& r, const float* starts, const float* pairs, const CtGates* gates, int K, int P, int p0,
                                       const float* norm0, int* error, Ahead ahead, Put put, Divide divide) {
    __shared__ double G[CT_TOKENS];
    __shared__ float left[CT_TOKENS], fade[CT_TOKENS], norms[3][CT_TOKENS];
    __shared__ __align__(16) float near[2][CT_TOKENS][4];
    const CtBlock c = ct_begin(error);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = 8 * warp + ct_row(lane), eight = lane & 3, token = 32 * (warp & 3) + lane, index = 4 * warp + (lane >> 3);
    const int state_stages = (K + CT_R - 1) / CT_R;
    float sum[32], q_norm[2] = {0.f, 0.f}, token_norm = 0.f;
    const bool ok = ct_products<false, true>(
        c, state_stages + (r.n + CT_R - 1) / CT_R,
        [&](int s, float (&v)[3][8]) {
            if (s < state_stages) {
#pragma unroll
                for (int i = 0; i < 2; ++i) ct_load(r.q + (size_t)(64 * i + row) * r.ld, CT_R * s + 8 * eight, K, 64 * i + row < r.n, v[i]);
                ct_load_planes(starts, K, CT_R * s + lane, p0 + 8 * warp, P, CT_R * s + lane < K, v[2]);
            } else {
                const int j0 = CT_R * (s - state_stages);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int j = j0 + 8 * ((warp >> 2) + 2 * i);
                    ct_load_planes(pairs, CT_TOKENS, token, j, CT_TOKENS, token >= j && token < r.n, v[i]);
                }
                ct_load(r.v + (size_t)(j0 + index) * r.ld, p0 + 8 * (lane & 7), P, j0 + index < r.n, v[2]);
            }
        },
        [&] {
            const int i = threadIdx.x & (CT_TOKENS - 1), half = threadIdx.x >> 7;
            if (half == 0) { G[i] = gates->G[i]; left[i] = gates->left[i]; fade[i] = gates->fade[i]; }
            *reinterpret_cast<float4*>(near[half][i]) = *reinterpret_cast<const float4*>(&gates->near[i][4 * half]);
        },
        [&](int s, float (&v)[3][8]) {
            if (s < state_stages) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float f = fade[64 * i + row];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[i][e] *= f;
                    if (norm0) {
                        float n0[8];
                        ct_load(norm0, CT_R * s + 8 * eight, K, true, n0);
#pragma unroll
                        for (int e = 0; e < 8; ++e) q_norm[i] += v[i][e] * n0[e];
                    }
                    ct_put(c.a, CT_A_PART, 64 * i + row, 4 * (s & 1) + eight, v[i]);
                }
                ct_put(c.b, CT_B_PART, CT_R * (s & 1) + lane, warp, v[2]);
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) {                       // the products times what is left of their tokens; 0 where none are loaded
                    const int j = CT_R * (s - state_stages) + 8 * ((warp >> 2) + 2 * i);
                    if (token >= j + 8) {
                        const float f = expf((float)(G[token] - G[j + 7]));
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[i][e] *= f * left[j + e];
                    } else if (token >= j) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[i][e] = token >= j + e ? v[i][e] * near[e >> 2][token][e & 3] : 0.f;
                    }
                    if (norm0) token_norm += ((v[i][0] + v[i][1]) + (v[i][2] + v[i][3])) + ((v[i][4] + v[i][5]) + (v[i][6] + v[i][7]));
                    ct_put(c.a, CT_A_PART, token, 4 * (s & 1) + (warp >> 2) + 2 * i, v[i]);
                }
                ct_put(c.b, CT_B_PART, CT_R * (s & 1) + index, lane & 7, v[2]);
            }
        },
        sum);
    if (ok && ct_lost(sum) && token < r.n) {
        const int p = p0 + 32 * (warp >> 2);
#pragma unroll 1
        for (int k = 0; k < K; ++k) ct_add(sum, fade[token] * r.q[(size_t)token * r.ld + k], 1.f, starts + ((size_t)(p / 4) * K + k) * 4, (size_t)K * 4, P - p);
#pragma unroll 1
        for (int j = 0; j <= token; ++j) {
            const float w = (token ^ j) < 8 ? near[(j >> 2) & 1][token][j & 3] : expf((float)(G[token] - G[j | 7])) * left[j];
            ct_add(sum, w * pairs[((size_t)(j / 4) * CT_TOKENS + token) * 4 + j % 4], 1.f, r.v + (size_t)j * r.ld + p, 4, P - p);
        }
    }
    if (ok) {                                                       // by way of shared memory, so that a row's values leave together
        float4* stage = reinterpret_cast<float4*>(c.a);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            stage[token * 16 + ((8 * (warp >> 2) + i) ^ (token & 7))] = make_float4(sum[4 * i], sum[4 * i + 1], sum[4 * i + 2], sum[4 * i + 3]);
        float4 own[8];                                              // asked for before the barrier
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = 16 * i + 2 * warp + (lane >> 4), p = p0 + 4 * (lane & 15);
            if (t < r.n && p < P) own[i] = ahead(t, p);
        }
        if (norm0) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float v = q_norm[i];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (eight == 0) norms[2][64 * i + row] = v;
            }
            norms[warp >> 2][token] = token_norm;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = 16 * i + 2 * warp + (lane >> 4), p = p0 + 4 * (lane & 15);
            if (t < r.n && p < P) put(t, p, stage[t * 16 + ((lane & 15) ^ (t & 7))], own[i]);
        }
        if (norm0 && (int)threadIdx.x < r.n) divide(threadIdx.x, norms[2][threadIdx.x] + (norms[0][threadIdx.x] + norms[1][threadIdx.x]));
    }
    ct_end(c);
}
