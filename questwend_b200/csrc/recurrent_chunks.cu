// Long prompts through the recurrences of recurrent.cu in chunks: inside a chunk the tokens meet in small matrix products,
// from chunk to chunk only the state is carried.  Everything is 32-bit: Mamba-2's products and the delta rule's outputs on the tensor cores
// as sums of products of bfloat16 parts (chunk_tc.cuh), the rest of the delta rule in plain multiply-adds.  Decays enter as sums of their
// logarithms, always of tokens between two others, so every exponential is of a number that is at most 0: nothing overflows, and
// what underflows is below the smallest float in truth too.
#include "chunk_tc.cuh"

// ---------------------------------------------------------------------------------
// Mamba-2 in chunks of 128 tokens.  With G_i the sum of a head's log decays (a dt) in the chunk up to token i and S0 the state
// at its start,
//     y_i   = e^(G_i) S0 C_i + sum_{j <= i} e^(G_i - G_j) dt_j (C_i . B_j) x_j + D x_i
//     S_end = e^(G_end) S0 + sum_j e^(G_end - G_j) dt_j x_j B_j^T
// Four kernels on chunk_tc.cuh: the gates; every chunk's own sum of outer products and, in the same launch, the products C_i . B_j,
// which the heads of a group share; the carries; the outputs.
// A step's sequences of at least `from` tokens go through these kernels, the others through the scan.  Chunk c of the z-th of them,
// b, is place cu_seqlens[b] / 128 + z + c of the scratch memory, which T / 128 and one for each of them hold:
//     own / starts [places, H, P / 4, N, 4], products [places, G, 32, 128 (i), 4 (j)], gates [places, H], total decays [places, H]
// The sums of logarithms are 64-bit (only their differences are used).  64 heads of 64 x 128 in 8 groups, 2,048 tokens, us under ncu (cold
// caches): gates 7, state 42, carries 19, outputs 68; with the convolution before it 158 in a run, where 8 x 8 sums a thread in plain
// multiply-adds took 233 (state 85, carries 14, outputs 113: bound by what shared memory hands to registers).  Errors against 64 bits, of the
// outputs 0.70e-7 (plain multiply-adds 0.79e-7), of the states 1.05 to 1.3e-7 (1.1 to 1.35e-7).
// ---------------------------------------------------------------------------------
#define SC_TOKENS CT_TOKENS
#define SC_FORGETS -128.f               // the exponential of this is 0 in 32-bit: a log decay below (-infinity too) counts as this much,
                                        // so that differences of sums are numbers and keep the digits of the other tokens' decays

struct ScArgs {
    const float *xbc, *dt_raw, *dt_bias, *A_log, *D;
    const int *cu_seqlens, *slots;
    float *state, *y, *own, *products, *totals;
    CtGates* gates;
    int* error;
    int ldx, ld_dt, H, P, N, G, write_state, B, from;
};

// a block's place, and its chunk's first token and tokens (0: none)
__device__ __forceinline__ int sc_chunk(const ScArgs& a, size_t& place, int& t0) {
    place = blockIdx.x;
    return rc_chunk<SC_TOKENS>(a.cu_seqlens, a.B, a.from, blockIdx.x, t0);
}
__device__ __forceinline__ CtRows sc_rows(const ScArgs& a, int t0, int n, int h, int g) {
    const float *x = a.xbc + (size_t)t0 * a.ldx, *bs = x + a.H * a.P + g * a.N;
    return {bs + a.G * a.N, bs, x + h * a.P, a.ldx, n};
}

// grid (places, H), 128 threads
__global__ void __launch_bounds__(SC_TOKENS)
ssm_chunk_gates_kernel(const ScArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float coef[SC_TOKENS];
    int t0;
    size_t place;
    const int n = sc_chunk(a, place, t0), h = blockIdx.y, i = threadIdx.x;
    if (n <= 0) return;
    float dt = 0.f, fade = 0.f;
    if (i < n) {
        dt = rc_softplus(a.dt_raw[(size_t)(t0 + i) * a.ld_dt + h] + a.dt_bias[h]);
        fade = -expf(a.A_log[h]) * dt;
        if (fade < SC_FORGETS) fade = SC_FORGETS;
    }
    ct_gates(fade, dt, a.gates + place * a.H + h, a.totals + place * a.H + h, coef);
}

// grid (places, 2 G + H * ptiles * ntiles): the products of a group's chunk with 64 of its tokens, or 64 values x 128 state rows of a head's own sum
__global__ void __launch_bounds__(CT_THREADS, 2)
ssm_chunk_state_kernel(const ScArgs a, int ptiles, int ntiles) {
    pdl_wait();
    pdl_launch_dependents();
    int t0;
    size_t place;
    const int n = sc_chunk(a, place, t0), i = (int)blockIdx.y - 2 * a.G;
    if (n <= 0) return;
    if (i < 0) {
        const int g = blockIdx.y / 2, j0 = blockIdx.y % 2 * 64;
        if (j0 < n) ct_pairs(sc_rows(a, t0, n, 0, g), a.N, j0, a.products + (place * a.G + g) * SC_TOKENS * SC_TOKENS, a.error);
        return;
    }
    const int h = i / (ptiles * ntiles), tile = i - h * ptiles * ntiles;
    ct_state(sc_rows(a, t0, n, h, h / (a.H / a.G)), a.gates + place * a.H + h, a.N, a.P, tile % ntiles * 128, tile / ntiles * 64,
             a.own + (place * a.H + h) * (size_t)a.P * a.N, a.error);
}

// grid (N * P / 1,024, H, B)
__global__ void __launch_bounds__(256, 4)
ssm_chunk_carry_kernel(const ScArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    const int h = blockIdx.y, b = rc_sequence(a.cu_seqlens, a.B, a.from, blockIdx.z);
    if (b < 0) return;
    const int t0 = a.cu_seqlens[b], n = a.cu_seqlens[b + 1] - t0;
    if (n <= 0) return;
    const size_t place = (size_t)(t0 / SC_TOKENS + blockIdx.z), size = (size_t)a.P * a.N;
    ct_carry(a.own + (place * a.H + h) * size, a.H * size, a.totals + place * a.H + h, a.H, (n + SC_TOKENS - 1) / SC_TOKENS,
             a.state + ((size_t)a.slots[b] * a.H + h) * size, a.N, a.P, blockIdx.x * 256 + threadIdx.x, a.write_state);
}

// grid (places, H * ptiles): a chunk's 128 tokens x 64 values
__global__ void __launch_bounds__(CT_THREADS, 2)
ssm_chunk_out_kernel(const ScArgs a, int ptiles) {
    pdl_wait();
    pdl_launch_dependents();
    int t0;
    size_t place;
    const int n = sc_chunk(a, place, t0), h = blockIdx.y / ptiles, p0 = (blockIdx.y - h * ptiles) * 64, g = h / (a.H / a.G);
    if (n <= 0) return;
    const CtRows rows = sc_rows(a, t0, n, h, g);
    float* y = a.y + (size_t)t0 * a.H * a.P + h * a.P;
    const float skip = a.D[h];                                      // added behind the sums: it is no product that was cut
    ct_out(rows, a.own + (place * a.H + h) * (size_t)a.P * a.N, a.products + (place * a.G + g) * SC_TOKENS * SC_TOKENS, a.gates + place * a.H + h, a.N, a.P, p0,
           nullptr, a.error,
           [&](int i, int p) { return *reinterpret_cast<const float4*>(rows.v + (size_t)i * rows.ld + p); },
           [&](int i, int p, float4 v, float4 x) {
               *reinterpret_cast<float4*>(y + (size_t)i * a.H * a.P + p) = make_float4(v.x + skip * x.x, v.y + skip * x.y, v.z + skip * x.z, v.w + skip * x.w);
           },
           [](int, float) {});
}

// Floats of scratch that qwb_ssm_chunked needs; 0: these sizes are not taken (more than a grid holds, or states that the scan refuses).
#define SC_MAX_N 512
extern "C" long long qwb_ssm_chunked_scratch(int T, int B, int from, int H, int P, int N, int G) {
    if (T <= 0 || B <= 0 || H <= 0 || P <= 0 || N <= 0 || G <= 0 || H % G || P % 4 || N % 4 || N > SC_MAX_N) return 0;
    if (B > 65535 || (long long)H * ((P + 63) / 64) * ((N + 127) / 128) + 3LL * G > 65535) return 0;
    return ((long long)T / SC_TOKENS + rc_planes(T, B, from)) * ((long long)H * ((long long)P * N + CT_GATE_FLOATS + 1) + (long long)G * SC_TOKENS * SC_TOKENS) + 4;
}

// The same step as qwb_ssm_scan for the sequences that bring at least `from` tokens (0: all), for 16-byte aligned tensors with rows of a
// multiple of 4 floats.  *error: set where a kernel's wait ran out.
extern "C" int qwb_ssm_chunked(const float* xbc, int ldx, const float* dt_raw, int ld_dt, const float* dt_bias, const float* A_log, const float* D,
                               float* state, const int* cu_seqlens, const int* slots, float* y, float* scratch, int T, int B, int max_new, int from, int H, int P,
                               int N, int G, int write_state, int* error, cudaStream_t stream) {
    if (T <= 0 || B <= 0 || max_new <= 0 || max_new < from) return 0;
    if (!qwb_ssm_chunked_scratch(T, B, from, H, P, N, G) || ldx % 4 || ldx < H * P + 2 * G * N || ld_dt < H || !error)
        return qwb_fail(QWB_ERR_ARG, "ssm_chunked: %d heads, %d groups, state %d x %d in rows of %d", H, G, N, P, ldx);
    for (const void* p : {(const void*)xbc, (const void*)state, (const void*)y, (const void*)scratch})
        if (!p || !rc_aligned16(p)) return qwb_fail(QWB_ERR_ARG, "ssm_chunked: a tensor is not 16-byte aligned");
    const int ptiles = (P + 63) / 64, ntiles = (N + 127) / 128, planes = rc_planes(T, B, from);
    const size_t places = (size_t)T / SC_TOKENS + planes;
    ScArgs a = {xbc, dt_raw, dt_bias, A_log, D, cu_seqlens, slots, state, y, nullptr, nullptr, nullptr, nullptr, error, ldx, ld_dt, H, P, N, G, write_state, B, from};
    a.own = scratch;
    a.products = a.own + places * H * P * N;
    a.gates = reinterpret_cast<CtGates*>(a.products + places * G * SC_TOKENS * SC_TOKENS);
    a.totals = reinterpret_cast<float*>(a.gates + places * H);
    cudaError_t e = cudaFuncSetAttribute(ssm_chunk_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CT_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ssm_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CT_SMEM);
    if (e != cudaSuccess) return qwb_fail(QWB_ERR_CUDA, "ssm_chunked: %s", cudaGetErrorString(e));
    qwb_launch(ssm_chunk_gates_kernel, dim3(rc_places(T, B, from, SC_TOKENS), H), SC_TOKENS, 0, stream, a);
    if (int rc = qwb_check_launch("ssm_chunk_gates")) return rc;
    qwb_launch(ssm_chunk_state_kernel, dim3(rc_places(T, B, from, SC_TOKENS), 2 * G + H * ptiles * ntiles), CT_THREADS, CT_SMEM, stream, a, ptiles, ntiles);
    if (int rc = qwb_check_launch("ssm_chunk_state")) return rc;
    qwb_launch(ssm_chunk_carry_kernel, dim3((N * (P / 4) + 255) / 256, H, planes), 256, 0, stream, a);
    if (int rc = qwb_check_launch("ssm_chunk_carry")) return rc;
    qwb_launch(ssm_chunk_out_kernel, dim3(rc_places(T, B, from, SC_TOKENS), H * ptiles), CT_THREADS, CT_SMEM, stream, a, ptiles);
    return qwb_check_launch("ssm_chunk_out");
}

// ---------------------------------------------------------------------------------
// The gated delta rule in chunks of 64 tokens.  Per head, S (K x P), with l_t the log decays of token t per key channel and
// e_ij = exp(sum of l over the tokens behind j up to i) per channel,
//     u_i = beta_i (v_i - S0^T (k_i e_i0) - sum_{j < i} A_ij u_j),    A_ij = k_i . (k_j e_ij)
//     o_i = S0^T (q_i e_i0) + sum_{j <= i} Q_ij u_j,                  Q_ij = q_i . (k_j e_ij)
//     S_end = e_end,0 S0 + sum_j (k_j e_end,j) u_j^T
// (S0: the state at the chunk's start, e_i0: the decays of its tokens up to i).  The equations of a chunk's u are triangular;
// solved for the right-hand sides beta v and beta k e_i0 instead of what depends on S0 they give u = U - W S0.  Three kernels:
//   delta_chunk_prep   every chunk by itself: A, Q, U and W by forward substitution, k e_end,j and q e_i0
//   delta_chunk_walk   a sequence's chunks in order: u = U - W S0, then the next S0; 16 value columns of a head a block
//   delta_chunk_out    every chunk by itself: o
// A decay per channel does not factor into a number of i and a number of j that are both small, so the tokens are taken in
// sub-blocks of 16: inside one, every pair and channel has an exponential of its own; between two, what decays behind j up to
// its sub-block's end, what decays in the sub-blocks between, and what decays from the start of i's sub-block to i are three
// factors of at most 1.  Sums of logarithms (base 2) span what they decay and nothing else.
// Chunk c of the z-th sequence that these kernels take, b, is place cu_seqlens[b] / 64 + z + c of the scratch memory.
// 16 heads of 128 x 128 with a decay per channel, the convolution before it, three sequences of 2,900 tokens in all: 1,194 us by the scan,
// 498 with plain multiply-adds in 8 x 8 sums a thread, 411 now (prep 157, walk 143, out 42, the convolution 35, norms 21).
// The first two are bound by what shared memory hands to registers (128 bytes a cycle).
// Scratch of a place and head:
//     W [64][K] | k e_end [64][K] | q e_0 [64][K] | Q [64 (i)][64 (j)] | U, then u [64][P] | decay of the chunk [K] | S0 [K][P]
// ---------------------------------------------------------------------------------
#define DC_TOKENS 64
#define DC_SUB 16
#define DC_WALK_ALONE (120 * 1024)        // bytes of shared memory of which an SM has no two
#define DC_MAX_K 128
#define DC_WALK_P 16

struct DcArgs {
    const float *qkv, *beta, *a_raw, *dt_bias, *A_log;
    const int *cu_seqlens, *slots;
    float *state, *o, *scratch;
    int* error;
    int ld, ld_a, H, Hk, K, P, decay_k, write_state, B, from;
};
struct DcPlace { float *w, *k_end, *q0, *q_pairs, *u, *decay, *start; };
__host__ __device__ __forceinline__ size_t dc_floats(int K, int P) {      // of one place and head: a multiple of 4
    return (size_t)3 * K * DC_TOKENS + DC_TOKENS * DC_TOKENS + (size_t)DC_TOKENS * P + K + (size_t)K * P;
}
__device__ __forceinline__ DcPlace dc_place(const DcArgs& a, size_t place, int h) {
    DcPlace p;
    p.w = a.scratch + (place * a.H + h) * dc_floats(a.K, a.P);
    p.k_end = p.w + a.K * DC_TOKENS;
    p.q0 = p.k_end + a.K * DC_TOKENS;
    p.q_pairs = p.q0 + a.K * DC_TOKENS;
    p.u = p.q_pairs + DC_TOKENS * DC_TOKENS;
    p.decay = p.u + DC_TOKENS * a.P;
    p.start = p.decay + a.K;
    return p;
}
__device__ __forceinline__ float dc_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Place of channel k of token `row` in a tile of 64 x 128: odd rows have their 16-byte pieces four apart exchanged, so that two
// threads' groups of four that read neighbouring rows at the same channels meet in no bank.
__device__ __forceinline__ int dc_at(int row, int k) { return row * DC_MAX_K + (k ^ ((row & 1) << 4)); }
// beta_i A_ij, token j by token j: behind each other the 16 rows of a sub-block's tokens, a row holding i from the sub-block's
// first token to 63 (64, 48, 32 or 16 values)
#define DC_A_FLOATS 2560
__device__ __forceinline__ int dc_row(int j) { const int s = j / DC_SUB; return 16 * (64 * s - 8 * s * (s - 1)) + (j % DC_SUB) * (64 - 16 * s) - 16 * s; }
__device__ __forceinline__ float dc_quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// grid (places, H), 256 threads; dynamic shared memory: 3 x [64][128], A, totals [4][128], beta [64] (two blocks an SM)
__global__ void __launch_bounds__(256, 2)
delta_chunk_prep_kernel(const DcArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) float dc_smem[];
    float* ks = dc_smem;                                            // k; then k times what decays behind it
    float* qs = ks + DC_TOKENS * DC_MAX_K;                             // q; then q times what decays from its sub-block's start on
    float* gs = qs + DC_TOKENS * DC_MAX_K;                             // logarithms of the decays; then k as q
    float* As = gs + DC_TOKENS * DC_MAX_K;                             // beta_i A_ij
    float* totals = As + DC_A_FLOATS;                               // [4][128]
    float* beta = totals + 4 * DC_MAX_K;
    int t0;
    const int h = blockIdx.y, n = rc_chunk<DC_TOKENS>(a.cu_seqlens, a.B, a.from, blockIdx.x, t0), tid = threadIdx.x, K = a.K, P = a.P;
    if (n <= 0) return;
    const DcPlace at = dc_place(a, blockIdx.x, h);
    const int kh = h / (a.H / a.Hk);
    const float rate = -expf(a.A_log[h]) * 1.4426950408889634f;
    if (tid < DC_TOKENS) beta[tid] = tid < n ? a.beta[(size_t)(t0 + tid) * a.H + h] : 0.f;
    const int warp = tid >> 5, e_lane = (tid & 31) * 4;             // a warp takes every eighth token, a lane four channels
    if (e_lane < K) {
        float bias[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) bias[i] = a.dt_bias[a.decay_k == 1 ? h : h * K + e_lane + i];
#pragma unroll
        for (int half = 0; half < 2; ++half) {                      // four tokens' loads at a time
            float4 q[4], k[4];
            float raw[4][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int j = warp + 8 * (4 * half + r);
                const float* row = a.qkv + (size_t)(t0 + (j < n ? j : 0)) * a.ld + kh * K + e_lane;
                q[r] = rc_load4(row, j < n);
                k[r] = rc_load4(row + a.Hk * K, j < n);
                const float* decays = a.a_raw + (size_t)(t0 + (j < n ? j : 0)) * a.ld_a + (a.decay_k == 1 ? h : h * K + e_lane);
#pragma unroll
                for (int i = 0; i < 4; ++i) raw[r][i] = decays[a.decay_k == 1 ? 0 : i];
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int j = warp + 8 * (4 * half + r);
                float g[4];
                g[0] = rate * rc_softplus(raw[r][0] + bias[0]);
#pragma unroll
                for (int i = 1; i < 4; ++i) g[i] = a.decay_k == 1 ? g[0] : rate * rc_softplus(raw[r][i] + bias[i]);
                *reinterpret_cast<float4*>(qs + dc_at(j, e_lane)) = q[r];
                *reinterpret_cast<float4*>(ks + dc_at(j, e_lane)) = k[r];
                *reinterpret_cast<float4*>(gs + dc_at(j, e_lane)) = j < n ? make_float4(g[0], g[1], g[2], g[3]) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    __syncthreads();
    // pairs of one sub-block, eight threads two tokens j: i goes down the tokens from j on, and what decays on the way is summed from j
    // on, never taken as the difference of two sums from the sub-block's start (after a token that forgets, the difference has
    // lost the digits of those that keep, and after a logarithm of -infinity it is no number).  Bound by the 16-byte loads, which cost
    // the same however many threads read one address: with four threads a token they served one j each, not two (29,000 of the
    // block's 75,000 cycles).
    {
        const int lane8 = (tid & 7) * 4, j0 = 8 * warp + ((tid >> 3) & 3), end = (j0 / DC_SUB + 1) * DC_SUB;       // tokens j0 and j0 + 4
        float4 kj[2][DC_MAX_K / 32], sum[2][DC_MAX_K / 32];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int c = 0; c < DC_MAX_K / 32; ++c) {
                kj[e][c] = lane8 + 32 * c < K ? *reinterpret_cast<const float4*>(ks + dc_at(j0 + 4 * e, lane8 + 32 * c)) : make_float4(0.f, 0.f, 0.f, 0.f);
                sum[e][c] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll 1
        for (int i = 8 * warp; i < end; ++i) {                      // from the first of the warp's eight tokens on
            float sa[2] = {0.f, 0.f}, sq[2] = {0.f, 0.f};
#pragma unroll
            for (int c = 0; c < DC_MAX_K / 32; ++c) {
                if (lane8 + 32 * c >= K) continue;
                const int pi = dc_at(i, lane8 + 32 * c);
                const float4 l = *reinterpret_cast<const float4*>(gs + pi), ki = *reinterpret_cast<const float4*>(ks + pi), qi = *reinterpret_cast<const float4*>(qs + pi);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float4& S = sum[e][c];
                    if (i > j0 + 4 * e) S = make_float4(S.x + l.x, S.y + l.y, S.z + l.z, S.w + l.w);
                    const float x = kj[e][c].x * dc_exp2(S.x), y = kj[e][c].y * dc_exp2(S.y), z = kj[e][c].z * dc_exp2(S.z), w = kj[e][c].w * dc_exp2(S.w);
                    sa[e] += ki.x * x + ki.y * y + ki.z * z + ki.w * w;
                    sq[e] += qi.x * x + qi.y * y + qi.z * z + qi.w * w;
                }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int j = j0 + 4 * e;
                float va = dc_quad_sum(sa[e]), vq = dc_quad_sum(sq[e]);
                va += __shfl_xor_sync(0xffffffffu, va, 4);
                vq += __shfl_xor_sync(0xffffffffu, vq, 4);
                if (lane8 == 0 && i >= j) {
                    if (i > j) As[dc_row(j) + i] = beta[i] * va;
                    at.q_pairs[i * DC_TOKENS + j] = vq;
                    if (i > j) at.q_pairs[j * DC_TOKENS + i] = 0.f;
                }
            }
        }
    }
    __syncthreads();
    // q and k by what decays from their sub-block's start on (k's into gs), k by what decays behind it in the sub-block, each
    // from a sum of its own; two channels of a sub-block's tokens a thread
    {
        const int s = tid >> 6, e = (tid & 63) * 2;
        if (e < K) {
            float2 l[DC_SUB];
            float x = 0.f, y = 0.f;
#pragma unroll
            for (int j = 0; j < DC_SUB; ++j) l[j] = *reinterpret_cast<const float2*>(gs + dc_at(s * DC_SUB + j, e));
#pragma unroll
            for (int j = 0; j < DC_SUB; ++j) {
                const int p = dc_at(s * DC_SUB + j, e);
                x += l[j].x; y += l[j].y;
                const float fx = dc_exp2(x), fy = dc_exp2(y);
                const float2 k = *reinterpret_cast<const float2*>(ks + p), q = *reinterpret_cast<const float2*>(qs + p);
                *reinterpret_cast<float2*>(gs + p) = make_float2(k.x * fx, k.y * fy);
                *reinterpret_cast<float2*>(qs + p) = make_float2(q.x * fx, q.y * fy);
            }
            *reinterpret_cast<float2*>(totals + s * DC_MAX_K + e) = make_float2(x, y);
            x = y = 0.f;
#pragma unroll
            for (int j = DC_SUB - 1; j >= 0; --j) {
                float2* kp = reinterpret_cast<float2*>(ks + dc_at(s * DC_SUB + j, e));
                *kp = make_float2(kp->x * dc_exp2(x), kp->y * dc_exp2(y));
                x += l[j].x; y += l[j].y;
            }
        }
    }
    // pairs of two sub-blocks: rows of sub-block s with all before it, 2 x 2 pairs to four threads
    for (int s = 1; s < 4; ++s) {
        __syncthreads();
        if (s > 1) {                                                // the sub-block between has decayed too
            for (int j = warp; j < (s - 1) * DC_SUB && e_lane < K; j += 8) {
                const int e = e_lane;
                float4* kp = reinterpret_cast<float4*>(ks + dc_at(j, e));
                const float4 k = *kp, tot = *reinterpret_cast<const float4*>(totals + (s - 1) * DC_MAX_K + e);
                *kp = make_float4(k.x * dc_exp2(tot.x), k.y * dc_exp2(tot.y), k.z * dc_exp2(tot.z), k.w * dc_exp2(tot.w));
            }
            __syncthreads();
        }
        for (int round = 0; round < s; ++round) {                   // sub-block `round` against sub-block s: 16 tiles of 4 x 4, 16 threads a tile
            const int kl = tid & 15, i0 = s * DC_SUB + (tid >> 6), j0 = round * DC_SUB + ((tid >> 4) & 3);      // rows i0 + 4 x, columns j0 + 4 y
            float v[32] = {};                                       // A: 4 x + y, Q: 16 + 4 x + y
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int k = 4 * kl + 64 * half;
                if (k >= K) continue;
                float4 r[4];
#pragma unroll
                for (int y = 0; y < 4; ++y) r[y] = *reinterpret_cast<const float4*>(ks + dc_at(j0 + 4 * y, k));
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float4 l = *reinterpret_cast<const float4*>(gs + dc_at(i0 + 4 * x, k)), q = *reinterpret_cast<const float4*>(qs + dc_at(i0 + 4 * x, k));
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        v[4 * x + y] += l.x * r[y].x + l.y * r[y].y + l.z * r[y].z + l.w * r[y].w;
                        v[16 + 4 * x + y] += q.x * r[y].x + q.y * r[y].y + q.z * r[y].z + q.w * r[y].w;
                    }
                }
            }
            // the 16 threads' parts: each step adds half of what is left across one bit of kl, which then says which half is kept
#pragma unroll
            for (int bit = 8, n = 16; bit > 0; bit >>= 1, n >>= 1) {
                const bool up = kl & bit;
#pragma unroll
                for (int e = 0; e < n; ++e) {
                    const float keep = up ? v[n + e] : v[e], give = up ? v[e] : v[n + e];
                    v[e] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
            }
            const int ii = i0 + 4 * ((kl >> 1) & 3);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int jj = j0 + 4 * (2 * (kl & 1) + e);
                if (kl < 8) {
                    As[dc_row(jj) + ii] = beta[ii] * v[e];
                } else {
                    at.q_pairs[ii * DC_TOKENS + jj] = v[e];
                    at.q_pairs[jj * DC_TOKENS + ii] = 0.f;
                }
            }
        }
    }
    __syncthreads();
    // k e_end: one more sub-block behind all but the last; q and k by what decays before their sub-block; the chunk's decay
    if (e_lane < K) {
        float4 before[4], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            before[s] = make_float4(dc_exp2(sum.x), dc_exp2(sum.y), dc_exp2(sum.z), dc_exp2(sum.w));
            const float4 tot = *reinterpret_cast<const float4*>(totals + s * DC_MAX_K + e_lane);
            sum = make_float4(sum.x + tot.x, sum.y + tot.y, sum.z + tot.z, sum.w + tot.w);
        }
        if (warp == 0) *reinterpret_cast<float4*>(at.decay + e_lane) = make_float4(dc_exp2(sum.x), dc_exp2(sum.y), dc_exp2(sum.z), dc_exp2(sum.w));
        const float4 last = *reinterpret_cast<const float4*>(totals + 3 * DC_MAX_K + e_lane);
        const float4 behind = make_float4(dc_exp2(last.x), dc_exp2(last.y), dc_exp2(last.z), dc_exp2(last.w));
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int j = warp + 8 * r, s = r / 2;                  // 16 tokens a sub-block
            float4 k = *reinterpret_cast<const float4*>(ks + dc_at(j, e_lane));
            if (s < 3) k = make_float4(k.x * behind.x, k.y * behind.y, k.z * behind.z, k.w * behind.w);
            *reinterpret_cast<float4*>(at.k_end + j * K + e_lane) = k;
            const float4 q = *reinterpret_cast<const float4*>(qs + dc_at(j, e_lane)), f = before[s];
            *reinterpret_cast<float4*>(at.q0 + j * K + e_lane) = make_float4(f.x * q.x, f.y * q.y, f.z * q.z, f.w * q.w);
            const float4 l = *reinterpret_cast<const float4*>(gs + dc_at(j, e_lane));
            const float w = beta[j];
            *reinterpret_cast<float4*>(gs + dc_at(j, e_lane)) = make_float4(w * f.x * l.x, w * f.y * l.y, w * f.z * l.z, w * f.w * l.w);
        }
    }
    // forward substitution of K + P columns, a column a thread: 128 at a time by each half of the block, in place in gs
    // (the columns of k) and, 128 at a time, in ks (those of v)
    const int half = tid >> 7, lane_col = tid & 127;
    for (int v0 = 0; v0 == 0 || v0 < P; v0 += 128) {
        __syncthreads();                                            // gs is whole, ks is read
        const bool key = half == 0;
        if (key ? (v0 > 0 || lane_col >= K) : v0 + lane_col >= P) continue;
        float* X = key ? gs : ks;
        if (!key) {
            const float* v = a.qkv + (size_t)t0 * a.ld + 2 * a.Hk * K + h * P + v0 + lane_col;
#pragma unroll 16
            for (int i = 0; i < DC_TOKENS; ++i) X[dc_at(i, lane_col)] = beta[i] * (i < n ? v[(size_t)i * a.ld] : 0.f);
        }
        float* out = key ? at.w + lane_col : at.u + v0 + lane_col;
        const int stride = key ? K : P;
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
            float x[DC_SUB];
#pragma unroll
            for (int i = 0; i < DC_SUB; ++i) x[i] = X[dc_at(s * DC_SUB + i, lane_col)];
#pragma unroll 4
            for (int j = 0; j < s * DC_SUB; ++j) {                  // the sub-blocks before
                const float xj = X[dc_at(j, lane_col)];
                const float4* m = reinterpret_cast<const float4*>(As + dc_row(j) + s * DC_SUB);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 f = m[i];
                    x[4 * i] -= f.x * xj; x[4 * i + 1] -= f.y * xj; x[4 * i + 2] -= f.z * xj; x[4 * i + 3] -= f.w * xj;
                }
            }
#pragma unroll
            for (int j = 0; j < DC_SUB; ++j) {                      // its own tokens, one after the other
                const float* m = As + dc_row(s * DC_SUB + j) + s * DC_SUB;
#pragma unroll
                for (int i = j / 4; i < 4; ++i) {
                    const float4 f = *reinterpret_cast<const float4*>(m + 4 * i);
                    if (4 * i > j) x[4 * i] -= f.x * x[j];
                    if (4 * i + 1 > j) x[4 * i + 1] -= f.y * x[j];
                    if (4 * i + 2 > j) x[4 * i + 2] -= f.z * x[j];
                    if (4 * i + 3 > j) x[4 * i + 3] -= f.w * x[j];
                }
            }
#pragma unroll
            for (int i = 0; i < DC_SUB; ++i) {
                X[dc_at(s * DC_SUB + i, lane_col)] = x[i];
                out[(s * DC_SUB + i) * stride] = x[i];
            }
        }
    }
}

// grid (ceil(P / 16), H, B), 256 threads; dynamic shared memory: W [64][K + 4], k e_end 2 x [64][K], S^T [16][K + 4], u [64][20].
// For u a thread sums 4 tokens x 4 values over a quarter of the channels, for the state 4 channels x 4 values over half of the tokens, and
// threads that hold parts of the same sums exchange halves of them by shuffles: 64 multiply-adds for eight 16-byte loads and 16 for two,
// where one value (16 for five) and two values a thread (8 for one and a half) were bound by the loads (8,200 of a chunk's 8,500 cycles).
// The state lives in registers, 4 channels x 2 values a thread, and in shared memory for u.  A chunk is two products in a chain, with two
// barriers.
__global__ void __launch_bounds__(256, 2)
delta_chunk_walk_kernel(const DcArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) float dc_smem[];
    constexpr int LU = DC_WALK_P + 4;
    const int h = blockIdx.y, b = rc_sequence(a.cu_seqlens, a.B, a.from, blockIdx.z), tid = threadIdx.x, K = a.K, P = a.P, p0 = blockIdx.x * DC_WALK_P, ldw = K + 4;
    if (b < 0) return;
    float* Ws = dc_smem;
    float* Ke = Ws + ldw * DC_TOKENS;
    float* Ss = Ke + 2 * K * DC_TOKENS;                             // [16][ldw]
    float* Us = Ss + DC_WALK_P * ldw;                               // [64][LU]
    const int t0 = a.cu_seqlens[b], n_tok = a.cu_seqlens[b + 1] - t0;
    if (n_tok <= 0) return;
    const int chunks = (n_tok + DC_TOKENS - 1) / DC_TOKENS;
    float* state = a.state + ((size_t)a.slots[b] * a.H + h) * P * K;
    const int warp = tid >> 5, lane4 = (tid & 31) * 4;
    auto copy = [&](float* dst, int ld, const float* src, bool wanted) {        // 64 rows of K, one commit group
        if (wanted && lane4 < K) {
#pragma unroll
            for (int i = 0; i < DC_TOKENS / 8; ++i) rc_copy16(dst + (warp + 8 * i) * ld + lane4, src + (warp + 8 * i) * K + lane4, true);
        }
        rc_commit();
    };
    DcPlace at = dc_place(a, a.cu_seqlens[b] / DC_TOKENS + blockIdx.z, h);
    const size_t step = a.H * dc_floats(K, P);
    copy(Ws, ldw, at.w, true);
    copy(Ke, K, at.k_end, true);
    const int lane = tid & 31, kq = lane >> 3, tg = (lane & 7) + 8 * (warp & 1), pv = 4 * (warp >> 1);     // u: tokens tg + 16 i, values pv .., channels 16 . + 4 kq ..
    const int mine = tg + 16 * kq;                                  // the token whose four sums this thread ends up with
    const int half = lane >> 4, kg = 4 * (4 * warp + ((lane >> 2) & 3)), pg = 4 * (lane & 3), ps = pg + 2 * half;    // state: channels kg .., of values pg .. in the end ps, ps + 1
    const bool p_ok = p0 + pv < P, s_ok = p0 + ps < P && kg < K;
    float S[2][4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float4 v = rc_load4(state + (size_t)(p0 + ps + e) * K + kg, s_ok);
        S[e][0] = v.x; S[e][1] = v.y; S[e][2] = v.z; S[e][3] = v.w;
        if (kg < K) *reinterpret_cast<float4*>(Ss + (ps + e) * ldw + kg) = v;
    }
    for (int c = 0; c < chunks; ++c) {
        const float4 own = rc_load4(at.u + (size_t)mine * P + p0 + pv, p_ok);      // U, asked for early
        const float4 fade = rc_load4(at.decay + kg, kg < K);
        rc_wait<0>();                                               // W and k e_end
        __syncthreads();                                            // and S is whole; the last chunk's k e_end is read
        copy(Ke + ((c + 1) & 1) * K * DC_TOKENS, K, at.k_end + step, c + 1 < chunks);
        if (s_ok) {                                                 // left for the outputs
#pragma unroll
            for (int k = 0; k < 4; ++k) *reinterpret_cast<float2*>(at.start + (size_t)(kg + k) * P + p0 + ps) = make_float2(S[0][k], S[1][k]);
        }
        {
            const float *w = Ws + tg * ldw, *s = Ss + pv * ldw;
            float part[16] = {};                                    // 4 i + e
#pragma unroll 2
            for (int k = 4 * kq; k < K; k += 16) {
                float4 x[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(w + 16 * i * ldw + k);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float4 y = *reinterpret_cast<const float4*>(s + e * ldw + k);
#pragma unroll
                    for (int i = 0; i < 4; ++i) part[4 * i + e] += x[i].x * y.x + x[i].y * y.y + x[i].z * y.z + x[i].w * y.w;
                }
            }
#pragma unroll
            for (int bit = 16, n = 8; bit >= 8; bit >>= 1, n >>= 1) {        // half of what is left across one bit of the lane, which says which is kept
                const bool up = lane & bit;
#pragma unroll
                for (int e = 0; e < n; ++e) {
                    const float keep = up ? part[n + e] : part[e], give = up ? part[e] : part[n + e];
                    part[e] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
            }
            const float4 u = make_float4(own.x - part[0], own.y - part[1], own.z - part[2], own.w - part[3]);
            *reinterpret_cast<float4*>(Us + mine * LU + pv) = u;
            if (p_ok) *reinterpret_cast<float4*>(at.u + (size_t)mine * P + p0 + pv) = u;
        }
        __syncthreads();                                            // u is whole; W is read
        copy(Ws, ldw, at.w + step, c + 1 < chunks);
#pragma unroll
        for (int e = 0; e < 2; ++e) { S[e][0] *= fade.x; S[e][1] *= fade.y; S[e][2] *= fade.z; S[e][3] *= fade.w; }
        const float* ke = Ke + (c & 1) * K * DC_TOKENS + (kg < K ? kg : 0);
        float sum[16] = {};                                         // 8 (value / 2) + 4 (value % 2) + channel
#pragma unroll 8
        for (int j = half * (DC_TOKENS / 2); j < (half + 1) * (DC_TOKENS / 2); ++j) {
            const float4 x = *reinterpret_cast<const float4*>(ke + j * K), y = *reinterpret_cast<const float4*>(Us + j * LU + pg);
            const float yv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) { sum[4 * e] += x.x * yv[e]; sum[4 * e + 1] += x.y * yv[e]; sum[4 * e + 2] += x.z * yv[e]; sum[4 * e + 3] += x.w * yv[e]; }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float keep = half ? sum[8 + 4 * e + k] : sum[4 * e + k], give = half ? sum[4 * e + k] : sum[8 + 4 * e + k];
                S[e][k] += keep + __shfl_xor_sync(0xffffffffu, give, 16);
            }
        if (kg < K) {
#pragma unroll
            for (int e = 0; e < 2; ++e) *reinterpret_cast<float4*>(Ss + (ps + e) * ldw + kg) = make_float4(S[e][0], S[e][1], S[e][2], S[e][3]);
        }
        at.w += step; at.k_end += step; at.u += step; at.decay += step; at.start += step;
    }
    if (a.write_state && s_ok) {
#pragma unroll
        for (int e = 0; e < 2; ++e) *reinterpret_cast<float4*>(state + (size_t)(p0 + ps + e) * K + kg) = make_float4(S[e][0], S[e][1], S[e][2], S[e][3]);
    }
}

// grid (places, H * ptiles): a chunk's 64 tokens x 128 values, from S0 and then from the chunk's own u, as o^T on tcgen05 (chunk_tc.cuh: the
// values are the product's 128 rows).  65 us with 8 x 8 sums a thread, 58 on mma.sync, 42 here (three prompts of 2,900 tokens in all)
__global__ void __launch_bounds__(CT_THREADS, 2)
delta_chunk_out_kernel(const DcArgs a, int ptiles) {
    pdl_wait();
    pdl_launch_dependents();
    int t0;
    const int h = blockIdx.y / ptiles, p0 = (blockIdx.y - h * ptiles) * 128, K = a.K, P = a.P, n = rc_chunk<DC_TOKENS>(a.cu_seqlens, a.B, a.from, blockIdx.x, t0);
    if (n <= 0) return;
    const DcPlace at = dc_place(a, blockIdx.x, h);
    const CtBlock block = ct_begin(a.error);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, state_stages = (K + CT_R - 1) / CT_R;
    const int index = 4 * warp + (lane >> 3), token = 8 * warp + ct_row(lane), eight = lane & 3;
    float sum[32];
    const bool ok = ct_products<true, false>(
        block, state_stages + (n + CT_R - 1) / CT_R,
        [&](int s, float (&v)[3][8]) {
            const bool state = s < state_stages;
            const int r = CT_R * (state ? s : s - state_stages) + index, col = CT_R * (state ? s : s - state_stages) + 8 * eight, cols = state ? K : DC_TOKENS;
            const float* from = (state ? at.start : at.u) + (size_t)r * P;
#pragma unroll
            for (int i = 0; i < 2; ++i) ct_load(from, p0 + 64 * i + 8 * (lane & 7), P, r < (state ? K : n), v[i]);
            ct_load((state ? at.q0 : at.q_pairs) + token * cols, col, cols, true, v[2]);
        },
        [] {},
        [&](int s, float (&v)[3][8]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) ct_put(block.a, CT_A_PART, 64 * i + CT_R * (s & 1) + index, lane & 7, v[i]);
            ct_put(block.b, CT_B_PART, token, 4 * (s & 1) + eight, v[2]);
        },
        sum);
    const int p = p0 + 32 * (warp & 3) + lane, first = 32 * (warp >> 2);
    if (ok && ct_lost(sum) && p < P) {                              // token `first` + i sees the chunk's tokens up to itself
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
            const float x = at.start[(size_t)k * P + p];
#pragma unroll
            for (int i = 0; i < 32; ++i) sum[i] += x * at.q0[(first + i) * K + k];
        }
#pragma unroll 1
        for (int j = 0; j < n; ++j) {
            const float x = at.u[(size_t)j * P + p];
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (j <= first + i) sum[i] += x * at.q_pairs[(first + i) * DC_TOKENS + j];
        }
    }
    if (ok && p < P) {
        float* out = a.o + (size_t)(t0 + first) * a.H * P + h * P + p;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (first + i < n) out[(size_t)i * a.H * P] = sum[i];
    }
    ct_end(block);
}

// Floats of scratch that qwb_delta_chunked needs; 0: these sizes are not taken.
extern "C" long long qwb_delta_chunked_scratch(int T, int B, int from, int H, int K, int P) {
    if (T <= 0 || B <= 0 || H <= 0 || K <= 0 || P <= 0 || K % 4 || P % 4 || K > DC_MAX_K) return 0;
    if (B > 65535 || (long long)H * ((P + 127) / 128) > 65535) return 0;
    return ((long long)T / DC_TOKENS + rc_planes(T, B, from)) * H * (long long)dc_floats(K, P);
}

// The same step as qwb_delta_prep and qwb_delta_scan with beta for the sequences that bring at least `from` tokens (0: all), after qwb_delta_prep made q and k unit vectors and beta; the raw
// decays come as qwb_delta_prep takes them.  16-byte aligned tensors, rows of a multiple of 4 floats.
extern "C" int qwb_delta_chunked(const float* qkv, int ld, const float* beta, const float* a_raw, int ld_a, const float* dt_bias, const float* A_log,
                                 float* state, const int* cu_seqlens, const int* slots, float* o, float* scratch, int T, int B, int max_new, int from, int H,
                                 int Hk, int K, int P, int decay_k, int write_state, int* error, cudaStream_t stream) {
    if (T <= 0 || B <= 0 || max_new <= 0 || max_new < from) return 0;
    if (!qwb_delta_chunked_scratch(T, B, from, H, K, P) || Hk <= 0 || H % Hk || ld % 4 || ld < 2 * Hk * K + H * P || (decay_k != K && decay_k != 1) || ld_a < H * decay_k || !error)
        return qwb_fail(QWB_ERR_ARG, "delta_chunked: %d heads, %d key heads, state %d x %d in rows of %d, %d decays a head", H, Hk, K, P, ld, decay_k);
    for (const void* p : {(const void*)qkv, (const void*)state, (const void*)o, (const void*)scratch})
        if (!p || !rc_aligned16(p)) return qwb_fail(QWB_ERR_ARG, "delta_chunked: a tensor is not 16-byte aligned");
    const int ptiles = (P + 127) / 128, planes = rc_planes(T, B, from);
    const unsigned places = rc_places(T, B, from, DC_TOKENS);
    const DcArgs a = {qkv, beta, a_raw, dt_bias, A_log, cu_seqlens, slots, state, o, scratch, error, ld, ld_a, H, Hk, K, P, decay_k, write_state, B, from};
    const size_t smem1 = (3 * DC_TOKENS * DC_MAX_K + DC_A_FLOATS + 4 * DC_MAX_K + DC_TOKENS) * sizeof(float);
    const size_t smem2 = ((3 * K + 4) * DC_TOKENS + DC_WALK_P * (K + 4) + DC_TOKENS * (DC_WALK_P + 4)) * sizeof(float);
    // The walk of one sequence is (P / 16) H blocks in a chain of chunks, which two on an SM slow down to 0.6.  Of a grid with room for other
    // sequences the SMs take neighbours two at a time, so where the longest sequence stands alone, or by far the most of the others take
    // the scan, a block asks for an SM's shared memory.  us, 16 heads of 128 x 128, two / one an SM: 2,048 tokens beside 16 single ones 371 / 293,
    // beside 31 of 100 1,262 / 1,184, beside 3 of 300 415 / 374; 2 x 2,048 469 / 502, 16 x 300 561 / 611.
    const bool alone = T < 2LL * max_new || T - max_new < (long long)(B - 1) * from;
    const size_t walk_smem = alone && smem2 < DC_WALK_ALONE ? DC_WALK_ALONE : smem2;
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CT_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem2 < DC_WALK_ALONE ? DC_WALK_ALONE : smem2));
    if (e != cudaSuccess) return qwb_fail(QWB_ERR_CUDA, "delta_chunked: %s", cudaGetErrorString(e));
    qwb_launch(delta_chunk_prep_kernel, dim3(places, H), 256, smem1, stream, a);
    if (int rc = qwb_check_launch("delta_chunk_prep")) return rc;
    qwb_launch(delta_chunk_walk_kernel, dim3((P + DC_WALK_P - 1) / DC_WALK_P, H, planes), 256, walk_smem, stream, a);
    if (int rc = qwb_check_launch("delta_chunk_walk")) return rc;
    qwb_launch(delta_chunk_out_kernel, dim3(places, H * ptiles), CT_THREADS, CT_SMEM, stream, a, ptiles);
    return qwb_check_launch("delta_chunk_out");
}
