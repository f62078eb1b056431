// Long prompts through the recurrences of recurrent.cu in chunks: inside a chunk the tokens meet in small matrix products,
// from chunk to chunk only the state is carried.  Everything is 32-bit (plain multiply-adds; the tensor cores have no product
// of 32-bit operands, and six products of bfloat16 parts in place of one would run no faster on mma.sync: 554 / 6 TFLOP/s
// against 72).  Decays enter as sums of their logarithms, always of tokens between two others, so every exponential is of a
// number that is at most 0: nothing overflows, and what underflows is below the smallest float in truth too.
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

// acc[8][8] += a[8] x b[8] for `STEPS` rows of two tiles in shared memory: row r of the first at A + r * lda, whose values
// a0 .. a0 + 3 and a1 .. a1 + 3 are this thread's, and the same for B.
template <int STEPS>
__device__ __forceinline__ void rc_outer(float (&acc)[8][8], const float* A, int lda, int a0, int a1, const float* B, int ldb, int b0, int b1) {
#pragma unroll 8
    for (int r = 0; r < STEPS; ++r) {
        const float4 x0 = *reinterpret_cast<const float4*>(A + r * lda + a0), x1 = *reinterpret_cast<const float4*>(A + r * lda + a1);
        const float4 y0 = *reinterpret_cast<const float4*>(B + r * ldb + b0), y1 = *reinterpret_cast<const float4*>(B + r * ldb + b1);
        const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w}, y[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] += x[i] * y[j];
    }
}

// ---------------------------------------------------------------------------------
// Mamba-2 in chunks of 128 tokens.  With G_i the sum of a head's log decays (a dt) in the chunk up to token i and S0 the state
// at its start,
//     y_i   = e^(G_i) S0 C_i + sum_{j <= i} e^(G_i - G_j) dt_j (C_i . B_j) x_j + D x_i
//     S_end = e^(G_end) S0 + sum_j e^(G_end - G_j) dt_j x_j B_j^T
// Three kernels: every chunk's own sum of outer products, and, in the same launch, the products C_i . B_j, which the heads of a
// group share; the carries, which run through a sequence's chunks and replace each sum by the state that its chunk starts from;
// the outputs.  A thread keeps 8 x 8 sums: four 16-byte loads from shared memory for 64 multiply-adds.  Tiles of 16 rows come
// by cp.async in three stages: while one is multiplied, the next one's rows are weighted in place and the one after is on its
// way, with one barrier a tile.  Scratch memory holds states and C row by row as the tiles want them (a state's row is a key
// row here), so that nothing is transposed on the way to a tile.
// Chunk c of sequence b is place cu_seqlens[b] / 128 + b + c of the scratch memory, which T / 128 + B places hold:
//     own / starts [places, H, N, P], total decays [places, H], products [places, G, 128 (j), 128 (i)], C [places, G, N, 128 (i)]
// The sums of logarithms are 64-bit (only their differences are used).  64 heads of 64 x 128 in 8 groups, with
// the convolution before it, the scan and now: 2,048 tokens 902 -> 222 us (85 + 14 + 113 us in ncu; the FMA pipe at 44 and 50 %,
// issue slots at 57 and 65 %), 4,096 tokens 1,804 -> 428 us, four sequences of 3,000 in all 1,115 -> 351 us.
// ---------------------------------------------------------------------------------
#define SC_TOKENS 128
#define SC_ROWS 16                      // rows of a tile
#define SC_LDA 132
#define SC_LDB 68

struct ScArgs {
    const float *xbc, *dt_raw, *dt_bias, *A_log, *D;
    const int *cu_seqlens, *slots;
    float *state, *y, *own, *totals, *products, *c_rows;
    int ldx, ld_dt, H, P, N, G, write_state;
};

// this head's step sizes [128], sums of log decays [128] and, if wanted, decays [128] (beyond the chunk's n tokens: 0, the last
// sum, 1); the caller synchronises
__device__ __forceinline__ void sc_steps(const ScArgs& a, int h, int t0, int n, float* dt, double* G, float* decay = nullptr) {
    const int lane = threadIdx.x;
    if (lane >= 32) return;
    const float rate = -expf(a.A_log[h]), bias = a.dt_bias[h];
    double own[4], sum = 0.0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int i = 4 * lane + e;
        const float d = i < n ? rc_softplus(a.dt_raw[(size_t)(t0 + i) * a.ld_dt + h] + bias) : 0.f;
        dt[i] = d;
        if (decay) decay[i] = expf(rate * d);
        sum += (double)(rate * d);
        own[e] = sum;
    }
    double run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    const double before = run - sum;
#pragma unroll
    for (int e = 0; e < 4; ++e) G[4 * lane + e] = before + own[e];
}

// grid (chunks, H * ptiles * ntiles + 3 G, B), 128 threads.  A state block makes 64 values (p) x 128 state rows (n); a product
// block one of the three 64 x 64 quarters with j <= i of a group's products.
__global__ void __launch_bounds__(128)
ssm_chunk_state_kernel(const ScArgs a, int ptiles, int ntiles) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int KB = 32;                                          // state rows of a tile of the products
    __shared__ __align__(16) float tiles[3][SC_ROWS][SC_LDA + SC_LDB];
    __shared__ float dt[SC_TOKENS], coef[SC_TOKENS];
    __shared__ double G[SC_TOKENS];
    const int c = blockIdx.x, b = blockIdx.z, tid = threadIdx.x;
    const int t0 = a.cu_seqlens[b] + c * SC_TOKENS, n = min(SC_TOKENS, a.cu_seqlens[b + 1] - t0);
    if (n <= 0) return;
    const size_t place = (size_t)(a.cu_seqlens[b] / SC_TOKENS + b + c);
    const int inner = a.H * a.P;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

    const int n_state = a.H * ptiles * ntiles;
    if ((int)blockIdx.y >= n_state) {                               // products
        const int g = ((int)blockIdx.y - n_state) / 3, quarter = ((int)blockIdx.y - n_state) % 3;
        const int i0 = quarter == 0 ? 0 : 64, j0 = quarter == 2 ? 64 : 0;
        if (i0 >= n) return;
        float (*As)[68] = reinterpret_cast<float (*)[68]>(&tiles[0][0][0]), (*Bs)[68] = As + KB;
        const float* Bg = a.xbc + (size_t)t0 * a.ldx + inner + g * a.N;
        const float* Cg = Bg + a.G * a.N;
        // 64 (i) x 64 (j) by 128 threads: i groups of 8 (tid >> 4), j groups of 4 (tid & 15)
        const int ig = (tid >> 4) * 4, jg = (tid & 15) * 4;
        for (int k0 = 0; k0 < a.N; k0 += KB) {
            __syncthreads();
            for (int idx = tid; idx < 64 * (KB / 4); idx += 128) {  // lanes walk tokens: the transposed stores do not collide
                const int i = idx & 63, k = (idx >> 6) * 4;
                const float4 cv = rc_load4(Cg + (size_t)(i0 + i) * a.ldx + k0 + k, i0 + i < n && k0 + k < a.N);
                const float4 bv = rc_load4(Bg + (size_t)(j0 + i) * a.ldx + k0 + k, j0 + i < n && k0 + k < a.N);
                As[k][i] = cv.x; As[k + 1][i] = cv.y; As[k + 2][i] = cv.z; As[k + 3][i] = cv.w;
                Bs[k][i] = bv.x; Bs[k + 1][i] = bv.y; Bs[k + 2][i] = bv.z; Bs[k + 3][i] = bv.w;
            }
            __syncthreads();
            if (quarter < 2)                                        // C, a state row a row, for the output blocks
                for (int idx = tid; idx < KB * 16; idx += 128) {
                    const int k = idx >> 4, e = (idx & 15) * 4;
                    if (k0 + k < a.N)
                        *reinterpret_cast<float4*>(a.c_rows + ((place * a.G + g) * a.N + k0 + k) * SC_TOKENS + i0 + e) = *reinterpret_cast<const float4*>(&As[k][e]);
                }
#pragma unroll 8
            for (int k = 0; k < KB; ++k) {
                const float4 x0 = *reinterpret_cast<const float4*>(&As[k][ig]), x1 = *reinterpret_cast<const float4*>(&As[k][32 + ig]);
                const float4 y = *reinterpret_cast<const float4*>(&Bs[k][jg]);
                const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w}, yv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] += xv[i] * yv[j];
            }
        }
        float* out = a.products + (place * a.G + g) * SC_TOKENS * SC_TOKENS;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float* row = out + (size_t)(j0 + jg + j) * SC_TOKENS + i0;
            *reinterpret_cast<float4*>(row + ig) = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
            *reinterpret_cast<float4*>(row + 32 + ig) = make_float4(acc[4][j], acc[5][j], acc[6][j], acc[7][j]);
        }
        return;
    }
    const int h = blockIdx.y / (ptiles * ntiles), tile = blockIdx.y - h * ptiles * ntiles, p0 = tile / ntiles * 64, n0 = tile % ntiles * 128;
    sc_steps(a, h, t0, n, dt, G);
    __syncthreads();
    coef[tid] = expf((float)(G[SC_TOKENS - 1] - G[tid])) * dt[tid];
    if (tid == 0 && tile == 0) a.totals[place * a.H + h] = expf((float)G[SC_TOKENS - 1]);
    const float* X = a.xbc + (size_t)t0 * a.ldx + h * a.P + p0;
    const float* Bh = a.xbc + (size_t)t0 * a.ldx + inner + (h / (a.H / a.G)) * a.N + n0;
    const int pg = (tid >> 4) * 4, ng = (tid & 15) * 4;
    const int n_tiles = (n + SC_ROWS - 1) / SC_ROWS;
    auto copy = [&](int t) {                                        // one commit group a tile, also beyond the last
        if (t < n_tiles) {
            float (*tile_rows)[SC_LDA + SC_LDB] = tiles[t % 3];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = (tid >> 5) + 4 * i, e = (tid & 31) * 4, j = t * SC_ROWS + r;
                const bool ok = j < n && n0 + e < a.N;
                rc_copy16(&tile_rows[r][e], Bh + (ok ? (size_t)j * a.ldx + e : 0), ok);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = (tid >> 4) + 8 * i, e = (tid & 15) * 4, j = t * SC_ROWS + r;
                const bool ok = j < n && p0 + e < a.P;
                rc_copy16(&tile_rows[r][SC_LDA + e], X + (ok ? (size_t)j * a.ldx + e : 0), ok);
            }
        }
        rc_commit();
    };
    auto weigh = [&](int t) {                                       // the values by their tokens' write strengths up to the chunk's end
        if (t >= n_tiles) return;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = (tid >> 4) + 8 * i;
            float4* v = reinterpret_cast<float4*>(&tiles[t % 3][r][SC_LDA + (tid & 15) * 4]);
            const float f = coef[t * SC_ROWS + r];
            const float4 x = *v;
            *v = make_float4(f * x.x, f * x.y, f * x.z, f * x.w);
        }
    };
    copy(0);
    copy(1);
    rc_wait<1>();
    __syncthreads();                                                // the write strengths are there too
    weigh(0);
    for (int t = 0; t < n_tiles; ++t) {
        rc_wait<0>();                                               // tile t + 1
        __syncthreads();
        copy(t + 2);
        weigh(t + 1);
        const float* rows = &tiles[t % 3][0][0];
        rc_outer<SC_ROWS>(acc, rows, SC_LDA + SC_LDB, ng, 64 + ng, rows + SC_LDA, SC_LDA + SC_LDB, pg, 32 + pg);
    }
    float* U = a.own + (place * a.H + h) * (size_t)a.P * a.N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = n0 + (i >> 2) * 64 + ng + (i & 3);
        if (m >= a.N) continue;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int p = p0 + 32 * half + pg;
            if (p < a.P) *reinterpret_cast<float4*>(U + (size_t)m * a.P + p) = make_float4(acc[i][4 * half], acc[i][4 * half + 1], acc[i][4 * half + 2], acc[i][4 * half + 3]);
        }
    }
}

// grid (tiles of 32 state rows x 32 values, H, B), 256 threads: four neighbouring values of a state row a thread, through the
// sequence's chunks in order.  The state itself lies column by column and is turned in shared memory.
__global__ void __launch_bounds__(256)
ssm_chunk_carry_kernel(const ScArgs a, int ptiles) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int AHEAD = 8;
    __shared__ float turn[32][33];
    const int h = blockIdx.y, b = blockIdx.z, t0 = a.cu_seqlens[b], n = a.cu_seqlens[b + 1] - t0;
    if (n <= 0) return;
    const int n0 = blockIdx.x / ptiles * 32, p0 = blockIdx.x % ptiles * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t size = (size_t)a.P * a.N;
    float* S = a.state + ((size_t)a.slots[b] * a.H + h) * size;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int p = warp + 8 * i;
        turn[p][lane] = p0 + p < a.P && n0 + lane < a.N ? S[(size_t)(p0 + p) * a.N + n0 + lane] : 0.f;
    }
    __syncthreads();
    const int row = threadIdx.x >> 3, p = (threadIdx.x & 7) * 4;
    float4 s = make_float4(turn[p][row], turn[p + 1][row], turn[p + 2][row], turn[p + 3][row]);
    if (n0 + row < a.N && p0 + p < a.P) {
        const int chunks = (n + SC_TOKENS - 1) / SC_TOKENS;
        const size_t place = (size_t)(t0 / SC_TOKENS + b), step = (size_t)a.H * size;
        float* at = a.own + (place * a.H + h) * size + (size_t)(n0 + row) * a.P + p0 + p;
        const float* total = a.totals + place * a.H + h;
        for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
            float4 u[AHEAD];
            float d[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
                if (c0 + i < chunks) { u[i] = *reinterpret_cast<const float4*>(at + (c0 + i) * step); d[i] = total[(size_t)(c0 + i) * a.H]; }
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
                if (c0 + i < chunks) {
                    *reinterpret_cast<float4*>(at + (c0 + i) * step) = s;
                    s = make_float4(d[i] * s.x + u[i].x, d[i] * s.y + u[i].y, d[i] * s.z + u[i].z, d[i] * s.w + u[i].w);
                }
        }
    }
    if (!a.write_state) return;
    turn[p][row] = s.x; turn[p + 1][row] = s.y; turn[p + 2][row] = s.z; turn[p + 3][row] = s.w;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int q = warp + 8 * i;
        if (p0 + q < a.P && n0 + lane < a.N) S[(size_t)(p0 + q) * a.N + n0 + lane] = turn[q][lane];
    }
}

// grid (chunks, H * ptiles, B), 128 threads: a chunk's 128 tokens x 64 values.  A thread weighs its token's products with a
// tile of tokens j, e^(G_i - G_j) dt_j, from the tile's last token to its first: one exponential, then a decay a token.
__global__ void __launch_bounds__(128, 4)
ssm_chunk_out_kernel(const ScArgs a, int ptiles) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ __align__(16) float tiles[3][SC_ROWS][SC_LDA + SC_LDB];
    __shared__ float dt[SC_TOKENS], decay[SC_TOKENS];
    __shared__ double G[SC_TOKENS];
    const int c = blockIdx.x, b = blockIdx.z, tid = threadIdx.x;
    const int h = blockIdx.y / ptiles, p0 = (blockIdx.y - h * ptiles) * 64;
    const int t0 = a.cu_seqlens[b] + c * SC_TOKENS, n = min(SC_TOKENS, a.cu_seqlens[b + 1] - t0);
    if (n <= 0) return;
    const size_t place = (size_t)(a.cu_seqlens[b] / SC_TOKENS + b + c);
    const int inner = a.H * a.P, g = h / (a.H / a.G);
    const float* X = a.xbc + (size_t)t0 * a.ldx + h * a.P + p0;
    const float* Cg = a.c_rows + (place * a.G + g) * (size_t)a.N * SC_TOKENS;
    const float* S0 = a.own + (place * a.H + h) * (size_t)a.P * a.N + p0;
    const float* products = a.products + (place * a.G + g) * SC_TOKENS * SC_TOKENS;
    const int state_tiles = (a.N + SC_ROWS - 1) / SC_ROWS, n_tiles = state_tiles + (n + SC_ROWS - 1) / SC_ROWS;
    auto copy = [&](int t) {                                        // one commit group a tile, also beyond the last
        if (t < n_tiles) {
            const bool from_state = t < state_tiles;
            const int row0 = (from_state ? t : t - state_tiles) * SC_ROWS, limit = from_state ? a.N : n;
            float (*tile_rows)[SC_LDA + SC_LDB] = tiles[t % 3];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = (tid >> 5) + 4 * i, e = (tid & 31) * 4;
                const bool ok = row0 + r < limit;
                rc_copy16(&tile_rows[r][e], (from_state ? Cg : products) + (ok ? (size_t)(row0 + r) * SC_TOKENS + e : 0), ok);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = (tid >> 4) + 8 * i, e = (tid & 15) * 4;
                const bool ok = row0 + r < limit && p0 + e < a.P;
                rc_copy16(&tile_rows[r][SC_LDA + e], from_state ? S0 + (ok ? (size_t)(row0 + r) * a.P + e : 0) : X + (ok ? (size_t)(row0 + r) * a.ldx + e : 0), ok);
            }
        }
        rc_commit();
    };
    copy(0);
    copy(1);
    sc_steps(a, h, t0, n, dt, G, decay);
    auto weigh = [&](int t) {                                       // this thread's token's weights of a tile of tokens, over their products
        if (t < state_tiles || t >= n_tiles) return;
        const int j0 = (t - state_tiles) * SC_ROWS;
        float* col = &tiles[t % 3][0][tid];
        float e = tid >= j0 + SC_ROWS ? expf((float)(G[tid] - G[j0 + SC_ROWS - 1])) : 0.f;
#pragma unroll
        for (int r = SC_ROWS - 1; r >= 0; --r) {
            if (r < SC_ROWS - 1) e *= decay[j0 + r + 1];
            if (tid == j0 + r) e = 1.f;
            col[r * (SC_LDA + SC_LDB)] = tid >= j0 + r ? col[r * (SC_LDA + SC_LDB)] * (e * dt[j0 + r]) : 0.f;
        }
    };
    const int ig = (tid >> 3) * 4, pg = (tid & 7) * 4;              // this thread's tokens ig .., 64 + ig ..; values pg .., 32 + pg ..
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    for (int t = 0; t < n_tiles; ++t) {
        rc_wait<0>();
        __syncthreads();                                            // tiles t and t + 1 are there (t's rows weighted)
        copy(t + 2);
        weigh(t + 1);
        const float* rows = &tiles[t % 3][0][0];
        if (t == state_tiles) {                                     // what came from the state fades with the chunk's decays
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float f = expf((float)G[(i >> 2) * 64 + ig + (i & 3)]);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] *= f;
            }
        }
        if (t < state_tiles + 64 / SC_ROWS) {
            rc_outer<SC_ROWS>(acc, rows, SC_LDA + SC_LDB, ig, 64 + ig, rows + SC_LDA, SC_LDA + SC_LDB, pg, 32 + pg);
        } else {                                                    // tokens of the chunk's second half: the first half sees nothing
#pragma unroll 8
            for (int r = 0; r < SC_ROWS; ++r) {
                const float* row = rows + r * (SC_LDA + SC_LDB);
                const float4 x = *reinterpret_cast<const float4*>(row + 64 + ig);
                const float4 y0 = *reinterpret_cast<const float4*>(row + SC_LDA + pg), y1 = *reinterpret_cast<const float4*>(row + SC_LDA + 32 + pg);
                const float xv[4] = {x.x, x.y, x.z, x.w}, yv[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[4 + i][j] += xv[i] * yv[j];
            }
        }
    }
    const float skip = a.D[h];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = (i >> 2) * 64 + ig + (i & 3);
        if (t >= n) continue;
        float* out = a.y + (size_t)(t0 + t) * inner + h * a.P + p0;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int p = 32 * half + pg;
            if (p0 + p >= a.P) continue;
            const float4 x = *reinterpret_cast<const float4*>(X + (size_t)t * a.ldx + p);
            *reinterpret_cast<float4*>(out + p) = make_float4(acc[i][4 * half] + skip * x.x, acc[i][4 * half + 1] + skip * x.y,
                                                              acc[i][4 * half + 2] + skip * x.z, acc[i][4 * half + 3] + skip * x.w);
        }
    }
}

// Floats of scratch that qwb_ssm_chunked needs; 0: these sizes are not taken.
extern "C" long long qwb_ssm_chunked_scratch(int T, int B, int H, int P, int N, int G) {
    if (T <= 0 || B <= 0 || H <= 0 || P <= 0 || N <= 0 || G <= 0 || H % G || P % 4 || N % 4) return 0;
    return ((long long)T / SC_TOKENS + B) * ((long long)H * P * N + H + (long long)G * SC_TOKENS * (SC_TOKENS + N)) + 4;
}

// The same step as qwb_ssm_scan, for 16-byte aligned tensors with rows of a multiple of 4 floats.
extern "C" int qwb_ssm_chunked(const float* xbc, int ldx, const float* dt_raw, int ld_dt, const float* dt_bias, const float* A_log, const float* D,
                               float* state, const int* cu_seqlens, const int* slots, float* y, float* scratch, int T, int B, int max_new, int H, int P,
                               int N, int G, int write_state, cudaStream_t stream) {
    if (T <= 0 || B <= 0 || max_new <= 0) return 0;
    if (!qwb_ssm_chunked_scratch(T, B, H, P, N, G) || ldx % 4 || ldx < H * P + 2 * G * N || ld_dt < H)
        return qwb_fail(QWB_ERR_ARG, "ssm_chunked: %d heads, %d groups, state %d x %d in rows of %d", H, G, N, P, ldx);
    for (const void* p : {(const void*)xbc, (const void*)state, (const void*)y, (const void*)scratch})
        if (!p || !rc_aligned16(p)) return qwb_fail(QWB_ERR_ARG, "ssm_chunked: a tensor is not 16-byte aligned");
    const int chunks = (max_new + SC_TOKENS - 1) / SC_TOKENS, ptiles = (P + 63) / 64, ntiles = (N + 127) / 128;
    if (B > 65535 || (long long)H * ptiles * ntiles + 3 * G > 65535) return qwb_fail(QWB_ERR_ARG, "ssm_chunked: %d sequences or %d heads of %d x %d are too many", B, H, N, P);
    const size_t places = (size_t)T / SC_TOKENS + B;
    ScArgs a = {xbc, dt_raw, dt_bias, A_log, D, cu_seqlens, slots, state, y, nullptr, nullptr, nullptr, nullptr, ldx, ld_dt, H, P, N, G, write_state};
    a.own = scratch;
    a.products = a.own + places * H * P * N;
    a.c_rows = a.products + places * G * SC_TOKENS * SC_TOKENS;
    a.totals = a.c_rows + places * G * N * SC_TOKENS;
    qwb_launch(ssm_chunk_state_kernel, dim3(chunks, H * ptiles * ntiles + 3 * G, B), 128, 0, stream, a, ptiles, ntiles);
    if (int rc = qwb_check_launch("ssm_chunk_state")) return rc;
    const int carry_p = (P + 31) / 32;
    qwb_launch(ssm_chunk_carry_kernel, dim3((N + 31) / 32 * carry_p, H, B), 256, 0, stream, a, carry_p);
    if (int rc = qwb_check_launch("ssm_chunk_carry")) return rc;
    qwb_launch(ssm_chunk_out_kernel, dim3(chunks, H * ptiles, B), 128, 0, stream, a, ptiles);
    return qwb_check_launch("ssm_chunk_out");
}
