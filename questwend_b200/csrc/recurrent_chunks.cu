// Long prompts through the recurrences of recurrent.cu in chunks: inside a chunk the tokens meet in small matrix products,
// from chunk to chunk only the state is carried.  Everything is 32-bit, in plain multiply-adds: the tensor cores have no product
// of 32-bit operands, and six products of bfloat16 parts in place of one, at mma.sync's rate 92 TFLOP/s (554 / 6) against 72, would
// gain little once the parts are made; on tcgen05 they would be faster, which is not written.  Decays enter as sums of their
// logarithms, always of tokens between two others, so every exponential is of a number that is at most 0: nothing overflows, and
// what underflows is below the smallest float in truth too.
#include "chunks.cuh"

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
// A step's sequences of at least `from` tokens go through these kernels, the others through the scan.  Chunk c of the z-th of them,
// b, is place cu_seqlens[b] / 128 + z + c of the scratch memory, which T / 128 and one for each of them hold:
//     own / starts [places, H, N, P], total decays [places, H], products [places, G, 128 (j), 128 (i)], C [places, G, N, 128 (i)]
// The sums of logarithms are 64-bit (only their differences are used).  64 heads of 64 x 128 in 8 groups, with
// the convolution before it, the scan and now: 2,048 tokens 902 -> 222 us (85 + 14 + 113 us in ncu; the FMA pipe at 44 and 50 %,
// issue slots at 57 and 65 %), 4,096 tokens 1,804 -> 428 us, four sequences of 3,000 in all 1,115 -> 351 us.
// ---------------------------------------------------------------------------------
#define SC_TOKENS 128
#define SC_ROWS 16                      // rows of a tile
#define SC_LDA 132
#define SC_LDB 68
#define SC_FORGETS -128.f               // the exponential of this is 0 in 32-bit: a log decay below (-infinity too) counts as this much,
                                        // so that differences of sums are numbers and keep the digits of the other tokens' decays

struct ScArgs {
    const float *xbc, *dt_raw, *dt_bias, *A_log, *D;
    const int *cu_seqlens, *slots;
    float *state, *y, *own, *totals, *products, *c_rows;
    int ldx, ld_dt, H, P, N, G, write_state, B, from;
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
        const float fade = i < n ? rate * d : 0.f;
        if (decay) decay[i] = expf(fade);
        sum += (double)(fade < SC_FORGETS ? SC_FORGETS : fade);
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
    const int c = blockIdx.x, b = rc_sequence(a.cu_seqlens, a.B, a.from, blockIdx.z), tid = threadIdx.x;
    if (b < 0) return;
    const int t0 = a.cu_seqlens[b] + c * SC_TOKENS, n = min(SC_TOKENS, a.cu_seqlens[b + 1] - t0);
    if (n <= 0) return;
    const size_t place = (size_t)(a.cu_seqlens[b] / SC_TOKENS + blockIdx.z + c);
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
    const int h = blockIdx.y, b = rc_sequence(a.cu_seqlens, a.B, a.from, blockIdx.z);
    if (b < 0) return;
    const int t0 = a.cu_seqlens[b], n = a.cu_seqlens[b + 1] - t0;
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
        const size_t place = (size_t)(t0 / SC_TOKENS + blockIdx.z), step = (size_t)a.H * size;
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
    const int c = blockIdx.x, b = rc_sequence(a.cu_seqlens, a.B, a.from, blockIdx.z), tid = threadIdx.x;
    const int h = blockIdx.y / ptiles, p0 = (blockIdx.y - h * ptiles) * 64;
    if (b < 0) return;
    const int t0 = a.cu_seqlens[b] + c * SC_TOKENS, n = min(SC_TOKENS, a.cu_seqlens[b + 1] - t0);
    if (n <= 0) return;
    const size_t place = (size_t)(a.cu_seqlens[b] / SC_TOKENS + blockIdx.z + c);
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

// Floats of scratch that qwb_ssm_chunked needs; 0: these sizes are not taken (more than a grid holds, or states that the scan refuses).
#define SC_MAX_N 512
extern "C" long long qwb_ssm_chunked_scratch(int T, int B, int from, int H, int P, int N, int G) {
    if (T <= 0 || B <= 0 || H <= 0 || P <= 0 || N <= 0 || G <= 0 || H % G || P % 4 || N % 4 || N > SC_MAX_N) return 0;
    if (B > 65535 || (long long)H * ((P + 63) / 64) * ((N + 127) / 128) + 3LL * G > 65535) return 0;
    return ((long long)T / SC_TOKENS + rc_planes(T, B, from)) * ((long long)H * P * N + H + (long long)G * SC_TOKENS * (SC_TOKENS + N)) + 4;
}

// The same step as qwb_ssm_scan for the sequences that bring at least `from` tokens (0: all), for 16-byte aligned tensors with rows of a
// multiple of 4 floats.
extern "C" int qwb_ssm_chunked(const float* xbc, int ldx, const float* dt_raw, int ld_dt, const float* dt_bias, const float* A_log, const float* D,
                               float* state, const int* cu_seqlens, const int* slots, float* y, float* scratch, int T, int B, int max_new, int from, int H, int P,
                               int N, int G, int write_state, cudaStream_t stream) {
    if (T <= 0 || B <= 0 || max_new <= 0 || max_new < from) return 0;
    if (!qwb_ssm_chunked_scratch(T, B, from, H, P, N, G) || ldx % 4 || ldx < H * P + 2 * G * N || ld_dt < H)
        return qwb_fail(QWB_ERR_ARG, "ssm_chunked: %d heads, %d groups, state %d x %d in rows of %d", H, G, N, P, ldx);
    for (const void* p : {(const void*)xbc, (const void*)state, (const void*)y, (const void*)scratch})
        if (!p || !rc_aligned16(p)) return qwb_fail(QWB_ERR_ARG, "ssm_chunked: a tensor is not 16-byte aligned");
    const int chunks = (max_new + SC_TOKENS - 1) / SC_TOKENS, ptiles = (P + 63) / 64, ntiles = (N + 127) / 128, planes = rc_planes(T, B, from);
    const size_t places = (size_t)T / SC_TOKENS + planes;
    ScArgs a = {xbc, dt_raw, dt_bias, A_log, D, cu_seqlens, slots, state, y, nullptr, nullptr, nullptr, nullptr, ldx, ld_dt, H, P, N, G, write_state, B, from};
    a.own = scratch;
    a.products = a.own + places * H * P * N;
    a.c_rows = a.products + places * G * SC_TOKENS * SC_TOKENS;
    a.totals = a.c_rows + places * G * N * SC_TOKENS;
    qwb_launch(ssm_chunk_state_kernel, dim3(chunks, H * ptiles * ntiles + 3 * G, planes), 128, 0, stream, a, ptiles, ntiles);
    if (int rc = qwb_check_launch("ssm_chunk_state")) return rc;
    const int carry_p = (P + 31) / 32;
    qwb_launch(ssm_chunk_carry_kernel, dim3((N + 31) / 32 * carry_p, H, planes), 256, 0, stream, a, carry_p);
    if (int rc = qwb_check_launch("ssm_chunk_carry")) return rc;
    qwb_launch(ssm_chunk_out_kernel, dim3(chunks, H * ptiles, planes), 128, 0, stream, a, ptiles);
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
// 16 heads of 128 x 128 with a decay per channel, the convolution before it, the scan and now: 2,048 tokens 955 -> 328 us (prep 123,
// walk 133, out 49 in ncu), three sequences of 2,900 in all 1,194 -> 484 us; a decay per head, four of 4,096 in all, 1,198 -> 596 us.
// Bound by what shared memory hands to registers (128 bytes a cycle), the walk more than the others.
// Scratch of a place and head:
//     W [64][K] | k e_end [64][K] | q e_0 [64][K] | Q [64 (j)][64 (i)] | U, then u [64][P] | decay of the chunk [K] | S0 [K][P]
// ---------------------------------------------------------------------------------
#define DC_TOKENS 64
#define DC_SUB 16
#define DC_MAX_K 128
#define DC_WALK_P 16

struct DcArgs {
    const float *qkv, *beta, *a_raw, *dt_bias, *A_log;
    const int *cu_seqlens, *slots;
    float *state, *o, *scratch;
    int ld, ld_a, H, Hk, K, P, decay_k, write_state, B, from;
};
struct DcPlace { float *w, *k_end, *q0, *q_pairs, *u, *decay, *start; };
__host__ __device__ __forceinline__ size_t dc_floats(int K, int P) {      // of one place and head: a multiple of 4
    return (size_t)3 * K * DC_TOKENS + DC_TOKENS * DC_TOKENS + (size_t)DC_TOKENS * P + K + (size_t)K * P;
}
__device__ __forceinline__ DcPlace dc_place(const DcArgs& a, int b, int c, int h) {      // in plane blockIdx.z of the grid
    const size_t place = (size_t)(a.cu_seqlens[b] / DC_TOKENS + blockIdx.z + c);
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

// grid (chunks, H, B), 256 threads; dynamic shared memory: 3 x [64][128], A, totals [4][128], beta [64] (two blocks an SM)
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
    const int c = blockIdx.x, h = blockIdx.y, b = rc_sequence(a.cu_seqlens, a.B, a.from, blockIdx.z), tid = threadIdx.x, K = a.K, P = a.P;
    if (b < 0) return;
    const int t0 = a.cu_seqlens[b] + c * DC_TOKENS, n = min(DC_TOKENS, a.cu_seqlens[b + 1] - t0);
    if (n <= 0) return;
    const DcPlace at = dc_place(a, b, c, h);
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
    // pairs of one sub-block, four threads a token j: i goes down the tokens from j on, and what decays on the way is summed from j
    // on, never taken as the difference of two sums from the sub-block's start (after a token that forgets, the difference has
    // lost the digits of those that keep, and after a logarithm of -infinity it is no number)
    const int lane4 = (tid & 3) * 4;
    {
        const int j = tid >> 2, end = (j / DC_SUB + 1) * DC_SUB;
        float4 kj[DC_MAX_K / 16], sum[DC_MAX_K / 16];
#pragma unroll
        for (int c = 0; c < DC_MAX_K / 16; ++c) {
            kj[c] = lane4 + 16 * c < K ? *reinterpret_cast<const float4*>(ks + dc_at(j, lane4 + 16 * c)) : make_float4(0.f, 0.f, 0.f, 0.f);
            sum[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll 1
        for (int i = 8 * warp; i < end; ++i) {                      // from the first of the warp's eight tokens on
            float sa = 0.f, sq = 0.f;
#pragma unroll
            for (int c = 0; c < DC_MAX_K / 16; ++c) {
                if (lane4 + 16 * c >= K) continue;
                const int pi = dc_at(i, lane4 + 16 * c);
                const float4 l = *reinterpret_cast<const float4*>(gs + pi), ki = *reinterpret_cast<const float4*>(ks + pi), qi = *reinterpret_cast<const float4*>(qs + pi);
                if (i > j) sum[c] = make_float4(sum[c].x + l.x, sum[c].y + l.y, sum[c].z + l.z, sum[c].w + l.w);
                const float x = kj[c].x * dc_exp2(sum[c].x), y = kj[c].y * dc_exp2(sum[c].y), z = kj[c].z * dc_exp2(sum[c].z), w = kj[c].w * dc_exp2(sum[c].w);
                sa += ki.x * x + ki.y * y + ki.z * z + ki.w * w;
                sq += qi.x * x + qi.y * y + qi.z * z + qi.w * w;
            }
            sa = dc_quad_sum(sa);
            sq = dc_quad_sum(sq);
            if (lane4 == 0 && i >= j) {
                if (i > j) As[dc_row(j) + i] = beta[i] * sa;
                at.q_pairs[j * DC_TOKENS + i] = sq;
                if (i > j) at.q_pairs[i * DC_TOKENS + j] = 0.f;
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
        for (int round = 0; round < s; ++round) {                   // sub-block `round` against sub-block s: 64 tiles of 2 x 2
            const int task = tid >> 2, i = task >> 3, j = task & 7;
            const int i0 = s * DC_SUB + i, j0 = round * DC_SUB + j;
            float sa[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, sq[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 2
            for (int k = lane4; k < K; k += 16) {
                float4 l[2], q[2], r[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    l[e] = *reinterpret_cast<const float4*>(gs + dc_at(i0 + 8 * e, k));
                    q[e] = *reinterpret_cast<const float4*>(qs + dc_at(i0 + 8 * e, k));
                    r[e] = *reinterpret_cast<const float4*>(ks + dc_at(j0 + 8 * e, k));
                }
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int y = 0; y < 2; ++y) {
                        sa[x][y] += l[x].x * r[y].x + l[x].y * r[y].y + l[x].z * r[y].z + l[x].w * r[y].w;
                        sq[x][y] += q[x].x * r[y].x + q[x].y * r[y].y + q[x].z * r[y].z + q[x].w * r[y].w;
                    }
            }
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const float va = dc_quad_sum(sa[x][y]), vq = dc_quad_sum(sq[x][y]);
                    if (lane4 == 4 * (2 * x + y)) {                 // one of the four threads each
                        const int ii = i0 + 8 * x, jj = j0 + 8 * y;
                        As[dc_row(jj) + ii] = beta[ii] * va;
                        at.q_pairs[jj * DC_TOKENS + ii] = vq;
                        at.q_pairs[ii * DC_TOKENS + jj] = 0.f;
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
// For u a thread sums 4 tokens x 1 value over all channels, four channels a load; the state lives in registers, 4 channels x 2
// values a thread, and in shared memory for u.  A chunk is two products in a chain, with two barriers.
__global__ void __launch_bounds__(256)
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
    DcPlace at = dc_place(a, b, 0, h);
    const size_t step = a.H * dc_floats(K, P);
    copy(Ws, ldw, at.w, true);
    copy(Ke, K, at.k_end, true);
    const int p = (tid & 3) + 4 * (warp & 3), ig = ((tid >> 2) & 7) + 8 * (warp >> 2);      // u: value p, tokens ig, ig + 16, ig + 32, ig + 48
    const int ps = (tid & 7) * 2, kg = (tid >> 3) * 4;              // state: values ps, ps + 1, channels kg ..
    const bool p_ok = p0 + p < P, s_ok = p0 + ps < P && kg < K;
    float S[2][4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float4 v = rc_load4(state + (size_t)(p0 + ps + e) * K + kg, s_ok);
        S[e][0] = v.x; S[e][1] = v.y; S[e][2] = v.z; S[e][3] = v.w;
        if (kg < K) *reinterpret_cast<float4*>(Ss + (ps + e) * ldw + kg) = v;
    }
    for (int c = 0; c < chunks; ++c) {
        float own[4];                                               // U, asked for early
#pragma unroll
        for (int i = 0; i < 4; ++i) own[i] = p_ok ? at.u[(size_t)(ig + 16 * i) * P + p0 + p] : 0.f;
        const float4 fade = rc_load4(at.decay + kg, kg < K);
        rc_wait<0>();                                               // W and k e_end
        __syncthreads();                                            // and S is whole; the last chunk's k e_end is read
        copy(Ke + ((c + 1) & 1) * K * DC_TOKENS, K, at.k_end + step, c + 1 < chunks);
        if (s_ok) {                                                 // left for the outputs
#pragma unroll
            for (int k = 0; k < 4; ++k) *reinterpret_cast<float2*>(at.start + (size_t)(kg + k) * P + p0 + ps) = make_float2(S[0][k], S[1][k]);
        }
        const float *w = Ws + ig * ldw, *s = Ss + p * ldw;
        float part[4][4] = {};                                      // four chains a sum: shorter ones round less
#pragma unroll 8
        for (int k = 0; k < K; k += 4) {
            const float4 y = *reinterpret_cast<const float4*>(s + k);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 x = *reinterpret_cast<const float4*>(w + 16 * i * ldw + k);
                part[i][0] += x.x * y.x; part[i][1] += x.y * y.y;
                part[i][2] += x.z * y.z; part[i][3] += x.w * y.w;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float u = own[i] - ((part[i][0] + part[i][1]) + (part[i][2] + part[i][3]));
            Us[(ig + 16 * i) * LU + p] = u;
            if (p_ok) at.u[(size_t)(ig + 16 * i) * P + p0 + p] = u;
        }
        __syncthreads();                                            // u is whole; W is read
        copy(Ws, ldw, at.w + step, c + 1 < chunks);
#pragma unroll
        for (int e = 0; e < 2; ++e) { S[e][0] *= fade.x; S[e][1] *= fade.y; S[e][2] *= fade.z; S[e][3] *= fade.w; }
        if (kg < K) {
            const float* ke = Ke + (c & 1) * K * DC_TOKENS + kg;
#pragma unroll 16
            for (int j = 0; j < DC_TOKENS; ++j) {
                const float4 x = *reinterpret_cast<const float4*>(ke + j * K);
                const float2 y = *reinterpret_cast<const float2*>(Us + j * LU + ps);
                S[0][0] += x.x * y.x; S[0][1] += x.y * y.x; S[0][2] += x.z * y.x; S[0][3] += x.w * y.x;
                S[1][0] += x.x * y.y; S[1][1] += x.y * y.y; S[1][2] += x.z * y.y; S[1][3] += x.w * y.y;
            }
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

// grid (chunks, H * ptiles, B), 128 threads: a chunk's 64 tokens x 128 values, from S0 and then from the chunk's own u
__global__ void __launch_bounds__(128, 3)
delta_chunk_out_kernel(const DcArgs a, int ptiles) {
    pdl_wait();
    pdl_launch_dependents();
    // a tile: 16 channels or tokens x 128 values, and q of 64 tokens x 16 channels or their pairs with 16 tokens, 16 x 64
    constexpr int ROWS = 16, LDV = 132, LDQ = ROWS + 4, LDP = 68;
    __shared__ __align__(16) float values[3][ROWS * LDV], lefts[3][DC_TOKENS * LDQ];
    const int c = blockIdx.x, h = blockIdx.y / ptiles, p0 = (blockIdx.y - h * ptiles) * 128, tid = threadIdx.x, K = a.K, P = a.P;
    const int b = rc_sequence(a.cu_seqlens, a.B, a.from, blockIdx.z);
    if (b < 0) return;
    const int t0 = a.cu_seqlens[b] + c * DC_TOKENS, n = min(DC_TOKENS, a.cu_seqlens[b + 1] - t0);
    if (n <= 0) return;
    const DcPlace at = dc_place(a, b, c, h);
    const int state_tiles = (K + ROWS - 1) / ROWS, n_tiles = state_tiles + (n + ROWS - 1) / ROWS;
    auto copy = [&](int t) {                                        // one commit group a tile, also beyond the last
        if (t < n_tiles) {
            const bool from_state = t < state_tiles;
            const int row0 = (from_state ? t : t - state_tiles) * ROWS, limit = from_state ? K : n;
            const float* right = from_state ? at.start : at.u;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (from_state) {
                    const int r = (tid >> 2) + 32 * i, e = (tid & 3) * 4;
                    const bool ok = row0 + e < K;
                    rc_copy16(&lefts[t % 3][r * LDQ + e], at.q0 + (ok ? r * K + row0 + e : 0), ok);
                } else {
                    const int r = (tid >> 4) + 8 * i, e = (tid & 15) * 4;
                    const bool ok = row0 + r < n;
                    rc_copy16(&lefts[t % 3][r * LDP + e], at.q_pairs + (ok ? (row0 + r) * DC_TOKENS + e : 0), ok);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = (tid >> 5) + 4 * i, e = (tid & 31) * 4;
                const bool ok = row0 + r < limit && p0 + e < P;
                rc_copy16(&values[t % 3][r * LDV + e], right + (ok ? (size_t)(row0 + r) * P + p0 + e : 0), ok);
            }
        }
        rc_commit();
    };
    copy(0);
    copy(1);
    const int ig = (tid >> 4) * 4, pg = (tid & 15) * 4;             // tokens ig .., 32 + ig ..; values pg .., 64 + pg ..
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    for (int t = 0; t < n_tiles; ++t) {
        rc_wait<1>();
        __syncthreads();
        copy(t + 2);
        const float *left = lefts[t % 3], *right = values[t % 3];
        if (t >= state_tiles) {
            rc_outer<ROWS>(acc, left, LDP, ig, 32 + ig, right, LDV, pg, 64 + pg);
        } else {
#pragma unroll
            for (int k = 0; k < ROWS; k += 4) {                     // q four channels a load
                float4 q[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) q[i] = *reinterpret_cast<const float4*>(left + ((i >> 2) * 32 + ig + (i & 3)) * LDQ + k);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float4 y0 = *reinterpret_cast<const float4*>(right + (k + r) * LDV + pg), y1 = *reinterpret_cast<const float4*>(right + (k + r) * LDV + 64 + pg);
                    const float y[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float x = r == 0 ? q[i].x : (r == 1 ? q[i].y : (r == 2 ? q[i].z : q[i].w));
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[i][j] += x * y[j];
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = (i >> 2) * 32 + ig + (i & 3);
        if (t >= n) continue;
        float* out = a.o + (size_t)(t0 + t) * a.H * P + h * P + p0;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int p = 64 * half + pg;
            if (p0 + p < P) *reinterpret_cast<float4*>(out + p) = make_float4(acc[i][4 * half], acc[i][4 * half + 1], acc[i][4 * half + 2], acc[i][4 * half + 3]);
        }
    }
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
                                 int Hk, int K, int P, int decay_k, int write_state, cudaStream_t stream) {
    if (T <= 0 || B <= 0 || max_new <= 0 || max_new < from) return 0;
    if (!qwb_delta_chunked_scratch(T, B, from, H, K, P) || Hk <= 0 || H % Hk || ld % 4 || ld < 2 * Hk * K + H * P || (decay_k != K && decay_k != 1) || ld_a < H * decay_k)
        return qwb_fail(QWB_ERR_ARG, "delta_chunked: %d heads, %d key heads, state %d x %d in rows of %d, %d decays a head", H, Hk, K, P, ld, decay_k);
    for (const void* p : {(const void*)qkv, (const void*)state, (const void*)o, (const void*)scratch})
        if (!p || !rc_aligned16(p)) return qwb_fail(QWB_ERR_ARG, "delta_chunked: a tensor is not 16-byte aligned");
    const int chunks = (max_new + DC_TOKENS - 1) / DC_TOKENS, ptiles = (P + 127) / 128, planes = rc_planes(T, B, from);
    const DcArgs a = {qkv, beta, a_raw, dt_bias, A_log, cu_seqlens, slots, state, o, scratch, ld, ld_a, H, Hk, K, P, decay_k, write_state, B, from};
    const size_t smem1 = (3 * DC_TOKENS * DC_MAX_K + DC_A_FLOATS + 4 * DC_MAX_K + DC_TOKENS) * sizeof(float);
    const size_t smem2 = ((3 * K + 4) * DC_TOKENS + DC_WALK_P * (K + 4) + DC_TOKENS * (DC_WALK_P + 4)) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
    if (e != cudaSuccess) return qwb_fail(QWB_ERR_CUDA, "delta_chunked: %s", cudaGetErrorString(e));
    qwb_launch(delta_chunk_prep_kernel, dim3(chunks, H, planes), 256, smem1, stream, a);
    if (int rc = qwb_check_launch("delta_chunk_prep")) return rc;
    qwb_launch(delta_chunk_walk_kernel, dim3((P + DC_WALK_P - 1) / DC_WALK_P, H, planes), 256, smem2, stream, a);
    if (int rc = qwb_check_launch("delta_chunk_walk")) return rc;
    qwb_launch(delta_chunk_out_kernel, dim3(chunks, H * ptiles, planes), 128, 0, stream, a, ptiles);
    return qwb_check_launch("delta_chunk_out");
}
