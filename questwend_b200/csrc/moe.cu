// Routed experts: the router's choice, and the experts' feed-forward for the tokens that chose them.
//
//   moe_route     scores of all experts (softmax or sigmoid of the logits, 32-bit); a choice by score, or by score plus a
//                 correction per expert, over all experts or inside the best groups of neighbours; the `top` largest,
//                 ties to the lower index; weights from the scores alone
//   moe_up        act[t, k, :] = silu(Wg[e] x_t) * (Wu[e] x_t) (gated) or f(Wu[e] x_t), e = the k-th choice of token t
//   moe_down      out[t, :] = sum_k weight[t, k] * Wd[e_k] act[t, k, :]
// The weights may stand on the experts' inputs instead: act = f(Wu[e] (w x_t)), formed as f(w (Wu[e] x_t)) in 32-bit (both
// factors of the gated form), and the sum over the choices is then plain.
// A shared expert (ungated, a width of its own) that every token uses rides in the same two kernels; its output is
// multiplied by a number per token.
//
// The products read each chosen expert's rows straight from the stacked weights (Wu [E, F, D], gated: [E, 2F, D] with the
// gate rows first; Wd [E, D, F]): a warp per few rows, 32-bit sums.  This is the form for a step of few tokens, where every
// token's experts are streamed once, and for the 32-bit engine.  moe_stream reads an expert once for all of its tokens, on mma.sync, from
// about as many choices on as there are experts.  Many bfloat16 tokens are sorted by expert instead
// and go through a library grouped product; moe_sort, moe_spread, moe_act and moe_combine are the kernels around it.
#include "common.cuh"

#define QWB_MOE_MAX_TOP 16
#define QWB_MOE_MAX_EXPERTS 1024
#define MOE_UP_BLOCKS 5         // blocks of moe_up an SM by registers: more loads on their way beat a few spills in the shared expert's part
#define MOE_SHARED_WARPS 4      // of moe_down, at most
#define QWB_MOE_GATED 16        // activation code of the gated form, silu(gate) * up; others: qwb_activate's codes

// ---------------------------------------------------------------------------------
// route: a warp per token.  logits rows hold ld values: E experts and, with gate_out, the shared expert's gate after them.
//   score[e]  softmax(z)[e] (sigmoid = 0) or 1 / (1 + exp(-z[e])) (sigmoid = 1)
//   choice[e] score[e] + correction[e]; a group's score is the sum of its two largest choices (of one, if it has one
//             expert), and the experts of all but the `keep` best groups (ties to the lower index) are out
//   weight    score of a chosen expert, / (their sum + sum_eps) if `renorm`, * weight_scale
//   gate_out  1 / (1 + exp(-z[E]))
// ---------------------------------------------------------------------------------
// The choice works on keys, the scores' bits in an order that unsigned integers keep; 0 (below every number's key) is out.
__device__ __forceinline__ unsigned order_key(float v) {
    const unsigned b = __float_as_uint(v);
    return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}
// The place of the largest of n keys in shared memory (the lowest of equal ones), which is then out; the whole warp calls.
__device__ __forceinline__ int take_best(unsigned* key, int n, int lane) {
    unsigned best = 0;
    int at = n;
    for (int e = lane; e < n; e += 32) {
        const unsigned v = key[e];
        if (v > best || at == n) { best = v; at = e; }
    }
    const unsigned top = __reduce_max_sync(0xffffffffu, best);
    const int first = (int)__reduce_min_sync(0xffffffffu, best == top && at < n ? (unsigned)at : 0x7fffffffu);
    if (lane == 0) key[first] = 0;
    __syncwarp();
    return first;
}

__global__ void moe_route_kernel(const float* logits, int ld, const float* __restrict__ correction, int* __restrict__ chosen,
                                 float* __restrict__ weight, float* __restrict__ gate_out, int T, int E, int top, int sigmoid,
                                 int groups, int keep, int renorm, float sum_eps, float weight_scale) {
    pdl_launch_dependents();            // the trigger first: see qwb_launch_link
    pdl_wait();
    extern __shared__ unsigned route_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= T) return;
    unsigned* key = route_smem + warp * (2 * E + groups);   // [E] keys of the choice scores
    float* score = reinterpret_cast<float*>(key + E);       // [E]
    unsigned* gkey = key + 2 * E;                           // [groups]
    const float* z = logits + (size_t)t * ld;
    float mx = 0.f, sum = 1.f;
    if (!sigmoid) {
        mx = -INFINITY;
        for (int e = lane; e < E; e += 32) mx = fmaxf(mx, __ldcg(z + e));
        mx = warp_max(mx);
        sum = 0.f;
        for (int e = lane; e < E; e += 32) sum += expf(__ldcg(z + e) - mx);
        sum = warp_sum(sum);
    }
    const bool by_logit = !sigmoid && !correction && groups == 1;       // a softmax keeps the logits' order
    for (int e = lane; e < E; e += 32) {
        const float v = __ldcg(z + e);
        const float s = sigmoid ? 1.f / (1.f + expf(-v)) : expf(v - mx) / sum;
        score[e] = s;
        key[e] = order_key(by_logit ? v : s + (correction ? correction[e] : 0.f));
    }
    __syncwarp();
    if (keep < groups) {
        const int size = E / groups;
        auto value = [&](int e) { const unsigned k = key[e]; return __uint_as_float((k >> 31) ? k ^ 0x80000000u : ~k); };
        for (int g = lane; g < groups; g += 32) {
            float a = value(g * size), b = -INFINITY;       // the two largest
            for (int e = g * size + 1; e < (g + 1) * size; ++e) {
                const float c = value(e);
                b = fmaxf(b, fminf(a, c));
                a = fmaxf(a, c);
            }
            gkey[g] = order_key(size > 1 ? a + b : a);
        }
        __syncwarp();
        for (int k = 0; k < keep; ++k) take_best(gkey, groups, lane);
        for (int e = lane; e < E; e += 32)
            if (gkey[e / size]) key[e] = 0;                 // of a group that was not taken
        __syncwarp();
    }
    int mine = 0;                                           // lane k's choice
    for (int k = 0; k < top; ++k) {
        const int at = take_best(key, E, lane);
        if (lane == k) mine = at;
    }
    const float s = lane < top ? score[mine] : 0.f;
    const float total = warp_sum(s);
    if (lane < top) {
        chosen[(size_t)t * top + lane] = mine;
        weight[(size_t)t * top + lane] = (renorm ? s / (total + sum_eps) : s) * weight_scale;
    }
    if (gate_out && lane == 31) gate_out[t] = 1.f / (1.f + expf(-__ldcg(z + E)));
}

extern "C" int qwb_moe_route(const float* logits, int ld, const float* correction, int* chosen, float* weight, float* gate_out, int T,
                             int E, int top, int sigmoid, int groups, int keep, int renorm, float sum_eps, float weight_scale,
                             cudaStream_t stream) {
    if (T <= 0) return 0;
    if (E <= 0 || E > QWB_MOE_MAX_EXPERTS || top <= 0 || top > E || top > QWB_MOE_MAX_TOP)
        return qwb_fail(QWB_ERR_ARG, "moe_route: %d of %d experts (at most %d of %d)", top, E, QWB_MOE_MAX_TOP, QWB_MOE_MAX_EXPERTS);
    if (groups <= 0 || E % groups || keep <= 0 || keep > groups || top > keep * (E / groups))
        return qwb_fail(QWB_ERR_ARG, "moe_route: %d of %d experts from %d of %d groups", top, E, keep, groups);
    if (ld < E + (gate_out ? 1 : 0)) return qwb_fail(QWB_ERR_ARG, "moe_route: rows of %d logits for %d experts", ld, E);
    const int warps = T >= 592 ? 4 : 1;                     // few tokens: a block each, side by side on the SMs
    const size_t smem = (size_t)warps * (2 * E + groups) * sizeof(float);   // at most 48 KB
    qwb_launch_link(T, QWB_LINK_ROWS_NORM, moe_route_kernel, (T + warps - 1) / warps, 32 * warps, smem, stream, logits, ld, correction, chosen, weight, gate_out, T, E, top,
               sigmoid, groups, keep, renorm, sum_eps, weight_scale);
    return qwb_check_launch("moe_route");
}

// ---------------------------------------------------------------------------------
// Rows of a matrix times vectors, a warp each: acc[r * NX + v] = this lane's part of w_r . x_v; rows `ldw` values apart, of
// which the first nr exist, vectors `ldx` apart, of which the first nx exist (a missing one repeats the last).
// ---------------------------------------------------------------------------------
template <typename T, int NR, int NX>
__device__ __forceinline__ void lane_dots(const T* __restrict__ w, size_t ldw, int nr, const T* __restrict__ x, size_t ldx, int nx, int n,
                                          int lane, float* acc) {
    constexpr int VEC = Vec16<T>::N;
#pragma unroll
    for (int i = 0; i < NR * NX; ++i) acc[i] = 0.f;
    const T* wr[NR];
    const T* xv[NX];
#pragma unroll
    for (int r = 0; r < NR; ++r) wr[r] = w + (size_t)(r < nr ? r : nr - 1) * ldw;
#pragma unroll
    for (int v = 0; v < NX; ++v) xv[v] = x + (size_t)(v < nx ? v : nx - 1) * ldx;
    if (n % VEC == 0 && ldw % VEC == 0 && (NX == 1 || ldx % VEC == 0) && (uintptr_t)w % 16 == 0 && (uintptr_t)x % 16 == 0) {
#pragma unroll 2
        for (int i = lane; i < n / VEC; i += 32) {
            float a[NR][VEC];
#pragma unroll
            for (int r = 0; r < NR; ++r) reinterpret_cast<const Vec16<T>*>(wr[r])[i].get(a[r]);
#pragma unroll
            for (int v = 0; v < NX; ++v) {
                float b[VEC];
                reinterpret_cast<const Vec16<T>*>(xv[v])[i].get(b);
#pragma unroll
                for (int r = 0; r < NR; ++r)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) acc[r * NX + v] += a[r][e] * b[e];
            }
        }
    } else {
        for (int i = lane; i < n; i += 32)
#pragma unroll
            for (int v = 0; v < NX; ++v) {
                const float b = to_f32(xv[v][i]);
#pragma unroll
                for (int r = 0; r < NR; ++r) acc[r * NX + v] += to_f32(wr[r][i]) * b;
            }
    }
}

// Blocks: per copy of a token (T * top) as many as its expert's features take, 8 warps each, then the shared expert's, with
// NT tokens a warp.
// A warp makes two features of a plain expert, one of a gated one (its gate and its up row), two of the shared expert.
template <typename T, int NT>
__global__ void __launch_bounds__(256, MOE_UP_BLOCKS)
moe_up_kernel(const T* __restrict__ x, const T* __restrict__ wu, const int* __restrict__ chosen, const float* __restrict__ weight_in, T* __restrict__ act,
              const T* __restrict__ wsu, T* __restrict__ act_s, int n_tok, int D, int F, int Fs, int top, int kind) {
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool gated = kind == QWB_MOE_GATED;
    const int per_slot = ((gated ? F : (F + 1) / 2) + 7) / 8, n_routed = n_tok * top * per_slot;
    if ((int)blockIdx.x < n_routed) {
        const int slot = blockIdx.x / per_slot, item = (blockIdx.x - slot * per_slot) * 8 + warp;
        const int f = gated ? item : 2 * item;
        if (f >= F) return;
        const size_t first = (size_t)chosen[slot] * (gated ? 2 * F : F) + f;
        float acc[2];
        lane_dots<T, 2, 1>(wu + first * D, gated ? (size_t)F * D : (size_t)D, gated ? 2 : min(2, F - f), x + (size_t)(slot / top) * D, 0, 1, D,
                           lane, acc);
        const float w = weight_in ? weight_in[slot] : 1.f;
        const float a = warp_sum(acc[0]) * w, b = warp_sum(acc[1]) * w;
        T* o = act + (size_t)slot * F + f;
        if (gated) { if (lane == 0) o[0] = from_f32<T>(a / (1.f + expf(-a)) * b); }
        else if (lane < min(2, F - f)) o[lane] = from_f32<T>(qwb_activate(lane ? b : a, kind));
    } else {
        const int per_group = ((Fs + 1) / 2 + 7) / 8, group = (blockIdx.x - n_routed) / per_group;
        const int t0 = group * NT, f = 2 * ((blockIdx.x - n_routed - group * per_group) * 8 + warp);
        if (f >= Fs) return;
        const int nt = min(NT, n_tok - t0), nf = min(2, Fs - f);
        float acc[2 * NT];
        lane_dots<T, 2, NT>(wsu + (size_t)f * D, D, nf, x + (size_t)t0 * D, D, nt, D, lane, acc);
#pragma unroll
        for (int i = 0; i < 2 * NT; ++i) {
            const float v = warp_sum(acc[i]);
            if (lane == i && i / NT < nf && i % NT < nt)
                act_s[(size_t)(t0 + i % NT) * Fs + f + i / NT] = from_f32<T>(qwb_activate(v, kind == QWB_MOE_GATED ? 3 : kind));
        }
    }
}

// grid (ceil(D / NR), T), a warp per choice and one or more for the shared expert: NR outputs of one token; the warps' products
// are weighted and summed in the order of the choices, the shared expert last.  out may be added onto (`onto`).  A shared expert
// about s times as wide as the others is cut into s warps' shares, as a block waits for its longest warp: by sizes alone, so that a token's
// sum has one order.  Both products, 6 of 64 experts of 2,048 x 1,408 and one of 2,816, us with a warp / shares: 1 token 19.7 / 17.6, 2 36.8 / 35.1, 3
// 48.2 / 46.4, 4 56.1 / 57.4, 7 88.4 / 91.3; experts of 2,048 x 704 7 58.6 / 57.3; 32-bit 1 38.3 / 33.7, 4 112.7 / 103.3, 16 377 / 356.
template <typename T, int NR>
__global__ void moe_down_kernel(const T* __restrict__ act, const T* __restrict__ wd, const int* __restrict__ chosen,
                                const float* __restrict__ weight, const T* __restrict__ act_s, const T* __restrict__ wsd,
                                const float* __restrict__ gate, float* out, int D, int F, int Fs, int top, int onto) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float part[QWB_MOE_MAX_TOP + MOE_SHARED_WARPS][NR];
    const int t = blockIdx.y, d = blockIdx.x * NR;
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nr = min(NR, D - d);
    float acc[NR], mul;
    if (k < top) {
        const size_t slot = (size_t)t * top + k;
        lane_dots<T, NR, 1>(wd + ((size_t)chosen[slot] * D + d) * F, F, nr, act + slot * F, 0, 1, F, lane, acc);
        mul = weight ? weight[slot] : 1.f;
    } else {
        const int warps = (blockDim.x >> 5) - top, share = warps == 1 ? Fs : (Fs / 8 + warps - 1) / warps * 8, from = min(Fs, (k - top) * share);
        lane_dots<T, NR, 1>(wsd + (size_t)d * Fs + from, Fs, nr, act_s + (size_t)t * Fs + from, 0, 1, min(share, Fs - from), lane, acc);
        mul = gate ? gate[t] : 1.f;
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const float v = warp_sum(acc[r]);
        if (lane == 0) part[k][r] = mul * v;
    }
    __syncthreads();
    if (threadIdx.x < nr) {
        float total = 0.f;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) total += part[i][threadIdx.x];
        float* o = out + (size_t)t * D + d + threadIdx.x;
        *o = onto ? *o + total : total;
    }
}

template <typename T>
static void launch_moe_experts(const void* x, const void* wu, const void* wd, const int* chosen, const float* weight_in, const float* weight, const void* wsu,
                               const void* wsd, const float* gate, void* act, void* act_s, float* out, int n_tok, int D, int F, int Fs,
                               int top, int kind, int onto, cudaStream_t stream) {
    const int per_slot = ((kind == QWB_MOE_GATED ? F : (F + 1) / 2) + 7) / 8, per_group = Fs > 0 ? ((Fs + 1) / 2 + 7) / 8 : 0;
    const int nt = n_tok > 1 ? 2 : 1;
    const dim3 g1(n_tok * top * per_slot + (n_tok + nt - 1) / nt * per_group), g2((D + 3) / 4, n_tok);
    if (nt == 1)
        qwb_launch(moe_up_kernel<T, 1>, g1, 256, 0, stream, (const T*)x, (const T*)wu, chosen, weight_in, (T*)act, (const T*)wsu, (T*)act_s, n_tok, D, F, Fs, top, kind);
    else
        qwb_launch(moe_up_kernel<T, 2>, g1, 256, 0, stream, (const T*)x, (const T*)wu, chosen, weight_in, (T*)act, (const T*)wsu, (T*)act_s, n_tok, D, F, Fs, top, kind);
    int shared_warps = Fs > 0 ? 1 : 0;
    if (Fs > F && Fs % 8 == 0) shared_warps = min((Fs + F / 2) / F, MOE_SHARED_WARPS);
    qwb_launch(moe_down_kernel<T, 4>, g2, 32 * (top + shared_warps), 0, stream, (const T*)act, (const T*)wd, chosen, weight, (const T*)act_s,
               (const T*)wsd, gate, out, D, F, Fs, top, onto);
}

// ---------------------------------------------------------------------------------
// The same for bfloat16 and sizes in multiples of 8, an expert's rows once for all the tokens that chose it: 16 rows of one expert a
// block on mma.sync (the rows are its 16-row operand, eight tokens its 8-column one), the contraction cut over the block's four warps.
// A step of few tokens is bound by the weights' bytes: a thread asks for 8 x 16 bytes of its two rows before the first product, seven
// blocks an SM, and the weights pass L1 by.  moe_lists finds the experts that are chosen and the copies of tokens that chose them, in order,
// so that a block's first weights are asked for one round trip after its start.  `down` leaves a row of D sums for every copy and for the
// shared expert of every token, which moe_merge adds up in the order of the choices.
// 32 tokens, 6 of 64 experts of 2,048 x 1,408 and a shared one, us: a row for each copy 328, the library's grouped products 224; here 168 with
// every block going through the choices by itself, 151 with lists, 136 with four instead of eight blocks of 32 values on their way, seven
// instead of four blocks an SM and early starts (the weights at 6.55 TB/s: 107).  8 tokens 104 -> 92.
// ---------------------------------------------------------------------------------
#define MS_WARPS 4
#define MS_AHEAD 4              // blocks of 32 values of two rows that are on their way
#define MS_MAX_COPIES 2048
#define MS_LINK_ROWS 128        // tokens up to which the four kernels start early

__device__ __forceinline__ uint4 ms_weight(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void ms_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// acc += rows lo and hi (of this lane; null: zeros) times NT x 8 vectors (vector(j): this lane's of the j-th eight, or null; called behind the
// rows' first loads), n values each (a multiple of 8), this warp's share.  A lane's 16 bytes are eight neighbouring values of the rows and
// the same eight of the vectors.
template <int NT, class Vector>
__device__ __forceinline__ void ms_tile(float (&acc)[NT][4], const bf16* lo, const bf16* hi, Vector vector, int n) {
    const int warp = threadIdx.x >> 5, t = threadIdx.x & 3, pieces = n / 8;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (int b0 = warp; 4 * b0 < pieces; b0 += MS_WARPS * MS_AHEAD) {
        uint4 w0[MS_AHEAD], w1[MS_AHEAD], v[NT == 1 ? MS_AHEAD : 1];
#pragma unroll
        for (int u = 0; u < MS_AHEAD; ++u) {
            const int p = 4 * (b0 + MS_WARPS * u) + t;
            w0[u] = lo && p < pieces ? ms_weight(reinterpret_cast<const uint4*>(lo) + p) : zero;
            w1[u] = hi && p < pieces ? ms_weight(reinterpret_cast<const uint4*>(hi) + p) : zero;
        }
        const bf16* x[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) x[j] = vector(j);
        if (NT == 1) {
#pragma unroll
            for (int u = 0; u < MS_AHEAD; ++u) {
                const int p = 4 * (b0 + MS_WARPS * u) + t;
                v[u] = x[0] && p < pieces ? reinterpret_cast<const uint4*>(x[0])[p] : zero;
            }
        }
#pragma unroll
        for (int u = 0; u < MS_AHEAD; ++u) {
            const int p = 4 * (b0 + MS_WARPS * u) + t;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const uint4 y = NT == 1 ? v[u] : (x[j] && p < pieces ? reinterpret_cast<const uint4*>(x[j])[p] : zero);
                ms_mma(acc[j], w0[u].x, w1[u].x, w0[u].y, w1[u].y, y.x, y.y);
                ms_mma(acc[j], w0[u].z, w1[u].z, w0[u].w, w1[u].w, y.z, y.w);
            }
        }
    }
}

// What moe_lists leaves: the experts that are chosen, in order, in slots of up to MS_SLOT copies, where each slot's copies begin (and the last
// one's end), the copies.  An expert that many tokens chose has several slots, whose blocks run side by side: with one slot an expert its blocks
// went through its copies 32 at a time, one pass behind the other.  us,
// tokens of which most chose the same experts, sorted through the grouped product / a slot an expert / now: 6 of 64 and a shared one, 64 tokens
// 122 / 115 / 97, 128 140 / 212 / 180; 8 of 128, 64 86 / 114 / 102, 128 122 / 194 / 167; 2 of 8 of 4,096 x 2,048, 64 65 / 125 / 78; evenly chosen, the first
// of these 204 / 150 / 149 and 208 / 204 / 188.
#define MS_SLOT 32
#define MS_MAX_SLOTS (QWB_MOE_MAX_EXPERTS + MS_MAX_COPIES / MS_SLOT)
struct MsLists { int n; int expert[MS_MAX_SLOTS], begin[MS_MAX_SLOTS + 1], copies[MS_MAX_COPIES]; };

struct MsArgs {
    const bf16 *in, *in_s, *w, *w_s;        // vectors of copies (up: of tokens) and of the shared expert's tokens; experts' and shared weights
    const MsLists* lists;
    const float* weight_in;
    bf16 *act, *act_s;                      // up
    float *y, *y_s;                         // down
    int T, top, K, K_s, rows, rows_s, kind;
};

// one block of 1,024 threads; a warp counts, then lists, the copies of every 32nd expert
__global__ void __launch_bounds__(1024)
moe_lists_kernel(const int* chosen, MsLists* lists, int S, int E) {
    pdl_launch_dependents();            // the trigger first: see qwb_launch_link
    pdl_wait();
    __shared__ int choice[MS_MAX_COPIES], count[QWB_MOE_MAX_EXPERTS], warps[2][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int c = tid; c < S; c += 1024) choice[c] = __ldcg(chosen + c);
    __syncthreads();
    for (int e = warp; e < E; e += 32) {
        int total = 0;
        for (int c = 0; c < S; c += 32) total += __popc(__ballot_sync(0xffffffffu, c + lane < S && choice[c + lane] == e));
        if (lane == 0) count[e] = total;
    }
    __syncthreads();
    const int mine = tid < E ? count[tid] : 0;
    const int own = (mine + MS_SLOT - 1) / MS_SLOT;
    int copies = mine, slots = own;                                 // sums over the experts up to this one
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, copies, o), b = __shfl_up_sync(0xffffffffu, slots, o);
        if (lane >= o) { copies += a; slots += b; }
    }
    if (lane == 31) { warps[0][warp] = copies; warps[1][warp] = slots; }
    __syncthreads();
    for (int w = 0; w < warp; ++w) { copies += warps[0][w]; slots += warps[1][w]; }
    for (int k = 0; k < own; ++k) { lists->expert[slots - own + k] = tid; lists->begin[slots - own + k + 1] = min(copies - mine + MS_SLOT * (k + 1), copies); }
    if (tid == 0) lists->begin[0] = 0;
    if (tid == 1023) lists->n = slots;
    if (tid < E) count[tid] = copies - mine;
    __syncthreads();
    for (int e = warp; e < E; e += 32) {
        int at = count[e];
        for (int c = 0; c < S; c += 32) {
            const bool is = c + lane < S && choice[c + lane] == e;
            const unsigned all = __ballot_sync(0xffffffffu, is);
            if (is) lists->copies[at + __popc(all & ((1u << lane) - 1u))] = c + lane;
            at += __popc(all);
        }
    }
}

// One 16-row tile with the vectors from `first` on, NT x 8 of them at a time
template <int NT, bool DOWN>
__device__ __forceinline__ void ms_rows(const MsArgs& a, bool shared, const bf16* lo, const bf16* hi, int f0, const int* copies, int n, int first, float* part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, K = shared ? a.K_s : a.K;
    int copy[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) copy[j] = first + 8 * j + g < n ? (shared ? first + 8 * j + g : __ldcg(copies + first + 8 * j + g)) : -1;
    float acc[NT][4] = {};
    ms_tile<NT>(acc, lo, hi, [&](int j) -> const bf16* {
        return copy[j] < 0 ? nullptr : (shared ? a.in_s + (size_t)copy[j] * K : a.in + (size_t)(DOWN ? copy[j] : copy[j] / a.top) * K);
    }, K);
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) part[((warp * NT + j) * 4 + r) * 32 + lane] = acc[j][r];
    __syncthreads();
    const int r = warp;                                             // thread: register r of every tile's lane
    const bool gated = !DOWN && !shared && a.kind == QWB_MOE_GATED;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        auto sum = [&](int reg) {
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < MS_WARPS; ++w) v += part[((w * NT + j) * 4 + reg) * 32 + lane];
            return v;
        };
        const int i = first + 8 * j + 2 * t + (r & 1), row = g + 8 * (r >> 1);
        if (i >= n || (gated && r >= 2)) continue;
        const int c = shared ? i : __ldcg(copies + i), f = f0 + row;
        if (f >= (shared ? a.rows_s : a.rows)) continue;
        float v = sum(r);
        if (DOWN) {
            (shared ? a.y_s : a.y)[(size_t)c * a.rows + f] = v;
        } else {
            const float w = a.weight_in && !shared ? a.weight_in[c] : 1.f;
            v *= w;
            if (gated) v = v / (1.f + expf(-v)) * (sum(r + 2) * w);
            else v = qwb_activate(v, shared && a.kind == QWB_MOE_GATED ? 3 : a.kind);
            (shared ? a.act_s + (size_t)c * a.rows_s : a.act + (size_t)c * a.rows)[f] = from_f32<bf16>(v);
        }
    }
}

// Blocks: the shared expert's tiles, once for every MS_SLOT tokens, then (slot, tile).  A tile is 16 rows, of a gated expert 8 gate rows and their 8 up rows.
template <bool DOWN>
__global__ void __launch_bounds__(32 * MS_WARPS, 7)
moe_stream_kernel(const MsArgs a, int tiles, int tiles_s) {
    pdl_launch_dependents();            // the trigger first: see qwb_launch_link
    pdl_wait();
    __shared__ float part[MS_WARPS * 4 * 4 * 32];
    const int lane = threadIdx.x & 31, g = lane >> 2;
    const int blocks_s = tiles_s * ((a.T + MS_SLOT - 1) / MS_SLOT);
    const bool shared = (int)blockIdx.x < blocks_s, gated = !DOWN && !shared && a.kind == QWB_MOE_GATED;
    const int item = (int)blockIdx.x - blocks_s, slot = item / tiles, tile = shared ? (int)blockIdx.x % tiles_s : item - slot * tiles;
    const int* copies = nullptr;
    int first = 0, n = 0, e = 0;
    if (shared) {
        first = (int)blockIdx.x / tiles_s * MS_SLOT;
        n = min(a.T, first + MS_SLOT);
    } else {
        const int begin = __ldcg(a.lists->begin + slot), end = __ldcg(a.lists->begin + slot + 1);
        e = __ldcg(a.lists->expert + slot);
        if (slot >= __ldcg(&a.lists->n)) return;
        copies = a.lists->copies + begin;
        n = end - begin;
    }
    const int rows = shared ? a.rows_s : a.rows, f0 = tile * (gated ? 8 : 16), K = shared ? a.K_s : a.K;
    const bf16* w = shared ? a.w_s : a.w + (size_t)e * (gated ? 2 * rows : rows) * K;
    const int r0 = f0 + g, r1 = gated ? rows + f0 + g : f0 + g + 8;
    const bf16 *lo = r0 < rows ? w + (size_t)r0 * K : nullptr, *hi = (gated ? r0 : r1) < rows ? w + (size_t)r1 * K : nullptr;
    if (n - first <= 8) ms_rows<1, DOWN>(a, shared, lo, hi, f0, copies, n, first, part);
    else if (n - first <= 16) ms_rows<2, DOWN>(a, shared, lo, hi, f0, copies, n, first, part);
    else ms_rows<4, DOWN>(a, shared, lo, hi, f0, copies, n, first, part);
}

// grid (ceil(D / 1,024), T), 256 threads: four outputs of a token a thread, from the rows of its copies
__global__ void __launch_bounds__(256)
moe_merge_kernel(const float* y, const float* y_s, const float* weight, const float* gate, float* out, int D, int top, int onto) {
    pdl_launch_dependents();            // the trigger first: see qwb_launch_link
    pdl_wait();
    const int t = blockIdx.y, d = (blockIdx.x * 256 + threadIdx.x) * 4;
    if (d >= D) return;
    float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](const float* row, float w) {
        const float4 v = *reinterpret_cast<const float4*>(row + d);
        total.x += w * v.x; total.y += w * v.y; total.z += w * v.z; total.w += w * v.w;
    };
#pragma unroll 4
    for (int k = 0; k < top; ++k) add(y + ((size_t)t * top + k) * D, weight ? weight[(size_t)t * top + k] : 1.f);
    if (y_s) add(y_s + (size_t)t * D, gate ? gate[t] : 1.f);
    float4* o = reinterpret_cast<float4*>(out + (size_t)t * D + d);
    if (onto) { const float4 v = *o; total.x += v.x; total.y += v.y; total.z += v.z; total.w += v.w; }
    *o = total;
}

// As qwb_moe_experts for bfloat16 and sizes in multiples of 8, every tensor 16-byte aligned; y [T * top + (Fs > 0 ? T : 0), D]: scratch,
// with qwb_moe_lists_floats() more behind it.
extern "C" int qwb_moe_lists_floats() { return (int)(sizeof(MsLists) / sizeof(float)) + 4; }
extern "C" int qwb_moe_stream(const void* x, const void* wu, const void* wd, const int* chosen, const float* weight, int on_input, const void* wsu, const void* wsd,
                              const float* gate, void* act, void* act_s, float* y, float* out, int T, int E, int D, int F, int Fs, int top, int kind, int onto,
                              cudaStream_t stream) {
    if (T <= 0) return 0;
    if (D <= 0 || F <= 0 || Fs < 0 || top <= 0 || top > QWB_MOE_MAX_TOP || E <= 0 || E > QWB_MOE_MAX_EXPERTS || D % 8 || F % 8 || Fs % 8 || T > MS_MAX_COPIES / top)
        return qwb_fail(QWB_ERR_ARG, "moe_stream: %d tokens x %d choices of %d experts, width %d, expert width %d, shared %d", T, top, E, D, F, Fs);
    if (Fs > 0 && (!wsu || !wsd || !act_s)) return qwb_fail(QWB_ERR_ARG, "moe_stream: a shared expert without its matrices");
    if (kind != QWB_MOE_GATED && !qwb_activation_known(kind)) return qwb_fail(QWB_ERR_ARG, "moe_stream: unknown activation %d", kind);
    for (const void* p : {x, wu, wd, wsu, wsd, (const void*)act, (const void*)act_s, (const void*)y, (const void*)out})
        if ((uintptr_t)p % 16) return qwb_fail(QWB_ERR_ARG, "moe_stream: a tensor is not 16-byte aligned");
    const int copies = T * top, slots = min(copies, min(copies, E) + copies / MS_SLOT);      // an expert's slots but for one are full
    const int passes = (T + MS_SLOT - 1) / MS_SLOT;                 // of the shared expert's tokens
    const int up_tiles = kind == QWB_MOE_GATED ? F / 8 : (F + 15) / 16, up_shared = (Fs + 15) / 16, down_tiles = (D + 15) / 16, down_shared = Fs > 0 ? down_tiles : 0;
    MsLists* lists = reinterpret_cast<MsLists*>(y + (size_t)T * (top + (Fs > 0 ? 1 : 0)) * D);
    float* y_s = Fs > 0 ? y + (size_t)T * top * D : nullptr;
    const MsArgs up = {(const bf16*)x, (const bf16*)x, (const bf16*)wu, (const bf16*)wsu, lists, on_input ? weight : nullptr, (bf16*)act, (bf16*)act_s, nullptr, nullptr,
                       T, top, D, D, F, Fs, kind};
    const MsArgs down = {(const bf16*)act, (const bf16*)act_s, (const bf16*)wd, (const bf16*)wsd, lists, nullptr, nullptr, nullptr, y, y_s, T, top, F, Fs, D, D, kind};
    qwb_launch_link(T, MS_LINK_ROWS, moe_lists_kernel, 1, 1024, 0, stream, chosen, lists, T * top, E);
    if (int rc = qwb_check_launch("moe_lists")) return rc;
    qwb_launch_link(T, MS_LINK_ROWS, moe_stream_kernel<false>, passes * up_shared + slots * up_tiles, 32 * MS_WARPS, 0, stream, up, up_tiles, up_shared);
    if (int rc = qwb_check_launch("moe_stream up")) return rc;
    qwb_launch_link(T, MS_LINK_ROWS, moe_stream_kernel<true>, passes * down_shared + slots * down_tiles, 32 * MS_WARPS, 0, stream, down, down_tiles, down_shared);
    if (int rc = qwb_check_launch("moe_stream down")) return rc;
    qwb_launch_link(T, MS_LINK_ROWS, moe_merge_kernel, dim3((D + 1023) / 1024, T), 256, 0, stream, (const float*)y, (const float*)y_s, on_input ? nullptr : weight, gate, out, D, top, onto);
    return qwb_check_launch("moe_merge");
}

// weight [T, top]: on the experts' inputs (on_input) or outputs.
// wsu [Fs, D], wsd [D, Fs], gate [T] (or null: 1), act_s [T, Fs]: the shared expert, Fs = 0 for none.
extern "C" int qwb_moe_experts(const void* x, const void* wu, const void* wd, const int* chosen, const float* weight, int on_input, const void* wsu,
                               const void* wsd, const float* gate, void* act, void* act_s, float* out, int dtype, int T, int D, int F,
                               int Fs, int top, int kind, int onto, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (D <= 0 || F <= 0 || Fs < 0 || top <= 0 || top > QWB_MOE_MAX_TOP)
        return qwb_fail(QWB_ERR_ARG, "moe_experts: width %d, expert width %d, shared %d, %d choices", D, F, Fs, top);
    if (Fs > 0 && (!wsu || !wsd || !act_s)) return qwb_fail(QWB_ERR_ARG, "moe_experts: a shared expert without its matrices");
    if (kind != QWB_MOE_GATED && !qwb_activation_known(kind)) return qwb_fail(QWB_ERR_ARG, "moe_experts: unknown activation %d", kind);
    if ((long long)T * top + T > 65535 || ((long long)T * top + T) * ((F > Fs ? F : Fs) / 8 + 1) > 0x7fffffffLL)
        return qwb_fail(QWB_ERR_ARG, "moe_experts: %d tokens x %d choices are too many for one launch", T, top);
    const float *weight_in = on_input ? weight : nullptr, *weight_out = on_input ? nullptr : weight;
    if (dtype == QWB_DT_F32)
        launch_moe_experts<float>(x, wu, wd, chosen, weight_in, weight_out, wsu, wsd, gate, act, act_s, out, T, D, F, Fs, top, kind, onto, stream);
    else if (dtype == QWB_DT_BF16)
        launch_moe_experts<bf16>(x, wu, wd, chosen, weight_in, weight_out, wsu, wsd, gate, act, act_s, out, T, D, F, Fs, top, kind, onto, stream);
    else return qwb_fail(QWB_ERR_ARG, "moe_experts: unknown dtype %d", dtype);
    return qwb_check_launch("moe_experts");
}

// ---------------------------------------------------------------------------------
// Around a grouped product over token copies sorted by expert (bfloat16; D and F multiples of 8):
//   moe_sort      place[c] = the row of copy c = t * top + k in the order (expert, copy); ends[e] = where expert e's run ends
//   moe_spread    xs[place[t, k], :] = x[t, :], and row_weight[place[t, k]] = weight[t, k] where the weights are on the inputs
//   moe_act       act[s, f] = f(u[s, f]), u [S, F], or silu(u[s, f]) * u[s, F + f], u [S, 2F]; u times row_weight[s] if given
//   moe_combine   out[t, :] (+)= sum_k weight[t, k] * y[place[t, k], :] + gate[t] * shared[t, :]
// ---------------------------------------------------------------------------------
// A block per expert: it counts the copies of lower experts (where its own run starts) and ranks its own ones.  Each warp
// walks over a run of neighbouring copies twice, 32 at a time (a ballot finds the ranks): once for its counts, then, knowing
// what the warps before it counted, to write the places.  Nothing depends on the order in which warps or blocks run.
#define MOE_SORT_WARPS 16
#define MOE_SORT_AHEAD 8          // groups of 32 whose loads are on their way together
__global__ void __launch_bounds__(MOE_SORT_WARPS * 32)
moe_sort_kernel(const int* __restrict__ chosen, int* __restrict__ place, int* __restrict__ ends, int S, int E) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ int own[MOE_SORT_WARPS], lower[MOE_SORT_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, expert = blockIdx.x;
    const unsigned full = 0xffffffffu, before = (1u << lane) - 1u;
    const int per = ((S + MOE_SORT_WARPS - 1) / MOE_SORT_WARPS + 31) & ~31;
    const int lo = min(S, warp * per), hi = min(S, lo + per);
    auto expert_of = [&](int i) { return i < hi ? min(max(chosen[i], 0), E - 1) : E; };        // E: not a copy
    int n_own = 0, n_lower = 0;
    for (int i0 = lo; i0 < hi; i0 += 32 * MOE_SORT_AHEAD) {
        int es[MOE_SORT_AHEAD];
#pragma unroll
        for (int a = 0; a < MOE_SORT_AHEAD; ++a) es[a] = expert_of(i0 + 32 * a + lane);
#pragma unroll
        for (int a = 0; a < MOE_SORT_AHEAD; ++a) {
            n_own += __popc(__ballot_sync(full, es[a] == expert));
            n_lower += __popc(__ballot_sync(full, es[a] < expert));
        }
    }
    if (lane == 0) { own[warp] = n_own; lower[warp] = n_lower; }
    __syncthreads();
    int at = 0, total = 0;                              // the next row of this warp's copies; where the run ends
    for (int w = 0; w < MOE_SORT_WARPS; ++w) {
        at += lower[w] + (w < warp ? own[w] : 0);
        total += lower[w] + own[w];
    }
    if (threadIdx.x == 0) ends[expert] = total;
    for (int i0 = lo; i0 < hi && n_own > 0; i0 += 32 * MOE_SORT_AHEAD) {
        int es[MOE_SORT_AHEAD];
#pragma unroll
        for (int a = 0; a < MOE_SORT_AHEAD; ++a) es[a] = expert_of(i0 + 32 * a + lane);
#pragma unroll
        for (int a = 0; a < MOE_SORT_AHEAD; ++a) {
            const unsigned mine = __ballot_sync(full, es[a] == expert);
            if (es[a] == expert) place[i0 + 32 * a + lane] = at + __popc(mine & before);
            at += __popc(mine);
        }
    }
}

extern "C" int qwb_moe_sort(const int* chosen, int* place, int* ends, int S, int E, cudaStream_t stream) {
    if (S <= 0) return 0;
    if (E <= 0 || E > QWB_MOE_MAX_EXPERTS) return qwb_fail(QWB_ERR_ARG, "moe_sort: %d experts (at most %d)", E, QWB_MOE_MAX_EXPERTS);
    qwb_launch(moe_sort_kernel, E, MOE_SORT_WARPS * 32, 0, stream, chosen, place, ends, S, E);
    return qwb_check_launch("moe_sort");
}

__global__ void moe_spread_kernel(const uint4* __restrict__ x, const int* __restrict__ place, uint4* __restrict__ xs, const float* __restrict__ weight,
                                  float* __restrict__ row_weight, int pieces, int top) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x;
    if (row_weight && (int)threadIdx.x < top) row_weight[place[(size_t)t * top + threadIdx.x]] = weight[(size_t)t * top + threadIdx.x];
    for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
        const uint4 v = x[(size_t)t * pieces + i];
        for (int k = 0; k < top; ++k) xs[(size_t)place[(size_t)t * top + k] * pieces + i] = v;
    }
}

// weight [T, top] and row_weight [T * top], or both null
extern "C" int qwb_moe_spread(const void* x, const int* place, void* xs, const float* weight, float* row_weight, int T, int D, int top,
                              cudaStream_t stream) {
    if (T <= 0 || D <= 0) return 0;
    if (D % 8) return qwb_fail(QWB_ERR_ARG, "moe_spread: rows of %d values", D);
    qwb_launch(moe_spread_kernel, T, D >= 2048 ? 256 : 128, 0, stream, (const uint4*)x, place, (uint4*)xs, weight, row_weight, D / 8, top);
    return qwb_check_launch("moe_spread");
}

__device__ __forceinline__ uint4 pack_bf16x8(const float* v) {
    uint4 o;
    uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&p);
    }
    return o;
}

// 8 values a thread and step, whatever row they are in; KIND: the activation code
template <int KIND>
__global__ void moe_act_kernel(const Vec16<bf16>* __restrict__ u, const float* __restrict__ row_weight, uint4* __restrict__ act, unsigned n, unsigned pieces) {
    pdl_wait();
    pdl_launch_dependents();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float a[8], b[8];
        const float w = row_weight ? row_weight[i / pieces] : 1.f;
        if (KIND == QWB_MOE_GATED) {
            const size_t gate = i + (size_t)(i / pieces) * pieces;          // row s: its gate pieces, then its up pieces
            u[gate].get(a);
            u[gate + pieces].get(b);
#pragma unroll
            for (int e = 0; e < 8; ++e) { const float g = a[e] * w; a[e] = g / (1.f + expf(-g)) * (b[e] * w); }
        } else {
            u[i].get(a);
#pragma unroll
            for (int e = 0; e < 8; ++e) a[e] = qwb_activate(a[e] * w, KIND);
        }
        act[i] = pack_bf16x8(a);
    }
}

// row_weight [S] or null
extern "C" int qwb_moe_act(const void* u, const float* row_weight, void* act, int S, int F, int kind, cudaStream_t stream) {
    if (S <= 0 || F <= 0) return 0;
    if (F % 8) return qwb_fail(QWB_ERR_ARG, "moe_act: rows of %d values", F);
    const long long n = (long long)S * (F / 8);
    if (n >= 1LL << 31) return qwb_fail(QWB_ERR_ARG, "moe_act: %d rows of %d values are too many for one launch", S, F);
    const int grid = (int)((n + 255) / 256 < 148 * 32 ? (n + 255) / 256 : 148 * 32);
#define QWB_MOE_ACT(KIND) \
    case KIND: qwb_launch(moe_act_kernel<KIND>, grid, 256, 0, stream, (const Vec16<bf16>*)u, row_weight, (uint4*)act, (unsigned)n, (unsigned)(F / 8)); break
    switch (kind) {
        QWB_MOE_ACT(0); QWB_MOE_ACT(1); QWB_MOE_ACT(2); QWB_MOE_ACT(3); QWB_MOE_ACT(5); QWB_MOE_ACT(QWB_MOE_GATED);
        default: return qwb_fail(QWB_ERR_ARG, "moe_act: unknown activation %d", kind);
    }
#undef QWB_MOE_ACT
    return qwb_check_launch("moe_act");
}

__global__ void moe_combine_kernel(const Vec16<bf16>* __restrict__ y, const int* __restrict__ place, const float* __restrict__ weight,
                                   const float* __restrict__ shared, const float* __restrict__ gate, float* out, int pieces, int top,
                                   int onto) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x;
    const float g = gate ? gate[t] : 1.f;
    for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
        float total[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) total[e] = 0.f;
#pragma unroll 4
        for (int k = 0; k < top; ++k) {
            float v[8];
            y[(size_t)place[(size_t)t * top + k] * pieces + i].get(v);
            const float w = weight ? weight[(size_t)t * top + k] : 1.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) total[e] += w * v[e];
        }
        float4* o = reinterpret_cast<float4*>(out) + ((size_t)t * pieces + i) * 2;
        const float4* sh = reinterpret_cast<const float4*>(shared) + ((size_t)t * pieces + i) * 2;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float4 r = make_float4(total[4 * j], total[4 * j + 1], total[4 * j + 2], total[4 * j + 3]);
            if (shared) { const float4 s = sh[j]; r.x += g * s.x; r.y += g * s.y; r.z += g * s.z; r.w += g * s.w; }
            if (onto) { const float4 s = o[j]; r.x += s.x; r.y += s.y; r.z += s.z; r.w += s.w; }
            o[j] = r;
        }
    }
}

// y [S, D] bfloat16; weight [T, top] (or null: 1); shared [T, D] float (or null) and gate [T] (or null: 1)
extern "C" int qwb_moe_combine(const void* y, const int* place, const float* weight, const float* shared, const float* gate, float* out,
                               int T, int D, int top, int onto, cudaStream_t stream) {
    if (T <= 0 || D <= 0) return 0;
    if (D % 8) return qwb_fail(QWB_ERR_ARG, "moe_combine: rows of %d values", D);
    qwb_launch(moe_combine_kernel, T, D >= 2048 ? 256 : 128, 0, stream, (const Vec16<bf16>*)y, place, weight, shared, gate, out, D / 8, top, onto);
    return qwb_check_launch("moe_combine");
}
