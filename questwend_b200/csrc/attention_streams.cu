// Prompt attention on the fifth-generation tensor cores (tcgen05), bfloat16, with TWO softmax streams a block that share the
// tiles of values (and, where they can, of keys) in shared memory.  Two uses:
//
//   latent_prefill_tc   attention of prompts that start a sequence, keys [unrotated part per head | rotated part shared by the
//                       heads] (qwb_latent_prefill_mma's contract).  The streams are 128 queries each of one head, the second
//                       behind the first; a tile of 64 keys serves both.
//   maps_prefill_tc     two score maps per head over the same values (qwb_maps_prefill_mma's contract with maps = 2).  The
//                       streams are the two maps of the same 128 (token, head of the group) rows; a tile's key rows hold both
//                       maps, its values serve both, and the difference, its norm and the gate are taken at the end.
//
// Per stream and tile: S = Q K^T into tensor memory (64 columns, two buffers), P = softmax by four warps, a thread a row, left as
// bfloat16 in tensor memory over the scores it came from, O += P V with P read from there, O in tensor memory (VD columns).  P is
// relative to the row's largest score so far, as with the mma.sync kernels: the largest probability is 1 and exact in bfloat16.  A
// reference that is moved only past 2^8 is faster (8,192 tokens 529 us where this takes 577, one latent prompt the same) but rounds
// the largest probability too: errors of 0.00213 and 0.00260 of the results in place of 0.00207 and 0.00252, more where few keys weigh.
// With two streams in one block the tensor cores work on one while the other is
// in its softmax, what two blocks an SM give attention_tc.cu, but the Q, K and V tiles of 192-value keys would not leave room for
// a second block (2 x 48 KB of Q, K and V in three stages: 216 KB), and K and V cross L2 once for 256 rows.  Every wait is bounded.
//
// Warps, in groups of four that have registers of their own (setmaxnreg): 0 loads, 1 and 2 issue a stream's products each, 4-7 and 8-11 are the
// streams' softmax warps, 12-15 multiply O by what a row's reference has moved: in most tiles some row of a warp's 32 moves it, and a
// softmax warp that did this itself waited for the product before, 780 to 1,830 of a tile's 3,000 cycles.  One warp for both streams'
// products spent 3,500 cycles a tile (65 to 80 a product, about 200 a wait, passed or not).  With capped scores the softmax's multiply-adds
// fill the schedulers and want the registers: there its warps move O themselves (8,192 tokens 673 us, with warps for it 760).  So they do for latent
// prompts, whose products of 192 values hide the wait: 4,096 tokens 85.2 us, with warps for it 87.2, 2,048 36.7 and 40.1, 32 of 64 18.0 and 19.0.  Two
// maps without a cap, the same: 4,096 154 and 140, 1,024 25.9 and 23.4, 32 of 64 12.7 and 13.1.
//
// Sizes that are no multiples of 64 are filled up by the TMA loads with zeros.  In the last tile, rows of V behind the last
// key that the block sees are overwritten with zeros before the product: they can belong to another sequence, and what stands
// there, infinite or not a number, must not meet a probability of 0.  Inside a sequence a value that is not finite does meet
// the zeros of the rows before it: up to 127 earlier tokens of a latent prompt (64-row tiles: 63) and 128 / (heads a group) - 1 of
// one with two maps.
//
// Bound by the issue of products of 64 keys and the softmax's chain, near each other.  16 heads: latent 128 + 64 / 128, one prompt of 4,096, with
// the mma.sync kernels 816 us, one issuing warp 108, now 85 (600 tokens 55 -> 15.3 -> 15.2); two maps of 64 over 4 key/value heads, values of 128,
// 8,192 tokens: 2,447 -> 583 -> 507 us (cap 50: 3,261 -> 696 -> 673), 2,048 tokens with a window of 1,024: 170 -> 51 -> 45 us.
#include "attention_tc.cuh"

#include <atomic>

#define AS_APART(maps, cap) ((maps) && !(cap))      // warps of their own move O
#define AS_THREADS(apart) ((apart) ? 512 : 384)
// Registers a thread of the loader's and issuers' warps, of the streams' softmax warps, of the warps that move O: as many in all as the block is
// launched with (128 a thread, all of an SM's), which is what setmaxnreg has to give.
#define AS_LAUNCH_REGS 128
#define AS_FEW_REGS 56
#define AS_SOFTMAX_REGS 184
#define AS_MOVE_REGS 88
static_assert(AS_FEW_REGS + 2 * AS_SOFTMAX_REGS + AS_MOVE_REGS == 4 * AS_LAUNCH_REGS, "four groups of 128 threads");
#define AS_MAX_STAGES 4
#define AS_SMEM (227 * 1024)

// A from tensor memory: a row a lane, two bfloat16 a column
__device__ __forceinline__ void as_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// as at_ld32 and at_st32, without their waits
__device__ __forceinline__ void as_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
}
__device__ __forceinline__ void as_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}
// VD sums of this lane's row times alpha
template <int VD>
__device__ __forceinline__ void as_rescale(uint32_t taddr, float alpha) {
#pragma unroll
    for (int c = 0; c < VD; c += 64) {                  // two loads and two stores on their way together
        uint32_t ov[2][32];
        as_ld32(taddr + c, ov[0]);
        as_ld32(taddr + c + 32, ov[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 64; ++e) ov[e / 32][e % 32] = __float_as_uint(__uint_as_float(ov[e / 32][e % 32]) * alpha);
        as_st32(taddr + c, ov[0]);
        as_st32(taddr + c + 32, ov[1]);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ uint64_t as_two(float lo, float hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ uint64_t as_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ uint64_t as_mul2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ float as_series(float v, float c0, float c1, float c2, float c3, float c4) {
    const float u = v * v;
    return fmaf(u, fmaf(u, fmaf(u, fmaf(u, c4, c3), c2), c1), c0);
}
// The largest of a row's 64 scores (ABS: of their sizes), in four chains: a chain of 64 would be the softmax's longest wait.
template <bool ABS>
__device__ __forceinline__ float as_max(const uint32_t (&sv)[2][32]) {
    float m[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) m[k] = ABS ? 0.f : -INFINITY;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
            const float a = __uint_as_float(sv[h][c]), b = __uint_as_float(sv[h][c + 1]);
            m[(c / 2) & 3] = fmaxf(m[(c / 2) & 3], ABS ? fmaxf(fabsf(a), fabsf(b)) : fmaxf(a, b));
        }
    return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}

// KA, VA: pieces of 64 values that a stream's keys and the values have.
template <int KA, int VA, bool MAPS>
struct AsSmem {
    static constexpr size_t Q_BYTES = (size_t)2 * KA * AT_ROWS * 128;                       // stream by stream, [128 rows][128 bytes] a piece
    static constexpr size_t K_BYTES = (size_t)(MAPS ? 2 : 1) * KA * AT_KEYS * 128;          // (map by map,) [64 keys][128 bytes] a piece
    static constexpr size_t V_BYTES = (size_t)VA * AT_KEYS * 128;
    static constexpr size_t MORE = 512 + 4 * AT_ROWS * sizeof(float);                       // barriers; factors of rows, see below
    static constexpr int FIT = (int)((AS_SMEM - MORE - Q_BYTES) / (K_BYTES + V_BYTES));
    static constexpr int STAGES = FIT < AS_MAX_STAGES ? FIT : AS_MAX_STAGES;
    static constexpr size_t TILES = Q_BYTES + STAGES * (K_BYTES + V_BYTES);
    static constexpr size_t BYTES = TILES + MORE;
    static_assert(STAGES >= 2, "the tiles do not fit");
};

struct AsArgs {
    const int *page_table, *cu_seqlens, *pos0;      // MAPS: the paged cache; else prompts that start at position 0
    bf16* out;
    int* error;
    const float *gate, *sink;                       // gate: rows of ld_gate floats, or null
    int ld_gate, H, Hkv, G, table_width, window, chunk, tok_per_block, vd;
    float scale, softcap, lambda, eps, out_scale;
    int norm_out, plain_pieces;                     // plain_pieces: of the keys' KA pieces, how many are the unrotated part's
};

template <int KA, int VA, bool MAPS, bool CAP>
__global__ void __launch_bounds__(AS_THREADS(AS_APART(MAPS, CAP)), 1)
attn_streams_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_q2, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_k2, const __grid_constant__ CUtensorMap map_v, const AsArgs p) {
    using Smem = AsSmem<KA, VA, MAPS>;
    constexpr int VD = 64 * VA, STAGES = Smem::STAGES;
    constexpr bool APART = AS_APART(MAPS, CAP);
    constexpr uint32_t K_BYTES = Smem::K_BYTES, V_BYTES = Smem::V_BYTES;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    if (at_smem(smem_raw) & 1023u) {                    // never seen; refuse rather than compute with a wrong layout
        if (threadIdx.x == 0) atomicExch(p.error, 7);
        return;
    }
    unsigned char* q_tile = smem_raw;
    unsigned char* k_tiles = q_tile + Smem::Q_BYTES;
    unsigned char* v_tiles = k_tiles + STAGES * K_BYTES;
    uint64_t* q_full = reinterpret_cast<uint64_t*>(smem_raw + Smem::TILES);
    uint64_t* k_full = q_full + 1;
    uint64_t* k_empty = k_full + STAGES;
    uint64_t* v_full = k_empty + STAGES;
    uint64_t* v_empty = v_full + STAGES;
    // [stream][tile & 1] each: a stream may be up to two tiles ahead of the tensor cores, and a barrier tells two phases apart
    uint64_t* s_full = v_empty + STAGES;
    uint64_t* p_full = s_full + 4;
    uint64_t* o_full = p_full + 4;
    uint64_t* a_full = o_full + 4;
    uint64_t* c_full = a_full + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(c_full + 4);
    // per stream two rows of 128: what a row's sums are multiplied by, of even and odd tiles; MAPS, in the end: factors and sums of squares
    float* swap = reinterpret_cast<float*>(smem_raw + Smem::TILES + 512);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.z;
    const int t0 = p.cu_seqlens[b], n_new = p.cu_seqlens[b + 1] - t0;
    // the blocks with the most keys first, of every head, as in attention_tc.cu
    const int q0 = (int)(gridDim.y - 1 - blockIdx.y) * p.tok_per_block;
    if (q0 >= n_new) return;
    const int p0 = MAPS ? p.pos0[b] : 0;
    // tiles of 64 keys that stream x sees: [first_tile + from(x), first_tile + to(x))
    int from_0 = 0, to_0 = 0, from_1 = 0, to_1 = 0, first_tile = 0, k_last = 0;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int tok0 = MAPS ? q0 : q0 + AT_ROWS * x, span = MAPS ? p.tok_per_block : AT_ROWS;
        const bool any = tok0 < n_new && (MAPS || tok0 < q0 + p.tok_per_block);
        const int last = p0 + min(n_new, tok0 + span) - 1, pos = p0 + tok0;
        int first = p.window > 0 ? max(0, pos - p.window + 1) : 0;
        if (MAPS && p.chunk > 0) first = max(first, (pos / p.chunk) * p.chunk);
        if (x == 0) first_tile = first / AT_KEYS;
        (x ? from_1 : from_0) = any ? first / AT_KEYS - first_tile : 0;
        (x ? to_1 : to_0) = any ? last / AT_KEYS + 1 - first_tile : 0;
        if (any) k_last = last;
    }
    const int n_tiles = max(to_0, to_1);
    auto from = [&](int x) { return x ? from_1 : from_0; };
    auto to = [&](int x) { return x ? to_1 : to_0; };
    const int* pages = MAPS ? p.page_table + (size_t)b * p.table_width : nullptr;

    if (threadIdx.x == 0) {
        at_bar_init(q_full, 1);
        for (int s = 0; s < STAGES; ++s) {
            at_bar_init(&k_full[s], 1); at_bar_init(&k_empty[s], 2);                   // both streams have read a tile
            at_bar_init(&v_full[s], 1); at_bar_init(&v_empty[s], 2);
        }
        for (int i = 0; i < 4; ++i) {
            at_bar_init(&s_full[i], 1); at_bar_init(&p_full[i], 4); at_bar_init(&o_full[i], 1);
            at_bar_init(&a_full[i], 4); at_bar_init(&c_full[i], 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    at_fence_before();
    __syncthreads();
    at_fence_after();
    const uint32_t tmem = *tmem_slot;                   // S of stream x: columns 128 x + {0, 64} ..; O of stream x: 256 + 128 x ..

    pdl_wait();
    pdl_launch_dependents();

    // what a warp does follows from its group of four, so that each group's registers are its own
    if (warp < 4) {
        if (APART) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AS_FEW_REGS));
    if (warp == 0) {
        if (lane == 0) {
            if (MAPS) {                                 // rows (token, head of the group): boxes of [128 / G tokens][G heads][1 map][64 d]
                at_expect_tx(q_full, (uint32_t)(2 * KA * p.tok_per_block * p.G * 128));
                for (int x = 0; x < 2; ++x)
                    for (int a = 0; a < KA; ++a)
                        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                                     ::"r"(at_smem(q_tile + (size_t)(x * KA + a) * AT_ROWS * 128)), "l"(&map_q), "r"(at_smem(q_full)), "r"(a * 64), "r"(x),
                                       "r"((int)blockIdx.x * p.G), "r"(t0 + q0) : "memory");
            } else {                                    // 128 tokens of one head a stream: the unrotated part, then the rotated one
                const int streams = to_1 > 0 ? 2 : 1;
                at_expect_tx(q_full, (uint32_t)(streams * KA * AT_ROWS * 128));
                for (int x = 0; x < streams; ++x)
                    for (int a = 0; a < KA; ++a) {
                        const bool rot = a >= p.plain_pieces;
                        at_tma_3d(q_tile + (size_t)(x * KA + a) * AT_ROWS * 128, rot ? &map_q2 : &map_q, q_full, (rot ? a - p.plain_pieces : a) * 64,
                                  (int)blockIdx.x, t0 + q0 + AT_ROWS * x);
                    }
            }
            bool ok = true;
            int k_issued = 0, v_issued = 0;
            auto load = [&](int j, bool is_k) -> bool {
                const int s = j % STAGES;
                uint64_t* empty = is_k ? &k_empty[s] : &v_empty[s];
                uint64_t* full = is_k ? &k_full[s] : &v_full[s];
                if (j >= STAGES && !at_wait(empty, ((j / STAGES) - 1) & 1)) return false;
                const uint32_t bytes = is_k ? K_BYTES : V_BYTES;
                unsigned char* dst = (is_k ? k_tiles : v_tiles) + (size_t)s * bytes;
                at_expect_tx(full, bytes);
                if (MAPS) {
                    const int row0 = (pages[first_tile + j] * p.Hkv + (int)blockIdx.x) * AT_KEYS;      // the (page, head) block's first row
                    if (is_k) {
                        for (int x = 0; x < 2; ++x)
                            for (int a = 0; a < KA; ++a) at_tma_3d(dst + (size_t)(x * KA + a) * AT_KEYS * 128, &map_k, full, a * 64, x, row0);
                    } else {
                        for (int a = 0; a < VA; ++a) at_tma_2d(dst + (size_t)a * AT_KEYS * 128, &map_v, full, a * 64, row0);
                    }
                } else {
                    const int key = t0 + (first_tile + j) * AT_KEYS;
                    if (is_k) {
                        for (int a = 0; a < KA; ++a) {
                            if (a < p.plain_pieces) at_tma_3d(dst + (size_t)a * AT_KEYS * 128, &map_k, full, a * 64, (int)blockIdx.x, key);
                            else at_tma_2d(dst + (size_t)a * AT_KEYS * 128, &map_k2, full, (a - p.plain_pieces) * 64, key);
                        }
                    } else {
                        for (int a = 0; a < VA; ++a) at_tma_3d(dst + (size_t)a * AT_KEYS * 128, &map_v, full, a * 64, (int)blockIdx.x, key);
                    }
                }
                if (is_k) k_issued = j + 1; else v_issued = j + 1;
                return true;
            };
            ok = load(0, true);
            for (int j = 0; j < n_tiles && ok; ++j) {
                if (j + 1 < n_tiles) ok = load(j + 1, true);
                if (ok) ok = load(j, false);
            }
            if (!ok) {
                atomicExch(p.error, 1);
                // copies already issued still write shared memory: wait for them (bounded) before the block ends
                at_wait(q_full, 0);
                for (int j = max(0, k_issued - STAGES); j < k_issued; ++j) at_wait(&k_full[j % STAGES], (j / STAGES) & 1);
                for (int j = max(0, v_issued - STAGES); j < v_issued; ++j) at_wait(&v_full[j % STAGES], (j / STAGES) & 1);
            }
        }
    } else if (warp == 1 || warp == 2) {                // a stream's products: all lanes wait, one issues
        constexpr uint32_t idesc_s = at_idesc(AT_ROWS, AT_KEYS, false), idesc_o = at_idesc(AT_ROWS, VD, true);
        const int x = warp - 1;
        auto all = [](bool ok) -> bool { return __all_sync(0xffffffffu, ok); };
        bool ok = all(at_wait(q_full, 0));
        auto active = [&](int j) { return j >= from(x) && j < to(x); };
        // S for tile j, two tiles ahead of its product with V: the buffer's last scores were read, and its P used by a product issued
        // before.  A tile that the stream does not see is waited for all the same, so that it is given back in its turn.
        auto issue_s = [&](int j) -> bool {
            const int i = j - from(x), s = j % STAGES;
            if (!all(at_wait(&k_full[s], (j / STAGES) & 1))) return false;
            at_fence_after();
            if (at_elect()) {
                if (active(j)) {
                    const unsigned char* qt = q_tile + (size_t)x * KA * AT_ROWS * 128;
                    const unsigned char* kt = k_tiles + (size_t)s * K_BYTES + (MAPS ? (size_t)x * KA * AT_KEYS * 128 : 0);
#pragma unroll
                    for (int k = 0; k < 4 * KA; ++k) {
                        const uint64_t da = at_desc_kmajor(qt + (size_t)(k / 4) * AT_ROWS * 128) + 2 * (k % 4);
                        const uint64_t db = at_desc_kmajor(kt + (size_t)(k / 4) * AT_KEYS * 128) + 2 * (k % 4);
                        at_mma(tmem + 128 * x + 64 * (i & 1), da, db, idesc_s, k > 0 ? 1u : 0u);
                    }
                    at_commit(&s_full[2 * x + (i & 1)]);
                    at_commit(&k_empty[s]);
                } else {
                    at_arrive(&k_empty[s]);
                }
            }
            __syncwarp();
            return true;
        };
        for (int j = 0; j < 2 && j < n_tiles && ok; ++j) ok = issue_s(j);
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int s = j % STAGES, i = j - from(x);
            unsigned char* vt = v_tiles + (size_t)s * V_BYTES;
            ok = all(at_wait(&v_full[s], (j / STAGES) & 1));
            if (!ok) break;
            if (active(j)) {
                const int kept = k_last + 1 - (first_tile + j) * AT_KEYS;
                if (kept < AT_KEYS) {                   // the last tile: rows behind the last key (both streams' warps write the same)
                    for (int e = lane; e < (AT_KEYS - kept) * VA * 8; e += 32) {
                        const int r = kept + e / (VA * 8), c = e % (VA * 8);
                        *reinterpret_cast<uint4*>(vt + (size_t)(c / 8) * AT_KEYS * 128 + r * 128 + (c % 8) * 16) = make_uint4(0, 0, 0, 0);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                }
                ok = all(at_wait(&p_full[2 * x + (i & 1)], (i >> 1) & 1) && (!APART || at_wait(&c_full[2 * x + (i & 1)], (i >> 1) & 1)));
                if (!ok) break;
                at_fence_after();
            }
            if (at_elect()) {
                if (active(j)) {
#pragma unroll
                    for (int k = 0; k < AT_KEYS / 16; ++k) {
                        const uint64_t db = at_desc_mnmajor(vt + (size_t)k * 16 * 128, AT_KEYS * 128);
                        as_mma_ts(tmem + 256 + 128 * x, tmem + 128 * x + 64 * (i & 1) + 8 * k, db, idesc_o, (i > 0 || k > 0) ? 1u : 0u);
                    }
                    at_commit(&o_full[2 * x + (i & 1)]);
                    at_commit(&v_empty[s]);
                } else {
                    at_arrive(&v_empty[s]);
                }
            }
            __syncwarp();
            if (j + 2 < n_tiles) ok = issue_s(j + 2);
        }
        if (!ok && at_elect()) {
            atomicExch(p.error, 2);
            for (int i = 2 * x; i < 2 * x + 2; ++i) { at_commit(&s_full[i]); at_commit(&o_full[i]); }
        }
    }
    } else if (APART && warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AS_MOVE_REGS));
        // O of both streams relative to the rows' new references, while the softmax warps go on
        const int lane_group = warp & 3, r = 32 * lane_group + lane;
        const uint32_t lane_off = (uint32_t)(32 * lane_group) << 16;
        bool ok = true;
        for (int j = 0; j < n_tiles && ok; ++j) {       // in the order in which the products are issued
#pragma unroll
            for (int x = 0; x < 2 && ok; ++x) {
                if (j < from(x) || j >= to(x)) continue;
                const int i = j - from(x), at = 2 * x + (i & 1);
                ok = at_wait(&a_full[at], (i >> 1) & 1);
                if (!ok) break;
                const float alpha = swap[at * AT_ROWS + r];
                if (i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                    ok = at_wait(&o_full[at ^ 1], ((i - 1) >> 1) & 1);      // what the products before have written
                    at_fence_after();
                    if (!ok) break;
                    as_rescale<VD>(tmem + 256 + 128 * x + lane_off, alpha);
                }
                at_fence_before();
                __syncwarp();
                if (lane == 0) at_arrive(&c_full[at]);
            }
        }
        if (!ok && lane == 0) atomicExch(p.error, 4);
    } else {
        if (APART) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AS_SOFTMAX_REGS));
        const int x = (warp - 4) >> 2, lane_group = warp & 3;
        const int r = 32 * lane_group + lane;                                          // this thread's row = tensor-memory lane
        const int tok = MAPS ? q0 + r / p.G : q0 + AT_ROWS * x + r, head = MAPS ? (int)blockIdx.x * p.G + r % p.G : (int)blockIdx.x;
        const bool row_ok = to(x) > 0 && tok < n_new && (!MAPS || r < p.tok_per_block * p.G);
        const int qp = row_ok ? p0 + tok : -1;
        const uint32_t lane_off = (uint32_t)(32 * lane_group) << 16;
        const uint32_t tmem_s = tmem + 128 * x, tmem_o = tmem + 256 + 128 * x;
        const float log2e = 1.4426950408889634f;
        // what turns a score (raw, or in units of log 2 when capped) into the exponent's argument, and the caps' factors
        const float sl2 = CAP ? 1.f : p.scale * log2e;
        const float to_t = CAP ? p.scale / p.softcap : 0.f, cap2 = p.softcap * log2e;
        // While every |t| of a tile is small, as capped scores mostly are, cap tanh(t), t = score / cap, is formed by its odd
        // series to t^9 (the next term is below 2^-24 of the value at 0.3), on raw scores as v (c0 + v^2 (c1 + ..)): packed
        // multiply-adds, where the form by ex2 and rcp keeps the special-function unit, which the probabilities need too,
        // busy for three turns a score.  One sequence of 8,192 tokens, 16 heads of 2 x 64, cap 50:
        // 795 us with it (P still in shared memory), 1,063 by ex2 and rcp alone.
        const float poly_up_to = CAP ? 0.3f / fabsf(to_t) : 0.f, tt = to_t * to_t;
        const float c0 = cap2 * to_t, c1 = c0 * tt * (-1.f / 3.f), c2 = c0 * tt * tt * (2.f / 15.f), c3 = c0 * tt * tt * tt * (-17.f / 315.f),
                    c4 = c0 * tt * tt * tt * tt * (62.f / 2835.f);
        int own = p.window > 0 ? max(0, qp - p.window + 1) : 0;                         // the first key that the row sees
        if (MAPS && p.chunk > 0 && qp >= 0) own = max(own, (qp / p.chunk) * p.chunk);
        float m_ref = -INFINITY, l = 0.f;
        bool ok = true;
        const int n_mine = to(x) - from(x);
        for (int i = 0; i < n_mine; ++i) {
            ok = at_wait(&s_full[2 * x + (i & 1)], (i >> 1) & 1);
            at_fence_after();
            if (!ok) { if (lane == 0) atomicExch(p.error, 3); break; }
            const int key0 = (first_tile + from(x) + i) * AT_KEYS;
            uint32_t sv[2][32];
            at_ld32(tmem_s + (i & 1) * 64 + lane_off, sv[0]);
            at_ld32(tmem_s + (i & 1) * 64 + lane_off + 32, sv[1]);
            const bool all_visible = key0 + AT_KEYS - 1 <= qp && key0 >= own;           // no mask needed
            float mx = -INFINITY;
            bool series = false;
            // in tiles that are not wholly visible the row sees the keys [lo, lo + span): one subtraction and one comparison a key
            const int lo = max(own - key0, 0), span = max(min(qp - key0 + 1, AT_KEYS) - lo, 0);
            auto mask = [&](uint32_t with) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if ((unsigned)(32 * h + c - lo) >= (unsigned)span) sv[h][c] = with;
            };
            if (CAP) {
                // which form the scores take follows from visible keys alone: behind them stand later tokens, and what an earlier
                // user of the page left there
                if (!all_visible) mask(0u);
                const float most = as_max<true>(sv);
                if (all_visible && most <= poly_up_to) {        // the series below, formed together with the exponent's argument
                    series = true;
                    mx = as_max<false>(sv);
                    mx *= as_series(mx, c0, c1, c2, c3, c4);
                } else if (most <= poly_up_to) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int c = 0; c < 32; ++c) {
                            const float raw = __uint_as_float(sv[h][c]);
                            sv[h][c] = __float_as_uint(raw * as_series(raw, c0, c1, c2, c3, c4));
                        }
                } else {
                    const float mul = 2.f * log2e * to_t;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int c = 0; c < 32; ++c) {
                            float rcp;
                            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rcp) : "f"(at_exp2(__uint_as_float(sv[h][c]) * mul) + 1.f));
                            sv[h][c] = __float_as_uint(fmaf(-2.f * cap2, rcp, cap2));
                        }
                }
            }
            if (!all_visible) mask(0xff800000u);                                       // -inf
            if (!series) mx = as_max<false>(sv);
            const bool rescale = mx > m_ref;
            const float m_new = rescale ? mx : m_ref;
            const float alpha = rescale ? at_exp2((m_ref - m_new) * sl2) : 1.f;        // m_ref = -inf gives 0
            const float base = m_new == -INFINITY ? 0.f : m_new * sl2;
            m_ref = m_new;
            if (APART) {                                                                // read before the tile after the next has scores
                swap[(2 * x + (i & 1)) * AT_ROWS + r] = alpha;
                __syncwarp();
                if (lane == 0) at_arrive(&a_full[2 * x + (i & 1)]);
            }
            uint32_t pk[32];                                                            // two keys' probabilities each
            float sum[4] = {l * alpha, 0.f, 0.f, 0.f};
            auto probabilities = [&](auto argument) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < 32; c += 2) {
                        float a0, a1;
                        argument(sv[h][c], sv[h][c + 1], a0, a1);
                        const float p0v = at_exp2(a0), p1v = at_exp2(a1);
                        sum[(c / 2) & 3] += p0v + p1v;
                        __nv_bfloat162 v = __floats2bfloat162_rn(p0v, p1v);
                        pk[16 * h + c / 2] = *reinterpret_cast<uint32_t*>(&v);
                    }
            };
            if (CAP && series) {
                const uint64_t k0 = as_two(c0, c0), k1 = as_two(c1, c1), k2 = as_two(c2, c2), k3 = as_two(c3, c3), k4 = as_two(c4, c4), off = as_two(-base, -base);
                probabilities([&](uint32_t x0, uint32_t x1, float& a0, float& a1) {
                    const uint64_t v = as_two(__uint_as_float(x0), __uint_as_float(x1)), u = as_mul2(v, v);
                    const uint64_t a = as_fma2(v, as_fma2(u, as_fma2(u, as_fma2(u, as_fma2(u, k4, k3), k2), k1), k0), off);
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(a));
                });
            } else {
                probabilities([&](uint32_t x0, uint32_t x1, float& a0, float& a1) {
                    a0 = fmaf(__uint_as_float(x0), sl2, -base);
                    a1 = fmaf(__uint_as_float(x1), sl2, -base);
                });
            }
            l = (sum[0] + sum[1]) + (sum[2] + sum[3]);
            if (!APART && i > 0 && __any_sync(0xffffffffu, rescale)) {                  // a row of this warp moves its reference: rescale O,
                ok = at_wait(&o_full[2 * x + ((i - 1) & 1)], ((i - 1) >> 1) & 1);       // which the product before this one has written
                at_fence_after();
                if (!ok) { if (lane == 0) atomicExch(p.error, 4); break; }
                as_rescale<VD>(tmem_o + lane_off, alpha);
            }
            at_st32(tmem_s + (i & 1) * 64 + lane_off, pk);                              // P over the scores it came from
            at_fence_before();
            __syncwarp();
            if (lane == 0) at_arrive(&p_full[2 * x + (i & 1)]);
        }
        if (ok && n_mine > 0) {
            ok = at_wait(&o_full[2 * x + ((n_mine - 1) & 1)], ((n_mine - 1) >> 1) & 1);
            at_fence_after();
            if (!ok && lane == 0) atomicExch(p.error, 5);
        }
        const float gate = p.gate && row_ok ? 1.f / (1.f + expf(-p.gate[(size_t)(t0 + tok) * p.ld_gate + head])) : 1.f;
        bf16* dst = p.out + ((size_t)(t0 + tok) * p.H + head) * p.vd;
        auto store32 = [&](const float* v, int c0) {                                    // 32 values from column c0 on
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
                uint32_t w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    __nv_bfloat162 two = __floats2bfloat162_rn(v[e + 2 * u], v[e + 2 * u + 1]);
                    w[u] = *reinterpret_cast<uint32_t*>(&two);
                }
                if (row_ok && c0 + e < p.vd) *reinterpret_cast<uint4*>(dst + c0 + e) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        };
        if (!MAPS) {
            if (ok && n_mine > 0) {
                // a sink: one more term of the denominator, exp(sink), relative to the row's reference
                if (p.sink && row_ok) l += at_exp2(p.sink[head] * log2e - (m_ref == -INFINITY ? 0.f : m_ref * sl2));
                const float inv = (l > 0.f ? 1.f / l : 0.f) * gate;
#pragma unroll 1
                for (int c = 0; c < VD; c += 32) {
                    uint32_t ov[32];
                    at_ld32(tmem_o + lane_off + c, ov);
                    float v[32];
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(ov[e]) * inv;
                    store32(v, c);
                }
            }
        } else {
            // both streams' threads of a row form half of the difference's columns each; every thread passes both barriers
            swap[2 * x * AT_ROWS + r] = (l > 0.f ? 1.f / l : 0.f) * (x ? p.lambda : 1.f);
            at_fence_before();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            at_fence_after();
            const float f0 = swap[r], f1 = swap[2 * AT_ROWS + r];
            float v[VA][32], squares = 0.f;
#pragma unroll
            for (int a = 0; a < VA; ++a) {
                const uint32_t col = 32 * (VA * x + a);
                uint32_t o0[32], o1[32];
                at_ld32(tmem + 256 + lane_off + col, o0);
                at_ld32(tmem + 384 + lane_off + col, o1);
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    v[a][e] = __uint_as_float(o0[e]) * f0 - __uint_as_float(o1[e]) * f1;
                    squares += v[a][e] * v[a][e];
                }
            }
            swap[(2 * x + 1) * AT_ROWS + r] = squares;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const float total = swap[AT_ROWS + r] + swap[3 * AT_ROWS + r];
            const float mul = (p.norm_out ? rsqrtf(total / (float)p.vd + p.eps) * p.out_scale : 1.f) * gate;
            if (ok) {
#pragma unroll
                for (int a = 0; a < VA; ++a) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[a][e] *= mul;
                    store32(v[a], 32 * (VA * x + a));
                }
            }
        }
    }
    at_fence_before();
    __syncthreads();
    if (warp == 1) {
        at_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------------------------------- host side
// a bfloat16 tensor of `rank` dimensions (innermost first; strides in bytes from the second one on), boxes of 128 swizzled bytes
static int as_map(const char* what, CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
    AtEncodeFn enc = at_encode();
    if (!enc) return qwb_fail(QWB_ERR_CUDA, "%s: cuTensorMapEncodeTiled is not available from this driver", what);
    cuuint32_t elem[4] = {1, 1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : qwb_fail(QWB_ERR_CUDA, "%s: cuTensorMapEncodeTiled failed with %d", what, (int)r);
}

// Whether the uncapped kernel for two maps was built with the registers that its warps share out among themselves (else they would wait for some that
// there are not): 1, 0, or -1 where that cannot be found out now.
template <int KA, int VA>
static int as_built() {
    static std::atomic<int> regs{0};
    if (regs == 0) {
        cudaFuncAttributes f;
        if (cudaFuncGetAttributes(&f, attn_streams_kernel<KA, VA, true, false>) != cudaSuccess) return -1;
        regs = f.numRegs;
    }
    return regs == AS_LAUNCH_REGS;
}

template <int KA, int VA, bool MAPS, bool CAP>
static int as_launch(const char* what, dim3 grid, const CUtensorMap* maps, const AsArgs& args, cudaStream_t stream) {
    constexpr size_t smem = AsSmem<KA, VA, MAPS>::BYTES;
    auto kernel = attn_streams_kernel<KA, VA, MAPS, CAP>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return qwb_fail(QWB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    if constexpr (AS_APART(MAPS, CAP))
        if (as_built<KA, VA>() != 1) return qwb_fail(QWB_ERR_CUDA, "%s: not built with %d registers a thread", what, AS_LAUNCH_REGS);
    e = qwb_launch(kernel, grid, AS_THREADS(AS_APART(MAPS, CAP)), smem, stream, maps[0], maps[1], maps[2], maps[3], maps[4], args);
    if (e != cudaSuccess) return qwb_fail(QWB_ERR_CUDA, "%s: launch failed: %s", what, cudaGetErrorString(e));
    return qwb_check_launch(what);
}

static int as_pieces(int n) { return (n + 63) / 64; }

// Whether uncapped prompts with two maps of these sizes may take this kernel as it was built; where they may not, the caller takes another one.
extern "C" int qwb_streams_built(int key_pieces, int value_pieces) {
    switch (10 * key_pieces + value_pieces) {
        case 11: return as_built<1, 1>() != 0;
        case 12: return as_built<1, 2>() != 0;
        case 21: return as_built<2, 1>() != 0;
        case 22: return as_built<2, 2>() != 0;
    }
    return 0;
}

static bool as_latent_fits(int K, int R, int DV) {
    return K > 0 && R >= 0 && DV > 0 && K % 8 == 0 && R % 8 == 0 && (K + R) % 16 == 0 && DV % 8 == 0 && DV <= 128 && as_pieces(K) + as_pieces(R) <= 3;
}

// Prompts that start their sequences: q [T, H, K + R], k_plain [T, H, K], R rotated values at kr + t * ld_kr, v [T, H, DV], out
// [T, H * DV], all bfloat16; sink [H] or null, gate: rows of ld_gate floats or null; `error` as for qwb_gemm_tc.
extern "C" int qwb_latent_prefill_tc(const void* q, const void* k_plain, const void* kr, int ld_kr, const void* v, const int* cu_seqlens,
                                     const float* sink, void* out, int B, int T, int max_new, int H, int K, int R, int DV, float scale,
                                     int window, const float* gate, int ld_gate, int* error, cudaStream_t stream) {
    if (B <= 0 || max_new <= 0 || T <= 0) return 0;
    if (H <= 0 || !as_latent_fits(K, R, DV) || ld_kr % 8 || ld_kr < R || !error || window < 0 || !(scale > 0.f) || (gate && ld_gate < H))
        return qwb_fail(QWB_ERR_ARG, "latent_prefill_tc: heads %d of %d + %d and %d values: multiples of 8, up to three pieces of 64 query values, up to 128 "
                        "values, a positive scale", H, K, R, DV);
    const int tok_per_block = (long long)H * B * ((max_new + 255) / 256) >= 148 ? 256 : 128;        // few blocks: one stream each, twice as many
    if (B > 65535 || (max_new + tok_per_block - 1) / tok_per_block > 65535)
        return qwb_fail(QWB_ERR_ARG, "latent_prefill_tc: batch %d or %d new tokens of a sequence are more than the grid takes", B, max_new);
    for (const void* x : {q, k_plain, kr, v, (const void*)out})
        if ((uintptr_t)x % 16) return qwb_fail(QWB_ERR_ARG, "latent_prefill_tc: a tensor is not 16-byte aligned");
    const int DQ = K + R;
    CUtensorMap maps[5];
    const char* what = "latent_prefill_tc";
    auto heads3 = [&](CUtensorMap* m, const void* base, int size, int row, int box_rows) {         // [T][H][row], `size` values of each
        const cuuint64_t dims[3] = {(cuuint64_t)size, (cuuint64_t)H, (cuuint64_t)T}, strides[2] = {(cuuint64_t)row * 2, (cuuint64_t)H * row * 2};
        const cuuint32_t box[3] = {64, 1, (cuuint32_t)box_rows};
        return as_map(what, m, base, 3, dims, strides, box);
    };
    if (int rc = heads3(&maps[0], q, K, DQ, AT_ROWS)) return rc;
    if (int rc = heads3(&maps[2], k_plain, K, K, AT_KEYS)) return rc;
    if (int rc = heads3(&maps[4], v, DV, DV, AT_KEYS)) return rc;
    maps[1] = maps[0]; maps[3] = maps[2];
    if (R > 0) {
        if (int rc = heads3(&maps[1], (const bf16*)q + K, R, DQ, AT_ROWS)) return rc;
        const cuuint64_t dims[2] = {(cuuint64_t)R, (cuuint64_t)T}, strides[1] = {(cuuint64_t)ld_kr * 2};
        const cuuint32_t box[2] = {64, AT_KEYS};
        if (int rc = as_map(what, &maps[3], kr, 2, dims, strides, box)) return rc;
    }
    AsArgs a = {};
    a.cu_seqlens = cu_seqlens; a.out = (bf16*)out; a.error = error; a.gate = gate; a.sink = sink; a.ld_gate = ld_gate; a.H = H; a.G = 1; a.Hkv = H;
    a.window = window; a.tok_per_block = tok_per_block; a.vd = DV; a.scale = scale; a.plain_pieces = as_pieces(K);
    const dim3 grid(H, (max_new + tok_per_block - 1) / tok_per_block, B);
    const int pieces = as_pieces(K) + as_pieces(R);
#define QWB_AS(KA) return DV <= 64 ? as_launch<KA, 1, false, false>(what, grid, maps, a, stream) : as_launch<KA, 2, false, false>(what, grid, maps, a, stream)
    if (pieces == 1) QWB_AS(1);
    if (pieces == 2) QWB_AS(2);
    QWB_AS(3);
#undef QWB_AS
}

static bool as_maps_fits(int dim, int vdim, int group) {
    return dim > 0 && vdim > 0 && dim % 8 == 0 && vdim % 8 == 0 && dim <= 128 && vdim <= 128 && group >= 1 && group <= AT_ROWS / 2;
}

// Two maps per head: q [T, H, 2, dim], pools [n_pages, Hkv, 64, 2 * dim] and [n_pages, Hkv, 64, vdim], out [T, H * vdim]; the rest as
// for qwb_maps_prefill_mma.
extern "C" int qwb_maps_prefill_tc(const void* q, const void* k_pool, const void* v_pool, const int* page_table, const int* cu_seqlens, const int* pos0,
                                   void* out, int B, int T, int max_new, int n_pages, int H, int Hkv, int dim, int vdim, int table_width, float scale,
                                   float softcap, int chunk, int window, float lambda, int norm_out, float eps, float out_scale, const float* gate,
                                   int ld_gate, int* error, cudaStream_t stream) {
    if (B <= 0 || max_new <= 0 || T <= 0) return 0;
    if (H <= 0 || Hkv <= 0 || H % Hkv || !as_maps_fits(dim, vdim, H / Hkv) || table_width <= 0 || n_pages <= 0 || !error || chunk < 0 || window < 0 ||
        !(scale > 0.f) || (gate && ld_gate < H))
        return qwb_fail(QWB_ERR_ARG, "maps_prefill_tc: %d heads over %d, keys of 2 x %d, values of %d: multiples of 8 up to 128, up to %d heads a group, a "
                        "positive scale", H, Hkv, dim, vdim, AT_ROWS / 2);
    for (const void* x : {q, k_pool, v_pool, (const void*)out})
        if ((uintptr_t)x % 16) return qwb_fail(QWB_ERR_ARG, "maps_prefill_tc: a tensor is not 16-byte aligned");
    const int G = H / Hkv, tok_per_block = AT_ROWS / G;
    if (B > 65535 || (max_new + tok_per_block - 1) / tok_per_block > 65535)
        return qwb_fail(QWB_ERR_ARG, "maps_prefill_tc: batch %d or %d new tokens of a sequence are more than the grid takes", B, max_new);
    CUtensorMap maps[5];
    const char* what = "maps_prefill_tc";
    {
        const cuuint64_t dims[4] = {(cuuint64_t)dim, 2, (cuuint64_t)H, (cuuint64_t)T};
        const cuuint64_t strides[3] = {(cuuint64_t)dim * 2, (cuuint64_t)dim * 4, (cuuint64_t)H * dim * 4};
        const cuuint32_t box[4] = {64, 1, (cuuint32_t)G, (cuuint32_t)tok_per_block};
        if (int rc = as_map(what, &maps[0], q, 4, dims, strides, box)) return rc;
    }
    {
        const cuuint64_t dims[3] = {(cuuint64_t)dim, 2, (cuuint64_t)n_pages * Hkv * AT_KEYS}, strides[2] = {(cuuint64_t)dim * 2, (cuuint64_t)dim * 4};
        const cuuint32_t box[3] = {64, 1, AT_KEYS};
        if (int rc = as_map(what, &maps[2], k_pool, 3, dims, strides, box)) return rc;
    }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)vdim, (cuuint64_t)n_pages * Hkv * AT_KEYS}, strides[1] = {(cuuint64_t)vdim * 2};
        const cuuint32_t box[2] = {64, AT_KEYS};
        if (int rc = as_map(what, &maps[4], v_pool, 2, dims, strides, box)) return rc;
    }
    maps[1] = maps[0]; maps[3] = maps[2];
    AsArgs a = {};
    a.page_table = page_table; a.cu_seqlens = cu_seqlens; a.pos0 = pos0; a.out = (bf16*)out; a.error = error; a.gate = gate; a.ld_gate = ld_gate;
    a.H = H; a.Hkv = Hkv; a.G = G; a.table_width = table_width; a.window = window; a.chunk = chunk; a.tok_per_block = tok_per_block; a.vd = vdim;
    a.scale = scale; a.softcap = softcap; a.lambda = lambda; a.eps = eps; a.out_scale = out_scale; a.norm_out = norm_out;
    const dim3 grid(Hkv, (max_new + tok_per_block - 1) / tok_per_block, B);
#define QWB_AS(KA, VA) return softcap > 0.f ? as_launch<KA, VA, true, true>(what, grid, maps, a, stream) : as_launch<KA, VA, true, false>(what, grid, maps, a, stream)
    if (dim <= 64) {
        if (vdim <= 64) QWB_AS(1, 1);
        QWB_AS(1, 2);
    }
    if (vdim <= 64) QWB_AS(2, 1);
    QWB_AS(2, 2);
#undef QWB_AS
}
