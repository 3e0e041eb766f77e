// Matrix products of float32 operands on the tensor cores, to float32's accuracy:
//
//     C[token, feature] (+)= scale (sum_k X[token, k] * W[feature, k] (+ bias))
//
// A float32 number is the sum of three bfloat16 numbers (hi: the number rounded to nearest; mid: what is left, rounded; lo: the rest, at most
// seven bits), and a product of two bfloat16 numbers is exact in float32.  Of the nine products of the parts the six largest are summed; the
// three left out (mid lo, lo mid, lo lo) are together at most 2^-24 (1 + 2^-10) of the product, of either sign.  What else decides the
// accuracy is the sum, and tensor memory's adds truncate.  So a tensor-memory accumulator only ever holds 32 products a term (one block
// of K): one the products of the leading parts, 16 bits each, another the five smaller terms; and the blocks are added up in registers with
// ordinary rounded float32 additions, in the order of K.  Measured against 64 bits, relative error of the result, this and the FMA pipe's
// chain of K fused multiply-adds: normal operands, K 132 7.3e-8 and 2.0e-7, K 2,048 2.1e-7 and 8.1e-7, K 5,632 3.4e-7 and 1.4e-6; 2,048
// products of one sign 1.8e-7 and 7.0e-7, with the low 15 bits of every operand set 1.8e-7 and 4.5e-6; rows with a single entry
// 2.6e-8 and 2.5e-8, at most 1.7 x 2^-24 and 2^-24.  (The parts cut off instead of rounded, as they were, lose up to 2^-21 of a product,
// always towards zero: single entries 1.0e-7, at most 9.7 x 2^-24.  mid lo and lo mid summed as well: single entries as the chain, but 1 row x
// 2,048 x 2,048 36.7 us instead of 31.5.)
//
// A result's operations depend on its own row of X, its row of W and K alone: not on the other rows of the launch, the tile
// sizes or the tile's place.  So a token's row has the same bits in a prompt's step and in a step of its own.
//
// Not every number is the sum of three such parts: not one that is infinite, or not a number, or so large that its first part would be
// infinite (from 2^128 - 2^119 on), or so small that its last one lies below the smallest bfloat16 (below 2^-110).  The splitting
// threads notice that a tile has one; the warps that add up then look for its rows of X and W, whose results, and no others, are summed on the
// FMA pipe instead, one chain over K as gemm_simt.cu has it.  So is a result that is not finite (a part's product may overflow where the
// product itself does not) or below 2^-100 (whose smaller parts' products are too small for float32).
//
// One block a tile of `feat_tile` (up to 128) features x N tokens; the weights are the rows of the product.  One thread sends for
// the float32 tiles (TMA) into a ring as deep as shared memory allows; groups of eight warps, a group every G-th block of K, split W into its
// parts and put them in tensor memory, from where the products read them: a product of 128 rows and n tokens takes 12 + n / 2 clocks so,
// 44 + n / 2 with W in shared memory (measured alone, back to back).  X goes to shared memory in its parts, split by the same warps or, for
// tiles of 64 tokens and more, once for all tiles by split_rows_kernel.  Two warps issue the products, every other one each, since one's round
// of waits, products and commits lasted longer than the products themselves; the last warps add the accumulators up, two sums an instruction,
// and store.  Blocks stay, one an SM, and every role runs across tile boundaries.  What bounds it: with few tokens the chain that a
// block of 32 of K goes through, 0.37 us with 16 tokens (splitting 0.13, the loads alone 0.2) whether 16 or 32 blocks share the features, the products
// and the adding up with many (0.84 us with 128 tokens, 0.5 of them the products).  Rows x features x K, us, cold weights; gemm_simt.cu, then W's parts
// in shared memory with one issuing warp, then a tile a block, then now: 8 x 2,048 x 2,048 190, 39, 34 and 37; 264 x 6,144 x 2,048 327, 111, 75 and 70;
// 1,777 x 6,144 x 2,048 1,817, 366, 314 and 284; the last three of 60 groups of 1,408 gated features, 17 tokens each 380, 340 and 304, 118 each
// 750, 650 and 610.
// Built and taken out: two blocks an SM with few tokens (60 groups of 17 tokens 333 us instead of 343, one of 24 groups the same); splitting warps
// that leave rows past a tile's features out (tiles of 64 features took what tiles of 128 take, 264 x 2,048 x 2,048 45 us instead of 41).  (With the
// float32 operands loaded into registers instead of by TMA 1,777 x 6,144 took 815: one load's latency a block lay bare.  Three loading
// threads instead of one changed nothing.)
// Grouped form as in gemm_simt.cu, with the rows of X already in the groups' order.
#define CJ_LIB "gemm_f32_tc"
#include "common.cuh"
#include "tc_common.cuh"

using namespace tc;

namespace {

constexpr int BK = 32;                    // K of a stage: 128 bytes of float32 (TMA's swizzle row), 64 bytes of bfloat16
// groups of eight splitting warps, each with stages of bfloat16 parts of its own, and warps that add up: as many as registers and issue slots bear
constexpr int GROUP_WARPS = 8;
constexpr int split_groups(int n) { return n <= 16 ? 3 : n <= 32 ? 2 : 1; }
constexpr int split_stages(int n) { return n <= 32 ? 6 : 4; }
// tiles of many tokens take X in its parts, which split_rows_kernel made once for all of them; the others split their rows of X themselves
constexpr bool ready_x(int n) { return n >= 64; }
constexpr int epi_warps(int n) { return n >= 64 ? 16 : n >= 32 ? 8 : 4; }
// warps: the splitting groups, two that issue products (every other unit each), two that load (one where the tile's X is not ready), adding up
constexpr int first_epi(int n) { return GROUP_WARPS * split_groups(n) + 4; }
constexpr int threads(int n) { return 32 * (first_epi(n) + epi_warps(n)); }

struct Args {
    const float* X; long long ldx;
    const int* x_index;                    // ready_x: the row of X that feeds a token (null: its own)
    const int* x_odd;                      // ready_x: tokens whose row has an entry that is not the sum of three parts
    const float* W; const float* W2;       // W2: the gated form's second weight
    const float* bias; const float* bias2;
    float* C; long long ldc;
    int tokens, features, K;
    int x_rows;                            // rows that X holds: nothing is read past them
    int accumulate;
    const int* group_offsets;
    int groups;
    float act_limit, act_alpha, act_cubic;
    int act, act_feats;
    float out_scale;
    int feat_tile;                         // features of a tile: at most 128, of the gated form at most 64
    int span, spans;                       // groups a place of the table, and its places
};

constexpr int SPANS = 1024;                // places of the table in shared memory that says where groups' tiles begin: of every group up to 1,024,
                                           // of every n-th beyond

template <int N, bool DUAL> struct Smem {
    static constexpr int STAGE = 3 * N * 64;                           // the bfloat16 parts of X (those of W lie in tensor memory)
    static constexpr int W_RAW = 128 * 128, X_RAW = ready_x(N) ? 0 : N * 128;       // one float32 tile
    static constexpr int RAW = W_RAW + X_RAW;
    static constexpr int STAGES = split_stages(N), GROUPS = split_groups(N);
    // a multiple of the groups, so that a slot is always read by the same group: a wait by phase parity must not be two phases off
    static constexpr int CROSS = DUAL ? epi_warps(N) * 1024 : 0;       // where the second weight's sums cross to the first's threads
    static constexpr int RING = (221 * 1024 - STAGES * STAGE - CROSS) / RAW / GROUPS * GROUPS;
    static constexpr int TOTAL = STAGES * STAGE + RING * RAW + CROSS + 1024 /* alignment */;
    static_assert(STAGES % GROUPS == 0, "a stage belongs to one group");
    // tensor memory: two accumulators of a unit of UNIT tokens (a tile of 128 tokens is two units), then the parts of W, three times 16
    // columns a stage
    static constexpr int UNIT = N < 64 ? N : 64, UNITS = N / UNIT;
    static constexpr int A_AT = 4 * UNIT, COLS_USED = A_AT + 48 * STAGES;
    static constexpr uint32_t TMEM_COLS = COLS_USED <= 256 ? 256 : 512;
    static_assert(COLS_USED <= 512, "tensor memory of an SM");
};

// eight float32 -> their three bfloat16 parts, packed; some bit of `odd` is set when one of the eight is not the sum of its parts: infinite,
// no number, so large that its first part rounds to infinity, or so small that its last part falls below the smallest bfloat16
__device__ __forceinline__ void split8(const float4 f0, const float4 f1, uint4& hi, uint4& mid, uint4& lo, uint32_t& odd) {
    const float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
    uint32_t h[4], m[4], l[4];
    auto pack = [](float a, float b) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
        return *(const uint32_t*)&t;
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = f[2 * i], b = f[2 * i + 1];
        h[i] = pack(a, b);
        const f32x2 r = sub2(pack2(a, b), pack2(__uint_as_float(h[i] << 16), __uint_as_float(h[i] & 0xffff0000u)));
        const float2 rs = unpack2(r);
        m[i] = pack(rs.x, rs.y);
        const float2 ls = unpack2(sub2(r, pack2(__uint_as_float(m[i] << 16), __uint_as_float(m[i] & 0xffff0000u))));
        l[i] = __byte_perm(__float_as_uint(ls.x), __float_as_uint(ls.y), 0x7632);        // (a remainder has eight bits at most)
        odd |= __float_as_uint(ls.x) | __float_as_uint(ls.y);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    mid = make_uint4(m[0], m[1], m[2], m[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// operand descriptor of a K-major bfloat16 tile of 64-byte rows, 64-byte swizzle (mode 4): 8-row groups 512 bytes apart; the other
// fields as in umma_desc_sw128
__device__ __forceinline__ uint64_t umma_desc_sw64(const void* smem_tile) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_u32(smem_tile) & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

// D[tmem] (+)= A[tmem] * B[smem] by the one thread of the warp with `on` set: A's rows are the lanes, two bfloat16 of neighbouring k a
// column; B's descriptor in two words.  (The whole warp walks the loop, so that addresses stay in uniform registers.)
__device__ __forceinline__ void umma_bf16_a_tmem(uint32_t on, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                                 uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "setp.ne.b32 q, %6, 0;\n\t"
        "mov.b64 b, {%2, %3};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(on)
        : "memory");
}
__device__ __forceinline__ void umma_commit_by(uint32_t on, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(on) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint4 a, const uint4 b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// whether `ok` holds in all of the block's THREADS threads that come here, after all of them have
template <int THREADS>
__device__ __forceinline__ bool all_of(bool ok) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 5, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)ok), "n"(THREADS)
        : "memory");
    return r != 0;
}

// (x null: a row of zeros)
__device__ __noinline__ float chain(const float* x, const float* w, int K) {
    float s = 0.0f;
    for (int k = 0; k < K; ++k) s = fmaf(x ? x[k] : 0.0f, w[k], s);
    return s;
}

// Which of `rows` (at most 64) rows have an entry that is not the sum of three parts, a bit a row; the warp goes over a row together.
__device__ __noinline__ unsigned long long odd_rows(const float* first, long long ld, int rows, int K) {
    unsigned long long found = 0;
    for (int r = 0; r < rows; ++r) {
        uint32_t odd = 0;
        for (int k = 4 * (threadIdx.x & 31); k < K; k += 128) {
            uint4 hi, mid, lo;
            split8(*(const float4*)(first + r * ld + k), make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi, mid, lo, odd);
        }
        if (__any_sync(0xffffffffu, (odd & 0xffffu) != 0)) found |= 1ull << r;
    }
    return found;
}

// whether a sum of the parts' products stands as it is (see the head of the file)
__device__ __forceinline__ bool chain_free(float v) { return (fabsf(v) >= 0x1p-100f && fabsf(v) <= 3.402823466e38f) || v == 0.0f; }

// A tile of the launch: tile index t is (token tile t / feat_tiles, feature tile t % feat_tiles), the token tiles of the groups after one another
struct Tile {
    int group, tok0, n_tok, feat0;
};
template <int N>
__device__ __forceinline__ int group_tiles(const Args& p, int g) { return (p.group_offsets[g + 1] - p.group_offsets[g] + N - 1) / N; }
template <int N>
__device__ __forceinline__ Tile locate(const Args& p, int t, int feat_tiles, const int* before) {
    const int tt = t / feat_tiles;
    Tile c;
    c.feat0 = (t - tt * feat_tiles) * p.feat_tile;
    c.group = 0;
    if (p.group_offsets) {
        int lo = 0, hi = p.spans;                             // before[lo] <= tt < before[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (before[mid] <= tt) lo = mid; else hi = mid;
        }
        int first = before[lo];
        c.group = lo * p.span;
        if (p.span > 1)                                       // (tt lies before the span's end, so some group of it holds it)
            for (int n; tt >= first + (n = group_tiles<N>(p, c.group)); ++c.group) first += n;
        c.tok0 = p.group_offsets[c.group] + (tt - first) * N;
        c.n_tok = min(p.group_offsets[c.group + 1] - c.tok0, N);
    } else {
        c.tok0 = tt * N;
        c.n_tok = min(p.tokens - c.tok0, N);
    }
    return c;
}

// Blocks stay, a block an SM, and take every gridDim.x-th tile; all roles run across tile boundaries, so that a tile's first loads and its last
// sums lie under its neighbours' products (they were 10 us of every tile bare).
template <int N, bool DUAL>
__global__ void __launch_bounds__(threads(N), 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                   const __grid_constant__ CUtensorMap map_w2, const Args p) {
    using S = Smem<N, DUAL>;
    // (blocks of K are counted without a sign: places in rings of odd sizes come cheaper so)
    constexpr unsigned G = S::GROUPS, STAGES = S::STAGES, RING = S::RING;
    constexpr int EPI_WARPS = epi_warps(N), ISSUE = GROUP_WARPS * G,
                  LOAD = ISSUE + 2, LOAD_X = LOAD + 1, FIRST_EPI = first_epi(N);
    constexpr bool READY = ready_x(N);
    constexpr int XP = READY ? 0 : 1;                         // rows of X a splitting thread takes (64 rows a pass)
    constexpr int UNIT = S::UNIT, UNITS = S::UNITS, UCOLS = UNIT * 4 / EPI_WARPS, COLS = UNITS * UCOLS;      // columns of an adding thread
    static_assert(UCOLS == 16 && UNITS <= 2, "sixteen columns of a unit an adding thread, a unit an accumulator");
    constexpr int FLAGS = 16;                                 // more tiles than splitting can be ahead of adding up: its stages and the accumulators
    extern __shared__ uint8_t smem_raw[];
    uint8_t* raw = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* stages = raw + RING * S::RAW;
    __shared__ uint64_t raw_full[RING], raw_empty[RING], full_bar[STAGES], empty_bar[STAGES], x_full[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int odd_flag[FLAGS];                           // some row of the tile has an entry that is not the sum of three parts
    __shared__ unsigned expired[threads(N) / 32];             // a warp's lanes whose waits ran out
    __shared__ int before[SPANS + 1];                         // token tiles of the groups before a span's first

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (lane == 0) expired[warp] = 0;
    if (tid == 0) {
        for (int s = 0; s < RING; ++s) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], GROUP_WARPS);
        }
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], GROUP_WARPS);
            mbar_init(&x_full[s], 1);
            mbar_init(&empty_bar[s], UNITS);                  // the products of every unit
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], EPI_WARPS);
        }
        for (int i = 0; i < FLAGS; ++i) odd_flag[i] = 0;
        fence_barrier_init();
    }
    if (warp == ISSUE) tmem_alloc(&tmem_slot, S::TMEM_COLS);
    const bool grouped = p.group_offsets != nullptr;
    if (grouped) cj::after_predecessor();
    if (grouped && warp == 0) {
        int carry = 0;
        for (int g0 = 0; g0 < p.groups; g0 += 32) {
            const int g = g0 + lane;
            const int n = g < p.groups ? group_tiles<N>(p, g) : 0;
            int inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (g < p.groups && g % p.span == 0) before[g / p.span] = carry + inc - n;
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) before[p.spans] = carry;
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    cj::release_successor();                                  // tensor memory is held
    const uint32_t tmem = tmem_slot;
    const int feat_tiles = (p.features + p.feat_tile - 1) / p.feat_tile;
    const int n_tiles = (grouped ? before[p.spans] : (p.tokens + N - 1) / N) * feat_tiles;
    const unsigned n_kb = (p.K + BK - 1) / BK;
    // the width of a unit's products; the parts of its X lie that many rows apart, side by side (those that came in parts UNIT rows)
    auto width = [](int n_tok, int u) { return (min(n_tok - u * UNIT, UNIT) + 15) & ~15; };

    if (warp == LOAD) {
        // ---- float32 tiles: the weights' first ones leave before the kernel before this one has ended (no kernel writes weights) ----
        if (elect_one()) {
            const uint32_t bytes = S::X_RAW + (DUAL ? 2u : 1u) * p.feat_tile * 128;
            auto weights = [&](unsigned kb, unsigned s, int w_row) {
                uint8_t* at = raw + s * S::RAW;
                tma_load_2d(at, &map_w, &raw_full[s], kb * BK, w_row);
                if (DUAL) tma_load_2d(at + 64 * 128, &map_w2, &raw_full[s], kb * BK, w_row);
            };
            unsigned early = 0;
            if (!grouped) {
                if ((int)blockIdx.x < n_tiles) {
                    const Tile c = locate<N>(p, blockIdx.x, feat_tiles, before);
                    for (; early < min(RING, n_kb); ++early) {
                        mbar_expect_tx(&raw_full[early], bytes);
                        weights(early, early, c.feat0);
                    }
                }
                if (!READY) cj::after_predecessor();
            }
            bool ok = true;
            unsigned it = 0;
            for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
                const Tile c = locate<N>(p, t, feat_tiles, before);
                for (unsigned kb = 0; kb < n_kb; ++kb, ++it) {
                    const unsigned s = it % RING;
                    if (it >= early) {
                        ok = mbar_wait(&raw_empty[s], ((it / RING) & 1) ^ 1, 15);
                        if (!ok) break;
                        mbar_expect_tx(&raw_full[s], bytes);
                        weights(kb, s, c.group * p.features + c.feat0);
                    }
                    if (!READY) tma_load_2d(raw + s * S::RAW + S::W_RAW, &map_x, &raw_full[s], kb * BK, c.tok0);
                }
            }
        }
    } else if (READY && warp == LOAD_X) {
        // ---- the parts of X, a stage's three side by side ----
        if (elect_one()) {
            if (!grouped) cj::after_predecessor();
            bool ok = true;
            unsigned it = 0;
            for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
                const Tile c = locate<N>(p, t, feat_tiles, before);
                const int units = (c.n_tok + UNIT - 1) / UNIT;
                for (unsigned kb = 0; kb < n_kb; ++kb, ++it) {
                    const unsigned s = it % STAGES;
                    ok = mbar_wait(&empty_bar[s], ((it / STAGES) & 1) ^ 1, 17);
                    if (!ok) break;
                    mbar_expect_tx(&x_full[s], units * 3 * UNIT * 64);
                    for (int u = 0; u < units; ++u)
                        tma_load_3d(stages + s * S::STAGE + u * 3 * UNIT * 64, &map_x, &x_full[s], kb * BK, c.tok0 + u * UNIT, 0);
                }
            }
        }
    } else if (warp < ISSUE) {
        // ---- splitting: of X a thread takes eight of a row's 32 float32 (a row of 64), of W half a row, its lane of tensor memory ----
        const unsigned g = warp / GROUP_WARPS;
        const int piece = tid & 3, row0 = (tid & (32 * GROUP_WARPS - 1)) >> 2;
        const int w_row = (warp & 3) * 32 + lane, half = warp >> 2 & 1;
        const bool w_live = (DUAL ? w_row & 63 : w_row) < p.feat_tile;      // (lanes past the tile's features: whatever they read, never stored)
        const uint32_t w_to = tmem + S::A_AT + half * 8 + ((uint32_t)((warp & 3) * 32) << 16);
        // 16-byte pieces 2 piece, 2 piece + 1 of a float32 row, piece `piece` of a bfloat16 row, each where its swizzle puts it
        const int src0 = row0 * 128 + (((2 * piece) ^ (row0 & 7)) << 4), src1 = row0 * 128 + (((2 * piece + 1) ^ (row0 & 7)) << 4);
        const int dst = row0 * 64 + ((piece ^ ((row0 >> 1) & 3)) << 4);
        bool ok = true;
        unsigned it = g, end = 0, nth = 0;                    // this group's next block of K of all tiles', one past the tile's last, tiles before it
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++nth) {
            end += n_kb;
            bool x_live = false;
            int x_part = 0;
            if (!READY) {
                const Tile c = locate<N>(p, t, feat_tiles, before);
                x_live = row0 < c.n_tok;
                x_part = width(c.n_tok, 0) * 64;
            }
            uint32_t odd = 0;
            for (; it < end; it += G) {
                const unsigned rs = it % RING, s = it % STAGES;
                ok = mbar_wait_warp(&raw_full[rs], (it / RING) & 1, 16, expired);
                if (!ok) break;
                const uint8_t* wr = raw + rs * S::RAW;
                const uint8_t* xr = wr + S::W_RAW;
                float4 w[4], x[2];
                auto read = [&]() {
#pragma unroll
                    for (int i = 0; i < 4; ++i) w[i] = *(const float4*)(wr + w_row * 128 + (((4 * half + i) ^ (w_row & 7)) << 4));
                    if (XP && x_live) {
                        x[0] = *(const float4*)(xr + src0);
                        x[1] = *(const float4*)(xr + src1);
                    }
                };
                // a lone group reads while the stage is still in use (1,777 x 6,144: 396 -> 375 us); several cover each other's
                if (G == 1) read();
                ok = mbar_wait_warp(&empty_bar[s], ((it / STAGES) & 1) ^ 1, 11, expired);
                if (!ok) break;
                tcgen05_fence_after();
                if (G > 1) read();
                {
                    uint4 hi[2], mid[2], lo[2];
                    uint32_t w_odd = 0;
                    split8(w[0], w[1], hi[0], mid[0], lo[0], w_odd);
                    split8(w[2], w[3], hi[1], mid[1], lo[1], w_odd);
                    if (w_live) odd |= w_odd;
                    const uint32_t to = w_to + s * 48;
                    tmem_st8(to, hi[0], hi[1]);
                    tmem_st8(to + 16, mid[0], mid[1]);
                    tmem_st8(to + 32, lo[0], lo[1]);
                }
                if (XP && x_live) {
                    uint4 hi, mid, lo;
                    split8(x[0], x[1], hi, mid, lo, odd);
                    uint8_t* at = stages + s * S::STAGE + dst;
                    *(uint4*)at = hi;
                    *(uint4*)(at + x_part) = mid;
                    *(uint4*)(at + 2 * x_part) = lo;
                }
                if (it + G >= end && (odd & 0xffffu)) odd_flag[nth % FLAGS] = 1;
                if (!READY) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // generic writes before the products' reads
                tmem_st_wait();
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&raw_empty[rs]);
                    mbar_arrive(&full_bar[s]);
                }
            }
        }
    } else if (warp == ISSUE || warp == ISSUE + 1) {
        // ---- product issue --------------------------------------------------------------------------
        // two accumulators a unit and block of K, D0 | D1, as wide as the unit each: D0 takes the products of the leading parts alone, whose
        // 16 bits an accumulator holds, D1 the others; the leading part of W meets the first two parts of X in one product twice as wide
        const uint32_t on = elect_one();
        const uint64_t first = umma_desc_sw64(stages);
        const uint32_t b_hi = (uint32_t)(first >> 32), b_first = (uint32_t)first;
        // tiles of one unit: every other block of K is a warp's (with the accumulator of its number), of two: every other unit
        const int mine = warp - ISSUE;
        const uint32_t acc0 = tmem + mine * 2 * UNIT;
        auto issue = [&](int wide, int u, unsigned s, unsigned times) {     // times: how often this warp has issued
            const uint32_t one = umma_idesc_bf16(128, wide), both = umma_idesc_bf16(128, 2 * wide);
            const uint32_t at = b_first + ((s * S::STAGE + u * 3 * UNIT * 64) >> 4), x_step = (READY ? UNIT : wide) * 64 >> 4;
            const uint32_t w = tmem + S::A_AT + s * 48, d1 = acc0 + wide;
            if (!mbar_wait_warp(&acc_empty[mine], (times & 1) ^ 1, 14, expired)) return false;
            tcgen05_fence_after();
            auto add = [&](int pw, int px) {                 // D1 += part pw of W . part px of X
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) umma_bf16_a_tmem(on, d1, w + pw * 16 + k * 8, at + px * x_step + 2 * k, b_hi, one, 1);
            };
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) {               // hi hi | hi mid
                const uint32_t wk = w + k * 8, xk = at + 2 * k;
                if (!READY || wide == UNIT) {
                    umma_bf16_a_tmem(on, acc0, wk, xk, b_hi, both, k > 0);
                } else {
                    umma_bf16_a_tmem(on, acc0, wk, xk, b_hi, one, k > 0);
                    umma_bf16_a_tmem(on, d1, wk, xk + x_step, b_hi, one, k > 0);
                }
            }
            add(1, 0); add(0, 2); add(1, 1); add(2, 0);
            umma_commit_by(on, &empty_bar[s]);
            umma_commit_by(on, &acc_full[mine]);
            return true;
        };
        bool ok = true;
        unsigned it = UNITS == 2 ? 0 : mine, end = 0, times = 0;
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            end += n_kb;
            const Tile c = locate<N>(p, t, feat_tiles, before);
            const int u = UNITS == 2 ? mine : 0;
            const bool live = u * UNIT < c.n_tok;
            const int wide = live ? width(c.n_tok, u) : 16;
            for (; it < end; it += UNITS == 2 ? 1 : 2) {
                const unsigned s = it % STAGES;
                ok = mbar_wait_warp(&full_bar[s], (it / STAGES) & 1, 12, expired) && (!READY || mbar_wait_warp(&x_full[s], (it / STAGES) & 1, 18, expired));
                if (!ok) break;
                if (live) {
                    ok = issue(wide, u, s, times);
                    if (!ok) break;
                    ++times;
                } else if (lane == 0) {
                    mbar_arrive(&empty_bar[s]);
                }
            }
        }
    } else if (warp >= FIRST_EPI) {
        // ---- adding up: a thread has one row of the product (a feature) and COLS of its tokens --------------
        const int quarter = warp & 3, r = quarter * 32 + lane, part = (warp - FIRST_EPI) >> 2, c_first = part * UCOLS;
        auto token = [&](int j) { return j / UCOLS * UNIT + c_first + j % UCOLS; };      // the token of the thread's column j
        if (!grouped) cj::after_predecessor();
        bool ok = true;
        unsigned it = 0, nth = 0, times[UNITS] = {};
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++nth) {
            const Tile c = locate<N>(p, t, feat_tiles, before);
            const int n_tok = c.n_tok, tok0 = c.tok0;
            f32x2 acc2[COLS / 2];
#pragma unroll
            for (int j = 0; j < COLS / 2; ++j) acc2[j] = pack2(0.0f, 0.0f);
            for (unsigned kb = 0; kb < n_kb && ok; ++kb, ++it) {
#pragma unroll
                for (int u = 0; u < UNITS; ++u) {
                    if (u * UNIT >= n_tok || !ok) break;
                    const int a = UNITS == 2 ? u : it & 1, wide = width(n_tok, u);
                    ok = mbar_wait_warp(&acc_full[a], (UNITS == 2 ? times[u] : it >> 1) & 1, 13, expired);
                    if (!ok) break;
                    ++times[u];
                    tcgen05_fence_after();
                    const uint32_t at = tmem + a * 2 * UNIT + c_first + ((uint32_t)(quarter * 32) << 16);
                    uint32_t v[16], h[16];                    // (columns past the unit's width hold whatever they held: nothing asks for them)
                    tmem_ld16(at + wide, v);
                    tmem_ld16(at, h);
                    tmem_ld_wait();
                    tcgen05_fence_before();                   // the accumulator is free before its sums are added
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[a]);
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        f32x2& s = acc2[(u * UCOLS + j) / 2];
                        s = add2(add2(s, pack2(__uint_as_float(v[j]), __uint_as_float(v[j + 1]))), pack2(__uint_as_float(h[j]), __uint_as_float(h[j + 1])));
                    }
                }
            }
            float acc[COLS];
#pragma unroll
            for (int j = 0; j < COLS; j += 2) {
                const float2 d = unpack2(acc2[j / 2]);
                acc[j] = d.x;
                acc[j + 1] = d.y;
            }
            const int fr = DUAL ? (r & 63) : r, feat = c.feat0 + fr;
            const bool live = ok && fr < p.feat_tile && feat < p.features;
            const bool odd_tile = odd_flag[nth % FLAGS] != 0;
            bool again = odd_tile;
            unsigned long long odd_x = 0;                     // the thread's tokens whose rows are not sums of three parts
            if (READY) {
#pragma unroll
                for (int u = 0; u < UNITS; ++u) {
                    const int tok = u * UNIT + c_first + lane;
                    odd_x |= (unsigned long long)__ballot_sync(0xffffffffu, lane < UCOLS && tok < n_tok && p.x_odd[tok0 + tok] != 0) << (u * UCOLS);
                }
                again = again || odd_x != 0;
            }
#pragma unroll
            for (int j = 0; j < COLS; ++j) again = again || (token(j) < n_tok && !chain_free(acc[j]));
            again = again && fr < p.feat_tile;                // the other rows' sums are of whatever lay behind the tile's weights
            if (__any_sync(0xffffffffu, again && ok)) {
                // (rarely: through an array in memory, so that the sums keep their registers)
                float sums[COLS];
#pragma unroll
                for (int j = 0; j < COLS; ++j) sums[j] = acc[j];
                const float* w = (DUAL && r >= 64 ? p.W2 : p.W) + ((size_t)c.group * p.features + feat) * p.K;
                bool odd_w = false;
                if (__any_sync(0xffffffffu, odd_tile)) {
                    // some row of the tile: which of the warp's (its live features are its first lanes')
                    // (rows from x_rows on are zeros, not memory of X)
                    if (!READY)
                        odd_x = odd_rows(p.X + (size_t)(tok0 + c_first) * p.ldx, p.ldx, max(0, min(UCOLS, min(n_tok, p.x_rows - tok0) - c_first)), p.K);
                    odd_w = odd_rows(w - (long long)lane * p.K, p.K, __popc(__ballot_sync(0xffffffffu, live)), p.K) >> lane & 1;
                }
#pragma unroll 1
                for (int j = 0; j < COLS; ++j) {
                    if (!live || token(j) >= n_tok || !(odd_w || (odd_x >> j & 1) || !chain_free(sums[j]))) continue;
                    const int row = READY && p.x_index ? p.x_index[tok0 + token(j)] : tok0 + token(j);
                    sums[j] = chain(row >= 0 && row < p.x_rows ? p.X + (size_t)row * p.ldx : nullptr, w, p.K);
                }
#pragma unroll
                for (int j = 0; j < COLS; ++j) acc[j] = sums[j];
            }
            const float b = p.bias && live ? p.bias[feat] : 0.0f;
            const float b2 = DUAL && p.bias2 && live ? p.bias2[feat] : 0.0f;
            float* out = p.C + (size_t)tok0 * p.ldc + feat;
            // the four warps of the same tokens
            auto together = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory"); };
            float* up = (float*)(stages + STAGES * S::STAGE) + part * 16 * 64;
#pragma unroll
            for (int u = 0; u < UNITS; ++u) {
                if (DUAL) {
                    // the second weight's sums cross to the threads that hold the first's, a unit at a time
                    if (u > 0) together();
                    if (r >= 64) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) up[j * 64 + fr] = acc[u * 16 + j];
                    }
                    together();
                }
                if (live && !(DUAL && r >= 64)) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (token(u * 16 + j) >= n_tok) break;
                        float v = p.bias ? acc[u * 16 + j] + b : acc[u * 16 + j];
                        if (DUAL) {
                            const float w2 = up[j * 64 + fr];
                            v = cj::gated_act(v, p.bias2 ? w2 + b2 : w2, p.act_limit, p.act_alpha, p.act_cubic);
                        } else if (p.act != cj::ACT_NONE && feat < p.act_feats) {
                            v = cj::plain_act(v, p.act);
                        }
                        v *= p.out_scale;
                        float* o = out + (size_t)token(u * 16 + j) * p.ldc;
                        *o = p.accumulate ? v + *o : v;
                    }
                }
            }
            // everyone has read the flag (and what crossed) before the next tile's; where a wait ran out, all of these warps leave together
            ok = all_of<EPI_WARPS * 32>(ok);
            if (warp == FIRST_EPI && lane == 0) odd_flag[nth % FLAGS] = 0;
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == ISSUE) {
        tcgen05_fence_after();
        tmem_dealloc(tmem, S::TMEM_COLS);
    }
}

// out[s, :] = x[index[s], :] for the rows of the groups (all rows without groups), zeros where the index names no row of x.  Rows outside
// the groups are left alone: no product reads them, and their indices may be anything.  A warp a row.
__global__ void __launch_bounds__(256) gather_group_rows_kernel(const float* __restrict__ x, long long ldx, int x_rows, const int* __restrict__ index,
                                                                const int* __restrict__ group_offsets, int groups, int rows, int K, float* __restrict__ out) {
    cj::after_predecessor();
    cj::release_successor();
    const int lane = threadIdx.x & 31, s = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lo = group_offsets ? group_offsets[0] : 0, hi = group_offsets ? min(rows, group_offsets[groups]) : rows;
    if (s < lo || s >= hi) return;
    const int from = index[s];
    const bool there = from >= 0 && from < x_rows;
    const float4* src = (const float4*)(x + (there ? from : 0) * ldx);
    float4* dst = (float4*)(out + (size_t)s * K);
#pragma unroll 4
    for (int i = lane; i < K / 4; i += 32) dst[i] = there ? src[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// The three parts of rows of x, [3][rows][Kp] bfloat16 (Kp: K rounded up to a block of K, the rest zeros), and whether a row has an entry that
// is not their sum.  Rows and index as above.  A warp a row.  Bound by memory: 1,777 rows of 2,048 out of HBM 11 us; a tile of 128 tokens x
// 128 features that splits its rows itself does so features / 128 times (1,777 x 6,144 x 2,048: see the head of the file).
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, long long ldx, int x_rows, const int* __restrict__ index,
                                                         const int* __restrict__ group_offsets, int groups, int rows, int K, int Kp,
                                                         __nv_bfloat16* __restrict__ out, int* __restrict__ odd_row) {
    cj::after_predecessor();
    cj::release_successor();
    const int lane = threadIdx.x & 31, s = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lo = group_offsets ? group_offsets[0] : 0, hi = group_offsets ? min(rows, group_offsets[groups]) : rows;
    if (s < lo || s >= hi) return;
    const int from = index ? index[s] : s;
    const bool there = from >= 0 && from < x_rows;
    const float4* src = (const float4*)(x + (there ? from : 0) * ldx);
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const size_t plane = (size_t)rows * Kp;
    __nv_bfloat16* dst = out + (size_t)s * Kp;
    uint32_t odd = 0;
#pragma unroll 4
    for (int i = lane; i < Kp / 8; i += 32) {
        uint4 h, m, l;
        split8(there && 8 * i < K ? src[2 * i] : zero, there && 8 * i + 4 < K ? src[2 * i + 1] : zero, h, m, l, odd);
        *(uint4*)(dst + 8 * i) = h;
        *(uint4*)(dst + plane + 8 * i) = m;
        *(uint4*)(dst + 2 * plane + 8 * i) = l;
    }
    const bool any = __any_sync(0xffffffffu, (odd & 0xffffu) != 0);
    if (lane == 0) odd_row[s] = any;
}

// the parts that split_rows_kernel left, in boxes of [3][box_rows][32] with the 64-byte swizzle; rows past the last read as zero
bool make_map_parts(CUtensorMap* map, const void* base, long long rows, long long Kp, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, 3};
    cuuint64_t strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)rows * Kp * 2};
    cuuint32_t box[3] = {BK, (cuuint32_t)box_rows, 3};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// a row-major float32 matrix in boxes of [box_rows, 32] with the 128-byte swizzle; out-of-range elements read as zero
bool make_map_f32(CUtensorMap* map, const float* base, long long rows, long long cols, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int N, bool DUAL>
int launch(const Args& a, const void* parts, int tok_tiles, cudaStream_t stream) {
    using S = Smem<N, DUAL>;
    auto kern = gemm_f32_tc_kernel<N, DUAL>;
    static bool sized = false;
    if (!sized) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL);
        if (e != cudaSuccess) return (int)e;
        sized = true;
    }
    const long long w_rows = (long long)(a.group_offsets ? a.groups : 1) * a.features;
    CUtensorMap mx, mw, mw2;
    if (ready_x(N)) {
        if (!make_map_parts(&mx, parts, a.tokens, (a.K + BK - 1) / BK * BK, S::UNIT)) return CJ_ERR_ARG;
    } else if (!make_map_f32(&mx, a.X, a.x_rows, a.K, a.ldx, N)) return CJ_ERR_ARG;
    if (!make_map_f32(&mw, a.W, w_rows, a.K, a.K, a.feat_tile)) return CJ_ERR_ARG;
    mw2 = mw;
    if (DUAL && !make_map_f32(&mw2, a.W2, w_rows, a.K, a.K, a.feat_tile)) return CJ_ERR_ARG;
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
    }
    const long long tiles = (long long)((a.features + a.feat_tile - 1) / a.feat_tile) * tok_tiles;
    if (tiles > 0x3fffffff) return CJ_ERR_SIZE;
    cj::launch(kern, dim3((unsigned)min(tiles, (long long)sms)), dim3(threads(N)), S::TOTAL, stream, mx, mw, mw2, a);
    return cj::launch_status();
}

}  // namespace

// Bytes of scratch that cj_gemm_f32_tc needs: the rows' parts and a flag a row for tiles of 64 tokens and more, the gathered rows for smaller ones
// with an index, else none.
CJ_EXPORT long long cj_gemm_f32_tc_scratch(int tokens, int K, int n_tok, int indexed) {
    const long long Kp = (long long)(K + BK - 1) / BK * BK;
    return n_tok >= 64 ? tokens * (6 * Kp + 4) : indexed ? (long long)tokens * K * 4 : 0;
}

// X [x_rows, K] float32 with row stride ldx; x_index (may be null): the row of X for each of `tokens` rows, those outside the groups left alone, an
// index that names no row of X for zeros; without it row s is row s, and those from x_rows on are zeros.  W (and W2) [groups, features, K]
// contiguous float32; the
// other arguments as cj_gemm_simt's.  n_tok: tokens of a tile (16, 32, 64 or 128); feat_tile: its features (32, 64 or 128; with W2 at most 64).
// scratch: scratch_bytes of memory, 16-byte aligned, at least what cj_gemm_f32_tc_scratch says.
CJ_EXPORT int cj_gemm_f32_tc(const float* X, long long ldx, int x_rows, const int* x_index, void* scratch, long long scratch_bytes, const float* W,
                             const float* W2, const float* bias, const float* bias2, float* C, long long ldc, int tokens, int features, int K,
                             int accumulate, const int* group_offsets, int groups, float act_limit, float act_alpha, float act_cubic, int act,
                             int act_feats, float out_scale, int n_tok, int feat_tile, cudaStream_t stream) {
    if (tokens <= 0 || features <= 0) return 0;
    if (!X || !W || !C || K <= 0 || x_rows <= 0) return CJ_ERR_ARG;
    if (group_offsets && groups <= 0) return CJ_ERR_ARG;
    if ((bias2 && !W2) || (act != cj::ACT_NONE && W2)) return CJ_ERR_ARG;
    if (feat_tile != 32 && feat_tile != 64 && !(feat_tile == 128 && !W2)) return CJ_ERR_SIZE;
    if (n_tok != 16 && n_tok != 32 && n_tok != 64 && n_tok != 128) return CJ_ERR_SIZE;
    if (K % 4 != 0 || ldx % 4 != 0 || ldx < K) return CJ_ERR_ALIGN;               // TMA: strides of 16 bytes
    if (((uintptr_t)X | (uintptr_t)W | (uintptr_t)W2 | (uintptr_t)scratch) & 15) return CJ_ERR_ALIGN;
    const int tok_tiles = (tokens + n_tok - 1) / n_tok + (group_offsets ? groups : 0);
    const long long room = cj_gemm_f32_tc_scratch(tokens, K, n_tok, x_index != nullptr);
    if (room > 0 && (!scratch || scratch_bytes < room)) return CJ_ERR_ARG;
    const int* x_odd = nullptr;
    if (n_tok >= 64) {
        const int Kp = (K + BK - 1) / BK * BK;
        int* odd = (int*)((__nv_bfloat16*)scratch + 3 * (size_t)tokens * Kp);
        cj::launch(split_rows_kernel, dim3((tokens + 7) / 8), dim3(256), 0, stream, X, ldx, x_rows, x_index, group_offsets, groups, tokens, K, Kp,
                   (__nv_bfloat16*)scratch, odd);
        x_odd = odd;
    } else if (x_index) {
        cj::launch(gather_group_rows_kernel, dim3((tokens + 7) / 8), dim3(256), 0, stream, X, ldx, x_rows, x_index, group_offsets, groups, tokens, K,
                   (float*)scratch);
        X = (const float*)scratch;
        ldx = K;
        x_rows = tokens;
        x_index = nullptr;
    }
    if (int st = cj::launch_status()) return st;
    Args a{X, ldx, x_index, x_odd, W, W2, bias, bias2, C, ldc, tokens, features, K, x_rows, accumulate, group_offsets, groups, act_limit, act_alpha, act_cubic, act,
           act_feats > 0 ? act_feats : features, out_scale, feat_tile, 1, 0};
    if (group_offsets) {
        a.span = (groups + SPANS - 1) / SPANS;
        a.spans = (groups + a.span - 1) / a.span;
    }
#define CASE(N) case N: return W2 ? launch<N, true>(a, scratch, tok_tiles, stream) : launch<N, false>(a, scratch, tok_tiles, stream);
    switch (n_tok) {
        CASE(16) CASE(32) CASE(64) CASE(128)
    }
#undef CASE
    return CJ_ERR_SIZE;
}

// 0, or the code of the first bounded wait that ran out (15 and 17 loads, 11 and 16 splitting, 12, 14 and 18 product issue, 13 adding up);
// reading it synchronises the device.
CJ_EXPORT int cj_gemm_f32_tc_error() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, tc::g_error_flag, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
