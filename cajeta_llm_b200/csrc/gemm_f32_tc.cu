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
// the float32 tiles (TMA) into a ring as deep as shared memory allows; groups of eight warps split them into the six bfloat16
// tiles of a stage, a group every G-th block of K; one warp issues the products; the last warps add the accumulators up
// and store.  A block of K is a chain of short waits for a group (tile landed, stage free, stores visible to the products: some
// 1,100 clocks, half of them waiting), so with few tokens several groups work side by side.  What bounds it: with few
// tokens that chain, with many one group's going through read, split, write and wait (issue slots 61 % used, shared memory 44 %, integer and
// conversion pipe 40 %, tensor pipe 33 %; shared memory has no room for a second group).
// Rows x features x K, us, gemm_simt.cu before and now (cold weights): 1 x 2,048 x 2,048 190 and 32; 250 x 6,144 x 2,048 327 and 100;
// 1,777 x 6,144 x 2,048 1,817 and 352; 64 groups of 1,408 gated features, 8 / 256 / 1,777 tokens of 4 picks among 60 of them
// 796 / 1,449 / 3,162 and 147 / 392 / 866.  (With the float32 operands loaded into registers instead of by TMA 1,777 x 6,144 took 815: one
// load's latency a block lay bare.  Three loading threads instead of one changed nothing.)
// Grouped form as in gemm_simt.cu, with the rows of X already in the groups' order.
#define CJ_LIB "gemm_f32_tc"
#include "common.cuh"
#include "tc_common.cuh"

using namespace tc;

namespace {

constexpr int BK = 32;                    // K of a stage: 128 bytes of float32 (TMA's swizzle row), 64 bytes of bfloat16
// groups of eight splitting warps, each with stages of bfloat16 parts of its own, and warps that add up: as many as registers
// and shared memory hold
constexpr int GROUP_WARPS = 8;
constexpr int split_groups(int n) { return n <= 32 ? 3 : n <= 64 ? 2 : 1; }
constexpr int split_stages(int n) { return n <= 32 ? 3 : 2; }
constexpr int epi_warps(int n) { return n >= 64 ? 8 : 4; }
// warps: the splitting groups, product issue, loads (and, so that the warps that add up begin at a multiple of four, idle ones), adding up
constexpr int first_epi(int n) { return (GROUP_WARPS * split_groups(n) + 2 + 3) / 4 * 4; }
constexpr int threads(int n) { return 32 * (first_epi(n) + epi_warps(n)); }

struct Args {
    const float* X; long long ldx;
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
};

template <int N> struct Smem {
    static constexpr int W_PART = 128 * 64, X_PART = N * 64;           // one bfloat16 tile
    static constexpr int STAGE = 3 * (W_PART + X_PART);
    static constexpr int W_RAW = 128 * 128, X_RAW = N * 128;           // one float32 tile
    static constexpr int RAW = W_RAW + X_RAW;
    static constexpr int STAGES = split_stages(N);
    // a multiple of the groups, so that a slot is always read by the same group: a wait by phase parity must not be two phases off
    static constexpr int RING = (225 * 1024 - STAGES * STAGE) / RAW / STAGES * STAGES;
    static constexpr int TOTAL = STAGES * STAGE + RING * RAW + 1024 /* alignment */;
    static_assert(STAGES % split_groups(N) == 0, "a stage belongs to one group");
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
        const float ra = a - __uint_as_float(h[i] << 16), rb = b - __uint_as_float(h[i] & 0xffff0000u);
        m[i] = pack(ra, rb);
        const float la = ra - __uint_as_float(m[i] << 16), lb = rb - __uint_as_float(m[i] & 0xffff0000u);
        l[i] = __byte_perm(__float_as_uint(la), __float_as_uint(lb), 0x7632);        // (a remainder has eight bits at most)
        odd |= __float_as_uint(la) | __float_as_uint(lb);
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

__device__ __noinline__ float chain(const float* x, const float* w, int K) {
    float s = 0.0f;
    for (int k = 0; k < K; ++k) s = fmaf(x[k], w[k], s);
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

template <int N, bool DUAL>
__global__ void __launch_bounds__(threads(N), 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                   const __grid_constant__ CUtensorMap map_w2, const Args p) {
    using S = Smem<N>;
    constexpr int G = split_groups(N), STAGES = S::STAGES, EPI_WARPS = epi_warps(N), RING = S::RING, ISSUE = GROUP_WARPS * G,
                  LOAD = ISSUE + 1, FIRST_EPI = first_epi(N);
    constexpr int XP = (N + 63) / 64;                         // rows of X a splitting thread takes (64 rows a pass)
    constexpr int COLS = N * 4 / EPI_WARPS;                   // columns of an adding thread
    constexpr uint32_t TMEM_COLS = 4 * N <= 64 ? 64 : 4 * N <= 128 ? 128 : 4 * N <= 256 ? 256 : 512;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* raw = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* stages = raw + RING * S::RAW;
    __shared__ uint64_t raw_full[RING], raw_empty[RING], full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int odd_flag;                                  // some row of the tile has an entry that is not the sum of three parts
    __shared__ int place[3];                                  // group, first row, one past the last; group -1: no work

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < RING; ++s) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], GROUP_WARPS);
        }
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], GROUP_WARPS);
            mbar_init(&empty_bar[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], EPI_WARPS);
        }
        odd_flag = 0;
        fence_barrier_init();
    }
    if (warp == ISSUE) tmem_alloc(&tmem_slot, TMEM_COLS);
    const bool grouped = p.group_offsets != nullptr;
    if (grouped) cj::after_predecessor();
    if (warp == 0) {
        // which rows: token tile blockIdx.y of the whole launch, or of the group that holds it
        if (grouped) {
            int before = 0, found = -1, lo = 0, hi = 0;
            for (int g0 = 0; g0 < p.groups; g0 += 32) {
                const int g = g0 + lane;
                const int a = g < p.groups ? p.group_offsets[g] : 0, b = g < p.groups ? p.group_offsets[g + 1] : 0;
                const int n = g < p.groups ? (b - a + N - 1) / N : 0;
                int inc = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += v;
                }
                const int t = (int)blockIdx.y - (before + inc - n);
                const unsigned who = __ballot_sync(0xffffffffu, t >= 0 && t < n);
                if (who) {
                    const int l = __ffs(who) - 1;
                    found = g0 + l;
                    lo = __shfl_sync(0xffffffffu, a, l) + __shfl_sync(0xffffffffu, t, l) * N;
                    hi = min(__shfl_sync(0xffffffffu, b, l), lo + N);
                    break;
                }
                before += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (lane == 0) { place[0] = found; place[1] = lo; place[2] = hi; }
        } else if (lane == 0) {
            place[0] = 0;
            place[1] = blockIdx.y * N;
            place[2] = min(p.tokens, place[1] + N);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    cj::release_successor();                                  // tensor memory is held
    const int group = place[0], tok0 = place[1], n_tok = place[2] - place[1];
    const uint32_t tmem = tmem_slot;
    const int feat0 = blockIdx.x * p.feat_tile;
    const int n_kb = (p.K + BK - 1) / BK;
    const bool work = group >= 0 && n_tok > 0;
    const int n16 = (n_tok + 15) & ~15;                       // the product's width; the parts of X lie n16 rows apart, side by side

    if (work && warp == LOAD) {
        // ---- float32 tiles: the weights' first ones leave before the kernel before this one has ended (no kernel writes weights) ----
        if (elect_one()) {
            const int w_row = group * p.features + feat0;
            const uint32_t bytes = S::X_RAW + (DUAL ? 2u : 1u) * p.feat_tile * 128;
            auto weights = [&](int kb, int s) {
                uint8_t* at = raw + s * S::RAW;
                tma_load_2d(at, &map_w, &raw_full[s], kb * BK, w_row);
                if (DUAL) tma_load_2d(at + 64 * 128, &map_w2, &raw_full[s], kb * BK, w_row);
            };
            const int early = grouped ? 0 : min(RING, n_kb);
            for (int kb = 0; kb < early; ++kb) {
                mbar_expect_tx(&raw_full[kb], bytes);
                weights(kb, kb);
            }
            if (!grouped) cj::after_predecessor();
            bool ok = true;
            for (int kb = 0; kb < n_kb && ok; ++kb) {
                const int s = kb % RING;
                if (kb >= early) {
                    ok = mbar_wait(&raw_empty[s], ((kb / RING) & 1) ^ 1, 15);
                    if (!ok) break;
                    mbar_expect_tx(&raw_full[s], bytes);
                    weights(kb, s);
                }
                tma_load_2d(raw + s * S::RAW + S::W_RAW, &map_x, &raw_full[s], kb * BK, tok0);
            }
        }
    } else if (work && warp < ISSUE) {
        // ---- splitting: thread = (row of 64, eight of the row's 32 float32) ------------------------
        const int g = warp / GROUP_WARPS, piece = tid & 3, row0 = (tid & (32 * GROUP_WARPS - 1)) >> 2;
        bool w_live[2], x_live[XP];
#pragma unroll
        for (int i = 0; i < 2; ++i) w_live[i] = (DUAL ? row0 : row0 + 64 * i) < p.feat_tile;      // (rows past the last feature: read as they are, never stored)
#pragma unroll
        for (int i = 0; i < XP; ++i) x_live[i] = row0 + 64 * i < n_tok;
        // 16-byte pieces 2 piece, 2 piece + 1 of a float32 row, piece `piece` of a bfloat16 row, each where its swizzle puts it
        // (64 rows apart the swizzles are the same)
        const int src0 = row0 * 128 + (((2 * piece) ^ (row0 & 7)) << 4), src1 = row0 * 128 + (((2 * piece + 1) ^ (row0 & 7)) << 4);
        const int dst = row0 * 64 + ((piece ^ ((row0 >> 1) & 3)) << 4);
        const int x_part = n16 * 64;
        uint32_t odd = 0;
        bool ok = true;
        for (int kb = g; kb < n_kb && ok; kb += G) {
            const int rs = kb % RING, s = kb % STAGES;
            ok = mbar_wait(&raw_full[rs], (kb / RING) & 1, 16);
            if (!ok) break;
            const uint8_t* wr = raw + rs * S::RAW;
            const uint8_t* xr = wr + S::W_RAW;
            float4 w[2][2], x[XP][2];
            auto read = [&]() {
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (w_live[i]) {
                        w[i][0] = *(const float4*)(wr + i * 64 * 128 + src0);
                        w[i][1] = *(const float4*)(wr + i * 64 * 128 + src1);
                    }
#pragma unroll
                for (int i = 0; i < XP; ++i)
                    if (x_live[i]) {
                        x[i][0] = *(const float4*)(xr + i * 64 * 128 + src0);
                        x[i][1] = *(const float4*)(xr + i * 64 * 128 + src1);
                    }
            };
            // a lone group reads while the stage is still in use (1,777 x 6,144: 396 -> 375 us); several cover each other's
            if (G == 1) read();
            ok = mbar_wait(&empty_bar[s], ((kb / STAGES) & 1) ^ 1, 11);
            if (!ok) break;
            if (G > 1) read();
            uint8_t* wt = stages + s * S::STAGE;
            uint8_t* xt = wt + 3 * S::W_PART;
            uint4 hi, mid, lo;
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (w_live[i]) {
                    split8(w[i][0], w[i][1], hi, mid, lo, odd);
                    uint8_t* at = wt + i * 64 * 64 + dst;
                    *(uint4*)at = hi;
                    *(uint4*)(at + S::W_PART) = mid;
                    *(uint4*)(at + 2 * S::W_PART) = lo;
                }
#pragma unroll
            for (int i = 0; i < XP; ++i)
                if (x_live[i]) {
                    split8(x[i][0], x[i][1], hi, mid, lo, odd);
                    uint8_t* at = xt + i * 64 * 64 + dst;
                    *(uint4*)at = hi;
                    *(uint4*)(at + x_part) = mid;
                    *(uint4*)(at + 2 * x_part) = lo;
                }
            if (kb + G >= n_kb && (odd & 0xffffu)) odd_flag = 1;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // generic writes before the products' reads
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&raw_empty[rs]);
                mbar_arrive(&full_bar[s]);
            }
        }
    } else if (work && warp == ISSUE) {
        // ---- product issue --------------------------------------------------------------------------
        if (elect_one()) {
            // two accumulators a block of K, D0 | D1, n16 columns each: D0 takes the products of the leading parts alone, whose 16 bits an
            // accumulator holds, D1 the others; the leading part of W meets the first two parts of X in one product twice as wide
            const uint32_t one = umma_idesc_bf16(128, n16), both = umma_idesc_bf16(128, 2 * n16);
            const uint64_t first = umma_desc_sw64(stages);
            const uint64_t w_step = S::W_PART >> 4, x_hi = 3 * w_step, x_step = (uint64_t)(n16 * 64 >> 4);
            bool ok = true;
            for (int kb = 0; kb < n_kb && ok; ++kb) {
                const int s = kb % STAGES, a = kb & 1;
                ok = mbar_wait(&acc_empty[a], ((kb >> 1) & 1) ^ 1, 14) && mbar_wait(&full_bar[s], (kb / STAGES) & 1, 12);
                if (!ok) break;
                tcgen05_fence_after();
                const uint64_t at = first + (uint64_t)((s * S::STAGE) >> 4);
                const uint32_t d0 = tmem + a * 2 * N, d1 = d0 + n16;
                auto add = [&](int pw, int px) {             // D1 += part pw of W . part px of X
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_bf16(d1, at + pw * w_step + 2 * k, at + x_hi + px * x_step + 2 * k, one, 1);
                };
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) umma_bf16(d0, at + 2 * k, at + x_hi + 2 * k, both, k > 0);                      // hi hi | hi mid
                add(1, 0); add(0, 2); add(1, 1); add(2, 0);
                umma_commit(&empty_bar[s]);
                umma_commit(&acc_full[a]);
            }
        }
    } else if (work && warp >= FIRST_EPI) {
        // ---- adding up: a thread has one row of the product (a feature) and COLS of its tokens --------------
        const int quarter = warp & 3, r = quarter * 32 + lane, c_first = ((warp - FIRST_EPI) >> 2) * COLS;
        float acc[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
        bool ok = true;
        for (int kb = 0; kb < n_kb && ok; ++kb) {
            const int a = kb & 1;
            ok = mbar_wait(&acc_full[a], (kb >> 1) & 1, 13);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t at = tmem + a * 2 * N + c_first + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
            for (int c = 0; c < COLS; c += 16) {
                if (c_first + c >= n16) break;
                uint32_t v[16];
                tmem_ld16(at + n16 + c, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(v[j]);
                tmem_ld16(at + c, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(v[j]);
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[a]);
        }
        if (!grouped) cj::after_predecessor();
        const int fr = DUAL ? (r & 63) : r, feat = feat0 + fr;
        const bool live = ok && fr < p.feat_tile && feat < p.features;
        bool again = odd_flag != 0;
#pragma unroll
        for (int j = 0; j < COLS; ++j) again = again || !chain_free(acc[j]);
        if (__any_sync(0xffffffffu, again)) {
            // (rarely: through an array in memory, so that the sums keep their registers)
            float sums[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) sums[j] = acc[j];
            const int cols = min(COLS, n_tok - c_first);
            const float* x = p.X + (size_t)(tok0 + c_first) * p.ldx;
            const float* w = (DUAL && r >= 64 ? p.W2 : p.W) + ((size_t)group * p.features + feat) * p.K;
            unsigned long long odd_x = 0;
            bool odd_w = false;
            if (__any_sync(0xffffffffu, odd_flag != 0)) {
                // some row of the tile: which of the warp's (its live features are its first lanes')
                odd_x = odd_rows(x, p.ldx, cols, p.K);
                odd_w = odd_rows(w - (long long)lane * p.K, p.K, __popc(__ballot_sync(0xffffffffu, live)), p.K) >> lane & 1;
            }
#pragma unroll 1
            for (int j = 0; j < cols && live; ++j)
                if (odd_w || (odd_x >> j & 1) || !chain_free(sums[j])) sums[j] = chain(x + (size_t)j * p.ldx, w, p.K);
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] = sums[j];
        }
        if (DUAL) {
            // the second weight's sums cross to the threads that hold the first's: through the ring, which nothing reads any more
            float* up = (float*)raw;
            if (r >= 64) {
#pragma unroll
                for (int j = 0; j < COLS; ++j) up[(c_first + j) * 64 + fr] = acc[j];
            }
            asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
        }
        if (live && !(DUAL && r >= 64)) {
            const float b = p.bias ? p.bias[feat] : 0.0f;
            const float b2 = DUAL && p.bias2 ? p.bias2[feat] : 0.0f;
            float* out = p.C + (size_t)(tok0 + c_first) * p.ldc + feat;
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                if (c_first + j >= n_tok) break;
                float v = p.bias ? acc[j] + b : acc[j];
                if (DUAL) {
                    const float u = ((const float*)raw)[(c_first + j) * 64 + fr];
                    v = cj::gated_act(v, p.bias2 ? u + b2 : u, p.act_limit, p.act_alpha, p.act_cubic);
                } else if (p.act != cj::ACT_NONE && feat < p.act_feats) {
                    v = cj::plain_act(v, p.act);
                }
                v *= p.out_scale;
                float* o = out + (size_t)j * p.ldc;
                *o = p.accumulate ? v + *o : v;
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == ISSUE) {
        tcgen05_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
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
int launch(const Args& a, int tok_tiles, cudaStream_t stream) {
    auto kern = gemm_f32_tc_kernel<N, DUAL>;
    static bool sized = false;
    if (!sized) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<N>::TOTAL);
        if (e != cudaSuccess) return (int)e;
        sized = true;
    }
    if (tok_tiles > 65535) return CJ_ERR_SIZE;
    const long long w_rows = (long long)(a.group_offsets ? a.groups : 1) * a.features;
    CUtensorMap mx, mw, mw2;
    if (!make_map_f32(&mx, a.X, a.x_rows, a.K, a.ldx, N) || !make_map_f32(&mw, a.W, w_rows, a.K, a.K, a.feat_tile)) return CJ_ERR_ARG;
    mw2 = mw;
    if (DUAL && !make_map_f32(&mw2, a.W2, w_rows, a.K, a.K, a.feat_tile)) return CJ_ERR_ARG;
    cj::launch(kern, dim3((a.features + a.feat_tile - 1) / a.feat_tile, tok_tiles), dim3(threads(N)), Smem<N>::TOTAL, stream, mx, mw, mw2, a);
    return cj::launch_status();
}

}  // namespace

// Rows of x (float32, row stride ldx, x_rows of them) in the groups' order, out [rows, K] contiguous: as cj_gemm_f32_tc takes them.
CJ_EXPORT int cj_gather_group_rows(const float* x, long long ldx, int x_rows, const int* index, const int* group_offsets, int groups, int rows,
                                   int K, float* out, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (!x || !index || !out || K <= 0 || x_rows <= 0 || (group_offsets && groups <= 0)) return CJ_ERR_ARG;
    if (K % 4 != 0 || ldx % 4 != 0 || ldx < K || (((uintptr_t)x | (uintptr_t)out) & 15)) return CJ_ERR_ALIGN;
    cj::launch(gather_group_rows_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, x, ldx, x_rows, index, group_offsets, groups, rows, K, out);
    return cj::launch_status();
}

// X [x_rows, K] float32 with row stride ldx (grouped: in the groups' order; no row from x_rows on is read), W (and W2) [groups, features, K]
// contiguous float32; the
// other arguments as cj_gemm_simt's.  n_tok: tokens of a tile (16, 32, 64 or 128); feat_tile: its features (32, 64 or 128; with W2 at most 64).
CJ_EXPORT int cj_gemm_f32_tc(const float* X, long long ldx, int x_rows, const float* W, const float* W2, const float* bias, const float* bias2, float* C,
                             long long ldc, int tokens, int features, int K, int accumulate, const int* group_offsets, int groups,
                             float act_limit, float act_alpha, float act_cubic, int act, int act_feats, float out_scale, int n_tok,
                             int feat_tile, cudaStream_t stream) {
    if (tokens <= 0 || features <= 0) return 0;
    if (!X || !W || !C || K <= 0 || x_rows <= 0) return CJ_ERR_ARG;
    if (group_offsets && groups <= 0) return CJ_ERR_ARG;
    if ((bias2 && !W2) || (act != cj::ACT_NONE && W2)) return CJ_ERR_ARG;
    if (feat_tile != 32 && feat_tile != 64 && !(feat_tile == 128 && !W2)) return CJ_ERR_SIZE;
    if (K % 4 != 0 || ldx % 4 != 0 || ldx < K) return CJ_ERR_ALIGN;               // TMA: strides of 16 bytes
    if (((uintptr_t)X | (uintptr_t)W | (uintptr_t)W2) & 15) return CJ_ERR_ALIGN;
    Args a{X, ldx, W, W2, bias, bias2, C, ldc, tokens, features, K, x_rows, accumulate, group_offsets, groups, act_limit, act_alpha, act_cubic, act,
           act_feats > 0 ? act_feats : features, out_scale, feat_tile};
    const int tok_tiles = (tokens + n_tok - 1) / max(n_tok, 1) + (group_offsets ? groups : 0);
#define CASE(N) case N: return W2 ? launch<N, true>(a, tok_tiles, stream) : launch<N, false>(a, tok_tiles, stream);
    switch (n_tok) {
        CASE(16) CASE(32) CASE(64) CASE(128)
    }
#undef CASE
    return CJ_ERR_SIZE;
}

// 0, or the code of the first bounded wait that ran out (15 loads, 11 and 16 splitting, 12 and 14 product issue, 13 adding up);
// reading it synchronises the device.
CJ_EXPORT int cj_gemm_f32_tc_error() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, tc::g_error_flag, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
