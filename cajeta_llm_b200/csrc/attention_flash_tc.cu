// Two more attentions for prompt portions on the 5th-generation tensor cores (tcgen05): differential attention over the paged
// cache, and latent attention in its plain form (keys and values of every head built in dense buffers).  bfloat16 storage, scores,
// softmaxes and sums in float32.
//
// A block runs two softmaxes side by side over the same tiles of 128 keys, so that the tensor core works on one while the other's
// exponentials are computed:
//   latent        two tiles of 128 query rows of one request and one head
//   differential  the two maps of the same 128 query rows; what leaves the block is a1 - lambda a2, normed over the head
// Per softmax and key tile: S = Q K^T into tensor memory (float32, 128 columns); four warps, a row a thread, turn 64 scores at a
// time into exp2(S - m) and put them back as bfloat16 over the columns they came from; O += P V with P read from tensor memory.
// TWO: a weight enters that product as two bfloat16 terms, its rounding and the rest, which together take just the columns of the
// scores they replace.  The running maximum moves (and O is rescaled) only when a half tile raises it by more than 2^8.
// Keys arrive as chunks of [128 keys x 64 columns], values as [64 keys x value size], each in a ring of its own that a warp of its
// own fills: with keys of 192 entries the two query tiles take 96 KB and whole tiles of keys and values would not fit twice.
// Rows of a values' tile that are no keys of the block (another request's tokens, the unwritten rest of a page) are cleared
// before the product reads them: a weight of zero times whatever lies there need not be zero.
//
// What bounds it: the tensor core's products of a key tile take 2,560 cycles a block in both forms (64 each 16 columns or keys deep;
// latent with two terms 3,584), the exponentials 2,048; a tile takes 3,500 (latent), 4,000 (latent, two terms) and 4,900 (differential,
// whose pages arrive in boxes of 2 KB).  One prompt of 2,048 tokens, 16 heads, cold L2, against the mma.sync kernels (attention_diff.cu,
// latent_prefill.cu): differential, maps of 64 and values of 128, 250 -> 66 us; latent, keys of 192 and values of 128, 168 -> 53 us, with
// two terms 197 -> 64 us; 4,000 tokens 780 -> 207, 512 -> 102 and 604 -> 118 us; 512 tokens 44 -> 23, 29 -> 20 and 31 -> 21 us.
// Every wait is bounded (tc_common.cuh).
#define CJ_LIB "attention_flash_tc"
#include "common.cuh"
#include "tc_common.cuh"

using namespace tc;

namespace {

constexpr int BM = 128;                           // query rows of a softmax
constexpr int BN = 128;                           // keys a tile
constexpr int THREADS = 352;                      // keys' warp, values' warp, products' warp, two times four softmax warps
constexpr int CHUNK = 128 * 64 * 2;               // a [128 x 64] bf16 chunk of queries or keys: 16 KB
constexpr float RESCALE_THRESHOLD = 8.0f;         // in log2 units
constexpr uint32_t TM_S = 0, TM_O = 256, TM_COLS = 512;      // tensor memory: two tiles of scores, two of outputs (128 columns each)

// MAPS: differential, DK the size of one map's key; otherwise latent, DK the key's size (64 more than a multiple of 64, or one)
template <bool MAPS, int DK, int DV>
struct Shape {
    static constexpr int WIDTH = MAPS ? 2 * DK : DK;                    // columns of a head's query row or key
    static constexpr int KC = (WIDTH + 63) / 64;                        // chunks a key tile
    static constexpr int QC = MAPS ? KC : 2 * KC;                       // chunks of queries a block
    static constexpr int V_BYTES = 64 * DV * 2;                         // 64 keys' values
    static constexpr int ROOM = 226 * 1024 - QC * CHUNK;                // for the rings
    static constexpr int VS = DV == 64 ? 4 : (QC >= 6 ? 3 : 4);
    static constexpr int KS_FIT = (ROOM - VS * V_BYTES) / CHUNK;
    static constexpr int KS = KS_FIT > 6 ? 6 : KS_FIT;
    static_assert(KS > KC, "a ring of keys holds a tile and part of the next");
    static constexpr int Q_AT = 0, K_AT = QC * CHUNK, V_AT = K_AT + KS * CHUNK, BAR_AT = V_AT + VS * V_BYTES;
    static constexpr int SMEM = BAR_AT + 512 + 512 + 1024;              // barriers, map 2's divisors, alignment
    static_assert(SMEM <= 232448, "shared memory of a block");
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *(uint32_t*)&v;
}
// what the two terms in `first` leave over, as the next terms
__device__ __forceinline__ uint32_t pack_rest(float a, float b, uint32_t first) {
    return pack_bf16(a - __uint_as_float(first << 16), b - __uint_as_float(first & 0xffff0000u));
}

struct Args {
    __nv_bfloat16* out;            // [T, n_heads * DV]
    const int* req_start;
    const int* req_prior;
    int n_requests, n_heads, window;
    float scale_log2;              // scores to units of log 2
    int block_rows;                // query rows a block takes: 256 (latent, both tiles) or 128
    // differential: the cache's pages
    const int* table;
    int table_stride, page_tokens, n_kv, plane_rows;
    float lambda, eps, out_scale;
    // latent: request i's token p lies at row req_base[i] + p of the dense buffers
    const int* req_base;
    const float* sink;             // null, or [n_heads]: exp(sink) joins the divisor
    // null, or float32 [T, gate_ld]: head h of row t is multiplied by sigmoid(gate[t, h]).  (A gate for every entry costs more here than in a
    // kernel of its own: the rows' results leave a row a thread, and the block waits for its gates - 29 to 40 us of 2,250 rows' 70 to 80.)
    const float* gate;
    int gate_ld;
};

// What a softmax of the block covers: its rows, the position of the first, and the key tiles it needs, counted from the block's
// first key tile (begin > end: none).
struct Rows {
    int n, p0, begin, end;
};

// map_k, map_k2, map_v: latent: the keys' own columns [tokens, heads * (DK - 64)], the shared last 64 [tokens, 64], the values
// [tokens, heads * DV]; differential: the planes as [pages * key heads * page_tokens, 2 DK] (map_k2 is not used) and [.., DV]
template <bool MAPS, int DK, int DV, bool TWO>
__global__ void __launch_bounds__(THREADS, 1)
flash_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_k2, const __grid_constant__ CUtensorMap map_v, Args p) {
    using S = Shape<MAPS, DK, DV>;
    constexpr int KC = S::KC, KS = S::KS, VS = S::VS, KSTEPS = DK / 16;
    constexpr uint32_t IDESC_QK = umma_idesc_bf16(BM, BN), IDESC_PV = umma_idesc_bf16(BM, DV) | (1u << 16);
    // blocks beyond the row blocks that the step's requests make (the grid covers the most the layout can hold) leave at once
    {
        int tiles = 0;
        for (int r = threadIdx.x & 31; r < p.n_requests; r += 32)
            tiles += (__ldcg(p.req_start + r + 1) - __ldcg(p.req_start + r) + p.block_rows - 1) / p.block_rows;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tiles += __shfl_xor_sync(0xffffffffu, tiles, o);
        if ((int)blockIdx.y >= tiles) {
            cj::after_predecessor();
            return;
        }
    }
    cj::after_predecessor();
    // The last rows of a request see the most keys: the last block_rows of every request come first, then those before them.
    int req = -1, row0 = 0, rows = 0;
    {
        int b = (int)blockIdx.y;
        for (int level = 0; req < 0; ++level) {
            bool any = false;
            for (int r = 0; r < p.n_requests; ++r) {
                const int lo = p.req_start[r], n = p.req_start[r + 1] - lo;
                const int tiles = (n + p.block_rows - 1) / p.block_rows;
                if (tiles <= level) continue;
                any = true;
                if (b-- == 0) {
                    req = r;
                    row0 = lo + (tiles - 1 - level) * p.block_rows;
                    rows = min(p.block_rows, lo + n - row0);
                    break;
                }
            }
            if (!any) return;
        }
    }
    const int h = blockIdx.x;
    const int p0 = p.req_prior[req] + (row0 - p.req_start[req]);
    const int p_last = p0 + rows - 1;
    const int key_from = (p.window > 0 && p0 + 1 > p.window) ? p0 + 1 - p.window : 0;
    const int kt_begin = key_from / BN;
    Rows part[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        const int skip = MAPS ? 0 : g * BM;
        part[g].n = max(0, min(BM, rows - skip));
        part[g].p0 = p0 + skip;
        const int from = (p.window > 0 && part[g].p0 + 1 > p.window) ? part[g].p0 + 1 - p.window : 0;
        part[g].begin = from / BN - kt_begin;
        part[g].end = part[g].n > 0 ? (part[g].p0 + part[g].n - 1) / BN - kt_begin : part[g].begin - 1;
    }
    const int n_tiles = max(part[0].end, part[1].end) + 1;        // the first softmax is never empty

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + S::BAR_AT);
    uint64_t* q_full = bars;                      // the queries landed
    uint64_t* k_full = bars + 1;                  // [KS] a chunk of keys landed
    uint64_t* k_empty = k_full + KS;              // [KS] the score products have read it
    uint64_t* v_full = k_empty + KS;              // [VS] 64 keys' values landed
    uint64_t* v_empty = v_full + VS;              // [VS] the output products have read them
    uint64_t* s_full = v_empty + VS;              // [2] a softmax's scores are complete (and every product before them)
    uint64_t* p_full = s_full + 2;                // [2][2] its weights of a tile's first / last 64 keys are written (and O rescaled)
    uint64_t* half_done = p_full + 4;             // [2] its output product over a tile's first 64 keys is done
    uint64_t* o_done = half_done + 2;             // [2] its last output product is done
    uint32_t* tmem_slot = (uint32_t*)(o_done + 2);
    float* inv2 = (float*)(smem + S::BAR_AT + 512);      // differential: 1 / divisor of the second map's rows
    static_assert((1 + 2 * KS + 2 * VS + 2 + 4 + 2 + 2) * 8 + 4 <= 512, "room for the barriers");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < KS; ++s) mbar_init(&k_full[s], 1), mbar_init(&k_empty[s], 1);
        for (int s = 0; s < VS; ++s) mbar_init(&v_full[s], 1), mbar_init(&v_empty[s], 1);
        for (int g = 0; g < 2; ++g) {
            mbar_init(&s_full[g], 1), mbar_init(&half_done[g], 1), mbar_init(&o_done[g], 1);
            mbar_init(&p_full[2 * g], BM), mbar_init(&p_full[2 * g + 1], BM);
        }
        fence_barrier_init();
    }
    if (warp == 2) tmem_alloc(tmem_slot, TM_COLS);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    // only now: a following kernel's block that took tensor memory first and waited for this kernel's end would starve this block
    cj::release_successor();
    const uint32_t tmem_base = *tmem_slot;

    const int kvh = MAPS ? h / (p.n_heads / p.n_kv) : 0;
    const int* tab = MAPS ? p.table + (size_t)req * p.table_stride : nullptr;
    const int base = MAPS ? 0 : p.req_base[req];
    // the plane's row of 16 keys from `key` on, or one past its end (read as zeros) where the block has no such keys
    auto plane_row = [&](int key) {
        if (key > p_last || key + 15 < key_from) return p.plane_rows;
        const int page = tab[key / p.page_tokens];
        return page >= 0 ? (page * p.n_kv + kvh) * p.page_tokens + key % p.page_tokens : p.plane_rows;
    };

    if (warp == 0) {
        // ---- queries, then keys, chunk by chunk -----------------------------------------------------
        // One lane issues; in the differential form a lane a page has looked up where the tile's pages lie (one lane doing both spent
        // 400 cycles a page on the lookup and its divisions: 71 us instead of 55 for 2,048 rows of 8 heads).
        const bool leader = elect_one();
        if (leader) {
            tma_prefetch_descriptor(&map_q);
            tma_prefetch_descriptor(&map_k);
            const int q_tiles = MAPS || part[1].n <= 0 ? 1 : 2;
            mbar_expect_tx(q_full, q_tiles * KC * CHUNK);
            for (int g = 0; g < q_tiles; ++g)
                for (int c = 0; c < KC; ++c)
                    tma_load_2d(smem + S::Q_AT + (g * KC + c) * CHUNK, &map_q, q_full, h * S::WIDTH + 64 * c, row0 + g * BM);
        }
        int slot = 0;
        uint32_t phase = 1;
        bool ok = true;
        int row = MAPS && lane < BN / 16 ? plane_row(kt_begin * BN + 16 * lane) : 0;
        for (int i = 0; i < n_tiles && ok; ++i) {
            const int key0 = (kt_begin + i) * BN;
            for (int c = 0; c < KC; ++c) {
                ok = mbar_wait_warp(&k_empty[slot], phase, 11);
                if (!ok) break;
                uint8_t* dst = smem + S::K_AT + slot * CHUNK;
                if (leader) mbar_expect_tx(&k_full[slot], CHUNK);
                if (MAPS) {
#pragma unroll
                    for (int k = 0; k < BN / 16; ++k) {
                        const int at = __shfl_sync(0xffffffffu, row, k);
                        if (leader) tma_load_2d(dst + k * 2048, &map_k, &k_full[slot], 64 * c, at);
                    }
                } else if (leader) {
                    if (c < KC - 1) tma_load_2d(dst, &map_k, &k_full[slot], h * (DK - 64) + 64 * c, base + key0);
                    else tma_load_2d(dst, &map_k2, &k_full[slot], 0, base + key0);
                }
                if (++slot == KS) slot = 0, phase ^= 1;
            }
            if (MAPS && lane < BN / 16) row = plane_row(key0 + BN + 16 * lane);
        }
    } else if (warp == 1) {
        // ---- values, 64 keys at a time --------------------------------------------------------------
        const bool leader = elect_one();
        if (leader) tma_prefetch_descriptor(&map_v);
        int slot = 0;
        uint32_t phase = 1;
        bool ok = true;
        int row = MAPS && lane < 4 ? plane_row(kt_begin * BN + 16 * lane) : 0;
        for (int i = 0; i < 2 * n_tiles && ok; ++i) {
            ok = mbar_wait_warp(&v_empty[slot], phase, 19);
            if (!ok) break;
            const int key0 = kt_begin * BN + i * 64;
            uint8_t* dst = smem + S::V_AT + slot * S::V_BYTES;
            if (leader) mbar_expect_tx(&v_full[slot], S::V_BYTES);
#pragma unroll
            for (int c = 0; c < DV / 64; ++c) {
                if (MAPS) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int at = __shfl_sync(0xffffffffu, row, k);
                        if (leader) tma_load_2d(dst + c * 8192 + k * 2048, &map_v, &v_full[slot], 64 * c, at);
                    }
                } else if (leader) {
                    tma_load_2d(dst + c * 8192, &map_v, &v_full[slot], h * DV + 64 * c, base + key0);
                }
            }
            if (++slot == VS) slot = 0, phase ^= 1;
            if (MAPS && lane < 4) row = plane_row(key0 + 64 + 16 * lane);
        }
    } else if (warp == 2) {
        // ---- products --------------------------------------------------------------------------------
        // In the order issued: S_a(0) S_b(0), then per key tile i: PV_a(i) S_a(i + 1) PV_b(i) S_b(i + 1), each PV in two halves of
        // 64 keys.  S_g(i + 1) overwrites the columns PV_g(i) reads the weights from; one thread's products run in the order they
        // were issued.  The whole warp walks the loop (it clears what the values' tiles must not hold); one lane issues.
        const bool leader = elect_one();
        bool ok = mbar_wait_warp(q_full, 0, 12);
        int k_slot = 0;                           // where the next tile's chunks lie, and the phase of the first
        uint32_t k_phase = 0;
        int v_slot = 0;
        uint32_t v_phase = 0, p_phase[2] = {0, 0};
        auto uses = [&](int g, int i) { return i >= part[g].begin && i <= part[g].end; };
        // the scores of softmax g over the tile whose chunks begin at k_slot
        auto scores = [&](int g) {
            const uint32_t acc = tmem_base + TM_S + g * BN;
            bool there = true;
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) {
                const int col = MAPS ? g * DK + 16 * k : 16 * k, c = col / 64, in = (col % 64) / 16;
                const int slot = k_slot + c >= KS ? k_slot + c - KS : k_slot + c;
                if ((k == 0 || in == 0) && there) {
                    there = mbar_wait_warp(&k_full[slot], k_phase ^ (k_slot + c >= KS ? 1u : 0u), 13);
                    tcgen05_fence_after();
                }
                if (there && leader)
                    umma_bf16(acc, umma_desc_sw128(smem + S::Q_AT + ((MAPS ? 0 : g * KC) + c) * CHUNK) + 2 * in,
                              umma_desc_sw128(smem + S::K_AT + slot * CHUNK) + 2 * in, IDESC_QK, k > 0);
            }
            if (there && leader) umma_commit(&s_full[g]);
            __syncwarp();
            return there;
        };
        auto keys_done = [&]() {                  // every chunk of the tile is free; on to the next tile
            for (int c = 0; c < KC; ++c) {
                if (leader) umma_commit(&k_empty[k_slot]);
                if (++k_slot == KS) k_slot = 0, k_phase ^= 1;
            }
        };
        // 64 keys' values have landed, and what are no keys of the block reads as zero
        auto values_there = [&](int slot, uint32_t phase, int key0) {
            if (!mbar_wait_warp(&v_full[slot], phase, 14)) return false;
            if (key0 < key_from || key0 + 63 > p_last) {
                uint8_t* v = smem + S::V_AT + slot * S::V_BYTES;
                for (int i = lane; i < 64 * (DV / 64) * 8; i += 32) {       // 16 bytes each
                    const int row = (i >> 3) & 63, key = key0 + row;
                    if (key < key_from || key > p_last) *(uint4*)(v + (i >> 9) * 8192 + row * 128 + (i & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_async_shared();
                __syncwarp();
            }
            return true;
        };
        if (ok) {
            tcgen05_fence_after();
#pragma unroll
            for (int g = 0; g < 2; ++g)
                if (ok && uses(g, 0)) ok = scores(g);
            if (ok) keys_done();
        }
        for (int i = 0; i < n_tiles && ok; ++i) {
            const bool next = i + 1 < n_tiles;
            bool there[2] = {false, false};
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                if (!ok) break;
                const uint32_t acc = tmem_base + TM_O + g * 128, pa = tmem_base + TM_S + g * BN;
                const bool mine = uses(g, i);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int slot = v_slot + half >= VS ? v_slot + half - VS : v_slot + half;
                    const uint32_t phase = v_phase ^ (v_slot + half >= VS ? 1u : 0u);
                    if (!there[half]) ok = values_there(slot, phase, (kt_begin + i) * BN + 64 * half);
                    there[half] = true;
                    if (!ok) break;
                    if (mine) {
                        ok = mbar_wait_warp(&p_full[2 * g + half], p_phase[g], 15);
                        if (!ok) break;
                        tcgen05_fence_after();
                        if (leader) {
                            const uint64_t dv = umma_desc_mn_sw128(smem + S::V_AT + slot * S::V_BYTES, 8192);
                            // 16 keys = 8 columns of weights = two 8-row groups of values = 2048 bytes
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                umma_bf16_a_tmem(acc, pa + 64 * half + 8 * k, dv + (uint64_t)(k * 2048 >> 4), IDESC_PV,
                                                 (i > part[g].begin || half > 0 || k > 0) ? 1u : 0u);
                                if (TWO) umma_bf16_a_tmem(acc, pa + 64 * half + 32 + 8 * k, dv + (uint64_t)(k * 2048 >> 4), IDESC_PV, 1u);
                            }
                            if (half == 0) umma_commit(&half_done[g]);
                        }
                    }
                    if (g == 1 && leader) umma_commit(&v_empty[slot]);
                    __syncwarp();
                }
                if (!ok) break;
                if (mine) {
                    p_phase[g] ^= 1;
                    if (i == part[g].end && leader) umma_commit(&o_done[g]);
                }
                if (next && uses(g, i + 1)) ok = scores(g);
                if (next && ok && g == 1) keys_done();
            }
            v_slot += 2;
            if (v_slot >= VS) v_slot -= VS, v_phase ^= 1;
        }
    } else {
        // ---- one softmax, one row per thread -----------------------------------------------------------
        const int g = (warp - 3) >> 2;
        const int quarter = warp & 3;                      // the quarter of the tensor-memory lanes this warp may touch
        const int r = quarter * 32 + lane;
        const Rows mine = g == 0 ? part[0] : part[1];
        const int pos = mine.p0 + r;
        const int from = (p.window > 0 && pos + 1 > p.window) ? pos + 1 - p.window : 0;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const uint32_t s_addr = tmem_base + TM_S + g * BN + lane_off;
        const uint32_t o_addr = tmem_base + TM_O + g * 128 + lane_off;
        float m_ref = -INFINITY, l = 0.0f;
        bool ok = true;
        const int n_mine = mine.end - mine.begin + 1;
        for (int j = 0; j < n_mine && ok; ++j) {
            ok = mbar_wait_warp(&s_full[g], j & 1, 16);
            if (!ok) break;
            tcgen05_fence_after();
            // columns [lo, lo + span] of this tile are keys this row may see (span < 0: none)
            const int kbase = (kt_begin + mine.begin + j) * BN;
            const int lo = max(from - kbase, 0);
            const int span = min(pos - kbase, BN - 1) - lo;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                constexpr int HC = BN / 2;
                uint32_t v[HC];
                tmem_ld32<0>(s_addr + half * HC, v);
                tmem_ld32<32>(s_addr + half * HC + 32, v);
                tmem_ld_wait();
                if (lo != 0 || span != BN - 1) {
#pragma unroll
                    for (int c = 0; c < HC; ++c)
                        if (!((unsigned)(half * HC + c - lo) <= (unsigned)span && span >= 0)) v[c] = 0xff800000u;       // -inf
                }
                // One pass with the reference maximum the row has so far gives the weights, their sum and these scores' maximum; only
                // when that raises the reference by more than the threshold (or the row had none yet) is the pass repeated.
                float m_use = m_ref, factor = 1.0f, sum;
                bool rescale = false;
                uint32_t hi[HC / 2], rest[HC / 2];
#pragma unroll 1
                for (int attempt = 0;; ++attempt) {
                    const float neg_sub = m_use == -INFINITY ? 0.0f : -m_use;
                    const f32x2 scale2 = pack2(p.scale_log2, p.scale_log2), sub2 = pack2(neg_sub, neg_sub);
                    f32x2 sum2a = pack2(0.0f, 0.0f), sum2b = sum2a;
                    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
                    for (int c = 0; c < HC; c += 4) {
                        const float2 t0 = unpack2(fma2(pack2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), scale2, sub2));
                        const float2 t1 = unpack2(fma2(pack2(__uint_as_float(v[c + 2]), __uint_as_float(v[c + 3])), scale2, sub2));
                        const float e0 = ex2(t0.x), e1 = ex2(t0.y), e2 = ex2(t1.x), e3 = ex2(t1.y);
                        sum2a = add2(sum2a, pack2(e0, e1));
                        sum2b = add2(sum2b, pack2(e2, e3));
                        hi[c >> 1] = pack_bf16(e0, e1);
                        hi[(c >> 1) + 1] = pack_bf16(e2, e3);
                        if (TWO) {
                            rest[c >> 1] = pack_rest(e0, e1, hi[c >> 1]);
                            rest[(c >> 1) + 1] = pack_rest(e2, e3, hi[(c >> 1) + 1]);
                        }
                        mx0 = max3(mx0, __uint_as_float(v[c]), __uint_as_float(v[c + 1]));
                        mx1 = max3(mx1, __uint_as_float(v[c + 2]), __uint_as_float(v[c + 3]));
                    }
                    const float2 sa = unpack2(sum2a), sb = unpack2(sum2b);
                    sum = (sa.x + sa.y) + (sb.x + sb.y);
                    if (attempt == 1) break;
                    const float mx = fmaxf(mx0, mx1) * p.scale_log2;          // scale > 0: the largest raw score is the largest score
                    float m_new = m_ref;
                    if (mx > m_ref + RESCALE_THRESHOLD || m_ref == -INFINITY) m_new = fmaxf(m_ref, mx);
                    if (!__any_sync(0xffffffffu, m_new != m_ref)) break;
                    rescale = m_new != m_ref && m_ref != -INFINITY;
                    factor = rescale ? exp2f(m_ref - m_new) : 1.0f;
                    m_use = m_new;
                }
                tmem_st32<0>(s_addr + half * HC, hi);
                if (TWO) tmem_st32<0>(s_addr + half * HC + 32, rest);
                l = l * factor + sum;
                m_ref = m_use;
                // O may be rescaled once the product before is done: the one over the last tile's second half was done before this
                // tile's scores were; the one over this tile's first half is waited for here
                if (half == 1) {
                    ok = mbar_wait_warp(&half_done[g], j & 1, 17);
                    if (!ok) break;
                    tcgen05_fence_after();
                }
                if (__any_sync(0xffffffffu, rescale)) {        // rare
#pragma unroll 1
                    for (int c0 = 0; c0 < DV; c0 += 16) {
                        uint32_t o[16];
                        tmem_ld16(o_addr + c0, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int q = 0; q < 16; ++q) o[q] = __float_as_uint(__uint_as_float(o[q]) * factor);
                        tmem_st16(o_addr + c0, o);
                    }
                }
                tmem_st_wait();
                tcgen05_fence_before();
                mbar_arrive(&p_full[2 * g + half]);
            }
        }
        // ---- the rows' results ---------------------------------------------------------------------------
        if (ok && n_mine > 0) ok = mbar_wait_warp(&o_done[g], 0, 18);
        if (MAPS) {
            // the second map's warps hand over what divides their rows; the first map's read both outputs from tensor memory
            if (g == 1) inv2[r] = ok && l > 0.0f ? 1.0f / l : 0.0f;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (g == 0 && ok) ok = mbar_wait_warp(&o_done[1], 0, 18);
            if (g == 0 && ok) {
                tcgen05_fence_after();
                const float ia = l > 0.0f ? 1.0f / l : 0.0f, ib = inv2[r];
                float d[DV], ss = 0.0f;
#pragma unroll
                for (int c0 = 0; c0 < DV; c0 += 16) {
                    uint32_t oa[16], ob[16];
                    tmem_ld16(o_addr + c0, oa);
                    tmem_ld16(o_addr + 128 + c0, ob);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        d[c0 + q] = __uint_as_float(oa[q]) * ia - p.lambda * (__uint_as_float(ob[q]) * ib);
                        ss = fmaf(d[c0 + q], d[c0 + q], ss);
                    }
                }
                const float norm = p.out_scale / sqrtf(ss / (float)DV + p.eps);
                if (r < mine.n) {
                    __nv_bfloat16* dst = p.out + ((size_t)(row0 + r) * p.n_heads + h) * DV;
#pragma unroll
                    for (int c0 = 0; c0 < DV; c0 += 8)
                        *(uint4*)(dst + c0) = make_uint4(pack_bf16(d[c0] * norm, d[c0 + 1] * norm), pack_bf16(d[c0 + 2] * norm, d[c0 + 3] * norm),
                                                         pack_bf16(d[c0 + 4] * norm, d[c0 + 5] * norm), pack_bf16(d[c0 + 6] * norm, d[c0 + 7] * norm));
                }
            }
        } else if (ok && n_mine > 0) {
            tcgen05_fence_after();
            const int row = row0 + g * BM + r;
            const bool live = r < mine.n;
            if (p.sink) l += exp2f(p.sink[h] * 1.4426950408889634f - m_ref);           // the key without a value
            float inv = l > 0.0f ? 1.0f / l : 0.0f;
            __nv_bfloat16* dst = p.out + ((size_t)row * p.n_heads + h) * DV;
            if (p.gate && live) inv *= 1.0f / (1.0f + expf(-p.gate[(size_t)row * p.gate_ld + h]));
#pragma unroll 1
            for (int c0 = 0; c0 < DV; c0 += 16) {
                uint32_t o[16];
                tmem_ld16(o_addr + c0, o);
                tmem_ld_wait();
                if (live) {
                    float x[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) x[q] = __uint_as_float(o[q]) * inv;
                    *(uint4*)(dst + c0) = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
                    *(uint4*)(dst + c0 + 8) = make_uint4(pack_bf16(x[8], x[9]), pack_bf16(x[10], x[11]), pack_bf16(x[12], x[13]), pack_bf16(x[14], x[15]));
                }
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 2) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, TM_COLS);
    }
}

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 1;
    }
    return n;
}

template <bool MAPS, int DK, int DV, bool TWO>
int start(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mk2, const CUtensorMap& mv, const Args& a, long long row_blocks,
          cudaStream_t stream) {
    auto kern = flash_tc_kernel<MAPS, DK, DV, TWO>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<MAPS, DK, DV>::SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    // heads run fastest: blocks start in the order of their length
    cj::launch(kern, dim3(a.n_heads, (unsigned)row_blocks), dim3(THREADS), Shape<MAPS, DK, DV>::SMEM, stream, mq, mk, mk2, mv, a);
    return cj::launch_status();
}

}  // namespace

// Differential attention of prompt portions: as cj_diff_attention_tile (attention_diff.cu) without stretches of keys; hd 64 or 128,
// vd 64 or 128, pages of a multiple of 16 tokens.
CJ_EXPORT int cj_diff_attention_tc(const void* q, void* out, const void* kplane, const void* vplane, int n_pages, const int* req_start,
                                   const int* req_prior, int n_requests, int T, const int* table, int table_stride, int page_tokens,
                                   int n_heads, int n_kv, int hd, int vd, int window, float scale, float lambda, float eps, float out_scale,
                                   cudaStream_t stream) {
    if (T <= 0 || n_requests <= 0) return 0;
    if (!q || !out || !kplane || !vplane || !req_start || !req_prior || !table) return CJ_ERR_ARG;
    if (n_heads <= 0 || n_kv <= 0 || n_heads % n_kv != 0 || n_pages <= 0 || page_tokens <= 0 || page_tokens % 16 != 0 || window < 0 || !(scale > 0.0f))
        return CJ_ERR_SIZE;
    if ((hd != 64 && hd != 128) || (vd != 64 && vd != 128)) return CJ_ERR_SIZE;
    if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)kplane | (uintptr_t)vplane) & 15) return CJ_ERR_ALIGN;
    const long long plane_rows = (long long)n_pages * n_kv * page_tokens, row_blocks = ((long long)T + BM - 1) / BM + n_requests;
    if (plane_rows > 0x7fffffffLL || row_blocks > 65535) return CJ_ERR_SIZE;
    CUtensorMap mq, mk, mv;
    if (!make_map_bf16(&mq, q, T, (long long)n_heads * 2 * hd, (long long)n_heads * 2 * hd, BM)) return CJ_ERR_ARG;
    if (!make_map_bf16(&mk, kplane, plane_rows, 2 * hd, 2 * hd, 16)) return CJ_ERR_ARG;
    if (!make_map_bf16(&mv, vplane, plane_rows, vd, vd, 16)) return CJ_ERR_ARG;
    Args a{};
    a.out = (__nv_bfloat16*)out;
    a.req_start = req_start, a.req_prior = req_prior, a.n_requests = n_requests, a.n_heads = n_heads, a.window = window;
    a.scale_log2 = scale * 1.4426950408889634f;
    a.block_rows = BM;
    a.table = table, a.table_stride = table_stride, a.page_tokens = page_tokens, a.n_kv = n_kv, a.plane_rows = (int)plane_rows;
    a.lambda = lambda, a.eps = eps, a.out_scale = out_scale;
    if (hd == 64) return vd == 64 ? start<true, 64, 64, true>(mq, mk, mk, mv, a, row_blocks, stream) : start<true, 64, 128, true>(mq, mk, mk, mv, a, row_blocks, stream);
    return vd == 64 ? start<true, 128, 64, true>(mq, mk, mk, mv, a, row_blocks, stream) : start<true, 128, 128, true>(mq, mk, mk, mv, a, row_blocks, stream);
}

// Latent attention's plain form.  q [T, heads, dim + 64]; kp [N, heads * dim], kr [N, 64] (the key part that the heads share), vp
// [N, heads * vdim]; out [T, heads * vdim]; all bfloat16.  dim and vdim 64 or 128.  Request i's token p lies at row req_base[i] + p.
// exact: weights as two bfloat16 terms.  sink: null or [heads]; gate: null or float32 with row stride gate_ld, a column a head.
CJ_EXPORT int cj_latent_attention_tc(const void* q, void* out, const void* kp, const void* kr, const void* vp, int N, const int* req_start,
                                     const int* req_prior, const int* req_base, int n_requests, int T, int heads, int dim, int vdim,
                                     int window, int exact, float scale, const float* sink, const float* gate, int gate_ld, cudaStream_t stream) {
    if (T <= 0 || n_requests <= 0) return 0;
    if (!q || !out || !kp || !kr || !vp || !req_start || !req_prior || !req_base || N <= 0) return CJ_ERR_ARG;
    if (heads <= 0 || window < 0 || !(scale > 0.0f) || (dim != 64 && dim != 128) || (vdim != 64 && vdim != 128)) return CJ_ERR_SIZE;
    if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)kp | (uintptr_t)kr | (uintptr_t)vp) & 15) return CJ_ERR_ALIGN;
    CUtensorMap mq, mk, mr, mv;
    const long long w = (long long)heads * (dim + 64);
    if (!make_map_bf16(&mq, q, T, w, w, BM)) return CJ_ERR_ARG;
    if (!make_map_bf16(&mk, kp, N, (long long)heads * dim, (long long)heads * dim, BN)) return CJ_ERR_ARG;
    if (!make_map_bf16(&mr, kr, N, 64, 64, BN)) return CJ_ERR_ARG;
    if (!make_map_bf16(&mv, vp, N, (long long)heads * vdim, (long long)heads * vdim, 64)) return CJ_ERR_ARG;
    Args a{};
    a.out = (__nv_bfloat16*)out;
    a.req_start = req_start, a.req_prior = req_prior, a.n_requests = n_requests, a.n_heads = heads, a.window = window;
    a.scale_log2 = scale * 1.4426950408889634f;
    // two tiles a block, unless that leaves more than half of the SMs without one
    const long long blocks_256 = (((long long)T + 255) / 256 + n_requests - 1) * heads;
    a.block_rows = 2 * blocks_256 <= sm_count() ? 128 : 256;
    const long long row_blocks = ((long long)T + a.block_rows - 1) / a.block_rows + n_requests;
    if (row_blocks > 65535) return CJ_ERR_SIZE;
    a.req_base = req_base, a.sink = sink, a.gate = gate, a.gate_ld = gate_ld;
#define START(D_, V_) (exact ? start<false, D_, V_, true>(mq, mk, mr, mv, a, row_blocks, stream) : start<false, D_, V_, false>(mq, mk, mr, mv, a, row_blocks, stream))
    if (dim == 64) return vdim == 64 ? START(128, 64) : START(128, 128);
    return vdim == 64 ? START(192, 64) : START(192, 128);
#undef START
}

CJ_EXPORT int cj_attention_flash_tc_error() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, tc::g_error_flag, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
