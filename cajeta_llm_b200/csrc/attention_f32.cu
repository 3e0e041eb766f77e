// Paged attention of the float32 path: float32 queries, cache and arithmetic, head sizes up to 128 that are multiples of four.
// The formulas are attention_paged.cu's (window, capped scores, a gate per row and head, a constant sink score).
//
// Two kernels, one result.  A portion of a prompt goes 64 or 32 rows of a request and one head a block, so that a key read from the cache
// serves as many rows; a request with few rows (a decoded token) goes a row and head a block, its warps sharing the keys.  A row
// must not depend on which of the two ran or on how its prompt was cut, so both do the same float32 operations for it, in this order:
//   keys in chunks of 64 that begin at multiples of 64;  s_t = (q . k_t) scale, one chain of fused multiply-adds over the head;
//   in a chunk m_c = max s_t, e_t = exp(s_t - m_c), l_c = sum e_t by a fixed tree, o_c = sum e_t v_t one chain over its keys;
//   chunks joined in order:  m' = max(m, m_c), l = l exp(m - m') + l_c exp(m_c - m'), o likewise.
// A score of -inf (a product that overflows) is a key without weight.
// Keys outside a row's [from, p] enter none of its sums (they are skipped, not multiplied by zero).
//
// The prompt form keeps a thread on 4 rows x 4 keys of the scores and 4 rows x 8 entries of the output, operands as float4 from
// shared memory, which gives an SM 128 bytes a clock: eight of them (32 clocks a warp) for 16 clocks of FMA, so shared memory bounds it, 315 us
// for the 1,777 rows of one prompt with 16 heads of 128; it takes 685, 785 before a chunk's keys travelled while the chunk before was summed up
// and its values while its scores were worked out (cold; a row and head a block with a key a lane took 12,700).  256 rows at 700 keys:
// 199 -> 134 us.  One row at 570 keys: 73 -> 33 us, at 4,000 293 -> 156.
#define CJ_LIB "attention_f32"
#include "common.cuh"

#include <type_traits>

using namespace cj;

namespace {

constexpr int KEYS = 64, MAX_DIM = 128;

struct Args {
    const float* q; float* out; const float* kplane; const float* vplane;
    const int* positions; const int* row_req; const int* req_start; int requests;
    const int* table; int table_stride, page_tokens;
    int n_heads, n_kv, hd, vd, window;
    float scale, softcap;
    const float* head_gate; int gate_ld;
    float sink;
    int few_rows;                  // requests with at most this many rows go row by row
};

__device__ __forceinline__ float score(float dot, const Args& p) {
    // (products rounded by themselves: contracted into the subtraction that follows, the two kernels could differ)
    float s = __fmul_rn(dot, p.scale);
    if (p.softcap > 0.0f) s = __fmul_rn(p.softcap, tanhf(s / p.softcap));
    return s;
}
// e^(s - top); with a top of -inf (every score so far is) zero: such a key has no weight, and the keys after it keep theirs
__device__ __forceinline__ float weight(float s, float top) { return expf(s - (top == -INFINITY ? 0.0f : top)); }
__device__ __forceinline__ int first_key(int pos, int window) { return window > 0 && pos + 1 > window ? pos + 1 - window : 0; }
__device__ __forceinline__ float chain4(float4 a, float4 b, float s) {
    s = fmaf(a.x, b.x, s);
    s = fmaf(a.y, b.y, s);
    s = fmaf(a.z, b.z, s);
    return fmaf(a.w, b.w, s);
}
__device__ __forceinline__ float gate_of(const Args& p, int row, int head) {
    return p.head_gate ? 1.0f / (1.0f + expf(-p.head_gate[(size_t)row * p.gate_ld + head])) : 1.0f;
}

// 16 bytes on their way to shared memory, zeros where `valid` is not set
__device__ __forceinline__ void cp_async16(float* smem, const float* gmem, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// VC: float4 of the output a thread holds per row (values of up to 64 VC entries); ROWS: rows of a tile, 64 or 32
template <int VC, int ROWS>
__global__ void __launch_bounds__(4 * ROWS, 2) attention_f32_tile_kernel(const Args p) {
    constexpr int TILE_THREADS = 4 * ROWS;
    cj::after_predecessor();
    cj::release_successor();
    extern __shared__ __align__(16) float smem[];
    const int ks = p.hd + 4;                        // row stride of queries and keys: 16 rows apart never share a bank
    float* Qs = smem;                               // [ROWS][ks]
    float* Ks = Qs + ROWS * ks;                     // [KEYS][ks]
    float* Vs = Ks + KEYS * ks;                     // [KEYS][vd]
    float* Ps = Vs + KEYS * p.vd;                   // [ROWS][KEYS + 4]
    __shared__ int place[3];                        // request, first row of the tile, rows

    const int tid = threadIdx.x, lane = tid & 31;
    const int head = blockIdx.y, kvh = head / (p.n_heads / p.n_kv);
    if (tid < 32) {
        // which rows: tile gridDim.x - 1 - blockIdx.x (a prompt's last rows, with the most keys, first) over all requests
        const int tile = gridDim.x - 1 - blockIdx.x;
        int before = 0, req = -1, row = 0, rows = 0;
        for (int r0 = 0; r0 < p.requests; r0 += 32) {
            const int r = r0 + lane;
            const int a = r < p.requests ? p.req_start[r] : 0, c = r < p.requests ? p.req_start[r + 1] - a : 0;
            const int n = c > p.few_rows ? (c + ROWS - 1) / ROWS : 0;
            int inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            const int t = tile - (before + inc - n);
            const unsigned who = __ballot_sync(0xffffffffu, t >= 0 && t < n);
            if (who) {
                const int l = __ffs(who) - 1;
                req = r0 + l;
                row = __shfl_sync(0xffffffffu, t, l) * ROWS;
                rows = min(ROWS, __shfl_sync(0xffffffffu, c, l) - row);
                row += __shfl_sync(0xffffffffu, a, l);
                break;
            }
            before += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) { place[0] = req; place[1] = row; place[2] = rows; }
    }
    __syncthreads();
    const int row0 = place[1], rows = place[2];
    if (place[0] < 0) return;
    const int* tab = p.table + (size_t)place[0] * p.table_stride;
    const int pos0 = p.positions[row0];             // the tile's rows are neighbours
    const int hd4 = p.hd / 4;
    for (int i = tid; i < ROWS * hd4; i += TILE_THREADS) {
        const int r = i / hd4, d = i - r * hd4;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < rows) v = *(const float4*)(p.q + ((size_t)(row0 + r) * p.n_heads + head) * p.hd + 4 * d);
        *(float4*)(Qs + r * ks + 4 * d) = v;
    }
    const int tx = tid & 15, ty = tid >> 4;
    const int first = first_key(pos0, p.window), last = pos0 + rows - 1;
    float m[4], l[4], acc[4][VC][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = p.sink;
        l[i] = p.sink == -INFINITY ? 0.0f : 1.0f;
#pragma unroll
        for (int c = 0; c < VC; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][c][e] = 0.0f;
    }
    // a chunk's keys travel while the chunk before is summed up, its values while its scores are worked out; four threads a key
    auto fetch = [&](int k0, const float* plane, int size, float* to, int stride) {
        const int size4 = size / 4;
        for (int i = tid; i < KEYS * 4; i += TILE_THREADS) {
            const int j = i >> 2, key = k0 + j;
            const bool held = key >= first && key <= last;
            size_t base = 0;
            if (held) base = ((size_t)tab[key / p.page_tokens] * p.n_kv + kvh) * p.page_tokens + key % p.page_tokens;
            const float* from = plane + base * size;
#pragma unroll 8
            for (int d = i & 3; d < size4; d += 4) cp_async16(to + j * stride + 4 * d, from + 4 * d, held);
        }
        cp_async_commit();
    };
    const int k_first = first & ~(KEYS - 1);
    fetch(k_first, p.kplane, p.hd, Ks, ks);
    for (int k0 = k_first; k0 <= last; k0 += KEYS) {
        if (k0 > k_first) __syncthreads();          // the values of the chunk before have been read
        fetch(k0, p.vplane, p.vd, Vs, p.vd);
        cp_async_wait<1>();
        __syncthreads();                            // the chunk's keys (and, the first time, the queries)
        // scores: rows 4 ty + i, keys tx + 16 j
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
#pragma unroll 2
        for (int d = 0; d < p.hd; d += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *(const float4*)(Qs + (4 * ty + i) * ks + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *(const float4*)(Ks + (tx + 16 * j) * ks + d);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = chain4(a[i], b[j], s[i][j]);
        }
        __syncthreads();                            // the keys have been read
        if (k0 + KEYS <= last) fetch(k0 + KEYS, p.kplane, p.hd, Ks, ks);
        else cp_async_commit();
        float keep[4], take[4];                     // factors of the sums so far and of this chunk's
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + 4 * ty + i, from = first_key(pos, p.window);
            float mc = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + tx + 16 * j;
                s[i][j] = key >= from && key <= pos ? score(s[i][j], p) : -INFINITY;
                mc = fmaxf(mc, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mc = fmaxf(mc, __shfl_xor_sync(0xffffffffu, mc, o));
            float e[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + tx + 16 * j;
                e[j] = key >= from && key <= pos ? weight(s[i][j], mc) : 0.0f;
                Ps[(4 * ty + i) * (KEYS + 4) + tx + 16 * j] = e[j];
            }
            float lc = __fadd_rn(__fadd_rn(e[0], e[2]), __fadd_rn(e[1], e[3]));
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) lc = __fadd_rn(lc, __shfl_xor_sync(0xffffffffu, lc, o));
            const bool any = from < k0 + KEYS && pos >= k0;          // the row sees a key of this chunk
            const float mn = any ? fmaxf(m[i], mc) : m[i];
            keep[i] = any ? weight(m[i], mn) : 1.0f;
            take[i] = any ? weight(mc, mn) : 0.0f;
            if (any) {
                l[i] = fmaf(lc, take[i], __fmul_rn(l[i], keep[i]));
                m[i] = mn;
            }
        }
        cp_async_wait<1>();
        __syncthreads();                            // the chunk's values (a row's weights were written by its warp's own lanes)
        float o[4][VC][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < VC; ++c)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[i][c][e] = 0.0f;
        // whether every row of the tile sees every key of the chunk
        const bool all = k0 + KEYS - 1 <= pos0 && k0 >= first_key(last, p.window);
        auto values = [&](auto whole) {
            constexpr bool ALL = decltype(whole)::value;
#pragma unroll 1
            for (int k = 0; k < KEYS; k += 4) {
                float4 w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = *(const float4*)(Ps + (4 * ty + i) * (KEYS + 4) + k);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    float4 v[VC];
#pragma unroll
                    for (int c = 0; c < VC; ++c) {
                        const int d = 4 * tx + 64 * c;
                        v[c] = d < p.vd ? *(const float4*)(Vs + (k + kk) * p.vd + d) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float e = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
                        const int key = k0 + k + kk, pos = pos0 + 4 * ty + i;
                        if (ALL || (key <= pos && key >= first_key(pos, p.window))) {
#pragma unroll
                            for (int c = 0; c < VC; ++c) {
                                o[i][c][0] = fmaf(e, v[c].x, o[i][c][0]);
                                o[i][c][1] = fmaf(e, v[c].y, o[i][c][1]);
                                o[i][c][2] = fmaf(e, v[c].z, o[i][c][2]);
                                o[i][c][3] = fmaf(e, v[c].w, o[i][c][3]);
                            }
                        }
                    }
                }
            }
        };
        if (all) values(std::true_type{});         // (the test a row and key is what the other chunks pay for)
        else values(std::false_type{});
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + 4 * ty + i;
            if (!(first_key(pos, p.window) < k0 + KEYS && pos >= k0)) continue;
#pragma unroll
            for (int c = 0; c < VC; ++c)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][c][e] = fmaf(o[i][c][e], take[i], __fmul_rn(acc[i][c][e], keep[i]));
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * ty + i;
        if (r >= rows) continue;
        const float inv = __fmul_rn(1.0f / l[i], gate_of(p, row0 + r, head));
        float* o = p.out + ((size_t)(row0 + r) * p.n_heads + head) * p.vd;
#pragma unroll
        for (int c = 0; c < VC; ++c) {
            const int d = 4 * tx + 64 * c;
            if (d < p.vd)
                *(float4*)(o + d) = make_float4(__fmul_rn(acc[i][c][0], inv), __fmul_rn(acc[i][c][1], inv), __fmul_rn(acc[i][c][2], inv),
                                                __fmul_rn(acc[i][c][3], inv));
        }
    }
}

// floats of a piece of a warp's chunk of keys or values in the kernel below
__host__ __device__ constexpr int piece_floats(int piece, int hd, int vd) { return piece * (hd + 4 > vd ? hd + 4 : vd); }

// A row and head a block: a warp a chunk of 64 keys, lane = keys lane and lane + 32 for the scores and four entries of the value for
// the sums; after every round of chunks thread d joins them, in order, into entry d of the output.  A chunk comes in pieces of PIECE keys, a warp
// a key (512 bytes side by side).  BUFS 2: its two halves of keys are sent for together and its values as soon as the keys have been read, so
// that a chunk is two round trips to memory; with a lane reading its own key's row, eight pieces at a time, it was twelve, in lines of 128 bytes
// for 16.  BUFS 1: one piece at a time, for room (a lane holds keys lane and lane + 32 whatever the piece).  Bound by the round trips with few blocks, by what an SM draws from memory with many.
template <int ROW_WARPS, int PIECE, int BUFS>
__global__ void __launch_bounds__(ROW_WARPS * 32) attention_f32_row_kernel(const Args p) {
    constexpr int PIECES = (KEYS + PIECE - 1) / PIECE;
    static_assert(PIECE <= 32 && (BUFS == 1 || PIECES == BUFS), "a lane has a key of a piece; all pieces of a chunk in buffers of their own, or one at a time");
    cj::after_predecessor();
    cj::release_successor();
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) float qs[MAX_DIM];
    __shared__ __align__(16) float oc[ROW_WARPS][MAX_DIM];
    __shared__ float mc_s[ROW_WARPS], lc_s[ROW_WARPS];
    __shared__ int place[2];
    const int head = blockIdx.y, kvh = head / (p.n_heads / p.n_kv);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (p.req_start) {
        // the rows of requests with few rows, in order: which is this block's
        if (warp == 0) {
            int before = 0, row = -1, req = 0;
            for (int r0 = 0; r0 < p.requests; r0 += 32) {
                const int r = r0 + lane;
                const int a = r < p.requests ? p.req_start[r] : 0, c = r < p.requests ? p.req_start[r + 1] - a : 0;
                const int n = c <= p.few_rows ? max(c, 0) : 0;
                int inc = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += v;
                }
                const int t = (int)blockIdx.x - (before + inc - n);
                const unsigned who = __ballot_sync(0xffffffffu, t >= 0 && t < n);
                if (who) {
                    const int l = __ffs(who) - 1;
                    req = r0 + l;
                    row = __shfl_sync(0xffffffffu, a + t, l);
                    break;
                }
                before += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (lane == 0) { place[0] = row; place[1] = req; }
        }
        __syncthreads();
        if (place[0] < 0) return;
    }
    const int row = p.req_start ? place[0] : blockIdx.x, req = p.req_start ? place[1] : p.row_req[row];
    const int pos = p.positions[row], from = first_key(pos, p.window);
    const int* tab = p.table + (size_t)req * p.table_stride;
    if (tid < p.hd / 4) *(float4*)(qs + 4 * tid) = *(const float4*)(p.q + ((size_t)row * p.n_heads + head) * p.hd + 4 * tid);
    __syncthreads();
    float* bufs[2];
    bufs[0] = smem + warp * BUFS * piece_floats(PIECE, p.hd, p.vd);
    bufs[1] = bufs[0] + (BUFS - 1) * piece_floats(PIECE, p.hd, p.vd);
    const int ks = p.hd + 4;
    float m = p.sink, l = p.sink == -INFINITY ? 0.0f : 1.0f, acc = 0.0f;
    for (int k0 = from & ~(KEYS - 1); k0 <= pos; k0 += KEYS * ROW_WARPS) {
        const int c0 = k0 + warp * KEYS;
        if (c0 <= pos) {
            float s[2], e[2];
            size_t base[2];
            bool seen[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int key = c0 + lane + 32 * j;
                seen[j] = key >= from && key <= pos;
                base[j] = 0;
                if (seen[j]) base[j] = ((size_t)tab[key / p.page_tokens] * p.n_kv + kvh) * p.page_tokens + key % p.page_tokens;
            }
            // whether key k of the chunk, in the piece that begins at `first`, is one of its second half
            auto half = [](int first, int k) { return (PIECE == 32 ? first : k) >= 32; };
            unsigned there[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) there[j] = __ballot_sync(0xffffffffu, seen[j]);
            // the chunk's keys or values [first, first + PIECE) into buffer h
            auto fetch = [&](int h, int first, const float* plane, int size, int stride) {
                __syncwarp();                       // what the buffer held has been read
#pragma unroll 4
                for (int j = 0; j < PIECE; ++j) {
                    const int k = first + j;
                    if (PIECE * PIECES > KEYS && k >= KEYS) break;
                    const size_t b = __shfl_sync(0xffffffffu, (unsigned long long)(half(first, k) ? base[1] : base[0]), k & 31);
                    if (4 * lane < size && ((half(first, k) ? there[1] : there[0]) >> (k & 31) & 1))
                        cp_async16(bufs[h] + j * stride + 4 * lane, plane + b * size + 4 * lane, true);
                }
                cp_async_commit();
            };
            fetch(0, 0, p.kplane, p.hd, ks);
            if (BUFS == 2) fetch(1, PIECE, p.kplane, p.hd, ks);
            s[0] = s[1] = -INFINITY;
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const int h = BUFS == 2 ? i : 0;
                cp_async_wait<BUFS - 1>();
                __syncwarp();
                const int row = (lane - i * PIECE) & 31, k = i * PIECE + row;          // this lane's key of the piece
                const bool second = half(i * PIECE, k);
                if (row < PIECE && k < KEYS && (second ? seen[1] : seen[0])) {
                    float dot = 0.0f;
                    const float* kr = bufs[h] + row * ks;
#pragma unroll 8
                    for (int d = 0; d < p.hd; d += 4) dot = chain4(*(const float4*)(qs + d), *(const float4*)(kr + d), dot);
                    dot = score(dot, p);
                    if (second) s[1] = dot; else s[0] = dot;
                }
                if (BUFS == 2) fetch(h, i * PIECE, p.vplane, p.vd, p.vd);
                else if (i + 1 < PIECES) fetch(0, (i + 1) * PIECE, p.kplane, p.hd, ks);
                else fetch(0, 0, p.vplane, p.vd, p.vd);
            }
            const float mc = warp_max(fmaxf(s[0], s[1]));
            e[0] = seen[0] ? weight(s[0], mc) : 0.0f;
            e[1] = seen[1] ? weight(s[1], mc) : 0.0f;
            // the tree of the other kernel: keys 32 apart, then 16 apart, then 1, 2, 4, 8
            float lc = __fadd_rn(e[0], e[1]);
            lc = __fadd_rn(lc, __shfl_xor_sync(0xffffffffu, lc, 16));
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) lc = __fadd_rn(lc, __shfl_xor_sync(0xffffffffu, lc, o));
            if (lane == 0) { mc_s[warp] = mc; lc_s[warp] = lc; }
            float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const bool mine = 4 * lane < p.vd;
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const int h = BUFS == 2 ? i : 0;
                if (BUFS == 1 && i > 0) fetch(0, i * PIECE, p.vplane, p.vd, p.vd);
                if (BUFS == 2 && i == 0) cp_async_wait<1>(); else cp_async_wait<0>();
                __syncwarp();
                const int lo = max(from - c0, i * PIECE), hi = min(pos - c0, min(KEYS, (i + 1) * PIECE) - 1);
#pragma unroll 4
                for (int k = lo; k <= hi; ++k) {
                    const float w = __shfl_sync(0xffffffffu, half(i * PIECE, k) ? e[1] : e[0], k & 31);
                    if (mine) {
                        const float4 v = *(const float4*)(bufs[h] + (k - i * PIECE) * p.vd + 4 * lane);
                        o.x = fmaf(w, v.x, o.x);
                        o.y = fmaf(w, v.y, o.y);
                        o.z = fmaf(w, v.z, o.z);
                        o.w = fmaf(w, v.w, o.w);
                    }
                }
            }
            if (mine) *(float4*)(oc[warp] + 4 * lane) = o;
        }
        __syncthreads();
        const int n = min(ROW_WARPS, (pos - k0) / KEYS + 1);
        for (int c = 0; c < n; ++c) {
            const float mc = mc_s[c], mn = fmaxf(m, mc), keep = weight(m, mn), take = weight(mc, mn);
            l = fmaf(lc_s[c], take, __fmul_rn(l, keep));
            if (tid < p.vd) acc = fmaf(oc[c][tid], take, __fmul_rn(acc, keep));
            m = mn;
        }
        __syncthreads();
    }
    if (tid < p.vd)
        p.out[((size_t)row * p.n_heads + head) * p.vd + tid] = __fmul_rn(acc, __fmul_rn(1.0f / l, gate_of(p, row, head)));
}

// multiprocessors, and the shared memory of one
int machine(int& n, int& bytes) {
    static int sms = 0, sm_bytes = 0;
    if (!sms) {
        int dev = 0, count = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        sms = count;
    }
    n = sms;
    bytes = sm_bytes;
    return 0;
}

}  // namespace

// Arguments as cj_paged_attention's, float32 throughout; req_start [requests + 1]: the step's rows by request (neighbouring rows of a
// request at neighbouring positions), or null: every row goes by itself.  tiles: an upper bound of the 64-row tiles of the
// requests with more than few_rows rows, 0 for none, tiles32 the same of 32 rows; singles: the rows of the others.
CJ_EXPORT int cj_attention_f32(const float* q, float* out, const float* kplane, const float* vplane, const int* positions, const int* row_req,
                               const int* req_start, int requests, const int* table, int table_stride, int page_tokens, int T, int n_heads,
                               int n_kv, int hd, int vd, int window, float scale, float softcap, const float* head_gate, int gate_ld,
                               float sink, int few_rows, int tiles, int tiles32, int singles, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (!q || !out || !kplane || !vplane || !positions || !row_req || !table || (tiles > 0 && !req_start)) return CJ_ERR_ARG;
    if (hd <= 0 || hd > MAX_DIM || hd % 4 != 0 || vd <= 0 || vd > MAX_DIM || vd % 4 != 0) return CJ_ERR_SIZE;
    if (n_heads <= 0 || n_heads > 65535 || n_kv <= 0 || n_heads % n_kv != 0 || page_tokens <= 0) return CJ_ERR_SIZE;
    if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)kplane | (uintptr_t)vplane) & 15) return CJ_ERR_ALIGN;
    Args a{q, out, kplane, vplane, positions, row_req, req_start, requests, table, table_stride, page_tokens, n_heads, n_kv, hd, vd, window,
           scale, softcap, head_gate, gate_ld, sink, few_rows};
    if (tiles > 0) {
        // Tiles of 64 rows where an SM holds two of them and the step has two for every SM, else of 32.  What an SM holds is what hides the
        // waits for keys: with heads of 128 a tile of 64 rows takes 115 KB and is alone (before keys travelled ahead: 1,777 rows of 16 heads 728 us,
        // with tiles of 32 713; 768 rows 187 and 172; 256 rows at 950 keys 185 and 137), with heads of 96 two fit (1,777 rows at 2,277 keys 925, 987).
        int sms, sm_bytes;
        if (int st = machine(sms, sm_bytes)) return st;
        auto smem = [](int rows, int h, int v) { return (int)sizeof(float) * ((rows + KEYS) * (h + 4) + KEYS * v + rows * (KEYS + 4)); };
        const bool two = 2 * (smem(64, hd, vd) + 1024) <= sm_bytes;
        const int rows = two && (long long)tiles * n_heads >= 2 * sms ? 64 : 32, wide = vd <= 64 ? 0 : 1;
        auto kern = rows == 64 ? (wide ? attention_f32_tile_kernel<2, 64> : attention_f32_tile_kernel<1, 64>)
                               : (wide ? attention_f32_tile_kernel<2, 32> : attention_f32_tile_kernel<1, 32>);
        static bool sized[2][2] = {};
        if (!sized[rows == 64][wide]) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(rows, MAX_DIM, MAX_DIM));
            if (e != cudaSuccess) return (int)e;
            sized[rows == 64][wide] = true;
        }
        cj::launch(kern, dim3(rows == 64 ? tiles : tiles32, n_heads), dim3(4 * rows), smem(rows, hd, vd), stream, a);
        if (int st = launch_status()) return st;
    }
    if (tiles <= 0) a.req_start = nullptr;                     // no tile: every row by itself, whatever its request has
    if (singles > 0 || tiles <= 0) {
        const int rows = a.req_start ? singles : T;
#define ROWS(W, PIECE, BUFS)                                                                                            \
    do {                                                                                                                \
        static bool row_sized = false;                                                                                  \
        if (!row_sized) {                                                                                               \
            cudaError_t e = cudaFuncSetAttribute(attention_f32_row_kernel<W, PIECE, BUFS>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                 BUFS * W * piece_floats(PIECE, MAX_DIM, MAX_DIM) * (int)sizeof(float)); \
            if (e != cudaSuccess) return (int)e;                                                                        \
            row_sized = true;                                                                                           \
        }                                                                                                               \
        cj::launch(attention_f32_row_kernel<W, PIECE, BUFS>, dim3(rows, n_heads), dim3(W * 32),                         \
                   BUFS * W * piece_floats(PIECE, hd, vd) * (int)sizeof(float), stream, a);                             \
    } while (0)
        // With a block an SM at most, six warps whose chunks travel whole (8 rows at 520 keys, 16 heads: 36 us, 63 with the kernel
        // before); with more, smaller blocks, one summing while another waits.  Those take a piece of 32, 24 or 16 keys at a time, so that an SM
        // holds three, four or six of them (heads of 128): the size with the fewest rounds, of those with as few the largest.  us with pieces of 32, 24
        // and 16, 16 heads, rows at 500 keys: 384 blocks 47, 51 and 53, 512 (32 decoding requests) 90, 73 and 72, 640 84, 86 and 63, 1,024 129,
        // 117 and 136, 2,048 186, 180 and 161 (with the kernel before 60, 77, 78, 145 and 199).
        int sms, sm_bytes;
        if (int st = machine(sms, sm_bytes)) return st;
        auto rounds = [&](int piece) {                         // (3.6 KB: what a block holds besides, and what an SM keeps for itself a block)
            const int held = min(16, sm_bytes / ((int)sizeof(float) * 4 * piece_floats(piece, hd, vd) + 3686));
            return ((long long)rows * n_heads + (long long)sms * held - 1) / ((long long)sms * held);
        };
        if ((long long)rows * n_heads <= sms) ROWS(6, 32, 2);
        else if (rounds(32) <= min(rounds(24), rounds(16))) ROWS(4, 32, 1);
        else if (rounds(24) <= rounds(16)) ROWS(4, 24, 1);
        else ROWS(4, 16, 1);
#undef ROWS
    }
    return launch_status();
}
