// Mixers that carry a fixed-size state per request instead of a growing cache, and the
// row-wise kernels of a block that norms a sublayer's OUTPUT.  Everything that enters a
// recurrence is float32: the state, decays and their logarithms, step sizes, gates, unit
// norms.  A step's rows are laid out request after request; every kernel finds a row's
// request, the request's first row and its state slot in the step's device metadata
// (row_req, req_start, req_slot), so the same launch serves prompt portions of any length
// beside single decoded tokens, and a request that a captured step is filled up with
// (slot -1, no rows) is left alone.
//
//   cast_rows          float32 rows -> the activation dtype (a sublayer reads the stream itself)
//   rmsnorm_add        hs += y / sqrt(mean(y^2) + eps) * w
//   scale_rows_gather  out[slot] = weight[pick] * x[token]  (a mixture whose score multiplies the expert's INPUT)
//   short_conv         causal convolution per channel over time (+ bias, + SiLU) whose first
//                      taps-1 inputs come from the request's state; short_conv_commit then
//                      stores the step's last taps-1 inputs
//   ssd_scan           S_t = exp(-A dt) S_(t-1) + dt B_t x_t^T ;  y_t = S_t^T C_t + D x_t
//   delta_scan         S <- g S ; u = beta (v - S^T k) ; S <- S + k u^T ; o = S^T q
//   gla_scan           S_t = diag(alpha_t) S_(t-1) + k_t v_t^T ;  o_t = S_t^T q_t   (a decay per state row)
//   mlstm_scan         m_t = max(f + m, i) ; S_t = e^(f + m - m_t) S + e^(i - m_t) k v^T ; n likewise with k alone ;
//                      o = S^T q / (max(|n . q|, e^(-m_t)) + floor)
//   gated_scan         S_t = (1 - z_t) S_(t-1) + z_t c_t per channel, out = S_t silu(g_t) (minGRU: gates of the current token only)
//   rmsnorm_mix2       out (+)= c (a / rms(a) * wa + b / rms(b) * wb)
//   softcap_rows       x <- cap tanh(x / cap), float32 in place (a head whose logits are capped)
//   gated_group_norm   y * silu(z) (or sigmoid(z)) and RMS over equal parts of a row, in either order
//
// The two scans give a thread one column of the state (one value dimension) for a share of
// its rows: a block is (request, head, tile of columns), a column's rows are dealt to DP
// neighbouring lanes, each holding NPER of them in registers, and a sum over the rows is a
// butterfly over those lanes.  Columns never talk to each other; the block's barriers only
// guard the staging of the tokens' inputs.  The tokens of a request are walked in order, which is what makes the result
// independent of how a prompt was cut: the state after token t is the same sequence of
// float32 operations whether t ended a step or not.
#define CJ_LIB "recurrent"
#include "common.cuh"

#include <type_traits>

using namespace cj;

namespace {

__device__ __forceinline__ float softplus_f(float v) { return v > 20.0f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float sigmoid_f(float v) { return 1.0f / (1.0f + expf(-v)); }

__device__ __forceinline__ float block_sum(float v, float* scratch) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float t = 0.0f;
    for (int i = 0; i < nw; ++i) t += scratch[i];
    return t;
}

template <typename TO>
__global__ void cast_rows_kernel(const float* __restrict__ x, TO* __restrict__ out, long long n) {
    cj::after_predecessor();
    cj::release_successor();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = from_f32<TO>(x[i]);
}

// The same, four at a time: 16-byte loads, 8- or 16-byte stores (n a multiple of four, both pointers on their boundaries).  2,048 rows of 2,048
// to bfloat16, cold: 8.8 us with the kernel above, 6.1 so
__device__ __forceinline__ void store_piece(float* dst, float4 v) { *(float4*)dst = v; }
__device__ __forceinline__ void store_piece(__nv_bfloat16* dst, float4 v) {
    __nv_bfloat162 two[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
    *(uint2*)dst = *(const uint2*)two;
}
template <typename TO>
__global__ void __launch_bounds__(256) cast_rows4_kernel(const float4* __restrict__ x, TO* __restrict__ out, long long n4) {
    cj::after_predecessor();
    cj::release_successor();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) store_piece(out + 4 * i, x[i]);
}

__global__ void rmsnorm_add_kernel(float* __restrict__ hs, const float* __restrict__ y, const float* __restrict__ w, float eps, int H) {
    cj::after_predecessor();
    cj::release_successor();
    __shared__ float scratch[32];
    const float* src = y + (size_t)blockIdx.x * H;
    float* dst = hs + (size_t)blockIdx.x * H;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) ss = fmaf(src[i], src[i], ss);
    ss = block_sum(ss, scratch);
    const float scale = 1.0f / sqrtf(ss / (float)H + eps);
    for (int i = threadIdx.x; i < H; i += blockDim.x) dst[i] += src[i] * scale * w[i];
}

// The same for widths that are multiples of four, up to 8,192, 16-byte aligned: a thread keeps its NV float4 of the row, which is read once.
// The squares are added in the order of the kernel above with `order` threads (from shared memory, a thread for one or two of that kernel's),
// so that both give the same bits.  Bound by memory: 2,048 rows of 2,048 out of HBM 21.6 us with the kernel above, 11.2 with this one (10.2
// with sums in the order of the float4); 8 rows 2.5 and 2.2.
template <int NV>
__global__ void __launch_bounds__(256) rmsnorm_add4_kernel(float* __restrict__ hs, const float* __restrict__ y,
                                                           const float* __restrict__ w, float eps, int H, int order) {
    cj::after_predecessor();
    cj::release_successor();
    __shared__ __align__(16) float row[1024 * NV];
    __shared__ float sums[16];
    const float4* src = (const float4*)(y + (size_t)blockIdx.x * H);
    float4* dst = (float4*)(hs + (size_t)blockIdx.x * H);
    const int n4 = H / 4;
    float4 v[NV], old[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        v[k] = old[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < n4) {
            v[k] = src[i];
            old[k] = dst[i];
            *(float4*)(row + 4 * i) = v[k];
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < order; t += 256) {
        float ss = 0.0f;
        for (int i = t; i < H; i += order) ss = fmaf(row[i], row[i], ss);
        ss = warp_sum(ss);
        if ((t & 31) == 0) sums[t >> 5] = ss;
    }
    __syncthreads();
    float total = 0.0f;
    for (int i = 0; i < order / 32; ++i) total += sums[i];
    const float scale = 1.0f / sqrtf(total / (float)H + eps);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        if (i >= n4) continue;
        const float4 g = ((const float4*)w)[i];
        dst[i] = make_float4(old[k].x + v[k].x * scale * g.x, old[k].y + v[k].y * scale * g.y, old[k].z + v[k].z * scale * g.z,
                             old[k].w + v[k].w * scale * g.w);
    }
}

template <typename TO>
__global__ void scale_rows_gather_kernel(const float* __restrict__ x, const int* __restrict__ slot_of_pick,
                                         const float* __restrict__ weight, int k, int H, TO* __restrict__ out) {
    cj::after_predecessor();
    cj::release_successor();
    const int pick = blockIdx.x;
    const float* src = x + (size_t)(pick / k) * H;
    TO* dst = out + (size_t)slot_of_pick[pick] * H;
    const float wt = weight[pick];
    for (int i = threadIdx.x; i < H; i += blockDim.x) dst[i] = from_f32<TO>(wt * src[i]);
}

// ---------------------------------------------------------------------------------
// short convolution over time with the request's last taps-1 inputs as state
// state of a slot: [taps-1][C] float32, oldest first
// ---------------------------------------------------------------------------------
template <typename TO>
__global__ void short_conv_kernel(const float* __restrict__ in, int ld_in, int C, int taps, const float* __restrict__ w,
                                  const float* __restrict__ bias, const float* __restrict__ state, long long slot_stride,
                                  const int* __restrict__ row_req, const int* __restrict__ req_start,
                                  const int* __restrict__ req_slot, TO* __restrict__ out, int ld_out, int act) {
    cj::after_predecessor();
    cj::release_successor();
    const int r = blockIdx.x;
    const int req = row_req[r];
    const int t = r - req_start[req];
    const int slot = req_slot[req];
    const float* st = state + (size_t)slot * slot_stride;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
        float acc = bias ? bias[c] : 0.0f;
        for (int j = taps - 1; j >= 0; --j) {          // oldest input first
            const int src_t = t - j;
            const float v = src_t >= 0 ? in[(size_t)(r - j) * ld_in + c] : st[(size_t)(taps - 1 + src_t) * C + c];
            acc = fmaf(w[(size_t)c * taps + (taps - 1 - j)], v, acc);
        }
        if (act) acc = acc / (1.0f + expf(-acc));
        out[(size_t)r * ld_out + c] = from_f32<TO>(acc);
    }
}

// The same for many rows: a thread takes four neighbouring channels (16-byte loads and stores) and CONV_ROWS rows after one another, so
// that an input is read once instead of once a tap.  The sums are the same, in the same order.  2,048 rows of 6,144 channels, 4 taps:
// 92 -> 33 us, of 4,096 channels 59 -> 21 us; 100 MB at 3 TB/s, bound by memory with the exponential beside it.
constexpr int CONV_ROWS = 16;
template <int N> struct alignas(4 * N) Floats { float v[N]; };
__device__ __forceinline__ void store_four(float* dst, const float (&v)[4]) { *(float4*)dst = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store_four(__nv_bfloat16* dst, const float (&v)[4]) {
    __nv_bfloat162 two[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
    *(uint2*)dst = *(const uint2*)two;
}

template <typename TO, int TAPS>
__global__ void __launch_bounds__(128) short_conv_tile_kernel(const float* __restrict__ in, int ld_in, int C, const float* __restrict__ w,
                                                              const float* __restrict__ bias, const float* __restrict__ state, long long slot_stride,
                                                              const int* __restrict__ row_req, const int* __restrict__ req_start,
                                                              const int* __restrict__ req_slot, TO* __restrict__ out, int ld_out, int act, int T) {
    cj::after_predecessor();
    cj::release_successor();
    const int c = (blockIdx.y * 128 + threadIdx.x) * 4;
    if (c >= C) return;
    const int r0 = blockIdx.x * CONV_ROWS, r1 = min(T, r0 + CONV_ROWS);
    float wt[TAPS][4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        b[i] = bias ? bias[c + i] : 0.0f;
#pragma unroll
        for (int k = 0; k < TAPS; ++k) wt[k][i] = w[(size_t)(c + i) * TAPS + k];
    }
    Floats<4> before[TAPS - 1];                             // the rows r0 - (TAPS - 1) .. r0 - 1 (those of another request are not used)
#pragma unroll
    for (int k = 0; k < TAPS - 1; ++k) {
        const int r = r0 - (TAPS - 1) + k;
        if (r >= 0) before[k] = *(const Floats<4>*)(in + (size_t)r * ld_in + c);
        else before[k] = Floats<4>{};
    }
    for (int g = r0; g < r1; g += 4) {
        Floats<4> row[TAPS + 3];                            // rows g - (TAPS - 1) .. g + 3
#pragma unroll
        for (int k = 0; k < TAPS - 1; ++k) row[k] = before[k];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (g + k < r1) row[TAPS - 1 + k] = *(const Floats<4>*)(in + (size_t)(g + k) * ld_in + c);
            else row[TAPS - 1 + k] = Floats<4>{};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = g + k;
            if (r >= r1) break;
            const int req = row_req[r], t = r - req_start[req];
            float acc[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = b[i];
            if (t >= TAPS - 1) {
#pragma unroll
                for (int j = TAPS - 1; j >= 0; --j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i] = fmaf(wt[TAPS - 1 - j][i], row[TAPS - 1 + k - j].v[i], acc[i]);
            } else {
                const float* st = state + (size_t)req_slot[req] * slot_stride;
#pragma unroll
                for (int j = TAPS - 1; j >= 0; --j)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        acc[i] = fmaf(wt[TAPS - 1 - j][i], t >= j ? row[TAPS - 1 + k - j].v[i] : st[(size_t)(TAPS - 1 + t - j) * C + c + i], acc[i]);
            }
            if (act) {
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] = acc[i] / (1.0f + expf(-acc[i]));
            }
            store_four(out + (size_t)r * ld_out + c, acc);
        }
#pragma unroll
        for (int k = 0; k < TAPS - 1; ++k) before[k] = row[4 + k];
    }
}

// A step in which every request brings one token: the convolution and the state's move in one kernel (a thread reads its
// channel's whole state before it writes it).
template <typename TO, int TAPS>
__global__ void __launch_bounds__(128) short_conv_single_kernel(const float* __restrict__ in, int ld_in, int C, const float* __restrict__ w,
                                                                const float* __restrict__ bias, float* __restrict__ state, long long slot_stride,
                                                                const int* __restrict__ row_req, const int* __restrict__ req_slot,
                                                                TO* __restrict__ out, int ld_out, int act) {
    cj::after_predecessor();
    cj::release_successor();
    const int r = blockIdx.x;
    const int slot = req_slot[row_req[r]];
    if (slot < 0) return;
    // (one round, unless there are more channels than a grid has threads)
    for (int c = blockIdx.y * 128 + threadIdx.x; c < C; c += gridDim.y * 128) {
        float* st = state + (size_t)slot * slot_stride + c;
        float v[TAPS], acc = bias ? bias[c] : 0.0f;
#pragma unroll
        for (int k = 0; k < TAPS - 1; ++k) v[k] = st[(size_t)k * C];
        v[TAPS - 1] = in[(size_t)r * ld_in + c];
#pragma unroll
        for (int k = 0; k < TAPS; ++k) acc = fmaf(w[(size_t)c * TAPS + k], v[k], acc);
        if (act) acc = acc / (1.0f + expf(-acc));
        out[(size_t)r * ld_out + c] = from_f32<TO>(acc);
#pragma unroll
        for (int k = 0; k < TAPS - 1; ++k) st[(size_t)k * C] = v[k + 1];
    }
}

__global__ void short_conv_commit_kernel(const float* __restrict__ in, int ld_in, int C, int taps, float* __restrict__ state,
                                         long long slot_stride, const int* __restrict__ req_start,
                                         const int* __restrict__ req_slot) {
    cj::after_predecessor();
    cj::release_successor();
    const int req = blockIdx.x;
    const int slot = req_slot[req];
    const int first = req_start[req], n = req_start[req + 1] - first;
    if (slot < 0 || n <= 0) return;
    float* st = state + (size_t)slot * slot_stride;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
        // ascending k: an entry that is kept moves down from k + n, which is read before it is written
        for (int k = 0; k < taps - 1; ++k) {
            const int src_t = n - (taps - 1) + k;
            st[(size_t)k * C + c] = src_t >= 0 ? in[(size_t)(first + src_t) * ld_in + c] : st[(size_t)(k + n) * C + c];
        }
    }
}

// ---------------------------------------------------------------------------------
// the scans
// ---------------------------------------------------------------------------------
struct ScanArgs {
    const float* x;      // the step's rows after convolution and activation, [T, ld]
    int ld;
    int off_a, off_b, off_v;   // ssd: B, C, x ; delta: q, k, v  (column offsets in x)
    const float* raw;    // the step's rows of the plain projections, [T, ld_raw]
    int ld_raw;
    int off_dt, off_beta;      // ssd: dt ; delta: the decay's input a, beta's input b
    const float* A_log; const float* dt_bias; const float* skip;    // per head (skip: ssd's D)
    float* state; long long slot_stride;     // per slot: the heads' matrices in the scan's own layout, float32
    const int* req_start; const int* req_slot;
    float* out;          // [T, heads * cols]
    int heads, groups, rows, cols;           // rows: state rows (N or key dim); cols: value dim
    float q_scale;
    int decays_ready;    // gla: raw holds the decays themselves
    float c0, c1;        // gla: c0 = 1 / tau ; mlstm: c0 = the gates' cap, c1 = the floor added to the read-out's divisor
};

constexpr int SCAN_SSD = 0, SCAN_DELTA = 1, SCAN_GLA = 2, SCAN_MLSTM = 3;

// log(sigmoid(v)) without overflow on either side
__device__ __forceinline__ float log_sigmoid_f(float v) { return fminf(v, 0.0f) - log1pf(expf(-fabsf(v))); }

__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A token's inputs (the two vectors over the state's rows, the block's columns of the value
// vector, the two gate inputs) are staged in shared memory TOK tokens at a time, the next
// TOK in flight (cp.async) while these are walked: a token's step then waits on shared
// memory, not on a round trip to L2.  One staged token: [a | b | v: block's columns | 4 scalars],
// a and b laid out so that a lane's NPER rows (part + DP i) are contiguous: index part * NPER + i.
// What does not depend on the state - the unit norms of q and k, softplus, the decay's
// exponential, beta - is worked out for all staged tokens side by side (a warp a token)
// before they are walked, so that the chain from one token's state to the next is only
// decay, one sum over the rows, the update.  The read-out's sum over the rows, which nothing
// waits for, is carried along with the next token's sum (two independent butterflies side by side).
//
// The state of a (slot, head) is kept in the order the threads hold it: element
// ((tile * NPER + i) * 128 + thread) is row part + DP i of column tile * cols_blk + lcol -
// a layout that depends on the state's shape alone, read and written with full coalescing.
// Nothing else reads the state (a slot is zeroed when it is admitted).
__device__ __forceinline__ float lanes_sum(float v, int first) {
    if (first == 1) return warp_sum(v);                     // a column's rows span the whole warp: unrolled
    for (int o = first; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// MODE 2 (gla) stages a third vector over the state's rows, the decays' inputs (from raw, columns off_dt +
// head * rows), which the scalar phase turns into the decays alpha = sigmoid(z)^(1/tau) = exp(log_sigmoid(z) / tau).
// MODE 3 (mlstm) keeps, beside a thread's share of its column, the same share of the vector n (every column of
// a tile holds it: what a block reads at its start no other block writes) and the running maximum m:
// a (slot, head, tile) holds [S: NPER x 128 | n: NPER x 128 | m: 128] floats.
template <int NPER, int MODE>
__global__ void __launch_bounds__(128) scan_kernel(ScanArgs p, int DP, int TOK) {
    constexpr bool DELTA = MODE == SCAN_DELTA;
    constexpr int NVEC = MODE == SCAN_GLA ? 3 : 2;
    constexpr int TILE_FLOATS = MODE == SCAN_MLSTM ? (2 * NPER + 1) * 128 : NPER * 128;
    cj::after_predecessor();
    cj::release_successor();
    extern __shared__ __align__(16) float staged[];
    const int req = blockIdx.x, head = blockIdx.y;
    const int slot = p.req_slot[req];
    const int first = p.req_start[req], n = p.req_start[req + 1] - first;
    if (slot < 0 || n <= 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cols_per_warp = 32 / DP, cols_blk = 4 * cols_per_warp;
    const int part = lane / cols_per_warp;                  // which share of the state's rows
    const int col0 = blockIdx.z * cols_blk;
    const int lcol = warp * cols_per_warp + (lane % cols_per_warp);
    const int col = col0 + lcol;
    const bool live = col < p.cols;
    const int rows = p.rows, padded = DP * NPER;            // rows rounded up to what the lanes hold
    const int group = head / (p.heads / p.groups);
    const int tail = NVEC * padded + cols_blk;              // where a staged token's four scalars begin
    const int stride = tail + 4;
    float* S = p.state + (size_t)slot * p.slot_stride + ((size_t)head * gridDim.z + blockIdx.z) * TILE_FLOATS;

    // Where a staged token's entries come from is the same for every token: a thread works out, once,
    // the source of the entries it copies (entry e = thread + 128 k) as an offset into the token's row
    // of x (kind 1) or of raw (kind 2), or nothing (kind 0: padding, written as zero).
    constexpr int OWN = 4;                                  // entries a thread remembers; longer tokens take the general loop
    int own_off[OWN], own_kind[OWN];
    auto source = [&](int e, int& off) -> int {
        if (e < NVEC * padded) {
            const int which = e / padded;
            const int v = e - which * padded;               // index part * NPER + i  ->  row part + DP i
            const int d = (v / NPER) + DP * (v % NPER);
            if (which == 2) {                               // gla: the decays' inputs, a row of raw per head
                off = p.off_dt + head * rows + d;
                return d < rows ? 2 : 0;
            }
            off = (which == 0 ? p.off_a : p.off_b) + group * rows + d;
            return d < rows ? 1 : 0;
        }
        if (e < tail) {
            const int c = col0 + e - NVEC * padded;
            off = p.off_v + head * p.cols + c;
            return c < p.cols ? 1 : 0;
        }
        if (MODE != SCAN_GLA && e == tail) { off = p.off_dt + head; return 2; }
        if ((DELTA || MODE == SCAN_MLSTM) && e == tail + 1) { off = p.off_beta + head; return 2; }
        off = 0;
        return 0;
    };
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
        const int e = threadIdx.x + 128 * k;
        own_kind[k] = e < stride ? source(e, own_off[k]) : -1;
        if (e >= stride) own_off[k] = 0;
    }
    auto stage = [&](int chunk, float* buf) {
        const int t0 = chunk * TOK, nt = min(TOK, n - t0);
        for (int tt = 0; tt < nt; ++tt) {
            const size_t row = (size_t)(first + t0 + tt);
            const float* xr = p.x + row * p.ld;
            const float* rr = p.raw + row * p.ld_raw;
            float* dst = buf + tt * stride;
#pragma unroll
            for (int k = 0; k < OWN; ++k) {
                const int e = threadIdx.x + 128 * k;
                if (own_kind[k] > 0) cp_async4(dst + e, (own_kind[k] == 1 ? xr : rr) + own_off[k]);
                else if (own_kind[k] == 0) dst[e] = 0.0f;
            }
            for (int e = threadIdx.x + 128 * OWN; e < stride; e += 128) {
                int off;
                const int kind = source(e, off);
                if (kind > 0) cp_async4(dst + e, (kind == 1 ? xr : rr) + off);
                else dst[e] = 0.0f;
            }
        }
    };

    const int chunks = (n + TOK - 1) / TOK;
    stage(0, staged);
    cp_async_commit();
    float s[NPER];
#pragma unroll
    for (int i = 0; i < NPER; ++i) s[i] = S[i * 128 + threadIdx.x];
    // ssd, delta: A = exp(A_log), bias = the step size's; mlstm: A = the forget gate's bias, bias = the input gate's
    const float A = MODE == SCAN_GLA ? 0.0f : (MODE == SCAN_MLSTM ? p.A_log[head] : expf(p.A_log[head]));
    const float bias = MODE == SCAN_GLA ? 0.0f : p.dt_bias[head];
    const float skip = MODE == SCAN_SSD ? p.skip[head] : 0.0f;
    float nvec[MODE == SCAN_MLSTM ? NPER : 1];
    float m_run = 0.0f;
    if (MODE == SCAN_MLSTM) {
#pragma unroll
        for (int i = 0; i < NPER; ++i) nvec[i] = S[(NPER + i) * 128 + threadIdx.x];
        m_run = S[2 * NPER * 128 + threadIdx.x];
    }
    float* out = p.out + (size_t)first * p.heads * p.cols + head * p.cols + col;
    const size_t out_ld = (size_t)p.heads * p.cols;
    const bool writer = live && part == 0;
    float y_prev = 0.0f;                                    // the token before's read-out, its sum over the lanes still owed
    int t_prev = -1;
    for (int chunk = 0; chunk < chunks; ++chunk) {
        float* cur = staged + (chunk & 1) * TOK * stride;
        if (chunk + 1 < chunks) stage(chunk + 1, staged + ((chunk + 1) & 1) * TOK * stride);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const int nt = min(TOK, n - chunk * TOK);
        // the staged tokens' scalars: a warp a token
        for (int tt = warp; tt < nt; tt += 4) {
            float* tk = cur + tt * stride;
            if (DELTA) {
                float qq = 0.0f, kk = 0.0f;
                for (int d = lane; d < padded; d += 32) {
                    qq = fmaf(tk[d], tk[d], qq);
                    kk = fmaf(tk[padded + d], tk[padded + d], kk);
                }
                qq = warp_sum(qq);
                kk = warp_sum(kk);
                if (lane == 0) {
                    const float g0 = tk[tail], g1 = tk[tail + 1];
                    tk[tail] = expf(-A * softplus_f(g0 + bias));          // the decay
                    tk[tail + 1] = sigmoid_f(g1);                         // beta
                    tk[tail + 2] = p.q_scale / sqrtf(qq + 1e-6f);         // q becomes a unit vector times q_scale
                    tk[tail + 3] = 1.0f / sqrtf(kk + 1e-6f);              // k a unit vector
                }
            } else if (MODE == SCAN_GLA) {
                for (int d = lane; d < padded; d += 32) tk[2 * padded + d] = expf(log_sigmoid_f(tk[2 * padded + d]) * p.c0);
            } else if (MODE == SCAN_MLSTM) {
                if (lane == 0) {
                    const float cap = p.c0;
                    tk[tail] = cap * tanhf((tk[tail] + bias) / cap);                          // log of the input gate
                    tk[tail + 1] = log_sigmoid_f(cap * tanhf((tk[tail + 1] + A) / cap));      // log of the forget gate
                }
            } else if (lane == 0) {
                const float dt = softplus_f(tk[tail] + bias);
                tk[tail] = dt;
                tk[tail + 1] = expf(-A * dt);
            }
        }
        __syncthreads();
        for (int tt = 0; tt < nt; ++tt) {
            const float* tk = cur + tt * stride;
            const float xv = tk[NVEC * padded + lcol];
            float a[NPER], b[NPER];
            if (NPER % 4 == 0) {
#pragma unroll
                for (int i = 0; i < NPER; i += 4) {
                    const float4 va = *(const float4*)(tk + part * NPER + i);
                    const float4 vb = *(const float4*)(tk + padded + part * NPER + i);
                    a[i] = va.x; a[i + 1] = va.y; a[i + 2] = va.z; a[i + 3] = va.w;
                    b[i] = vb.x; b[i + 1] = vb.y; b[i + 2] = vb.z; b[i + 3] = vb.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < NPER; ++i) {
                    a[i] = tk[part * NPER + i];
                    b[i] = tk[padded + part * NPER + i];
                }
            }
            if (DELTA) {
                const float decay = tk[tail], beta = tk[tail + 1], qs = tk[tail + 2], ks = tk[tail + 3];
                float dot = 0.0f;
#pragma unroll
                for (int i = 0; i < NPER; ++i) {
                    b[i] *= ks;
                    s[i] *= decay;
                    dot = fmaf(s[i], b[i], dot);
                }
                // this token's S^T k and the token before's read-out: two sums over the lanes, side by side
                if (cols_per_warp == 1) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        dot += __shfl_xor_sync(0xffffffffu, dot, o);
                        y_prev += __shfl_xor_sync(0xffffffffu, y_prev, o);
                    }
                } else {
                    for (int o = cols_per_warp; o < 32; o <<= 1) {
                        dot += __shfl_xor_sync(0xffffffffu, dot, o);
                        y_prev += __shfl_xor_sync(0xffffffffu, y_prev, o);
                    }
                }
                if (writer && t_prev >= 0) out[(size_t)t_prev * out_ld] = y_prev;
                const float u = beta * (xv - dot);
                float y = 0.0f;
#pragma unroll
                for (int i = 0; i < NPER; ++i) {
                    s[i] = fmaf(b[i], u, s[i]);
                    y = fmaf(s[i], a[i] * qs, y);
                }
                y_prev = y;
                t_prev = chunk * TOK + tt;
            } else if (MODE == SCAN_GLA) {
                // a = q, b = k, a row's decay from the third staged vector
                float y = 0.0f;
#pragma unroll
                for (int i = 0; i < NPER; ++i) {
                    s[i] = fmaf(tk[2 * padded + part * NPER + i], s[i], b[i] * xv);
                    y = fmaf(s[i], a[i] * p.q_scale, y);
                }
                y = lanes_sum(y, cols_per_warp);
                if (writer) out[(size_t)(chunk * TOK + tt) * out_ld] = y;
            } else if (MODE == SCAN_MLSTM) {
                const float li = tk[tail], lf = tk[tail + 1];
                const float m_new = fmaxf(lf + m_run, li);
                const float keep = expf(lf + m_run - m_new), take = expf(li - m_new);
                m_run = m_new;
                float y = 0.0f, nq = 0.0f;
#pragma unroll
                for (int i = 0; i < NPER; ++i) {
                    const float kb = take * b[i], qa = a[i] * p.q_scale;
                    s[i] = fmaf(keep, s[i], kb * xv);
                    nvec[i] = fmaf(keep, nvec[i], kb);
                    y = fmaf(s[i], qa, y);
                    nq = fmaf(nvec[i], qa, nq);
                }
                if (cols_per_warp == 1) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        y += __shfl_xor_sync(0xffffffffu, y, o);
                        nq += __shfl_xor_sync(0xffffffffu, nq, o);
                    }
                } else {
                    for (int o = cols_per_warp; o < 32; o <<= 1) {
                        y += __shfl_xor_sync(0xffffffffu, y, o);
                        nq += __shfl_xor_sync(0xffffffffu, nq, o);
                    }
                }
                if (writer) out[(size_t)(chunk * TOK + tt) * out_ld] = y / (fmaxf(fabsf(nq), expf(-m_run)) + p.c1);
            } else {
                // a = B, b = C
                const float dt = tk[tail], decay = tk[tail + 1];
                const float dx = dt * xv;
                float y = 0.0f;
#pragma unroll
                for (int i = 0; i < NPER; ++i) {
                    s[i] = fmaf(decay, s[i], a[i] * dx);
                    y = fmaf(s[i], b[i], y);
                }
                y = lanes_sum(y, cols_per_warp);
                if (writer) out[(size_t)(chunk * TOK + tt) * out_ld] = fmaf(skip, xv, y);
            }
        }
        __syncthreads();                       // everyone has walked this buffer before it is staged into again
    }
    if (DELTA) {
        y_prev = lanes_sum(y_prev, cols_per_warp);
        if (writer && t_prev >= 0) out[(size_t)t_prev * out_ld] = y_prev;
    }
#pragma unroll
    for (int i = 0; i < NPER; ++i) S[i * 128 + threadIdx.x] = s[i];
    if (MODE == SCAN_MLSTM) {
#pragma unroll
        for (int i = 0; i < NPER; ++i) S[(NPER + i) * 128 + threadIdx.x] = nvec[i];
        S[2 * NPER * 128 + threadIdx.x] = m_run;
    }
}

// The same scans for steps that bring many tokens a request.  scan_kernel's chain a token (shared-memory loads, a row's partial sum,
// a butterfly, the store, one after the other) takes 600 to 700 ns whatever the state's size.  Here a thread keeps C columns, so that a
// token's two vectors are loaded once for them; U tokens are walked before their C U read-outs are summed over the DP lanes all at once,
// by halving (each lane hands half of its values to its partner: DP - 1 shuffles for DP values instead of log2 DP for one), after which
// every lane holds one finished value; and what needs no state is worked out for WALK_TOK tokens side by side, a lane a token.
// Every float32 operation on a (column, token) is scan_kernel's, in its order - the partial sums over a lane's rows, the butterfly's
// tree, the update - so a state or a row has the same bits whichever of the two walked it.  Half of a block's warps walk; the other half
// fetch the next tokens and work out what needs no state (unit norms, gates, decays' exponentials), a batch ahead.  2,048 tokens of
// one prompt, scan_kernel, this kernel with every warp doing both, and as it is: state-space, 64 heads of 128 x 64, 1,266, 356 and
// 274 us; delta rule, 16 of 128 x 128, 1,412, 565 and 333 us; gated linear attention, 4 of 128 x 256, 1,214, 427 and 385 us (217 with its
// decays worked out ahead, gla_decays_kernel);
// matrix memory, 8 of 128 x 256, 1,488, 369 and 296 us.  Two columns a thread: with one 20 to 35 % slower (twice the loads), with
// four up to 60 % (too few warps).  What bounds it: latencies with one walking warp a scheduler (an instruction every 3.3 clocks, the FMA
// pipe at most 47 % busy), in the delta rule the chain from one token's state to the next (four dependent shuffles).  Two rows packed
// into one instruction (f32x2), operands read a token ahead and eight walking warps of a column each changed nothing or cost time
// (state-space 282, 286 and 379 us).
constexpr int WALK_COLS = 2, WALK_BUFS = 3;
constexpr int walk_tok(int mode) { return mode == SCAN_GLA ? 16 : 32; }      // (with the decays staged too, 32 would leave an SM room for one block)

// Sums of V values over the DP lanes that share a column; lane `part` is left, in v[0], with the value its bits name, the first
// exchanged the most significant.  The order of the exchanges is scan_kernel's: neighbouring parts first, but with a whole warp a
// column the farthest.  (Written as a recursion, so that every index is a constant.)
template <int DP, int N, int STEP, int V> __device__ __forceinline__ void halve_sum(float (&v)[V], int lane) {
    constexpr int STEPS = DP == 8 ? 3 : DP == 16 ? 4 : 5;
    if constexpr (STEP < STEPS) {
        constexpr int O = DP == 32 ? 16 >> STEP : (32 / DP) << STEP;
        if constexpr (N > 1) {
            const bool up = (lane & O) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                const float give = up ? v[i] : v[N / 2 + i], keep = up ? v[N / 2 + i] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, O);
            }
            halve_sum<DP, N / 2, STEP + 1>(v, lane);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            halve_sum<DP, 1, STEP + 1>(v, lane);
        }
    }
}

// The decays of gated linear attention for a step's rows, once: each of the walk's blocks of 8 or so columns (4 heads of 256 columns: 32 a
// head) would work out all of its head's otherwise, and its walking warps wait for them: 2,048 tokens, 4 heads of 128 x 256, 388 us so,
// 217 with this kernel before it (its own 4 included).
__global__ void gla_decays_kernel(const float* __restrict__ raw, int ld, int off, int width, long long n, float c0, float* __restrict__ out) {
    cj::after_predecessor();
    cj::release_successor();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = expf(log_sigmoid_f(raw[i / width * ld + off + i % width]) * c0);
}

template <int DP, int NPER, int MODE, int C>
__global__ void __launch_bounds__(256, 1) walk_kernel(ScanArgs p) {
    constexpr bool DELTA = MODE == SCAN_DELTA;
    constexpr int TOK = walk_tok(MODE);
    constexpr int NVEC = MODE == SCAN_GLA ? 3 : 2, ROWS = DP * NPER, CPW = 32 / DP, CB = 4 * CPW * C, U = DP / C, V = U * C;
    constexpr int OLD_CB = 4 * CPW;                                       // columns of a tile of the state's layout
    constexpr int TILE_FLOATS = MODE == SCAN_MLSTM ? (2 * NPER + 1) * 128 : NPER * 128;
    constexpr int TAIL = NVEC * ROWS + CB, STRIDE = TAIL + 4;             // a staged token: [a | b | (decays) | v: CB columns | 4 scalars]
    constexpr int OWN = (STRIDE + 127) / 128;
    cj::after_predecessor();
    cj::release_successor();
    extern __shared__ __align__(16) float staged[];         // WALK_BUFS batches of TOK tokens: one walked, one made ready, one landing
    __shared__ float m_last;
    const int req = blockIdx.x, head = blockIdx.y;
    const int slot = p.req_slot[req];
    const int first = p.req_start[req], n = p.req_start[req + 1] - first;
    if (slot < 0 || n <= 0) return;
    // threads 0-127 walk, threads 128-255 fetch the tokens and work out what needs no state; both count from 0
    const bool walker = threadIdx.x < 128;
    const int tid = threadIdx.x & 127, lane = tid & 31, warp = tid >> 5;
    const int part = lane / CPW;
    const int lcol = warp * CPW * C + lane % CPW;                         // the thread's columns: lcol + CPW k of the block's
    const int col0 = blockIdx.z * CB;
    const int group = head / (p.heads / p.groups);
    const int batches = (n + TOK - 1) / TOK;
    const float A = MODE == SCAN_GLA ? 0.0f : (MODE == SCAN_MLSTM ? p.A_log[head] : expf(p.A_log[head]));
    const float bias = MODE == SCAN_GLA ? 0.0f : p.dt_bias[head];
    const int old_tiles = (p.cols + OLD_CB - 1) / OLD_CB;

    if (!walker) {
        // the sources of the entries of a staged token that this thread copies (entry tid + 128 k), for the request's first row; null: none
        const float* src[OWN];
        int ld[OWN];
#pragma unroll
        for (int k = 0; k < OWN; ++k) {
            const int e = tid + 128 * k;
            src[k] = nullptr;
            ld[k] = p.ld;
            const float* x = p.x + (size_t)first * p.ld;
            const float* raw = p.raw + (size_t)first * p.ld_raw;
            if (e < NVEC * ROWS) {
                const int which = e / ROWS, v = e - which * ROWS, d = v / NPER + DP * (v % NPER);      // index part * NPER + i -> row part + DP i
                if (which == 2) { src[k] = raw + p.off_dt + head * ROWS + d; ld[k] = p.ld_raw; }
                else src[k] = x + (which == 0 ? p.off_a : p.off_b) + group * ROWS + d;
            } else if (e < TAIL) {
                const int c = col0 + e - NVEC * ROWS;
                if (c < p.cols) src[k] = x + p.off_v + head * p.cols + c;
            } else if (e == TAIL && MODE != SCAN_GLA) { src[k] = raw + p.off_dt + head; ld[k] = p.ld_raw; }
            else if (e == TAIL + 1 && (DELTA || MODE == SCAN_MLSTM)) { src[k] = raw + p.off_beta + head; ld[k] = p.ld_raw; }
        }
        auto stage = [&](int t0, float* buf) {
            const int nt = min(TOK, n - t0);
#pragma unroll
            for (int k = 0; k < OWN; ++k) {
                if (!src[k]) continue;
                const float* s = src[k] + (size_t)t0 * ld[k];
                float* d = buf + tid + 128 * k;
#pragma unroll 4
                for (int tt = 0; tt < nt; ++tt, s += ld[k], d += STRIDE) cp_async4(d, s);
            }
        };
        auto prepare_sync = []() { asm volatile("bar.sync 1, 128;" ::: "memory"); };      // the fetching threads alone
        float m_run = 0.0f;
        if (MODE == SCAN_MLSTM) {
            // every tile and thread of the layout holds the maximum; this block's first tile is its own, whatever a thread's columns
            m_run = p.state[(size_t)slot * p.slot_stride + ((size_t)head * old_tiles + col0 / OLD_CB) * TILE_FLOATS + 2 * NPER * 128];
        }
        auto prepare = [&](int batch) {
            float* cur = staged + batch % WALK_BUFS * TOK * STRIDE;
            const int nt = min(TOK, n - batch * TOK);
            // what needs no state
            if (DELTA) {
                // unit vectors: a warp sums a token's squares (eight tokens a warp, their butterflies side by side)
#pragma unroll 2
                for (int tt = warp; tt < nt; tt += 4) {
                    float* tk = cur + tt * STRIDE;
                    float qq = 0.0f, kk = 0.0f;
#pragma unroll
                    for (int d = 0; d < ROWS; d += 32)
                        if (d + lane < ROWS) {
                            qq = fmaf(tk[d + lane], tk[d + lane], qq);
                            kk = fmaf(tk[ROWS + d + lane], tk[ROWS + d + lane], kk);
                        }
                    qq = warp_sum(qq);
                    kk = warp_sum(kk);
                    const float qs = p.q_scale / sqrtf(qq + 1e-6f), ks = 1.0f / sqrtf(kk + 1e-6f);
#pragma unroll
                    for (int d = 0; d < ROWS; d += 32)
                        if (d + lane < ROWS) {
                            tk[d + lane] *= qs;
                            tk[ROWS + d + lane] *= ks;
                        }
                }
                if (tid < nt) {
                    float* tk = cur + tid * STRIDE + TAIL;
                    tk[0] = expf(-A * softplus_f(tk[0] + bias));                                   // the decay
                    tk[1] = sigmoid_f(tk[1]);                                                      // beta
                }
            } else if (MODE == SCAN_GLA) {
#pragma unroll 4
                for (int e = tid; e < nt * ROWS; e += 128) {
                    float* tk = cur + (e / ROWS) * STRIDE + e % ROWS;
                    tk[0] *= p.q_scale;
                    if (!p.decays_ready) tk[2 * ROWS] = expf(log_sigmoid_f(tk[2 * ROWS]) * p.c0);
                }
            } else if (MODE == SCAN_MLSTM) {
                float li = 0.0f, lf = 0.0f;
                if (warp == 0) {
                    // the running maximum, token after token in every lane; a lane keeps its own token's
                    if (lane < nt) {
                        const float* tk = cur + lane * STRIDE + TAIL;
                        li = p.c0 * tanhf((tk[0] + bias) / p.c0);                                  // log of the input gate
                        lf = log_sigmoid_f(p.c0 * tanhf((tk[1] + A) / p.c0));                      // log of the forget gate
                    }
                    float m = m_run, before = m_run, after = m_run;
                    for (int tt = 0; tt < nt; ++tt) {
                        const float i = __shfl_sync(0xffffffffu, li, tt), f = __shfl_sync(0xffffffffu, lf, tt);
                        const float mn = fmaxf(f + m, i);
                        if (lane == tt) { before = m; after = mn; }
                        m = mn;
                    }
                    if (lane < nt) {
                        float* tk = cur + lane * STRIDE + TAIL;
                        tk[0] = expf(lf + before - after);                                         // keep
                        tk[1] = expf(li - after);                                                  // take
                        tk[2] = expf(-after);
                        tk[3] = after;
                    }
                }
                prepare_sync();
                m_run = cur[(nt - 1) * STRIDE + TAIL + 3];
                if (tid == 0 && batch == batches - 1) m_last = m_run;
#pragma unroll 4
                for (int e = tid; e < nt * ROWS; e += 128) {
                    float* tk = cur + (e / ROWS) * STRIDE;
                    tk[e % ROWS] *= p.q_scale;
                    tk[ROWS + e % ROWS] *= tk[TAIL + 1];
                }
            } else if (tid < nt) {
                float* tk = cur + tid * STRIDE + TAIL;
                const float dt = softplus_f(tk[0] + bias);
                tk[0] = dt;
                tk[1] = expf(-A * dt);
            }
        };
        // columns past the last read as zero in every staged token
        for (int i = tid; i < WALK_BUFS * TOK * CB; i += 128) {
            const int t = i / CB, c = i - t * CB;
            if (col0 + c >= p.cols) staged[t * STRIDE + NVEC * ROWS + c] = 0.0f;
        }
        stage(0, staged);
        cp_async_commit();
        if (batches > 1) stage(TOK, staged + TOK * STRIDE);
        cp_async_commit();
        cp_async_wait<1>();
        prepare_sync();
        prepare(0);
        for (int batch = 0; batch < batches; ++batch) {
            __syncthreads();                    // batch is ready, and the one before it walked: its buffer takes the one after next
            if (batch + 2 < batches) stage((batch + 2) * TOK, staged + (batch + 2) % WALK_BUFS * TOK * STRIDE);
            cp_async_commit();
            if (batch + 1 < batches) {
                cp_async_wait<1>();
                prepare_sync();
                prepare(batch + 1);
            }
        }
        return;
    }

    // the state, in scan_kernel's layout: (tile of OLD_CB columns, i, thread of that kernel)
    float* S[C];
    bool live[C];
    float s[C][NPER];
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const int col = col0 + lcol + CPW * k, in = col % OLD_CB;
        live[k] = col / OLD_CB < old_tiles;                               // (columns that only pad the last tile belong to the layout)
        S[k] = p.state + (size_t)slot * p.slot_stride + ((size_t)head * old_tiles + col / OLD_CB) * TILE_FLOATS
               + (in / CPW) * 32 + part * CPW + in % CPW;
#pragma unroll
        for (int i = 0; i < NPER; ++i) s[k][i] = live[k] ? S[k][i * 128] : 0.0f;
    }
    const float skip = MODE == SCAN_SSD ? p.skip[head] : 0.0f;
    float nvec[MODE == SCAN_MLSTM ? NPER : 1];
    if (MODE == SCAN_MLSTM) {
#pragma unroll
        for (int i = 0; i < NPER; ++i) nvec[i] = live[0] ? S[0][(NPER + i) * 128] : 0.0f;
    }
    // which finished value a lane is left with: token `my_u` of the batch, column `my_k` of the thread's
    int my = 0;
#pragma unroll
    for (int b = 0, w = V >> 1; w > 0; ++b, w >>= 1) my += (lane & (DP == 32 ? 16 >> b : CPW << b)) ? w : 0;
    const int my_u = my / C, my_k = my % C, my_col = lcol + CPW * my_k;
    float* out = p.out + (size_t)first * p.heads * p.cols + head * p.cols + col0 + my_col;
    const size_t out_ld = (size_t)p.heads * p.cols;
    const bool writer = col0 + my_col < p.cols;

    for (int batch = 0; batch < batches; ++batch) {
        const float* cur = staged + batch % WALK_BUFS * TOK * STRIDE;
        const int t0 = batch * TOK, nt = min(TOK, n - t0);
        __syncthreads();                        // the batch is ready
        auto walk = [&](int b0, int nu, auto whole) {
            constexpr bool WHOLE = decltype(whole)::value;
            float y[V], nq[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!WHOLE && u >= nu) {
#pragma unroll
                    for (int k = 0; k < C; ++k) y[u * C + k] = 0.0f;
                    nq[u] = 0.0f;
                    continue;
                }
                const float* tk = cur + (b0 + u) * STRIDE;
                float a[NPER], b[NPER], xv[C];
#pragma unroll
                for (int i = 0; i < NPER; i += 4) {
                    const float4 va = *(const float4*)(tk + part * NPER + i);
                    const float4 vb = *(const float4*)(tk + ROWS + part * NPER + i);
                    a[i] = va.x; a[i + 1] = va.y; a[i + 2] = va.z; a[i + 3] = va.w;
                    b[i] = vb.x; b[i + 1] = vb.y; b[i + 2] = vb.z; b[i + 3] = vb.w;
                }
#pragma unroll
                for (int k = 0; k < C; ++k) xv[k] = tk[NVEC * ROWS + lcol + CPW * k];
                if (DELTA) {
                    const float decay = tk[TAIL], beta = tk[TAIL + 1];
                    float dot[C];
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        dot[k] = 0.0f;
#pragma unroll
                        for (int i = 0; i < NPER; ++i) {
                            s[k][i] *= decay;
                            dot[k] = fmaf(s[k][i], b[i], dot[k]);
                        }
                    }
#pragma unroll
                    for (int st = 0; st < (DP == 8 ? 3 : DP == 16 ? 4 : 5); ++st)
#pragma unroll
                        for (int k = 0; k < C; ++k) dot[k] += __shfl_xor_sync(0xffffffffu, dot[k], DP == 32 ? 16 >> st : CPW << st);
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        const float w = beta * (xv[k] - dot[k]);
                        float sum = 0.0f;
#pragma unroll
                        for (int i = 0; i < NPER; ++i) {
                            s[k][i] = fmaf(b[i], w, s[k][i]);
                            sum = fmaf(s[k][i], a[i], sum);
                        }
                        y[u * C + k] = sum;
                    }
                } else if (MODE == SCAN_GLA) {
#pragma unroll
                    for (int k = 0; k < C; ++k) y[u * C + k] = 0.0f;
#pragma unroll
                    for (int i = 0; i < NPER; i += 4) {
                        const float4 d4 = *(const float4*)(tk + 2 * ROWS + part * NPER + i);
                        const float d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j)
#pragma unroll
                            for (int k = 0; k < C; ++k) {
                                s[k][i + j] = fmaf(d[j], s[k][i + j], __fmul_rn(b[i + j], xv[k]));
                                y[u * C + k] = fmaf(s[k][i + j], a[i + j], y[u * C + k]);
                            }
                    }
                } else if (MODE == SCAN_MLSTM) {
                    const float keep = tk[TAIL];
                    nq[u] = 0.0f;
#pragma unroll
                    for (int i = 0; i < NPER; ++i) {
                        nvec[i] = fmaf(keep, nvec[i], b[i]);
                        nq[u] = fmaf(nvec[i], a[i], nq[u]);
                    }
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        float sum = 0.0f;
#pragma unroll
                        for (int i = 0; i < NPER; ++i) {
                            s[k][i] = fmaf(keep, s[k][i], __fmul_rn(b[i], xv[k]));
                            sum = fmaf(s[k][i], a[i], sum);
                        }
                        y[u * C + k] = sum;
                    }
                } else {
                    const float dt = tk[TAIL], decay = tk[TAIL + 1];
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        const float dx = dt * xv[k];
                        float sum = 0.0f;
#pragma unroll
                        for (int i = 0; i < NPER; ++i) {
                            s[k][i] = fmaf(decay, s[k][i], __fmul_rn(a[i], dx));
                            sum = fmaf(s[k][i], b[i], sum);
                        }
                        y[u * C + k] = sum;
                    }
                }
            }
            halve_sum<DP, V, 0>(y, lane);
            if (MODE == SCAN_MLSTM) halve_sum<DP, U, 0>(nq, lane);
            if (writer && (WHOLE || my_u < nu)) {
                const float* tk = cur + (b0 + my_u) * STRIDE;
                float v = y[0];
                if (MODE == SCAN_SSD) v = fmaf(skip, tk[NVEC * ROWS + my_col], v);
                if (MODE == SCAN_MLSTM) v = v / (fmaxf(fabsf(nq[0]), tk[TAIL + 2]) + p.c1);
                out[(size_t)(t0 + b0 + my_u) * out_ld] = v;
            }
        };
        int b0 = 0;
#pragma unroll 1
        for (; b0 + U <= nt; b0 += U) walk(b0, U, std::true_type{});
        if (b0 < nt) walk(b0, nt - b0, std::false_type{});
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
        if (!live[k]) continue;
#pragma unroll
        for (int i = 0; i < NPER; ++i) S[k][i * 128] = s[k][i];
        if (MODE == SCAN_MLSTM) {
#pragma unroll
            for (int i = 0; i < NPER; ++i) S[k][(NPER + i) * 128] = nvec[i];
            S[k][2 * NPER * 128] = m_last;        // (written before the last barrier)
        }
    }
}

// ---------------------------------------------------------------------------------
// y * silu(z) and an RMS over equal parts of the row, in either order:
//   gate_first:  v = y * silu(z);  out = v / rms_part(v) * w
//   else:        out = y / rms_part(y) * w * silu(z)
// (bit 0 of `gate_first` is the order; bit 1 set: the gate is sigmoid(z) instead of silu(z))
// w has w_len entries and is indexed by (column % w_len): a weight per column of the row,
// or one shared by all parts.  One warp per part.
// ---------------------------------------------------------------------------------
template <typename TO>
__global__ void gated_group_norm_kernel(const float* __restrict__ y, int n, int part_len, const float* __restrict__ z, int ld_z,
                                        const float* __restrict__ w, int w_len, float eps, int gate_first,
                                        TO* __restrict__ out) {
    cj::after_predecessor();
    cj::release_successor();
    const int r = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int parts = n / part_len;
    const bool plain_sigmoid = (gate_first & 2) != 0;
    gate_first &= 1;
    for (int g = blockIdx.y * nw + warp; g < parts; g += gridDim.y * nw) {
        const float* yr = y + (size_t)r * n + (size_t)g * part_len;
        const float* zr = z + (size_t)r * ld_z + (size_t)g * part_len;
        float ss = 0.0f;
        for (int i = lane; i < part_len; i += 32) {
            float v = yr[i];
            if (gate_first) { const float zz = zr[i]; v *= (plain_sigmoid ? 1.0f : zz) / (1.0f + expf(-zz)); }
            ss = fmaf(v, v, ss);
        }
        ss = warp_sum(ss);
        const float scale = 1.0f / sqrtf(ss / (float)part_len + eps);
        for (int i = lane; i < part_len; i += 32) {
            const float zz = zr[i];
            const float gate = (plain_sigmoid ? 1.0f : zz) / (1.0f + expf(-zz));
            const int c = g * part_len + i;
            float v = yr[i];
            v = gate_first ? (v * gate) * scale * w[c % w_len] : v * scale * w[c % w_len] * gate;
            out[(size_t)r * n + c] = from_f32<TO>(v);
        }
    }
}

// The same for parts of 32 NV entries: a lane keeps its entries, so y and z are read and the gate is worked out once.  The operations and
// their order are the kernel's above, so both give the same bits.  2,048 rows of 8 parts of 512 out of HBM: 49.9 us with the kernel above,
// 16.1 with this one; of 16 parts of 128: 24.9 and 11.4.
template <typename TO, int NV>
__global__ void gated_group_norm_kept_kernel(const float* __restrict__ y, int n, const float* __restrict__ z, int ld_z, const float* __restrict__ w,
                                             int w_len, float eps, int gate_first, TO* __restrict__ out) {
    cj::after_predecessor();
    cj::release_successor();
    constexpr int PART = 32 * NV;
    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, parts = n / PART;
    const bool plain_sigmoid = (gate_first & 2) != 0, first = (gate_first & 1) != 0;
    for (int g = blockIdx.y * nw + warp; g < parts; g += gridDim.y * nw) {
        const int c0 = g * PART + lane;
        const float* yr = y + (size_t)r * n + c0;
        const float* zr = z + (size_t)r * ld_z + c0;
        float v[NV], gate[NV], ss = 0.0f;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            v[k] = yr[32 * k];
            gate[k] = zr[32 * k];
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            gate[k] = (plain_sigmoid ? 1.0f : gate[k]) / (1.0f + expf(-gate[k]));
            if (first) v[k] *= gate[k];
            ss = fmaf(v[k], v[k], ss);
        }
        ss = warp_sum(ss);
        const float scale = 1.0f / sqrtf(ss / (float)PART + eps);
        const float* wp = w + c0 % w_len;                    // (w_len is a multiple of the part)
        TO* o = out + (size_t)r * n + c0;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const float u = v[k] * scale * wp[32 * k];
            o[32 * k] = from_f32<TO>(first ? u : u * gate[k]);
        }
    }
}

// out (+)= c (a / rms(a) * wa + b / rms(b) * wb): the results of two mixers that read the same input, each
// RMS-normed over the row with a weight of its own, averaged (c = 1/2) or summed.  A block a row.
__global__ void rmsnorm_mix2_kernel(const float* __restrict__ a, const float* __restrict__ wa, const float* __restrict__ b,
                                    const float* __restrict__ wb, float eps, float c, int accumulate, float* __restrict__ out, int H) {
    cj::after_predecessor();
    cj::release_successor();
    __shared__ float scratch[32];
    const float* ra = a + (size_t)blockIdx.x * H;
    const float* rb = b + (size_t)blockIdx.x * H;
    float* dst = out + (size_t)blockIdx.x * H;
    float sa = 0.0f, sb = 0.0f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        sa = fmaf(ra[i], ra[i], sa);
        sb = fmaf(rb[i], rb[i], sb);
    }
    sa = block_sum(sa, scratch);
    sb = block_sum(sb, scratch);
    const float fa = 1.0f / sqrtf(sa / (float)H + eps), fb = 1.0f / sqrtf(sb / (float)H + eps);
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const float v = c * (ra[i] * fa * wa[i] + rb[i] * fb * wb[i]);
        dst[i] = accumulate ? dst[i] + v : v;
    }
}

// The same for widths that are multiples of four, 512 to 4,096, everything on 16 bytes: a thread keeps its NV float4 of both rows, which are read
// once.  The squares are added in the order of the kernel above with `order` threads, from shared memory, as in rmsnorm_add4_kernel: the
// same bits.  Bound by memory: 1,511 rows of 2,048, cold, 20.2 us with the kernel above, 12.4 so
template <int NV>
__global__ void __launch_bounds__(256) rmsnorm_mix2_vec_kernel(const float* __restrict__ a, const float* __restrict__ wa, const float* __restrict__ b,
                                                               const float* __restrict__ wb, float eps, float c, int accumulate, float* __restrict__ out,
                                                               int H, int order) {
    cj::after_predecessor();
    cj::release_successor();
    __shared__ __align__(16) float row[2][1024 * NV];
    __shared__ float sums[2][16];
    const float4* ra = (const float4*)(a + (size_t)blockIdx.x * H);
    const float4* rb = (const float4*)(b + (size_t)blockIdx.x * H);
    float4* dst = (float4*)(out + (size_t)blockIdx.x * H);
    const int n4 = H / 4;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 va[NV], vb[NV], old[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        va[k] = vb[k] = old[k] = zero;
        if (i < n4) {
            va[k] = ra[i];
            vb[k] = rb[i];
            if (accumulate) old[k] = dst[i];
            *(float4*)(row[0] + 4 * i) = va[k];
            *(float4*)(row[1] + 4 * i) = vb[k];
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < order; t += 256) {
        float sa = 0.0f, sb = 0.0f;
        for (int i = t; i < H; i += order) {
            sa = fmaf(row[0][i], row[0][i], sa);
            sb = fmaf(row[1][i], row[1][i], sb);
        }
        sa = warp_sum(sa);
        sb = warp_sum(sb);
        if ((t & 31) == 0) { sums[0][t >> 5] = sa; sums[1][t >> 5] = sb; }
    }
    __syncthreads();
    float sa = 0.0f, sb = 0.0f;
    for (int i = 0; i < order / 32; ++i) {
        sa += sums[0][i];
        sb += sums[1][i];
    }
    const float fa = 1.0f / sqrtf(sa / (float)H + eps), fb = 1.0f / sqrtf(sb / (float)H + eps);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        if (i >= n4) continue;
        const float4 ga = ((const float4*)wa)[i], gb = ((const float4*)wb)[i];
        auto mixed = [&](float x, float g, float y, float h, float o) {
            const float v = c * (x * fa * g + y * fb * h);
            return accumulate ? o + v : v;
        };
        dst[i] = make_float4(mixed(va[k].x, ga.x, vb[k].x, gb.x, old[k].x), mixed(va[k].y, ga.y, vb[k].y, gb.y, old[k].y),
                             mixed(va[k].z, ga.z, vb[k].z, gb.z, old[k].z), mixed(va[k].w, ga.w, vb[k].w, gb.w, old[k].w));
    }
}

// x <- cap tanh(x / cap), in place, float32
__global__ void softcap_rows_kernel(float* __restrict__ x, float cap, long long n) {
    cj::after_predecessor();
    cj::release_successor();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] = cap * tanhf(x[i] / cap);
}

// ---------------------------------------------------------------------------------
// A gated recurrence channel by channel whose gates read the current token alone (minGRU):
//     z = sigmoid(zp) ; c = u + 1/2 for u >= 0, sigmoid(u) below ; S_t = (1 - z) S_(t-1) + z c ; out = S_t silu(g)
// zp, u and g are columns off_z + k, off_x + k, off_g + k of the step's projected rows (biases included).  Because the
// gates do not read the state, a stretch of tokens is one affine map S -> A S + B, and stretches compose: a block takes
// CT neighbouring channels of one request, a thread PER consecutive tokens of a channel (their a = 1 - z and b = z c in
// registers), a warp composes the maps of a channel's stretches by a prefix scan, and every thread
// then walks its tokens from the state its stretch begins with.  A request is cut into tiles from its own first row of the
// step; requests of a few tokens (single decoded ones) are walked by a thread a channel instead, in the leading blocks.
// Everything is float32 but the result.
// ---------------------------------------------------------------------------------
struct GatedScanArgs {
    const float* x;
    int ld, off_z, off_x, off_g, width;
    float* state;
    long long slot_stride;
    const int* req_start;
    const int* req_slot;
    int vec;         // rows and column offsets on 16-byte boundaries
    int single;      // every request brings one token
};

// e^x, 1 / x: CUDA's own for float32 results; FAST (results rounded to bfloat16): the special-function unit's, a few units in
// the last place of float32
template <bool FAST> __device__ __forceinline__ float gs_exp(float x) {
    if (!FAST) return expf(x);
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
    return y;
}
template <bool FAST> __device__ __forceinline__ float gs_rcp(float x) {
    if (!FAST) return 1.0f / x;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <bool FAST> __device__ __forceinline__ float gs_silu(float x) { return x * gs_rcp<FAST>(1.0f + gs_exp<FAST>(-fmaxf(x, -80.0f))); }

// a = 1 - z and b = z c; both sides of the sigmoid come from one exponential, so neither loses digits near 0 or 1
template <bool FAST>
__device__ __forceinline__ void gated_step(float zp, float u, float& a, float& b) {
    const float e = gs_exp<FAST>(-fabsf(zp)), big = gs_rcp<FAST>(1.0f + e), small = e * big;
    const float z = zp >= 0.0f ? big : small;
    a = zp >= 0.0f ? small : big;
    const float below = gs_rcp<FAST>(1.0f + gs_exp<FAST>(fminf(-u, 80.0f)));      // sigmoid(u); the bound keeps e^(-u) finite
    b = z * (u >= 0.0f ? u + 0.5f : below);
}

constexpr int GS_WALK = 16;          // a request of at most this many tokens is walked by a thread a channel

// 16 bytes, or four times 4 where the rows are not aligned for that, on their way to shared memory
__device__ __forceinline__ void cp_async16(float* smem, const float* gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}

// A block takes CT (8, 16 or 32) neighbouring channels and 32 CT threads: 32 stretches of PER tokens each make a tile.  The
// next tile's pre-activations travel to shared memory (cp.async) while this one is worked on; a stretch's tokens lie CT floats
// apart and stretches CT (PER + 1), which keeps the reads of a warp (CT channels of 32 / CT stretches) in different banks.
constexpr int GS_SEG = 32;
template <int CT, int PER> struct GatedScanTile {
    static constexpr int TOKENS = GS_SEG * PER, PLANE = GS_SEG * CT * (PER + 1), FLOATS = 3 * PLANE, BYTES = 2 * FLOATS * 4;
};

template <typename TO, int CT, int PER, int BLOCKS>
__global__ void __launch_bounds__(32 * CT, BLOCKS) gated_scan_kernel(GatedScanArgs p, TO* __restrict__ out) {
    cj::after_predecessor();
    cj::release_successor();
    constexpr bool FAST = sizeof(TO) == 2;
    using Tile = GatedScanTile<CT, PER>;
    constexpr int THREADS = 32 * CT;
    extern __shared__ __align__(16) float gs_buf[];             // [2][z | x | g]
    __shared__ float As[GS_SEG][CT + 1], Bs[GS_SEG][CT + 1];      // a stretch's map, then (in Bs) the state it begins with
    __shared__ float carry[CT];
    const int req = blockIdx.y;
    const int slot = p.req_slot[req];
    const int first = p.req_start[req], n = p.req_start[req + 1] - first;
    if (slot < 0 || n <= 0) return;
    float* st = p.state + (size_t)slot * p.slot_stride;
    if (n <= GS_WALK || p.single) {
        // a thread a channel: the launch has at least enough blocks of its size for all channels
        const int c = blockIdx.x * blockDim.x + threadIdx.x;
        if (c >= p.width) return;
        float S = st[c];
        for (int t = 0; t < n; ++t) {
            const float* row = p.x + (size_t)(first + t) * p.ld;
            const float g = row[p.off_g + c];
            float a, b;
            gated_step<FAST>(row[p.off_z + c], row[p.off_x + c], a, b);
            S = fmaf(a, S, b);
            out[(size_t)(first + t) * p.width + c] = from_f32<TO>(S * gs_silu<FAST>(g));
        }
        st[c] = S;
        return;
    }
    const int c0 = blockIdx.x * CT, nch = min(CT, p.width - c0);
    const int ch = threadIdx.x % CT, seg = threadIdx.x / CT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool live = ch < nch;
    auto fetch = [&](int tile0, float* buf) {
        const int rows = min(Tile::TOKENS, n - tile0);
        const float* src = p.x + (size_t)(first + tile0) * p.ld + c0;
        if (p.vec && nch == CT) {
            for (int e = threadIdx.x; e < Tile::TOKENS * (CT / 4); e += THREADS) {
                const int t = e / (CT / 4), h = (e % (CT / 4)) * 4;
                if (t >= rows) break;
                const float* r = src + (size_t)t * p.ld + h;
                float* d = buf + (t + t / PER) * CT + h;
                cp_async16(d, r + p.off_z);
                cp_async16(d + Tile::PLANE, r + p.off_x);
                cp_async16(d + 2 * Tile::PLANE, r + p.off_g);
            }
        } else {
            for (int e = threadIdx.x; e < Tile::TOKENS * CT; e += THREADS) {
                const int t = e / CT, k = e % CT;
                if (t >= rows) break;
                if (k >= nch) continue;
                const float* r = src + (size_t)t * p.ld + k;
                float* d = buf + (t + t / PER) * CT + k;
                cp_async4(d, r + p.off_z);
                cp_async4(d + Tile::PLANE, r + p.off_x);
                cp_async4(d + 2 * Tile::PLANE, r + p.off_g);
            }
        }
    };
    if (threadIdx.x < CT) carry[threadIdx.x] = live ? st[c0 + ch] : 0.0f;
    fetch(0, gs_buf);
    cp_async_commit();
    int cur = 0;
    for (int tile0 = 0; tile0 < n; tile0 += Tile::TOKENS, cur ^= 1) {
        if (tile0 + Tile::TOKENS < n) fetch(tile0 + Tile::TOKENS, gs_buf + (cur ^ 1) * Tile::FLOATS);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const float* mine = gs_buf + cur * Tile::FLOATS + seg * CT * (PER + 1) + ch;
        const int t0 = tile0 + seg * PER;
        const int have = live ? min(PER, n - t0) : 0;           // tokens of this stretch (none: zero or below)
        float a[PER], b[PER];
        float A = 1.0f, B = 0.0f;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            float ai, bi;
            gated_step<FAST>(mine[i * CT], mine[Tile::PLANE + i * CT], ai, bi);
            a[i] = i < have ? ai : 1.0f;                        // past the end (whatever lies there): the map that changes nothing
            b[i] = i < have ? bi : 0.0f;
            A *= a[i];
            B = fmaf(a[i], B, b[i]);
        }
        As[seg][ch] = A;
        Bs[seg][ch] = B;
        __syncthreads();
        {
            // a warp a channel: its 32 stretches' maps composed by a prefix scan over the lanes
            float ta = As[lane][warp], tb = Bs[lane][warp];
            const float S0 = carry[warp];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float pa = __shfl_up_sync(0xffffffffu, ta, o), pb = __shfl_up_sync(0xffffffffu, tb, o);
                if (lane >= o) {
                    tb = fmaf(ta, pb, tb);
                    ta *= pa;
                }
            }
            const float end = fmaf(ta, S0, tb);                 // the state after this lane's stretch
            float begin = __shfl_up_sync(0xffffffffu, end, 1);
            if (lane == 0) begin = S0;
            Bs[lane][warp] = begin;
            __syncwarp();
            if (lane == 31) carry[warp] = end;
        }
        __syncthreads();
        float S = Bs[seg][ch];
        TO* dst = out + (size_t)(first + t0) * p.width + c0 + ch;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            S = fmaf(a[i], S, b[i]);
            if (i < have) dst[(size_t)i * p.width] = from_f32<TO>(S * gs_silu<FAST>(mine[2 * Tile::PLANE + i * CT]));
        }
        __syncthreads();                                        // this buffer and Bs are read before the next tile writes them
    }
    if (threadIdx.x < nch) st[c0 + threadIdx.x] = carry[threadIdx.x];
}

}  // namespace

// Lanes a column's rows are dealt to (4, 8, 16 or 32).  Every (column, token) costs a warp its staging,
// its butterflies and its store whatever the lanes hold, so fewer lanes a column - more columns a
// warp - mean fewer instructions in all; but one request's scan is a chain, and with too few warps
// the chain's latencies lie bare.  So: the fewest lanes (at least 8 where there are 8 rows) that
// still give ONE request's scan a warp for each of a B200's 592 warp schedulers; and few enough rows
// a lane (64) to stay in registers.  Measured on two scans of a 2,048-token prompt, 8 / 16 / 32 lanes:
// 32 + 8 heads 2.40 / 2.46 / 2.36 ms (all short of warps), 64 + 16 heads 2.63 / 2.85 / 3.64 ms.
// The state's layout follows from this number, so it depends on the state's shape alone.
static int scan_lanes(int heads, int rows, int cols) {
    int dp = 4;
    while (dp < 32 && dp < rows && (dp < 8 || (long long)heads * cols * dp / 32 < 592)) dp <<= 1;
    while (dp < 32 && (rows + dp - 1) / dp > 64) dp <<= 1;
    return dp;
}

CJ_EXPORT int cj_cast_rows(const float* x, void* out, int out_dtype, long long n, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (!x || !out) return CJ_ERR_ARG;
    if (out_dtype != CJ_F32 && out_dtype != CJ_BF16) return CJ_ERR_DTYPE;
    if (n % 4 == 0 && (((uintptr_t)x | (uintptr_t)out) & 15) == 0) {
        const dim3 grid((unsigned)min((n / 4 + 255) / 256, (long long)148 * 16));
        if (out_dtype == CJ_F32) cj::launch(cast_rows4_kernel<float>, grid, dim3(256), 0, stream, (const float4*)x, (float*)out, n / 4);
        else cj::launch(cast_rows4_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, (const float4*)x, (__nv_bfloat16*)out, n / 4);
        return launch_status();
    }
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (out_dtype == CJ_F32) cj::launch(cast_rows_kernel<float>, dim3((unsigned)blocks), dim3(256), 0, stream, x, (float*)out, n);
    else cj::launch(cast_rows_kernel<__nv_bfloat16>, dim3((unsigned)blocks), dim3(256), 0, stream, x, (__nv_bfloat16*)out, n);
    return launch_status();
}

CJ_EXPORT int cj_rmsnorm_add(float* hs, const float* y, const float* w, float eps, int rows, int H, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (!hs || !y || !w || H <= 0) return CJ_ERR_ARG;
    const int threads = H >= 2048 ? 512 : (H >= 512 ? 256 : 128);
    if (H % 4 == 0 && H <= 8192 && (((uintptr_t)hs | (uintptr_t)y | (uintptr_t)w) & 15) == 0) {
#define LAUNCH_NV(NV) cj::launch(rmsnorm_add4_kernel<NV>, dim3(rows), dim3(256), 0, stream, hs, y, w, eps, H, threads)
        if (H <= 1024) LAUNCH_NV(1);
        else if (H <= 2048) LAUNCH_NV(2);
        else if (H <= 4096) LAUNCH_NV(4);
        else LAUNCH_NV(8);
#undef LAUNCH_NV
        return launch_status();
    }
    cj::launch(rmsnorm_add_kernel, dim3(rows), dim3(threads), 0, stream, hs, y, w, eps, H);
    return launch_status();
}

CJ_EXPORT int cj_scale_rows_gather(const float* x, const int* slot_of_pick, const float* weight, int picks, int k, int H,
                                   void* out, int out_dtype, cudaStream_t stream) {
    if (picks <= 0) return 0;
    if (!x || !slot_of_pick || !weight || !out || k < 1 || H <= 0) return CJ_ERR_ARG;
    int threads = H >= 1024 ? 256 : 128;
    if (out_dtype == CJ_F32) cj::launch(scale_rows_gather_kernel<float>, dim3(picks), dim3(threads), 0, stream, x, slot_of_pick, weight, k, H, (float*)out);
    else if (out_dtype == CJ_BF16) cj::launch(scale_rows_gather_kernel<__nv_bfloat16>, dim3(picks), dim3(threads), 0, stream, x, slot_of_pick, weight, k, H, (__nv_bfloat16*)out);
    else return CJ_ERR_DTYPE;
    return launch_status();
}

constexpr int CONV_MIN_ROWS = 128;

CJ_EXPORT int cj_short_conv(const float* in, int ld_in, int C, int taps, const float* w, const float* bias, const float* state,
                            long long slot_stride, const int* row_req, const int* req_start, const int* req_slot, void* out,
                            int ld_out, int out_dtype, int act, int T, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (!in || !w || !state || !row_req || !req_start || !req_slot || !out || C <= 0 || taps < 1) return CJ_ERR_ARG;
    // many rows: four channels and 16 rows a thread.  From 128 rows on: 8 x 12 blocks for 6,144 channels, a block an SM nearly
    const int out_bytes = out_dtype == CJ_F32 ? 16 : 8;
    if (T >= CONV_MIN_ROWS && taps >= 2 && taps <= 4 && C <= 65535 * 512 && (C | ld_in | ld_out) % 4 == 0 && ((uintptr_t)in & 15) == 0 && (uintptr_t)out % out_bytes == 0
        && (out_dtype == CJ_F32 || out_dtype == CJ_BF16)) {
        const dim3 tiles((T + CONV_ROWS - 1) / CONV_ROWS, (C + 511) / 512);
#define LAUNCH_TILE(TO, N) cj::launch(short_conv_tile_kernel<TO, N>, tiles, dim3(128), 0, stream, in, ld_in, C, w, bias, state, slot_stride, row_req, \
                                      req_start, req_slot, (TO*)out, ld_out, act, T)
#define LAUNCH_TAPS(TO)                                                                                                 \
        if (taps == 2) LAUNCH_TILE(TO, 2);                                                                              \
        else if (taps == 3) LAUNCH_TILE(TO, 3);                                                                         \
        else LAUNCH_TILE(TO, 4)
        if (out_dtype == CJ_F32) { LAUNCH_TAPS(float); }
        else { LAUNCH_TAPS(__nv_bfloat16); }
#undef LAUNCH_TAPS
#undef LAUNCH_TILE
        return launch_status();
    }
    int threads = C >= 512 ? 256 : 128;
    int by = (C + threads - 1) / threads;
    if (by > 64) by = 64;
    dim3 grid(T, by);
    if (out_dtype == CJ_F32) cj::launch(short_conv_kernel<float>, grid, dim3(threads), 0, stream, in, ld_in, C, taps, w, bias, state, slot_stride, row_req, req_start, req_slot, (float*)out, ld_out, act);
    else if (out_dtype == CJ_BF16) cj::launch(short_conv_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream, in, ld_in, C, taps, w, bias, state, slot_stride, row_req, req_start, req_slot, (__nv_bfloat16*)out, ld_out, act);
    else return CJ_ERR_DTYPE;
    return launch_status();
}

// Every request brings one token: convolution and commit.  taps 2 to 4 (CJ_ERR_SIZE otherwise: cj_short_conv and cj_short_conv_commit).
CJ_EXPORT int cj_short_conv_single(const float* in, int ld_in, int C, int taps, const float* w, const float* bias, float* state,
                                   long long slot_stride, const int* row_req, const int* req_slot, void* out, int ld_out, int out_dtype, int act,
                                   int T, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (!in || !w || !state || !row_req || !req_slot || !out || C <= 0) return CJ_ERR_ARG;
    if (taps < 2 || taps > 4) return CJ_ERR_SIZE;
    const dim3 grid(T, min((C + 127) / 128, 65535));
#define LAUNCH_ONE(TO, N) cj::launch(short_conv_single_kernel<TO, N>, grid, dim3(128), 0, stream, in, ld_in, C, w, bias, state, slot_stride, row_req, \
                                     req_slot, (TO*)out, ld_out, act)
#define LAUNCH_TAPS(TO)                                                                                                 \
    if (taps == 2) LAUNCH_ONE(TO, 2);                                                                                   \
    else if (taps == 3) LAUNCH_ONE(TO, 3);                                                                              \
    else LAUNCH_ONE(TO, 4)
    if (out_dtype == CJ_F32) { LAUNCH_TAPS(float); }
    else if (out_dtype == CJ_BF16) { LAUNCH_TAPS(__nv_bfloat16); }
    else return CJ_ERR_DTYPE;
#undef LAUNCH_TAPS
#undef LAUNCH_ONE
    return launch_status();
}

CJ_EXPORT int cj_short_conv_commit(const float* in, int ld_in, int C, int taps, float* state, long long slot_stride,
                                   const int* req_start, const int* req_slot, int requests, cudaStream_t stream) {
    if (requests <= 0 || taps <= 1) return 0;
    if (!in || !state || !req_start || !req_slot || C <= 0) return CJ_ERR_ARG;
    int threads = C >= 512 ? 256 : 128;
    int by = (C + threads - 1) / threads;
    if (by > 64) by = 64;
    cj::launch(short_conv_commit_kernel, dim3(requests, by), dim3(threads), 0, stream, in, ld_in, C, taps, state, slot_stride, req_start, req_slot);
    return launch_status();
}

// mode 0: the state-space scan (off_a = B, off_b = C, off_v = x; off_dt in raw);
// mode 1: the gated delta rule (off_a = q, off_b = k, off_v = v; off_dt = decay input, off_beta in raw);
// mode 2: gated linear attention (off_a = q, off_b = k, off_v = v; raw columns off_dt + head * rows + d = the decays'
//         inputs; c0 = 1 / tau; A_log, dt_bias unused);
// mode 3: the matrix memory with exponential gating (off_a = q, off_b = k, off_v = v; raw columns off_dt + head = the
//         input gate's, off_beta + head = the forget gate's pre-activation; dt_bias = the input gate's bias, A_log = the
//         forget gate's; c0 = the gates' cap, c1 = the floor added to the read-out's divisor).
static long long scan_tile_floats(int mode, int nper) { return mode == 3 ? (long long)(2 * nper + 1) * 128 : (long long)nper * 128; }

// Tokens a request, on average over the step, from which on walk_kernel takes over: at 8 tokens for each of 8 requests it takes 18, 27,
// 17 and 19 us against scan_kernel's 27, 29, 30 and 30 (the four modes at the sizes above); at 4 the delta rule takes 24 against 18.
constexpr int WALK_MIN_ROWS = 8;

template <int DP, int NPER, int MODE, int C>
static int launch_walk_as(const ScanArgs& p, int requests, cudaStream_t stream) {
    constexpr int CB = 4 * (32 / DP) * C;
    constexpr int bytes = WALK_BUFS * walk_tok(MODE) * ((MODE == SCAN_GLA ? 3 : 2) * DP * NPER + CB + 4) * (int)sizeof(float);
    // more than half of an SM's shared memory: one block an SM
    constexpr int alone = bytes > 116 * 1024 ? bytes : 116 * 1024;
    static bool sized = false;
    static int sms = 0;
    if (!sized) {
        cudaError_t e = cudaFuncSetAttribute(walk_kernel<DP, NPER, MODE, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, alone);
        int dev = 0;
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        sized = true;
    }
    const dim3 grid(requests, p.heads, (p.cols + CB - 1) / CB);
    if (grid.z > 65535) return CJ_ERR_SIZE;
    // A grid that the machine holds a block an SM is made to spread: set up while the kernel before still runs, two of its blocks may
    // otherwise land on one SM, and the scan takes as long as those two (64 heads of 128 x 64, 2,048 tokens: 650 us instead of 274).
    const bool spread = (long long)grid.x * grid.y * grid.z <= sms;
    cj::launch(walk_kernel<DP, NPER, MODE, C>, grid, dim3(256), spread ? alone : bytes, stream, p);
    return launch_status();
}

static bool walk_built(int DP, int nper) { return DP * nper == 64 ? DP <= 16 : DP * nper == 128 && DP >= 8; }
// CJ_ERR_SIZE: not built for this share of the rows
static int launch_walk(int mode, int DP, int nper, const ScanArgs& p, int requests, cudaStream_t stream) {
#define WALK(D, N)                                                                                                      \
    if (DP == D && nper == N) {                                                                                         \
        switch (mode) {                                                                                                 \
            case SCAN_SSD: return launch_walk_as<D, N, SCAN_SSD, WALK_COLS>(p, requests, stream);                       \
            case SCAN_DELTA: return launch_walk_as<D, N, SCAN_DELTA, WALK_COLS>(p, requests, stream);                   \
            case SCAN_GLA: return launch_walk_as<D, N, SCAN_GLA, WALK_COLS>(p, requests, stream);                       \
            default: return launch_walk_as<D, N, SCAN_MLSTM, WALK_COLS>(p, requests, stream);                           \
        }                                                                                                               \
    }
    // 64 or 128 rows a state
    WALK(8, 8) WALK(8, 16) WALK(16, 4) WALK(16, 8) WALK(32, 4)
#undef WALK
    return CJ_ERR_SIZE;
}

// Whether cj_state_scan takes the kernel that walks several columns and tokens at a time (in mode 2 with a kernel ahead of it that works out the
// decays, where it is given room for them).
CJ_EXPORT int cj_state_scan_walks(int mode, int heads, int rows, int cols, int requests, int total_rows, long long state_floats) {
    if (heads <= 0 || rows <= 0 || cols <= 0 || requests <= 0 || heads > 65535 || total_rows < (long long)WALK_MIN_ROWS * requests) return 0;
    const int DP = scan_lanes(heads, rows, cols), per = (rows + DP - 1) / DP, cols_per_block = 4 * (32 / DP);
    int nper = 1;
    while (nper < per) nper <<= 1;
    const int tiles = (cols + cols_per_block - 1) / cols_per_block;
    return rows == DP * nper && walk_built(DP, nper) && state_floats >= (long long)heads * tiles * scan_tile_floats(mode, nper);
}

CJ_EXPORT int cj_state_scan(int mode, const float* x, int ld, int off_a, int off_b, int off_v, const float* raw, int ld_raw,
                            int off_dt, int off_beta, const float* A_log, const float* dt_bias, const float* skip, float* state,
                            long long slot_stride, long long state_floats, const int* req_start, const int* req_slot, float* out,
                            int requests, int total_rows, int heads, int groups, int rows, int cols, float q_scale, float c0, float c1,
                            float* decays, int single, cudaStream_t stream) {
    if (requests <= 0) return 0;
    if (mode < 0 || mode > 3) return CJ_ERR_ARG;
    if (!x || !raw || !state || !req_start || !req_slot || !out) return CJ_ERR_ARG;
    if (mode != 2 && (!A_log || !dt_bias)) return CJ_ERR_ARG;
    if (mode == 0 && !skip) return CJ_ERR_ARG;
    if ((mode == 2 || mode == 3) && !(c0 > 0.0f)) return CJ_ERR_ARG;
    if (heads <= 0 || groups <= 0 || heads % groups != 0 || rows <= 0 || cols <= 0) return CJ_ERR_SIZE;
    const int DP = scan_lanes(heads, rows, cols);
    const int per = (rows + DP - 1) / DP;
    if (per > 64) return CJ_ERR_SIZE;
    int nper = 1;
    while (nper < per) nper <<= 1;
    ScanArgs p{x, ld, off_a, off_b, off_v, raw, ld_raw, off_dt, off_beta, A_log, dt_bias, skip, state, slot_stride,
               req_start, req_slot, out, heads, groups, rows, cols, q_scale, 0, c0, c1};
    const int cols_per_block = 4 * (32 / DP);
    dim3 grid(requests, heads, (cols + cols_per_block - 1) / cols_per_block);
    if (cj_state_scan_walks(mode, heads, rows, cols, requests, total_rows, state_floats)) {
        // many tokens a request: the same results from the kernel that walks several columns and tokens at a time, where it is built
        ScanArgs w = p;
        if (mode == SCAN_GLA && decays) {
            const long long n = (long long)total_rows * heads * rows;
            cj::launch(gla_decays_kernel, dim3((unsigned)min((n + 255) / 256, (long long)148 * 16)), dim3(256), 0, stream, raw, ld_raw, off_dt,
                       heads * rows, n, c0, decays);
            w.raw = decays;
            w.ld_raw = heads * rows;
            w.off_dt = 0;
            w.decays_ready = 1;
        }
        const int st = launch_walk(mode, DP, nper, w, requests, stream);
        if (st != CJ_ERR_SIZE) return st;
    }
    if (grid.y > 65535 || grid.z > 65535) return CJ_ERR_SIZE;
    if (state_floats < (long long)heads * grid.z * scan_tile_floats(mode, nper)) return CJ_ERR_SIZE;
    // tokens staged at a time: up to 16, as many as 96 KB of shared memory hold twice
    const size_t token_bytes = (size_t)((mode == 2 ? 3 : 2) * DP * nper + cols_per_block + 4) * sizeof(float);
    int TOK = (int)((96 * 1024) / (2 * token_bytes));
    if (TOK > 16) TOK = 16;
    // single tokens: seven blocks an SM instead of six (8 requests, state-space and delta rule, cold: 13.0 and 13.6 us -> 11.2 and 11.4).  Said by
    // the caller: fewer rows than requests may also be a few of them with many, in a layout filled up with requests that bring none
    if (TOK > 1 && single) TOK = 1;
    if (TOK < 1) return CJ_ERR_SIZE;
    const size_t smem = 2 * (size_t)TOK * token_bytes;
#define LAUNCH_MODE(N, M)                                                                                               \
    do {                                                                                                                \
        static bool sized = false;                                                                                      \
        if (!sized) {                                                                                                   \
            cudaFuncSetAttribute(scan_kernel<N, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);            \
            sized = true;                                                                                               \
        }                                                                                                               \
        cj::launch(scan_kernel<N, M>, grid, dim3(128), smem, stream, p, DP, TOK);                                       \
    } while (0)
#define LAUNCH(N)                                                                                                       \
    do {                                                                                                                \
        if (mode == 0) LAUNCH_MODE(N, SCAN_SSD);                                                                        \
        else if (mode == 1) LAUNCH_MODE(N, SCAN_DELTA);                                                                 \
        else if (mode == 2) LAUNCH_MODE(N, SCAN_GLA);                                                                   \
        else LAUNCH_MODE(N, SCAN_MLSTM);                                                                                \
    } while (0)
    switch (nper) {
        case 1: LAUNCH(1); break;
        case 2: LAUNCH(2); break;
        case 4: LAUNCH(4); break;
        case 8: LAUNCH(8); break;
        case 16: LAUNCH(16); break;
        case 32: LAUNCH(32); break;
        default: LAUNCH(64);
    }
#undef LAUNCH
#undef LAUNCH_MODE
    return launch_status();
}

// floats of state one (slot, schedule entry) needs for heads matrices of rows x cols in the scan's own layout
// (mode 3 keeps a vector over the rows and a scalar beside every tile of a matrix)
CJ_EXPORT long long cj_state_scan_floats_mode(int mode, int heads, int rows, int cols) {
    if (heads <= 0 || rows <= 0 || cols <= 0) return 0;
    const int DP = scan_lanes(heads, rows, cols);
    const int per = (rows + DP - 1) / DP;
    int nper = 1;
    while (nper < per) nper <<= 1;
    const int cols_per_block = 4 * (32 / DP);
    return (long long)heads * ((cols + cols_per_block - 1) / cols_per_block) * scan_tile_floats(mode, nper);
}

CJ_EXPORT long long cj_state_scan_floats(int heads, int rows, int cols) { return cj_state_scan_floats_mode(0, heads, rows, cols); }

CJ_EXPORT int cj_gated_group_norm(const float* y, int n, int part_len, const float* z, int ld_z, const float* w, int w_len,
                                  float eps, int gate_first, void* out, int out_dtype, int rows, cudaStream_t stream) {
    // gate_first: bit 0 the gate multiplies before the norm's statistics, bit 1 the gate is sigmoid(z), not silu(z)
    if (rows <= 0) return 0;
    if (!y || !z || !w || !out || n <= 0 || part_len <= 0 || w_len <= 0) return CJ_ERR_ARG;
    if (n % part_len != 0) return CJ_ERR_SIZE;
    const int parts = n / part_len;
    int warps = parts < 8 ? parts : 8;
    int by = (parts + warps - 1) / warps;
    if (by > 64) by = 64;
    dim3 grid(rows, by);
    if ((part_len == 128 || part_len == 256 || part_len == 512 || part_len == 1024) && w_len % part_len == 0
        && (out_dtype == CJ_F32 || out_dtype == CJ_BF16)) {
#define LAUNCH_NV(TO, NV) cj::launch(gated_group_norm_kept_kernel<TO, NV>, grid, dim3(warps * 32), 0, stream, y, n, z, ld_z, w, w_len, eps, gate_first, (TO*)out)
#define LAUNCH_PART(TO)                                                                                                 \
        if (part_len == 128) LAUNCH_NV(TO, 4);                                                                          \
        else if (part_len == 256) LAUNCH_NV(TO, 8);                                                                     \
        else if (part_len == 512) LAUNCH_NV(TO, 16);                                                                    \
        else LAUNCH_NV(TO, 32)
        if (out_dtype == CJ_F32) { LAUNCH_PART(float); }
        else { LAUNCH_PART(__nv_bfloat16); }
#undef LAUNCH_PART
#undef LAUNCH_NV
        return launch_status();
    }
    if (out_dtype == CJ_F32) cj::launch(gated_group_norm_kernel<float>, grid, dim3(warps * 32), 0, stream, y, n, part_len, z, ld_z, w, w_len, eps, gate_first, (float*)out);
    else if (out_dtype == CJ_BF16) cj::launch(gated_group_norm_kernel<__nv_bfloat16>, grid, dim3(warps * 32), 0, stream, y, n, part_len, z, ld_z, w, w_len, eps, gate_first, (__nv_bfloat16*)out);
    else return CJ_ERR_DTYPE;
    return launch_status();
}

// x: float32 rows with stride ld holding the gate's, the candidate's and the output gate's pre-activations (biases included) at
// columns off_z, off_x, off_g; state: per slot `width` float32 from the given pointer on, slot_stride apart.  single: every
// request of the step brings one token.  out: [T, width] in out_dtype.
CJ_EXPORT int cj_gated_scan(const float* x, int ld, int off_z, int off_x, int off_g, int width, float* state, long long slot_stride,
                            const int* req_start, const int* req_slot, int requests, int single, void* out, int out_dtype,
                            cudaStream_t stream) {
    if (requests <= 0) return 0;
    if (!x || !state || !req_start || !req_slot || !out) return CJ_ERR_ARG;
    if (width <= 0 || ld < width || slot_stride < width || requests > 65535) return CJ_ERR_SIZE;
    const int vec = (ld | off_z | off_x | off_g) % 4 == 0 && ((uintptr_t)x & 15) == 0;
    GatedScanArgs p{x, ld, off_z, off_x, off_g, width, state, slot_stride, req_start, req_slot, vec, single};
    // single tokens: small blocks, a thread a channel, no tile.  Otherwise 16 channels a block (64-byte pieces of a row; measured
    // on 2,048 and 8,192 rows of 6,144 channels 55 / 184 us against 64 / 217 us with 8), or 8 where that leaves room on the SMs
    // (3,072 channels: 37 / 118 us against 41 / 127 us)
    const bool wide = (long long)((width + 15) / 16) * requests >= 2 * 148;
#define LAUNCH_CT(TO, CT, BLOCKS)                                                                                       \
    do {                                                                                                                \
        constexpr int bytes = GatedScanTile<CT, 8>::BYTES;                                                              \
        static bool sized = false;                                                                                      \
        if (!sized) {                                                                                                   \
            cudaFuncSetAttribute(gated_scan_kernel<TO, CT, 8, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); \
            sized = true;                                                                                               \
        }                                                                                                               \
        const dim3 grid(single ? (width + 127) / 128 : (width + CT - 1) / CT, requests);                                \
        cj::launch(gated_scan_kernel<TO, CT, 8, BLOCKS>, grid, dim3(single ? 128 : 32 * CT), single ? 0 : bytes, stream, p, (TO*)out); \
    } while (0)
#define LAUNCH(TO)                                                                                                      \
    do {                                                                                                                \
        if (wide) LAUNCH_CT(TO, 16, 2);                                                                                 \
        else LAUNCH_CT(TO, 8, 3);                                                                                       \
    } while (0)
    if (out_dtype == CJ_F32) LAUNCH(float);
    else if (out_dtype == CJ_BF16) LAUNCH(__nv_bfloat16);
    else return CJ_ERR_DTYPE;
#undef LAUNCH
#undef LAUNCH_CT
    return launch_status();
}

CJ_EXPORT int cj_rmsnorm_mix2(const float* a, const float* wa, const float* b, const float* wb, float eps, float c, int accumulate,
                              float* out, int rows, int H, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (!a || !wa || !b || !wb || !out || H <= 0) return CJ_ERR_ARG;
    int threads = H >= 2048 ? 512 : (H >= 512 ? 256 : 128);
    // (narrower rows leave most of its threads idle: 4,000 rows, us with the plain kernel and this one, 128 entries 10.2 and 15.6, 384 14.3 and 16.4, 448 16.4
    // and 17.0)
    if (H % 4 == 0 && H >= 512 && H <= 4096 && (((uintptr_t)a | (uintptr_t)wa | (uintptr_t)b | (uintptr_t)wb | (uintptr_t)out) & 15) == 0) {
#define MIX(NV) cj::launch(rmsnorm_mix2_vec_kernel<NV>, dim3(rows), dim3(256), 0, stream, a, wa, b, wb, eps, c, accumulate, out, H, threads)
        if (H <= 1024) MIX(1);
        else if (H <= 2048) MIX(2);
        else MIX(4);
#undef MIX
        return launch_status();
    }
    cj::launch(rmsnorm_mix2_kernel, dim3(rows), dim3(threads), 0, stream, a, wa, b, wb, eps, c, accumulate, out, H);
    return launch_status();
}

CJ_EXPORT int cj_softcap_rows(float* x, float cap, long long n, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (!x || !(cap > 0.0f)) return CJ_ERR_ARG;
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    cj::launch(softcap_rows_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, x, cap, n);
    return launch_status();
}
