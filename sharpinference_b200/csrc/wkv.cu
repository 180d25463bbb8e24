// The WKV recurrence (time mixing with a per-token, per-channel decay) in float32 from per-request state.
//
// Per head, key channel i and value channel j, for the rows of a request in order:
//     w_t = exp(-exp(wraw_t + w0))                                   the decay, in (0, 1)
//     o_t[j] = sum_i r_t[i] (S[i][j] + u[i] k_t[i] v_t[j])           the bonus u reaches the current token only
//     S[i][j] <- w_t[i] S[i][j] + k_t[i] v_t[j]
// then (sharpi_wkv_out) every head's o is divided by its root mean square, multiplied by a weight and by
// silu(gate), and rounded for the output projection.
//
// What does not depend on the state runs first, over all rows at once (wkv_prepare_kernel): the decay with its two
// exponentials, written over wraw, and the bonus' scalar b_t = sum_i r_t[i] u[i] k_t[i], so that
// o_t[j] = sum_i r_t[i] S[i][j] + b_t v_t[j].  The walk itself (wkv_scan_kernel) is one block a (request, head): a
// thread owns a tile of S (eight key channels of four value columns) in registers; r, k, w and v of the next rows
// arrive in shared memory by cp.async, two chunks of rows on their way while a third is walked (a chunk of sixteen
// rows is walked in less time than a chunk takes to arrive).  A request's rows are walked one after the
// other and a column's parts are added in a fixed order, so a row's result is the same sequence of operations
// whether it came in a prompt portion or alone.  Heads of more than 128 elements take the form in which
// a column's key channels are dealt over several threads (wkv_recurrence_kernel).
// Requests of many rows may run in chunks of 64 rows that work side by side, on the tensor cores (below).
#include "chunk_mma.cuh"
#include "common.cuh"

struct WkvArgs {
    const float* r;        // [T, heads * d]
    const float* k;
    const float* v;
    const float* wraw;     // [T, heads * d]: the decay before its two exponentials, without w0
    const float* w0;       // [heads * d]
    const float* u;        // [heads * d]
    const int* row_offsets;
    const int* state_slots;
    float* state;          // [slots, heads * d * d], [head][key][value]
    long long state_stride;
    float* o;              // [T, heads * d]
    int heads, d;
};

template <int KT>
__global__ void __launch_bounds__(1024) wkv_recurrence_kernel(WkvArgs a) {
    extern __shared__ float sm[];
    pdl_wait();
    const int d = a.d, head = blockIdx.x, b = blockIdx.y;
    const int parts = (d + KT - 1) / KT, dp = parts * KT;
    const int j = threadIdx.x % d, part = threadIdx.x / d;
    // shared: two buffers of (r, k, w, uk) [dp] each, two buffers of partial sums [parts][d]
    float* stage = sm;                        // [2][4][dp]
    float* red = sm + 2 * 4 * dp;             // [2][parts][d]
    const int first = a.row_offsets[b], end = a.row_offsets[b + 1];
    float* S_g = a.state + (size_t)a.state_slots[b] * a.state_stride + (size_t)head * d * d;
    float S[KT];
#pragma unroll
    for (int i = 0; i < KT; ++i) {
        const int key = part * KT + i;
        S[i] = key < d ? S_g[(size_t)key * d + j] : 0.0f;
    }
    const size_t hd = (size_t)a.heads * d, col = (size_t)head * d;
    auto load = [&](int t, int buf) {
        float* s = stage + buf * 4 * dp;
        for (int i = threadIdx.x; i < dp; i += blockDim.x) {
            float rv = 0.0f, kv = 0.0f, wv = 0.0f, uv = 0.0f;
            if (i < d) {
                rv = a.r[(size_t)t * hd + col + i];
                kv = a.k[(size_t)t * hd + col + i];
                wv = expf(-expf(a.wraw[(size_t)t * hd + col + i] + a.w0[col + i]));
                uv = a.u[col + i] * kv;
            }
            s[i] = rv; s[dp + i] = kv; s[2 * dp + i] = wv; s[3 * dp + i] = uv;
        }
    };
    if (first < end) load(first, 0);
    __syncthreads();
    for (int t = first; t < end; ++t) {
        const int buf = (t - first) & 1;
        const float* s = stage + buf * 4 * dp + part * KT;
        const float vj = a.v[(size_t)t * hd + col + j];
        float acc = 0.0f;
#pragma unroll
        for (int i = 0; i < KT; ++i) {
            const float kv = s[dp + i] * vj;
            acc += s[i] * (S[i] + s[3 * dp + i] * vj);
            S[i] = s[2 * dp + i] * S[i] + kv;
        }
        red[(buf * parts + part) * d + j] = acc;
        if (t + 1 < end) load(t + 1, buf ^ 1);
        __syncthreads();
        if (part == 0) {
            float total = 0.0f;
            for (int p = 0; p < parts; ++p) total += red[(buf * parts + p) * d + j];
            a.o[(size_t)t * hd + col + j] = total;
        }
    }
#pragma unroll
    for (int i = 0; i < KT; ++i) {
        const int key = part * KT + i;
        if (key < d) S_g[(size_t)key * d + j] = S[i];
    }
}

__global__ void __launch_bounds__(256)
wkv_prepare_kernel(const float* r, const float* k, float* wraw, const float* __restrict__ w0,
                   const float* __restrict__ u, float* bonus, long long work, int heads, int d) {
    pdl_wait();
    const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= work) return;
    const int lane = threadIdx.x & 31;
    const int head = (int)(item % heads);
    const size_t base = (size_t)item * d;
    float acc = 0.0f;
    for (int i = lane; i < d; i += 32) {
        wraw[base + i] = expf(-expf(wraw[base + i] + w0[(size_t)head * d + i]));
        acc += r[base + i] * u[(size_t)head * d + i] * k[base + i];
    }
    acc = warp_sum(acc);
    if (lane == 0) bonus[item] = acc;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct WkvScanArgs {
    const float* r;        // [T, heads * d]
    const float* k;
    const float* v;
    const float* w;        // the decay itself
    const float* bonus;    // [T, heads]
    const int* row_offsets;
    const int* state_slots;
    float* state;
    long long state_stride;
    float* o;
    int heads, d, aligned;
    int ch;                // rows a chunk (at most WKV_CH; fewer when no request brings that many)
    int skip;              // requests of this many rows or more are not walked (the chunk kernels serve them)
};

constexpr int WKV_CH = 16;     // rows a chunk at most
constexpr int WKV_STAGES = 3;  // chunks in shared memory: one being walked, two on their way

// Thread (kg, jg) keeps KT key channels (kg * KT ...) of CPT value columns (jg * CPT ...) of S in registers.  Per row
// it adds its part of sum_i r[i] S[i][j] into shared memory and moves its tile of S on; nothing is exchanged between
// threads inside a chunk of WKV_CH rows.  After the chunk the parts of a column are added in the order of the key
// groups, the bonus b_t v_t[j] joins, and the rows' outputs are written.
template <int KT, int CPT, int MAXT>
__global__ void __launch_bounds__(MAXT) wkv_scan_kernel(WkvScanArgs a) {
    extern __shared__ __align__(16) float sm[];
    pdl_wait();
    const int d = a.d, head = blockIdx.x, b = blockIdx.y;
    const int KG = (d + KT - 1) / KT, DKP = KG * KT;          // key groups, keys padded
    const int JG = (d + CPT - 1) / CPT, DVP = JG * CPT;       // column groups, columns padded
    const int jg = threadIdx.x % JG, kg = threadIdx.x / JG;
    const int j0 = jg * CPT, k0 = kg * KT;
    const int CH = a.ch;
    float* stage = sm;                                        // [STAGES][CH][3][DKP]
    float* v_s = stage + WKV_STAGES * CH * 3 * DKP;           // [STAGES][CH][DVP]
    float* part = v_s + WKV_STAGES * CH * DVP;                // [CH][KG][DVP]
    float* bon = part + CH * KG * DVP;                        // [STAGES][CH]
    const int first = a.row_offsets[b], end = a.row_offsets[b + 1];
    if (end - first >= a.skip) return;
    const size_t hd = (size_t)a.heads * d, col = (size_t)head * d;
    float* S_g = a.state + (size_t)a.state_slots[b] * a.state_stride + (size_t)head * d * d;
    float S[KT][CPT];
#pragma unroll
    for (int i = 0; i < KT; ++i) {
#pragma unroll
        for (int c = 0; c < CPT; ++c)
            S[i][c] = (k0 + i < d && j0 + c < d) ? S_g[(size_t)(k0 + i) * d + j0 + c] : 0.0f;
    }
    // keys and columns beyond the head's own stay zero in both buffers
    if (DKP != d)
        for (int i = threadIdx.x; i < WKV_STAGES * CH * 3 * DKP; i += blockDim.x)
            if (i % DKP >= d) stage[i] = 0.0f;
    if (DVP != d)
        for (int i = threadIdx.x; i < WKV_STAGES * CH * DVP; i += blockDim.x)
            if (i % DVP >= d) v_s[i] = 0.0f;
    auto fetch = [&](int t0, int buf) {
        const int rows = max(0, min(CH, end - t0));           // none: an empty group keeps the count of groups even
        float* st = stage + buf * CH * 3 * DKP;
        float* vs = v_s + buf * CH * DVP;
        if (a.aligned) {
            const int q = d >> 2;                              // 16-byte pieces a row and array
            for (int i = threadIdx.x; i < rows * q; i += blockDim.x) {
                const int tt = i / q, piece = (i % q) * 4;
                const size_t g = (size_t)(t0 + tt) * hd + col + piece;
                cp_async16(st + (tt * 3 + 0) * DKP + piece, a.r + g);
                cp_async16(st + (tt * 3 + 1) * DKP + piece, a.k + g);
                cp_async16(st + (tt * 3 + 2) * DKP + piece, a.w + g);
                cp_async16(vs + tt * DVP + piece, a.v + g);
            }
        } else {
            for (int i = threadIdx.x; i < rows * d; i += blockDim.x) {
                const int tt = i / d, e = i % d;
                const size_t g = (size_t)(t0 + tt) * hd + col + e;
                st[(tt * 3 + 0) * DKP + e] = a.r[g];
                st[(tt * 3 + 1) * DKP + e] = a.k[g];
                st[(tt * 3 + 2) * DKP + e] = a.w[g];
                vs[tt * DVP + e] = a.v[g];
            }
        }
        if (threadIdx.x < rows) cp_async4(bon + buf * CH + threadIdx.x, a.bonus + (size_t)(t0 + threadIdx.x) * a.heads + head);
        cp_async_commit();
    };
    fetch(first, 0);
    fetch(first + CH, 1);
    int buf = 0;
    for (int t0 = first; t0 < end; t0 += CH, buf = (buf + 1) % WKV_STAGES) {
        const int rows = min(CH, end - t0);
        cp_async_wait<1>();       // all but the newest group: this chunk is here, the next may still be on its way
        __syncthreads();          // ... for everyone; the buffer of the chunk before and the parts have been read
        fetch(t0 + 2 * CH, (buf + 2) % WKV_STAGES);          // two chunks ahead: a chunk is walked faster than one arrives
        const float* st = stage + buf * CH * 3 * DKP + k0;
        const float* vs = v_s + buf * CH * DVP + j0;
        if (kg < KG) {
#pragma unroll 2
            for (int tt = 0; tt < rows; ++tt) {
                float rk[KT], kk[KT], wk[KT], vv[CPT], acc[CPT];
#pragma unroll
                for (int i = 0; i < KT; i += 4) {
                    const float4 r4 = *reinterpret_cast<const float4*>(st + (tt * 3 + 0) * DKP + i);
                    const float4 k4 = *reinterpret_cast<const float4*>(st + (tt * 3 + 1) * DKP + i);
                    const float4 w4 = *reinterpret_cast<const float4*>(st + (tt * 3 + 2) * DKP + i);
                    rk[i] = r4.x; rk[i + 1] = r4.y; rk[i + 2] = r4.z; rk[i + 3] = r4.w;
                    kk[i] = k4.x; kk[i + 1] = k4.y; kk[i + 2] = k4.z; kk[i + 3] = k4.w;
                    wk[i] = w4.x; wk[i + 1] = w4.y; wk[i + 2] = w4.z; wk[i + 3] = w4.w;
                }
                if (CPT == 4) {
                    const float4 v4 = *reinterpret_cast<const float4*>(vs + tt * DVP);
                    vv[0] = v4.x; vv[1 % CPT] = v4.y; vv[2 % CPT] = v4.z; vv[3 % CPT] = v4.w;
                } else {
#pragma unroll
                    for (int c = 0; c < CPT; ++c) vv[c] = vs[tt * DVP + c];
                }
#pragma unroll
                for (int c = 0; c < CPT; ++c) acc[c] = 0.0f;
#pragma unroll
                for (int i = 0; i < KT; ++i) {
#pragma unroll
                    for (int c = 0; c < CPT; ++c) {
                        acc[c] = fmaf(rk[i], S[i][c], acc[c]);
                        S[i][c] = fmaf(wk[i], S[i][c], kk[i] * vv[c]);
                    }
                }
                if (CPT == 4) {
                    *reinterpret_cast<float4*>(part + (tt * KG + kg) * DVP + j0) =
                        make_float4(acc[0], acc[1 % CPT], acc[2 % CPT], acc[3 % CPT]);
                } else {
#pragma unroll
                    for (int c = 0; c < CPT; ++c) part[(tt * KG + kg) * DVP + j0 + c] = acc[c];
                }
            }
        }
        __syncthreads();
        if (CPT == 4) {           // four columns a thread: d is a multiple of four and the rows of o start on 16 bytes
            for (int i = threadIdx.x; i < rows * JG; i += blockDim.x) {
                const int tt = i / JG, j = (i % JG) * 4;
                float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                for (int g = 0; g < KG; ++g) {
                    const float4 p = *reinterpret_cast<const float4*>(part + (tt * KG + g) * DVP + j);
                    total.x += p.x; total.y += p.y; total.z += p.z; total.w += p.w;
                }
                const float bt = bon[buf * CH + tt];
                const float4 v4 = *reinterpret_cast<const float4*>(v_s + (buf * CH + tt) * DVP + j);
                *reinterpret_cast<float4*>(a.o + (size_t)(t0 + tt) * hd + col + j) =
                    make_float4(fmaf(bt, v4.x, total.x), fmaf(bt, v4.y, total.y), fmaf(bt, v4.z, total.z), fmaf(bt, v4.w, total.w));
            }
        } else {
            for (int i = threadIdx.x; i < rows * d; i += blockDim.x) {
                const int tt = i / d, j = i % d;
                float total = 0.0f;
                for (int g = 0; g < KG; ++g) total += part[(tt * KG + g) * DVP + j];
                a.o[(size_t)(t0 + tt) * hd + col + j] = fmaf(bon[buf * CH + tt], v_s[(buf * CH + tt) * DVP + j], total);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < KT; ++i) {
#pragma unroll
        for (int c = 0; c < CPT; ++c)
            if (k0 + i < d && j0 + c < d) S_g[(size_t)(k0 + i) * d + j0 + c] = S[i][c];
    }
}

template <int KT, int CPT, int MAXT>
static int launch_wkv_scan(WkvScanArgs a, int B, int T, cudaStream_t stream) {
    const int d = a.d, KG = (d + KT - 1) / KT, JG = (d + CPT - 1) / CPT;
    const int DKP = KG * KT, DVP = JG * CPT;
    const int threads = (KG * JG + 31) / 32 * 32;
    if (threads > MAXT) return SHARPI_BAD_ARGUMENT;
    a.ch = T - B + 1 < WKV_CH ? (T - B + 1 < 1 ? 1 : T - B + 1) : WKV_CH;      // no request brings more rows than T - B + 1
    const size_t per_row = (size_t)(WKV_STAGES * 3 * DKP + WKV_STAGES * DVP + WKV_STAGES + KG * DVP) * sizeof(float);
    if (a.ch * per_row > 160 * 1024) a.ch = (int)(160 * 1024 / per_row);
    if (a.ch < 1) return SHARPI_BAD_ARGUMENT;
    const size_t smem = a.ch * per_row;
    auto kern = wkv_scan_kernel<KT, CPT, MAXT>;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return SHARPI_LAUNCH_FAILED;
    const dim3 grid(a.heads, B);
    SHARPI_LAUNCH_PDL(kern, grid, threads, smem, stream, a);
    return SHARPI_OK;
}

// -------------------------------------------------------------------------------------------------------------
// Chunks of 64 rows for heads of up to 64 elements.  With W_(s,t] the product of the decays of rows s + 1 .. t, per channel:
//   (1) wkv_sums_kernel    U = sum_s (W_(s,last] k_s) v_s^T and the chunk's decay per channel; wraw <- the decays
//   (2) wkv_carry_kernel   the state before each chunk in U's place
//   (3) wkv_outs_kernel    o_t = (W_(first-1,t-1] r_t)^T S + sum_(s<t) A_ts v_s + (r_t . u k_t) v_t,
//                          A_ts = sum_i r_t[i] W_(s,t-1][i] k_s[i]
// A decay per channel cannot be taken out of A as a factor of its row (1 / W overflows).  The chunk is four blocks of sixteen
// rows, a warp's each: between blocks A is a product of r times the decays since its block began (and of the whole
// blocks between) with k times the decays up to its block's end, every factor at most 1; inside a block lanes walk their two
// channels.  All other products run on the tensor cores in bfloat16 pieces of 24 bits (chunk_mma.cuh).
// -------------------------------------------------------------------------------------------------------------
constexpr int WC_D = 64, WC_LD = WC_D + 8, WC_PLANE = chunked::ROWS * WC_LD, WC_THREADS = chunked::THREADS, WC_R = WC_D + 4;

struct WkvChunkArgs {
    const float *r, *k, *v, *w0, *u;
    float* w;              // [T, heads * d]: raw, then the decay
    const int* row_offsets;
    const int* state_slots;
    int B, least;
    float* state;
    long long state_stride;
    float* o;
    int heads, d;
    float* sums;           // [chunks][heads][d][d]
    float* total;          // [chunks][heads][64]
};

__device__ __forceinline__ void store_pieces(bf16* planes, int at, float x) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const bf16 b = __float2bfloat16_rn(x);
        planes[p * WC_PLANE + at] = b;
        x -= __bfloat162float(b);
    }
}

__global__ void __launch_bounds__(WC_THREADS, 3) wkv_sums_kernel(WkvChunkArgs a) {
    extern __shared__ __align__(16) uint8_t wkv_smem[];
    bf16* k_s = reinterpret_cast<bf16*>(wkv_smem);            // three planes [64 rows][64 channels]
    bf16* v_s = k_s + 3 * WC_PLANE;
    __shared__ float half_s[WC_D];
    chunked::Place p;
    if (!chunked::find_chunk(a.row_offsets, a.B, a.least, blockIdx.y, p)) return;
    const int head = blockIdx.x, d = a.d, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t hd = (size_t)a.heads * d, at0 = (size_t)p.row0 * hd + (size_t)head * d;
    chunked::load_split<chunked::ROWS, WC_D>(v_s, a.v + at0, hd, p.rows, d);
    {
        constexpr int HALF = chunked::ROWS / 2;
        const int c = threadIdx.x % WC_D, half = threadIdx.x / WC_D;
        float w[HALF], k[HALF];
        const float w0 = c < d ? a.w0[(size_t)head * d + c] : 0.0f;
#pragma unroll
        for (int r = 0; r < HALF; ++r) {
            const int row = half * HALF + r;
            const bool ok = row < p.rows && c < d;
            w[r] = ok ? a.w[at0 + (size_t)row * hd + c] : 0.0f;
            k[r] = ok ? a.k[at0 + (size_t)row * hd + c] : 0.0f;
        }
        float tail = 1.0f;                                   // the decays behind a row, inside its half
#pragma unroll
        for (int r = HALF - 1; r >= 0; --r) {
            const int row = half * HALF + r;
            const bool ok = row < p.rows && c < d;
            const float x = ok ? expf(-expf(w[r] + w0)) : 1.0f;
            if (ok) a.w[at0 + (size_t)row * hd + c] = x;
            k[r] *= tail;
            tail *= x;
        }
        if (half == 1) half_s[c] = tail;
        __syncthreads();
        const float after = half == 0 ? half_s[c] : 1.0f;
        if (half == 0) a.total[((size_t)blockIdx.y * a.heads + head) * WC_D + c] = tail * after;
#pragma unroll
        for (int r = 0; r < HALF; ++r) store_pieces(k_s, (half * HALF + r) * WC_LD + c, k[r] * after);
    }
    __syncthreads();
    float acc[8][4], small[8][4];
    chunked::clear(acc);
    chunked::clear(small);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        uint32_t x[3][4];
#pragma unroll
        for (int q = 0; q < 3; ++q)                          // stored [row][channel], taken transposed
            mma16::ldmatrix_x4_trans(x[q], k_s + q * WC_PLANE + (kk * 16 + (lane / 16) * 8 + lane % 8) * WC_LD + warp * 16 + ((lane / 8) % 2) * 8);
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            uint32_t b[3][4][2];
            chunked::right_operand<WC_LD, WC_PLANE>(b, v_s, kk * 16, n * 8, lane);
            chunked::mma_pieces(acc + n, small + n, x, b);
        }
    }
    chunked::add_small(acc, small);
    float* out = a.sums + ((size_t)blockIdx.y * a.heads + head) * d * d;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int row = warp * 16 + lane / 4 + 8 * e;
        if (row >= d) continue;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int c = n * 8 + (lane % 4) * 2;
            if (c < d) *reinterpret_cast<float2*>(out + (size_t)row * d + c) = make_float2(acc[n][2 * e], acc[n][2 * e + 1]);
        }
    }
}

__global__ void __launch_bounds__(chunked::CARRY_THREADS) wkv_carry_kernel(WkvChunkArgs a) {
    const int b = blockIdx.z, head = blockIdx.y, d = a.d, rows = a.row_offsets[b + 1] - a.row_offsets[b];
    if (rows < a.least) return;
    const int base = chunked::chunks_before(a.row_offsets, b, a.least);
    const int i = (blockIdx.x * chunked::CARRY_THREADS + threadIdx.x) * 4;
    if (i >= d * d) return;
    const int n = (rows + chunked::ROWS - 1) / chunked::ROWS;
    const float* total = a.total + ((size_t)base * a.heads + head) * WC_D + i / d;
    float4* s = reinterpret_cast<float4*>(a.state + (size_t)a.state_slots[b] * a.state_stride + (size_t)head * d * d + i);
    const size_t step = (size_t)a.heads * d * d;
    float* u = a.sums + ((size_t)base * a.heads + head) * d * d + i;
    constexpr int AHEAD = 8;
    float4 S = *s, next[AHEAD];
    float decay[AHEAD];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k)
        if (k < n) {
            next[k] = *reinterpret_cast<const float4*>(u + k * step);
            decay[k] = total[(size_t)k * a.heads * WC_D];
        }
    for (int c = 0; c < n; c += AHEAD) {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            if (c + k >= n) break;
            const float4 own = next[k];
            const float A = decay[k];
            if (c + k + AHEAD < n) {
                next[k] = *reinterpret_cast<const float4*>(u + (size_t)(c + k + AHEAD) * step);
                decay[k] = total[(size_t)(c + k + AHEAD) * a.heads * WC_D];
            }
            *reinterpret_cast<float4*>(u + (size_t)(c + k) * step) = S;
            S = make_float4(fmaf(A, S.x, own.x), fmaf(A, S.y, own.y), fmaf(A, S.z, own.z), fmaf(A, S.w, own.w));
        }
    }
    *s = S;
}

constexpr size_t WC_OUTS_SMEM = (size_t)6 * WC_PLANE * sizeof(bf16) + (size_t)(chunked::ROWS * WC_R + 4 * 16 * 17 + 4 * WC_D) * sizeof(float);

__global__ void __launch_bounds__(WC_THREADS, 2) wkv_outs_kernel(WkvChunkArgs a) {
    extern __shared__ __align__(16) uint8_t wkv_smem[];
    bf16* k_s = reinterpret_cast<bf16*>(wkv_smem);            // k times the decays up to its block's end; then the state
    bf16* v_s = k_s + 3 * WC_PLANE;
    float* r_s = reinterpret_cast<float*>(v_s + 3 * WC_PLANE);  // [64][WC_R]: r times the decays since its block began
    float* A_s = r_s + chunked::ROWS * WC_R;                   // [warp][16][17]: A inside a block
    float* W_s = A_s + 4 * 16 * 17;                            // [block][64]: a block's decay
    chunked::Place p;
    if (!chunked::find_chunk(a.row_offsets, a.B, a.least, blockIdx.y, p)) return;
    const int head = blockIdx.x, d = a.d, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / 4, t = lane % 4;
    const size_t hd = (size_t)a.heads * d, at0 = (size_t)p.row0 * hd + (size_t)head * d;
    bool finite;                                               // whether the values that this thread loaded are
    {
        float r[16][2], k[16][2], w[16][2], u[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) u[e] = lane + 32 * e < d ? a.u[(size_t)head * d + lane + 32 * e] : 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int row = warp * 16 + i, c = lane + 32 * e;
                const bool ok = row < p.rows && c < d;
                const size_t at = at0 + (size_t)row * hd + c;
                r[i][e] = ok ? a.r[at] : 0.0f;
                k[i][e] = ok ? a.k[at] : 0.0f;
                w[i][e] = ok ? a.w[at] : 1.0f;
            }
        finite = chunked::load_split<chunked::ROWS, WC_D>(v_s, a.v + at0, hd, p.rows, d);
        // columns s and s + 1 of the block's A: a lane's channels down the rows, then lane 16 e + t has A of row t, column s + e
#pragma unroll
        for (int s = 0; s < 16; s += 2) {
            float acc[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = s + e;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    acc[16 * e + col] = fmaf(r[col][c] * u[c], k[col][c], acc[16 * e + col]);
                    float x = k[col][c];
#pragma unroll
                    for (int i = col + 1; i < 16; ++i) {
                        acc[16 * e + i] = fmaf(r[i][c], x, acc[16 * e + i]);
                        x *= w[i][c];
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < o; ++i) {
                    const bool up = lane & o;
                    const float give = up ? acc[i] : acc[i + o], keep = up ? acc[i + o] : acc[i];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            A_s[(warp * 16 + lane % 16) * 17 + s + lane / 16] = acc[0];
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = lane + 32 * e;
            float x = 1.0f;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                r_s[(warp * 16 + i) * WC_R + c] = r[i][e] * x;
                x *= w[i][e];
            }
            W_s[warp * WC_D + c] = x;
            x = 1.0f;
#pragma unroll
            for (int i = 15; i >= 0; --i) {
                store_pieces(k_s, (warp * 16 + i) * WC_LD + c, k[i][e] * x);
                x *= w[i][e];
            }
        }
    }
    const bool odd = __syncthreads_or(!finite);
    // the left operand of this warp's rows: r_s times the decays of the whole blocks `from` .. warp - 1, sixteen channels
    auto left = [&](uint32_t (&x)[3][4], int kk, int from) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = kk * 16 + 2 * t + 8 * h;
            float m0 = 1.0f, m1 = 1.0f;
            for (int b = from; b < warp; ++b) {
                const float2 f = *reinterpret_cast<const float2*>(W_s + b * WC_D + c);
                m0 *= f.x; m1 *= f.y;
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float2 v = *reinterpret_cast<const float2*>(r_s + (warp * 16 + g + 8 * e) * WC_R + c);
                const mma16::Pieces s = mma16::split3(v.x * m0, v.y * m1);
#pragma unroll
                for (int q = 0; q < 3; ++q) x[q][2 * h + e] = s.v[q];
            }
        }
    };
    float score[3][2][4];
#pragma unroll
    for (int J = 0; J < 3; ++J) {
        chunked::clear(score[J]);
        if (J >= warp) continue;
        float few[2][4];
        chunked::clear(few);
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
            uint32_t b[2][3][2][2];
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    uint32_t m[4];
                    mma16::ldmatrix_x4(m, k_s + q * WC_PLANE + (J * 16 + n * 8 + lane % 8) * WC_LD + k2 * 32 + (lane / 8) * 8);
                    b[0][q][n][0] = m[0]; b[0][q][n][1] = m[1]; b[1][q][n][0] = m[2]; b[1][q][n][1] = m[3];
                }
#pragma unroll
            for (int k1 = 0; k1 < 2; ++k1) {
                uint32_t x[3][4];
                left(x, 2 * k2 + k1, J + 1);
                chunked::mma_pieces(score[J], few, x, b[k1]);
            }
        }
        chunked::add_small(score[J], few);
    }
    __syncthreads();                                           // the keys are free
    chunked::load_split<WC_D, WC_D>(k_s, a.sums + ((size_t)blockIdx.y * a.heads + head) * d * d, d, d, d);
    __syncthreads();
    float acc[8][4], small[8][4];
    chunked::clear(acc);
    chunked::clear(small);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        uint32_t x[3][4];
        left(x, kk, 0);
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            uint32_t b[3][4][2];
            chunked::right_operand<WC_LD, WC_PLANE>(b, k_s, kk * 16, n * 8, lane);
            chunked::mma_pieces(acc + n, small + n, x, b);
        }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        if (kk > warp || (odd && kk == warp)) continue;
        uint32_t x[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int n = e >> 1, row = g + 8 * (e & 1);
            float u0 = 0.0f, u1 = 0.0f;
            if (kk == warp) {
                u0 = A_s[(warp * 16 + row) * 17 + n * 8 + 2 * t];
                u1 = A_s[(warp * 16 + row) * 17 + n * 8 + 2 * t + 1];
            } else if (kk < 3) {
                u0 = score[kk < 3 ? kk : 0][n][2 * (e & 1)];
                u1 = score[kk < 3 ? kk : 0][n][2 * (e & 1) + 1];
            }
            const mma16::Pieces s = mma16::split3(u0, u1);
#pragma unroll
            for (int q = 0; q < 3; ++q) x[q][e] = s.v[q];
        }
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            uint32_t b[3][4][2];
            chunked::right_operand<WC_LD, WC_PLANE>(b, v_s, kk * 16, n * 8, lane);
            chunked::mma_pieces(acc + n, small + n, x, b);
        }
    }
    chunked::add_small(acc, small);
    if (odd) {                                                 // this warp's own rows, left out above
        float own[4][2];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int i = 0; i < 2; ++i) own[e][i] = A_s[(warp * 16 + g + 8 * (e & 1)) * 17 + (e >> 1) * 8 + 2 * t + i];
        chunked::own_rows_exact(acc, own, a.v + at0 + (size_t)(warp * 16) * hd, hd, p.rows - warp * 16, d, lane);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int row = warp * 16 + g + 8 * e;
        if (row >= p.rows) continue;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int c = n * 8 + 2 * t;
            if (c < d) *reinterpret_cast<float2*>(a.o + at0 + (size_t)row * hd + c) = make_float2(acc[n][2 * e], acc[n][2 * e + 1]);
        }
    }
}

static int launch_wkv_chunks(const WkvChunkArgs& a, int chunks, cudaStream_t stream) {
    constexpr size_t smem_sums = (size_t)6 * WC_PLANE * sizeof(bf16);
    if (cudaFuncSetAttribute(wkv_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_sums) != cudaSuccess ||
        cudaFuncSetAttribute(wkv_outs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WC_OUTS_SMEM) != cudaSuccess)
        return SHARPI_LAUNCH_FAILED;
    const dim3 grid(a.heads, chunks);
    wkv_sums_kernel<<<grid, WC_THREADS, smem_sums, stream>>>(a);
    SHARPI_CHECK_LAUNCH();
    wkv_carry_kernel<<<dim3((a.d * a.d / 4 + chunked::CARRY_THREADS - 1) / chunked::CARRY_THREADS, a.heads, a.B), chunked::CARRY_THREADS, 0, stream>>>(a);
    SHARPI_CHECK_LAUNCH();
    wkv_outs_kernel<<<grid, WC_THREADS, WC_OUTS_SMEM, stream>>>(a);
    SHARPI_CHECK_LAUNCH();
    return SHARPI_OK;
}

// `sums` (nullable; `chunks` * heads * (d * d + 64) floats): requests of at least `least` rows run in chunks, `chunks` of them
// at most, on the tensor cores (d <= 64); the others, and without it all, are walked (`walk` = 0: there are no others).
SHARPI_API int sharpi_wkv_recurrence(const float* r, const float* k, const float* v, float* wraw,
                                     const float* w0, const float* u, const int* row_offsets, const int* state_slots,
                                     float* state, long long state_stride, float* o, float* bonus, int T, int B,
                                     int heads, int d, float* sums, int chunks, int least, int walk,
                                     cudaStream_t stream) {
    if (B <= 0) return SHARPI_OK;
    if (heads <= 0 || d <= 0 || d > 256 || T <= 0) return SHARPI_BAD_ARGUMENT;
    int skip = 0x7fffffff;
    if (sums) {
        const uintptr_t bases = (uintptr_t)v | (uintptr_t)sums | (uintptr_t)state | (uintptr_t)o;
        if (d > WC_D || d % 4 != 0 || (bases & 15) != 0 || state_stride % 4 != 0 || chunks < 1 || chunks > 65535 || B > 65535 ||
            heads > 65535 || least < 1)
            return SHARPI_BAD_ARGUMENT;
        WkvChunkArgs c;
        c.r = r; c.k = k; c.v = v; c.w = wraw; c.w0 = w0; c.u = u; c.row_offsets = row_offsets; c.state_slots = state_slots;
        c.B = B; c.least = least; c.state = state; c.state_stride = state_stride; c.o = o; c.heads = heads; c.d = d;
        c.sums = sums; c.total = sums + (size_t)chunks * heads * d * d;
        const int rc = launch_wkv_chunks(c, chunks, stream);
        if (rc != SHARPI_OK || !walk) return rc;
        skip = least;
    }
    if (d <= 128) {
        // the decay and the bonus' scalar for all rows at once, then the walk
        const long long work = (long long)T * heads;
        SHARPI_LAUNCH_PDL(wkv_prepare_kernel, (unsigned)((work + 7) / 8), 256, 0, stream, r, k, wraw, w0, u, bonus, work,
                          heads, d);
        WkvScanArgs s;
        s.r = r; s.k = k; s.v = v; s.w = wraw; s.bonus = bonus; s.row_offsets = row_offsets; s.state_slots = state_slots;
        s.state = state; s.state_stride = state_stride; s.o = o; s.heads = heads; s.d = d; s.skip = skip;
        const uintptr_t ptrs = reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(k) |
                               reinterpret_cast<uintptr_t>(wraw) | reinterpret_cast<uintptr_t>(v);
        s.aligned = (d % 4 == 0 && (ptrs & 15) == 0) ? 1 : 0;
        if (d % 4 == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) return launch_wkv_scan<8, 4, 512>(s, B, T, stream);
        if (d <= 88) return launch_wkv_scan<8, 1, 1024>(s, B, T, stream);
        return launch_wkv_scan<16, 1, 1024>(s, B, T, stream);
    }
    WkvArgs a;
    a.r = r; a.k = k; a.v = v; a.wraw = wraw; a.w0 = w0; a.u = u; a.row_offsets = row_offsets;
    a.state_slots = state_slots; a.state = state; a.state_stride = state_stride; a.o = o; a.heads = heads; a.d = d;
    const dim3 grid(heads, B);
    {
        constexpr int KT = 64;
        const int parts = (d + KT - 1) / KT;
        const size_t smem = (size_t)(8 * parts * KT + 2 * parts * d) * sizeof(float);
        SHARPI_LAUNCH_PDL(wkv_recurrence_kernel<KT>, grid, d * parts, smem, stream, a);
    }
    return SHARPI_OK;
}

// o / rms(o) * weight * silu(gate), one warp a (row, head)
template <typename TO>
__global__ void __launch_bounds__(256)
wkv_out_kernel(const float* o, const float* gate, const float* __restrict__ weight, TO* out, long long work, int heads,
               int d, float eps) {
    pdl_wait();
    const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= work) return;
    const int lane = threadIdx.x & 31;
    const int head = (int)(item % heads);
    const size_t base = (size_t)item * d;
    float ss = 0.0f;
    for (int i = lane; i < d; i += 32) ss += o[base + i] * o[base + i];
    ss = warp_sum(ss);
    const float scale = 1.0f / sqrtf(ss / (float)d + eps);
    for (int i = lane; i < d; i += 32) {
        const float g = gate[base + i];
        out[base + i] = from_float<TO>(o[base + i] * scale * weight[(size_t)head * d + i] * (g / (1.0f + expf(-g))));
    }
}

// The same for heads of 4 LANES elements on 16 bytes: LANES lanes a (row, head), four elements each, loads all under way at once.
// 2048 rows of 32 heads of 64: 25 us with a warp a (row, head), 11 us so.
template <typename TO, int LANES>
__global__ void __launch_bounds__(256)
wkv_out_vec_kernel(const float* o, const float* gate, const float* __restrict__ weight, TO* out, long long work, int heads, float eps) {
    pdl_wait();
    constexpr int d = 4 * LANES;
    const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const int e = threadIdx.x % LANES * 4;
    const bool ok = item < work;
    const size_t at = (size_t)(ok ? item : 0) * d + e;
    const float4 v = *reinterpret_cast<const float4*>(o + at), g = *reinterpret_cast<const float4*>(gate + at);
    const float4 w = *reinterpret_cast<const float4*>(weight + (size_t)((ok ? item : 0) % heads) * d + e);
    float ss = v.x * v.x + v.y * v.y + (v.z * v.z + v.w * v.w);
#pragma unroll
    for (int x = LANES / 2; x > 0; x >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, x);
    const float scale = 1.0f / sqrtf(ss / (float)d + eps);
    const float y[4] = {v.x * scale * w.x * (g.x / (1.0f + expf(-g.x))), v.y * scale * w.y * (g.y / (1.0f + expf(-g.y))),
                        v.z * scale * w.z * (g.z / (1.0f + expf(-g.z))), v.w * scale * w.w * (g.w / (1.0f + expf(-g.w)))};
    if (!ok) return;
    store_four(out + at, y);
}

SHARPI_API int sharpi_wkv_out(const float* o, const float* gate, const float* weight, void* out, int out_dtype, int T,
                              int heads, int d, float eps, cudaStream_t stream) {
    if (T <= 0) return SHARPI_OK;
    if (heads <= 0 || d <= 0) return SHARPI_BAD_ARGUMENT;
    const long long work = (long long)T * heads;
    const unsigned blocks = (unsigned)((work + 7) / 8);
    const uintptr_t bases = (uintptr_t)o | (uintptr_t)gate | (uintptr_t)weight | (uintptr_t)out;
    if ((d == 64 || d == 128) && (bases & 15) == 0 && (out_dtype == SHARPI_F32 || out_dtype == SHARPI_BF16)) {
        const unsigned n = (unsigned)((work * (d / 4) + 255) / 256);
        if (d == 64 && out_dtype == SHARPI_F32) SHARPI_LAUNCH_PDL((wkv_out_vec_kernel<float, 16>), n, 256, 0, stream, o, gate, weight, (float*)out, work, heads, eps);
        else if (d == 64) SHARPI_LAUNCH_PDL((wkv_out_vec_kernel<bf16, 16>), n, 256, 0, stream, o, gate, weight, (bf16*)out, work, heads, eps);
        else if (out_dtype == SHARPI_F32) SHARPI_LAUNCH_PDL((wkv_out_vec_kernel<float, 32>), n, 256, 0, stream, o, gate, weight, (float*)out, work, heads, eps);
        else SHARPI_LAUNCH_PDL((wkv_out_vec_kernel<bf16, 32>), n, 256, 0, stream, o, gate, weight, (bf16*)out, work, heads, eps);
        return SHARPI_OK;
    }
    if (out_dtype == SHARPI_F32)
        SHARPI_LAUNCH_PDL(wkv_out_kernel<float>, blocks, 256, 0, stream, o, gate, weight, (float*)out, work, heads, d, eps);
    else if (out_dtype == SHARPI_BF16)
        SHARPI_LAUNCH_PDL(wkv_out_kernel<bf16>, blocks, 256, 0, stream, o, gate, weight, (bf16*)out, work, heads, d, eps);
    else
        return SHARPI_BAD_ARGUMENT;
    return SHARPI_OK;
}
