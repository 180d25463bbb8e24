// Recurrences with one decay a row and head,
//
//     S_t = a_t S_(t-1) + b_t k_t v_t^T   (d x dv a head) ;   o_t = S_t^T q_t ,
//
// over the rows of long portions, in chunks of 64 rows that work side by side, every product on the tensor cores:
//
//   sums_kernel    per chunk and head   U = sum_j (b_j a_(j+1) .. a_last) k_j v_j^T   and   A = a_first .. a_last
//   carry_kernel   over the chunks of a request: the state before each chunk in U's place, S <- A S + U
//   outs_kernel    per chunk and head   o_i = sum_(j <= i) D_ij (q_i . k_j) v_j + (a_first .. a_i) S^T q_i ,
//                  D_ij = b_j a_(j+1) .. a_i
//
// Operands are float32 numbers in three bfloat16 pieces (24 bits together), products the six of nine piece products that
// reach 24 bits, added in float32 (m16n8k16).  Decays are products of the a themselves: differences of summed
// logarithms would lose what the sums have in common.
// Several heads may share keys and queries (a key head); their scores q . k are then formed once.
//
// One prompt of 2048 rows, walked row by row / in chunks: matrix memory, 8 heads of 128 x 256, 321 / 120 us; state-space
// duality, 64 heads of 128 x 64 on one key head, 646 / 180 us.  Two CTAs of four warps an SM (255 registers hold the queries' or keys'
// pieces); the chunk kernels wait for one warp's products, conversions and barriers in turn (a fifth to a quarter of the issue
// slots, the tensor pipe a third of the time).  1777 rows of the duality, outputs / sums: 113 / 52 us when a tile's values were fetched
// as it began, a head's 64 x 64 decays formed by chains of 64 products, and what joins an output was read behind a store
// (which it might alias: sixteen trips to L2, one after the other); 86 / 46 us now.
#pragma once

#include "common.cuh"
#include "mma_sync.cuh"

namespace chunked {

constexpr int ROWS = 64;          // rows of a chunk
constexpr int COLS = 64;          // value columns of a tile
constexpr int THREADS = 128;
constexpr int BLOCK = 16;         // rows of a block of a chunk (a warp's)
constexpr int LD_D = BLOCK + 1;   // floats between two rows of a block's D in shared memory
constexpr int CARRY_THREADS = 256;

struct Args {
    const float *q, *k, *v;       // row t, key head g: q[t ld_q + g d ..], k likewise; head h: v[t ld_v + h dv ..]
    int ld_q, ld_k, ld_v;
    int d, dv, heads, key_heads;  // multiples of 4; heads / key_heads neighbouring heads share a key head
    int group;                    // tiles a CTA works through
    const int* row_offsets;       // [B + 1]
    const int* state_slots;       // [B]
    int B, least;                 // requests of at least `least` rows are served
    float* sums;                  // [chunks][heads][d][dv], then (NORM) [chunks][heads][d]
    float* total;                 // [chunks][heads]
    long long norms;              // floats in front of the second part of sums
    float* out;                   // [T, heads dv]
};

// Chunk number `want` of the step: the chunks of the requests that are served, one request after the other.
struct Place { int req, row0, rows; };

template <int LEN = ROWS>                 // rows of a chunk
__device__ __forceinline__ bool find_chunk(const int* row_offsets, int B, int least, int want, Place& p) {
    __shared__ int place_s[3];
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int base = 0, found = 0;
        for (int b0 = 0; b0 < B && !found; b0 += 32) {
            const int b = b0 + lane, first = b < B ? row_offsets[b] : 0, n = b < B ? row_offsets[b + 1] - first : 0;
            const int c = n >= least ? (n + LEN - 1) / LEN : 0;
            int upto = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += x;
            }
            const int mine = want - (base + upto - c);
            if (mine >= 0 && mine < c) {
                place_s[0] = b; place_s[1] = first + mine * LEN; place_s[2] = min(LEN, n - mine * LEN);
                found = 1;
            }
            found = __any_sync(0xffffffffu, found);
            base += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (!found && lane == 0) place_s[0] = -1;
    }
    __syncthreads();
    p.req = place_s[0]; p.row0 = place_s[1]; p.rows = place_s[2];
    return p.req >= 0;
}

// The chunks in front of request b's, for every thread of a block
template <int LEN = ROWS>
__device__ __forceinline__ int chunks_before(const int* row_offsets, int b, int least) {
    __shared__ int base_s;
    if (threadIdx.x < 32) {
        int c = 0;
        for (int i = threadIdx.x; i < b; i += 32) {
            const int n = row_offsets[i + 1] - row_offsets[i];
            c += n >= least ? (n + LEN - 1) / LEN : 0;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (threadIdx.x == 0) base_s = c;
    }
    __syncthreads();
    return base_s;
}

// R x C floats (C a power of two; those with r < rows and c < cols, zeros elsewhere) as three planes of bfloat16 pieces,
// rows C + 8 apart (neighbouring rows start in other banks).  All of a thread's loads are under way before the first is
// split.  Returns whether all that this thread loaded is finite.
template <int R, int C>
__device__ __forceinline__ bool load_split(bf16* dst, const float* src, size_t ld, int rows, int cols) {
    constexpr int LD = C + 8, PLANE = R * LD, N = R * C / 4 / THREADS;
    float4 x[N];
#pragma unroll
    for (int p = 0; p < N; ++p) {
        const int i = threadIdx.x + p * THREADS, r = i / (C / 4), e = (i % (C / 4)) * 4;
        x[p] = r < rows && e < cols ? *reinterpret_cast<const float4*>(src + (size_t)r * ld + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float zero = 0.0f;                                         // a NaN as soon as one of them is not
#pragma unroll
    for (int p = 0; p < N; ++p) {
        const int i = threadIdx.x + p * THREADS, r = i / (C / 4), e = (i % (C / 4)) * 4;
        zero = fmaf(x[p].x, 0.0f, fmaf(x[p].y, 0.0f, fmaf(x[p].z, 0.0f, fmaf(x[p].w, 0.0f, zero))));
        const mma16::Pieces lo = mma16::split3(x[p].x, x[p].y), hi = mma16::split3(x[p].z, x[p].w);
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * PLANE + r * LD + e) = make_uint2(lo.v[q], hi.v[q]);
    }
    return zero == 0.0f;
}

// The same in two parts: R x C floats on their way into shared memory (a thread's pieces of four lie where it alone reads them: no
// barrier), and, when they are there, their pieces; a row of block b times f(r).
template <int R, int C>
__device__ __forceinline__ void fetch_raw(float* raw, const float* src, size_t ld, int rows, int cols) {
#pragma unroll
    for (int p = 0; p < R * C / 4 / THREADS; ++p) {
        const int i = threadIdx.x + p * THREADS, r = i / (C / 4), e = (i % (C / 4)) * 4;
        const bool ok = r < rows && e < cols;
        mma16::cp_async_16(raw + 4 * i, ok ? src + (size_t)r * ld + e : src, ok ? 16 : 0);
    }
}
template <int R, int C, class W>
__device__ __forceinline__ bool split_raw(bf16* dst, const float* raw, const W& f) {
    constexpr int LD = C + 8, PLANE = R * LD;
    float zero = 0.0f;
#pragma unroll
    for (int p = 0; p < R * C / 4 / THREADS; ++p) {
        const int i = threadIdx.x + p * THREADS, r = i / (C / 4), e = (i % (C / 4)) * 4;
        float4 x = *reinterpret_cast<const float4*>(raw + 4 * i);
        zero = fmaf(x.x, 0.0f, fmaf(x.y, 0.0f, fmaf(x.z, 0.0f, fmaf(x.w, 0.0f, zero))));
        const float s = f(p, r);
        const mma16::Pieces lo = mma16::split3(x.x * s, x.y * s), hi = mma16::split3(x.z * s, x.w * s);
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * PLANE + r * LD + e) = make_uint2(lo.v[q], hi.v[q]);
    }
    return zero == 0.0f;
}

// x b[n] for N neighbouring n-tiles, all pieces, a tile after the other for each.  The tensor core's own additions cut off what
// does not fit: over the 72 of a row's sums that was the largest error (5.3e-7 of the result against 7.7e-8 of a float32 walk).
// So the large product of a step starts from zero and joins `acc` by a rounded addition; the five small ones, which start 8 bits
// lower, run on in `small` and join at the end (add_small), or with JOIN right in front of the large one.
template <int N, bool JOIN = false>
__device__ __forceinline__ void mma_pieces(float (*acc)[4], float (*small)[4], const uint32_t (&x)[3][4], const uint32_t (&b)[3][N][2]) {
    constexpr int X[5] = {2, 1, 0, 1, 0}, Y[5] = {0, 1, 2, 0, 1};
#pragma unroll
    for (int s = 0; s < 5; ++s)
#pragma unroll
        for (int n = 0; n < N; ++n) mma16::mma_bf16(small[n], x[X[s]], b[Y[s]][n][0], b[Y[s]][n][1]);
    float large[N][4];
#pragma unroll
    for (int n = 0; n < N; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) large[n][e] = 0.0f;
        mma16::mma_bf16(large[n], x[0], b[0][n][0], b[0][n][1]);
    }
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = (JOIN ? acc[n][e] + small[n][e] : acc[n][e]) + large[n][e];
}
template <int N>
__device__ __forceinline__ void clear(float (&t)[N][4]) {
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) t[n][e] = 0.0f;
}
template <int N>
__device__ __forceinline__ void add_small(float (*acc)[4], const float (&small)[N][4]) {
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] += small[n][e];
}

// The right operand of four n-tiles from planes stored [k][n] (row k0 .. k0 + 15, columns n0 .. n0 + 31)
template <int LD, int PLANE>
__device__ __forceinline__ void right_operand(uint32_t (&b)[3][4][2], const bf16* planes, int k0, int n0, int lane) {
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
            uint32_t r[4];
            mma16::ldmatrix_x4_trans(r, planes + p * PLANE + (k0 + (lane % 8) + ((lane / 8) % 2) * 8) * LD + n0 + n * 8 + (lane / 16) * 8);
            b[p][n][0] = r[0]; b[p][n][1] = r[1]; b[p][n + 1][0] = r[2]; b[p][n + 1][1] = r[3];
        }
}

// A warp's own sixteen rows among themselves where a value is not finite: the tensor core multiplies what a row must not see by
// zero, and zero times a NaN is NaN.  acc += u v over the rows up to each one: u as the left operand's elements lie in the
// lanes (rows lane / 4 and + 8), v the sixteen rows' values from column `c` on (two a lane and n-tile), cols of them, rows rows.
__device__ __forceinline__ void own_rows_exact(float (&acc)[8][4], const float (&u)[4][2], const float* v, size_t ld, int rows, int cols, int lane) {
    const int g = lane / 4, t = lane % 4;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int e = 2 * (j / 8), src = g * 4 + (j % 8) / 2;
        const float w0 = __shfl_sync(0xffffffffu, u[e][j % 2], src), w1 = __shfl_sync(0xffffffffu, u[e + 1][j % 2], src);
        if (j >= rows) continue;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int c = n * 8 + 2 * t;
            if (c >= cols) continue;
            const float2 x = *reinterpret_cast<const float2*>(v + (size_t)j * ld + c);
            if (j <= g) { acc[n][0] = fmaf(w0, x.x, acc[n][0]); acc[n][1] = fmaf(w0, x.y, acc[n][1]); }
            if (j <= g + 8) { acc[n][2] = fmaf(w1, x.x, acc[n][2]); acc[n][3] = fmaf(w1, x.y, acc[n][3]); }
        }
    }
}

// a_t and b_t of row threadIdx.x of the chunk for head h, in the threads of the first two warps (1 and 0 behind the last row)
template <class F>
__device__ __forceinline__ void load_decays(const F& f, const Place& p, int h, float& al, float& be) {
    al = 1.0f; be = 0.0f;
    if ((int)threadIdx.x < p.rows) f.decay(p.row0 + threadIdx.x, h, al, be);
}

// In the first two warps, a row a thread: b of the row times the decays behind it in its block of 16 rows, and every block's decay.
// With them D_ij of rows in different blocks is three factors: the decays up to i in its block, those of the blocks between, and
// this.  (The decays are at most 1, so a product of some is not zero where that of all is not; b may be larger than 1 and joins the
// decays behind it in one product, which is zero where it falls below float32's least number.)
__device__ __forceinline__ void block_tails(float al, float be, float* tail_s, float* block_s) {
    const int l = threadIdx.x % BLOCK;
    float z = al;
#pragma unroll
    for (int o = 1; o < BLOCK; o <<= 1) {
        const float y = __shfl_down_sync(0xffffffffu, z, o, BLOCK);
        if (l + o < BLOCK) z *= y;
    }
    const float behind = __shfl_down_sync(0xffffffffu, z, 1, BLOCK);
    tail_s[threadIdx.x] = l == BLOCK - 1 ? be : be * behind;
    if (l == 0) block_s[threadIdx.x / BLOCK] = z;
}

// DP: the key size padded to 64 or 128.  A CTA holds the chunk's keys as left operands in registers (warp w: DP / 4 of the
// state's rows) and works through `group` tiles of the key head's heads; a tile's values come in while the one before is multiplied.
template <class F, int DP>
__global__ void __launch_bounds__(THREADS, 2) sums_kernel(Args a, F f) {
    extern __shared__ __align__(16) uint8_t chunk_smem[];
    constexpr int LDK = DP + 8, PLANE_K = ROWS * LDK, LDV = COLS + 8, PLANE_V = ROWS * LDV, MT = DP / 64;
    bf16* k_s = reinterpret_cast<bf16*>(chunk_smem);
    bf16* v_s = k_s + 3 * PLANE_K;
    float* raw = reinterpret_cast<float*>(v_s + 3 * PLANE_V);
    __shared__ float tail_s[ROWS], block_s[ROWS / BLOCK];
    pdl_wait();
    Place p;
    if (!find_chunk(a.row_offsets, a.B, a.least, blockIdx.z, p)) return;
    const int kh = blockIdx.y, per = a.heads / a.key_heads, tiles = (a.dv + COLS - 1) / COLS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* keys = a.k + (size_t)p.row0 * a.ld_k + (size_t)kh * a.d;
    const int first = blockIdx.x * a.group, last = min(first + a.group, per * tiles);
    auto fetch = [&](int tl) {
        const int h = kh * per + tl / tiles, c0 = (tl % tiles) * COLS;
        fetch_raw<ROWS, COLS>(raw, a.v + (size_t)p.row0 * a.ld_v + (size_t)h * a.dv + c0, a.ld_v, p.rows, a.dv - c0);
    };
    float al = 1.0f, be = 0.0f;
    fetch(first);
    if (warp < 2) load_decays(f, p, kh * per + first / tiles, al, be);
    load_split<ROWS, DP>(k_s, keys, a.ld_k, p.rows, a.d);
    __syncthreads();
    uint32_t x[MT][4][3][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int q = 0; q < 3; ++q)      // stored [row][key channel], taken transposed
                mma16::ldmatrix_x4_trans(x[m][kk][q], k_s + q * PLANE_K + (kk * 16 + (lane / 16) * 8 + lane % 8) * LDK +
                                                          (warp * MT + m) * 16 + ((lane / 8) % 2) * 8);
    int have = -1;
    for (int tl = first; tl < last; ++tl) {
        const int h = kh * per + tl / tiles, c0 = (tl % tiles) * COLS;
        const size_t head = (size_t)blockIdx.z * a.heads + h;
        if (h != have && warp < 2) block_tails(al, be, tail_s, block_s);
        have = h;
        mma16::cp_async_wait_all();
        __syncthreads();                     // the tails are here; the tile before has been multiplied
        const float after[4] = {block_s[1] * block_s[2] * block_s[3], block_s[2] * block_s[3], block_s[3], 1.0f};
        // rows 8 p + thread / 16: what the row's term is worth behind the last one
        split_raw<ROWS, COLS>(v_s, raw, [&](int pc, int r) { return tail_s[r] * after[pc / 2]; });
        if (tl % tiles == 0) {
            if (threadIdx.x == 0) a.total[head] = block_s[0] * after[0];
            if (F::NORM && (int)threadIdx.x < a.d) {
                float n = 0.0f;
#pragma unroll
                for (int b = 0; b < ROWS / BLOCK; ++b)
                    for (int j = b * BLOCK; j < min((b + 1) * BLOCK, p.rows); ++j)
                        n = fmaf(tail_s[j] * after[b], keys[(size_t)j * a.ld_k + threadIdx.x], n);
                a.sums[a.norms + head * a.d + threadIdx.x] = n;
            }
        }
        __syncthreads();
        if (tl + 1 < last) {
            fetch(tl + 1);
            if (warp < 2 && (tl + 1) % tiles == 0) load_decays(f, p, h + 1, al, be);
        }
        float* out = a.sums + head * a.d * a.dv;
#pragma unroll
        for (int n0 = 0; n0 < COLS / 8; n0 += 4) {
            float acc[MT][4][4], small[MT][4][4];
#pragma unroll
            for (int m = 0; m < MT; ++m) clear(acc[m]), clear(small[m]);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint32_t b[3][4][2];
                right_operand<LDV, PLANE_V>(b, v_s, kk * 16, n0 * 8, lane);
#pragma unroll
                for (int m = 0; m < MT; ++m) mma_pieces(acc[m], small[m], x[m][kk], b);
            }
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                add_small(acc[m], small[m]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int row = (warp * MT + m) * 16 + lane / 4 + 8 * e;
                    if (row >= a.d) continue;
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        const int c = c0 + (n0 + n) * 8 + (lane % 4) * 2;
                        if (c < a.dv)
                            *reinterpret_cast<float2*>(out + (size_t)row * a.dv + c) = make_float2(acc[m][n][2 * e], acc[m][n][2 * e + 1]);
                    }
                }
            }
        }
    }
}

// S before every chunk into the place of its sum; four neighbouring columns a thread.  The last block of a head (NORM) has
// the normaliser, a thread an element.
template <class F>
__global__ void __launch_bounds__(CARRY_THREADS) carry_kernel(Args a, F f) {
    pdl_wait();
    const int b = blockIdx.z, h = blockIdx.y, rows = a.row_offsets[b + 1] - a.row_offsets[b];
    if (rows < a.least) return;
    const int base = chunks_before(a.row_offsets, b, a.least);
    const int n = (rows + ROWS - 1) / ROWS, slot = a.state_slots[b];
    const float* total = a.total + (size_t)base * a.heads + h;
    constexpr int AHEAD = 8;                       // sums asked for ahead of the walk
    if (F::NORM && blockIdx.x == gridDim.x - 1) {
        for (int i = threadIdx.x; i < a.d; i += CARRY_THREADS) {
            float* s = f.norm(slot, h, i);
            float* u = a.sums + a.norms + ((size_t)base * a.heads + h) * a.d + i;
            float S = *s;
            for (int c = 0; c < n; ++c) {
                const size_t at = (size_t)c * a.heads * a.d;
                const float own = u[at];
                u[at] = S;
                S = fmaf(total[(size_t)c * a.heads], S, own);
            }
            *s = S;
        }
        return;
    }
    const int i = (blockIdx.x * CARRY_THREADS + threadIdx.x) * 4, size = a.d * a.dv;
    if (i >= size) return;
    float4* s = reinterpret_cast<float4*>(f.state(slot, h, i / a.dv, i % a.dv));
    const size_t step = (size_t)a.heads * size;
    float* u = a.sums + ((size_t)base * a.heads + h) * size + i;
    float4 S = *s, next[AHEAD];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k)
        if (k < n) next[k] = *reinterpret_cast<const float4*>(u + k * step);
    for (int c = 0; c < n; c += AHEAD) {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            if (c + k >= n) break;
            const float4 own = next[k];
            if (c + k + AHEAD < n) next[k] = *reinterpret_cast<const float4*>(u + (size_t)(c + k + AHEAD) * step);
            *reinterpret_cast<float4*>(u + (size_t)(c + k) * step) = S;
            const float A = total[(size_t)(c + k) * a.heads];
            S = make_float4(fmaf(A, S.x, own.x), fmaf(A, S.y, own.y), fmaf(A, S.z, own.z), fmaf(A, S.w, own.w));
        }
    }
    *s = S;
}

// Warp w has rows 16 w .. 16 w + 15 of the chunk: its queries are left operands in registers, its scores stay in registers as
// accumulators, and weighted by D they are at once the left operand of the product with the values.
template <class F, int DP>
__global__ void __launch_bounds__(THREADS, 2) outs_kernel(Args a, F f) {
    extern __shared__ __align__(16) uint8_t chunk_smem[];
    constexpr int LDK = DP + 8, PLANE_K = ROWS * LDK, LDV = COLS + 8, PLANE_V = ROWS * LDV, PLANE_S = DP * LDV, KT = DP / 16;
    constexpr int KS = 3 * (PLANE_K > PLANE_S ? PLANE_K : PLANE_S);
    bf16* k_s = reinterpret_cast<bf16*>(chunk_smem);           // the keys; then the state before the chunk
    bf16* v_s = k_s + KS;
    float* raw = reinterpret_cast<float*>(v_s + 3 * PLANE_V);   // the next tile's values
    float* D_s = raw + ROWS * COLS;                            // [block][16][LD_D]: D inside a block
    __shared__ float head_s[ROWS], tail_s[ROWS], block_s[ROWS / BLOCK];   // decays from a block's first row up to a row; block_tails
    pdl_wait();
    Place p;
    if (!find_chunk(a.row_offsets, a.B, a.least, blockIdx.z, p)) return;
    const int kh = blockIdx.y, per = a.heads / a.key_heads, tiles = (a.dv + COLS - 1) / COLS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / 4, t = lane % 4;
    const int i0 = warp * 16 + g, i1 = i0 + 8;                 // this lane's rows
    const float* queries = a.q + (size_t)p.row0 * a.ld_q + (size_t)kh * a.d;
    const int first = blockIdx.x * a.group, last = min(first + a.group, per * tiles);
    auto fetch_values = [&](int tl) {
        const int h = kh * per + tl / tiles, c0 = (tl % tiles) * COLS;
        fetch_raw<ROWS, COLS>(raw, a.v + (size_t)p.row0 * a.ld_v + (size_t)h * a.dv + c0, a.ld_v, p.rows, a.dv - c0);
    };
    float al = 1.0f, be = 0.0f;
    fetch_values(first);
    if (warp < 2) load_decays(f, p, kh * per + first / tiles, al, be);
    load_split<ROWS, DP>(k_s, a.k + (size_t)p.row0 * a.ld_k + (size_t)kh * a.d, a.ld_k, p.rows, a.d);
    uint32_t x[KT][3][4];
#pragma unroll
    for (int kk = 0; kk < KT; ++kk)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = e & 1 ? i1 : i0, c = kk * 16 + 2 * t + 8 * (e >> 1);
            float2 v = make_float2(0.0f, 0.0f);
            if (r < p.rows && c < a.d) v = *reinterpret_cast<const float2*>(queries + (size_t)r * a.ld_q + c);
            const mma16::Pieces s = mma16::split3(v.x, v.y);
#pragma unroll
            for (int q = 0; q < 3; ++q) x[kk][q][e] = s.v[q];
        }
    __syncthreads();
    float score[8][4];
    clear(score);
#pragma unroll
    for (int n = 0; n < 8; n += 4) {
        if (n * 8 > warp * 16 + 15) continue;                  // columns above the diagonal
        float small[4][4];
        clear(small);
#pragma unroll
        for (int k2 = 0; k2 < KT / 2; ++k2) {
            uint32_t b[2][3][4][2];
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    uint32_t r[4];
                    mma16::ldmatrix_x4(r, k_s + q * PLANE_K + ((n + m) * 8 + lane % 8) * LDK + k2 * 32 + (lane / 8) * 8);
                    b[0][q][m][0] = r[0]; b[0][q][m][1] = r[1]; b[1][q][m][0] = r[2]; b[1][q][m][1] = r[3];
                }
            float two[4][4];                                   // two steps join before they join the sum: half its roundings
            clear(two);
            mma_pieces(two, small, x[2 * k2], b[0]);
            mma_pieces(two, small, x[2 * k2 + 1], b[1]);
            add_small(score + n, two);
        }
        add_small(score + n, small);
    }
    int have = -1;
    for (int tl = first; tl < last; ++tl) {
        const int h = kh * per + tl / tiles, c0 = (tl % tiles) * COLS;
        const size_t head = (size_t)blockIdx.z * a.heads + h;
        const float* values = a.v + (size_t)p.row0 * a.ld_v + (size_t)h * a.dv + c0;
        mma16::cp_async_wait_all();
        __syncthreads();                                       // the keys, or the tile before: done with
        load_split<DP, COLS>(k_s, a.sums + head * a.d * a.dv + c0, a.dv, a.d, a.dv - c0);
        const bool odd = __syncthreads_or(!split_raw<ROWS, COLS>(v_s, raw, [](int, int) { return 1.0f; }));
        if (h != have && warp < 2) {
            const int l = lane % BLOCK;
            float z = al, w = 0.0f;
#pragma unroll
            for (int o = 1; o < BLOCK; o <<= 1) {
                const float y = __shfl_up_sync(0xffffffffu, z, o, BLOCK);
                if (l >= o) z *= y;
            }
            head_s[threadIdx.x] = z;
            block_tails(al, be, tail_s, block_s);
#pragma unroll
            for (int i = 0; i < BLOCK; ++i) {                  // column l of the block's D
                const float ai = __shfl_sync(0xffffffffu, al, i, BLOCK);
                w = i == l ? be : w * ai;
                D_s[(threadIdx.x / BLOCK * BLOCK + i) * LD_D + l] = w;
            }
        }
        have = h;
        float acc[8][4];
        clear(acc);
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            float small[4][4];
            clear(small);
#pragma unroll
            for (int kk = 0; kk < KT; ++kk) {
                uint32_t b[3][4][2];
                right_operand<LDV, PLANE_S>(b, k_s, kk * 16, n * 8, lane);
                mma_pieces(acc + n, small, x[kk], b);
            }
            add_small(acc + n, small);
        }
        __syncthreads();                                       // D is here
        if (tl + 1 < last) {
            fetch_values(tl + 1);
            if (warp < 2 && (tl + 1) % tiles == 0) load_decays(f, p, h + 1, al, be);
        }
        float before = 1.0f;                                   // the decays of the blocks in front of this warp's
#pragma unroll
        for (int b = 0; b < 3; ++b)
            if (b < warp) before *= block_s[b];
        const float h0 = head_s[i0], h1 = head_s[i1], p0 = before * h0, p1 = before * h1;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            acc[n][0] *= p0; acc[n][1] *= p0;
            acc[n][2] *= p1; acc[n][3] *= p1;
        }
        float row0 = 0.0f, row1 = 0.0f;                        // NORM: this lane's part of the rows' sums of weighted scores
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            if (kk > warp) continue;
            uint32_t w[3][4];
            float u[4][2], m = 1.0f;                           // the decays of the blocks between
#pragma unroll
            for (int b = kk + 1; b < 3; ++b)
                if (b < warp) m *= block_s[b];
            const float m0 = m * h0, m1 = m * h1;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = e & 1 ? i1 : i0, n = 2 * kk + (e >> 1), c = n * 8 + 2 * t;
                float d0, d1;
                if (kk == warp) {
                    d0 = D_s[r * LD_D + c % BLOCK]; d1 = D_s[r * LD_D + c % BLOCK + 1];
                } else {
                    d0 = (e & 1 ? m1 : m0) * tail_s[c]; d1 = (e & 1 ? m1 : m0) * tail_s[c + 1];
                }
                // (selected, not multiplied by zero: what a later row's key brings must not reach this one through a NaN; for its
                // values see own_rows_exact)
                const float u0 = c <= r ? score[n][2 * (e & 1)] * d0 : 0.0f;
                const float u1 = c + 1 <= r ? score[n][2 * (e & 1) + 1] * d1 : 0.0f;
                if (F::NORM) (e & 1 ? row1 : row0) += u0 + u1;
                u[e][0] = u0; u[e][1] = u1;
                const mma16::Pieces s = mma16::split3(u0, u1);
#pragma unroll
                for (int q = 0; q < 3; ++q) w[q][e] = s.v[q];
            }
            if (odd && kk == warp) {
                own_rows_exact(acc, u, values + (size_t)(warp * 16) * a.ld_v, a.ld_v, p.rows - warp * 16, a.dv - c0, lane);
                continue;
            }
#pragma unroll
            for (int n = 0; n < 8; n += 4) {
                uint32_t b[3][4][2];
                float small[4][4];
                clear(small);
                right_operand<LDV, PLANE_V>(b, v_s, kk * 16, n * 8, lane);
                mma_pieces<4, true>(acc + n, small, w, b);
            }
        }
        if (F::NORM && tl % tiles == 0) {
            const float* n0 = a.sums + a.norms + head * a.d;
            float s0 = 0.0f, s1 = 0.0f;
            for (int c = 4 * t; c < a.d; c += 16) {
                const float4 n = *reinterpret_cast<const float4*>(n0 + c);
                const float4 q0 = i0 < p.rows ? *reinterpret_cast<const float4*>(queries + (size_t)i0 * a.ld_q + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 q1 = i1 < p.rows ? *reinterpret_cast<const float4*>(queries + (size_t)i1 * a.ld_q + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                s0 = fmaf(n.x, q0.x, fmaf(n.y, q0.y, fmaf(n.z, q0.z, fmaf(n.w, q0.w, s0))));
                s1 = fmaf(n.x, q1.x, fmaf(n.y, q1.y, fmaf(n.z, q1.z, fmaf(n.w, q1.w, s1))));
            }
            row0 = fmaf(p0, s0, row0);
            row1 = fmaf(p1, s1, row1);
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                row0 += __shfl_xor_sync(0xffffffffu, row0, o);
                row1 += __shfl_xor_sync(0xffffffffu, row1, o);
            }
            if (t == 0) {
                if (i0 < p.rows) f.store_norm(p.row0 + i0, h, row0);
                if (i1 < p.rows) f.store_norm(p.row0 + i1, h, row1);
            }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = e ? i1 : i0;
            if (r >= p.rows) continue;
#pragma unroll
            for (int n = 0; n < 8; ++n) {                      // (what joins is read before the first store: a load behind one waits for it)
                const int c = c0 + n * 8 + 2 * t;
                if (c < a.dv) f.finish(p.row0 + r, h, c, acc[n][2 * e], acc[n][2 * e + 1]);
            }
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int c = c0 + n * 8 + 2 * t;
                if (c < a.dv)
                    *reinterpret_cast<float2*>(a.out + ((size_t)(p.row0 + r) * a.heads + h) * a.dv + c) = make_float2(acc[n][2 * e], acc[n][2 * e + 1]);
            }
        }
    }
}

// Whether these sizes and addresses can be served (the rows read 16 bytes at a time)
inline bool takes(const Args& a) {
    const uintptr_t p = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.sums | (uintptr_t)a.out;
    return a.d > 0 && a.d <= 128 && a.d % 4 == 0 && a.dv > 0 && a.dv % 4 == 0 && a.ld_q % 4 == 0 && a.ld_k % 4 == 0 &&
           a.ld_v % 4 == 0 && (p & 15) == 0 && a.heads % a.key_heads == 0 && a.key_heads <= 65535 && a.heads <= 65535 &&
           (long long)a.d * a.dv <= (1 << 24);
}

template <class F, int DP>
static int launch(Args a, const F& f, int chunks, cudaStream_t stream) {
    constexpr int LDV = COLS + 8, KS = 3 * (ROWS * (DP + 8) > DP * LDV ? ROWS * (DP + 8) : DP * LDV);
    constexpr size_t smem_sums = (size_t)(3 * ROWS * (DP + 8) + 3 * ROWS * LDV) * sizeof(bf16) + ROWS * COLS * sizeof(float);
    constexpr size_t smem_outs = (size_t)(KS + 3 * ROWS * LDV) * sizeof(bf16) + (ROWS * COLS + ROWS * LD_D) * sizeof(float);
    if (cudaFuncSetAttribute(sums_kernel<F, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_sums) != cudaSuccess ||
        cudaFuncSetAttribute(outs_kernel<F, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_outs) != cudaSuccess)
        return SHARPI_LAUNCH_FAILED;
    // a CTA's keys and scores (about a tile's work) serve `group` tiles: the group with the shortest sum of waves over the
    // resident places, two an SM.  29 chunks of 64 one-tile heads on one key head: groups of 7 in one wave, where groups of 6
    // left 23 CTAs to a second one (outputs 160 -> 115 us, sums 70 -> 56 us).
    // Several requests leave the true number of chunks open by up to one each: the middle is taken.
    const int tiles = a.heads / a.key_heads * ((a.dv + COLS - 1) / COLS), expected = a.B == 1 ? chunks : chunks - (a.B < chunks / 3 ? a.B : chunks / 3) / 2;
    long long best = 0;
    a.group = 1;
    for (int g = 1; g <= tiles && g <= 16; ++g) {
        const long long ctas = (long long)((tiles + g - 1) / g) * a.key_heads * expected, cost = (ctas + 295) / 296 * (g + 1);
        if (g == 1 || cost < best) { best = cost; a.group = g; }
    }
    const dim3 grid((tiles + a.group - 1) / a.group, a.key_heads, chunks);
    // (each may start beside the tail of the one before: 2 us less a kernel)
    SHARPI_LAUNCH_PDL((sums_kernel<F, DP>), grid, THREADS, smem_sums, stream, a, f);
    const dim3 carry((a.d * a.dv / 4 + CARRY_THREADS - 1) / CARRY_THREADS + (F::NORM ? 1 : 0), a.heads, a.B);
    SHARPI_LAUNCH_PDL(carry_kernel<F>, carry, CARRY_THREADS, 0, stream, a, f);
    SHARPI_LAUNCH_PDL((outs_kernel<F, DP>), grid, THREADS, smem_outs, stream, a, f);
    return SHARPI_OK;
}

// `chunks`: at least as many as the requests that are served have together
template <class F>
static int launch(const Args& a, const F& f, int chunks, cudaStream_t stream) {
    if (chunks <= 0 || chunks > 65535 || a.B > 65535 || !takes(a)) return SHARPI_BAD_ARGUMENT;
    return a.d <= 64 ? launch<F, 64>(a, f, chunks, stream) : launch<F, 128>(a, f, chunks, stream);
}

}  // namespace chunked
