// Paged attention for any head size, head count and grouping, in fp32 or bf16 storage:
// the kernel of the true 32-bit path, and the one every other attention kernel is checked
// against on the device.  One block serves one (token row, query head): it walks the keys
// the row may see in tiles of 128, through the request's block table, with an online
// softmax; scores, maxima, exponentials, sums and the weighted value sum are fp32.
//
// The reference's counterpart is llm_attention (one block per query head, scores in shared
// memory, three-phase softmax, serial value sum; src/SharpInference.Cuda/CudaTextKernels.cs:7384)
// with the score formula of src/SharpInference.Engine/ForwardPass.cs:1850-1911:
// s_t = (q . k_t) / sqrt(d) over the visible t, p = softmax(s), o = sum_t p_t v_t, query head
// h reading kv head h / (nq / nkv).  Chunked and windowed visibility are not in the
// reference; `visible_lo` in common.cuh defines them.
//
// The tiles start at the row's lowest visible position (in the kernel for float32 rows below: at absolute multiples of 64
// keys), which depends on the row's own position only, so a row's result does not depend on how the step was cut or batched.
//
// Three further rules, each off by default.  `kv_planes` = 1: a page holds keys only and a value is the
// key row itself (its leading `d` elements): attention whose values are its keys, or keys and values that are
// two readings of one cached latent.  `keep_first` > 0 (window mask): the first `keep_first` positions of a
// sequence stay visible beyond the window; the walk then runs over the kept positions below the window first and
// the window after them.  `dist_bias` [far + 1, nq]: a number added to the scaled score by the distance
// pos - key (distances beyond `far` read row `far`).  `softcap` > 0 bends the scaled score to softcap * tanh(s /
// softcap) (before any bias); `sinks` [nq] adds exp(sink) of the head to the softmax's denominator.
#include "common.cuh"
#include "mma_sync.cuh"

#include <type_traits>

constexpr int ATT_THREADS = 128;
constexpr int ATT_TILE = 128;
constexpr int ATT_MAX_D = 1024;

struct PagedAttnArgs {
    const void* q;           // [T, nq, d]
    const void* kv_base;     // [page][2][nkv][page_size][d]
    const int* block_table;  // [B, max_blocks]
    const int* row_req;      // [T]
    const int* positions;    // [T]
    void* out;               // [T, nq * d]
    int T, nq, nkv, d, max_blocks, page_size;
    int mask_kind, mask_span;
    float scale;
    int kv_planes;           // 2: [K|V] planes a page; 1: keys only, values are the keys
    int keep_first;          // window mask: positions below this stay visible
    const float* dist_bias;  // [dist_far + 1, nq] or null
    int dist_far;
    float softcap;           // > 0: the scaled score s becomes softcap * tanh(s / softcap)
    const float* sinks;      // [nq] or null: exp(sinks[h]) joins the softmax's denominator, with no key and no value
};

template <typename TS>
__global__ void paged_attention_generic_kernel(PagedAttnArgs a) {
    __shared__ float q_s[ATT_MAX_D];
    __shared__ float p_s[ATT_TILE];
    __shared__ long long off_s[ATT_TILE];  // element offset of the key row inside the K plane; V adds `plane`
    __shared__ float scratch[32];

    const int t = blockIdx.x;
    const int h = blockIdx.y;
    const int d = a.d;
    const int kvh = h / (a.nq / a.nkv);
    const int pos = a.positions[t];
    const int lo = visible_lo(pos, a.mask_kind, a.mask_span);
    const int* table = a.block_table + (size_t)a.row_req[t] * a.max_blocks;
    const size_t plane = (size_t)a.nkv * a.page_size * d;
    const size_t vplane = a.kv_planes == 2 ? plane : 0;
    const TS* kv = (const TS*)a.kv_base;
    // kept positions below the window come first in the walk, the window behind them
    const int n_first = (a.mask_kind == SHARPI_MASK_WINDOW && a.keep_first > 0) ? min(a.keep_first, lo) : 0;
    const int n_keys_all = n_first + pos - lo + 1;

    const TS* qrow = (const TS*)a.q + ((size_t)t * a.nq + h) * d;
    for (int i = threadIdx.x; i < d; i += ATT_THREADS) q_s[i] = to_float(qrow[i]);
    __syncthreads();

    constexpr int DPT = ATT_MAX_D / ATT_THREADS;  // output dims per thread
    float acc[DPT];
#pragma unroll
    for (int r = 0; r < DPT; ++r) acc[r] = 0.0f;
    float m_run = -INFINITY, l_run = 0.0f;

    for (int tile = 0; tile < n_keys_all; tile += ATT_TILE) {
        const int at = tile + threadIdx.x;
        const int key = at < n_first ? at : lo + (at - n_first);
        float s = -INFINITY;
        long long off = -1;
        if (at < n_keys_all) {
            const int page = table[key / a.page_size];
            if (page >= 0) {
                off = (long long)page * a.kv_planes * plane + ((long long)kvh * a.page_size + key % a.page_size) * d;
                const TS* krow = kv + off;
                float dot = 0.0f;
                for (int i = 0; i < d; ++i) dot += q_s[i] * to_float(krow[i]);
                s = dot * a.scale;
                if (a.softcap > 0.0f) s = a.softcap * tanhf(s / a.softcap);
                if (a.dist_bias) s += a.dist_bias[(size_t)min(pos - key, a.dist_far) * a.nq + h];
            }
        }
        const float m_tile = block_max(s, scratch);
        const float m_new = fmaxf(m_run, m_tile);
        // m_new is finite: the row's own key is always visible and present.
        const float p = (off >= 0) ? expf(s - m_new) : 0.0f;
        const float corr = (m_run == -INFINITY) ? 0.0f : expf(m_run - m_new);
        __syncthreads();  // the previous tile's p_s / off_s are no longer read
        p_s[threadIdx.x] = p;
        off_s[threadIdx.x] = off;
        const float l_tile = block_sum(p, scratch);  // has __syncthreads inside: p_s/off_s are visible after it
        l_run = l_run * corr + l_tile;
        m_run = m_new;
        const int n_keys = min(ATT_TILE, n_keys_all - tile);
#pragma unroll
        for (int r = 0; r < DPT; ++r) {
            const int i = threadIdx.x + r * ATT_THREADS;
            if (i < d) {
                float sum = 0.0f;
                for (int k = 0; k < n_keys; ++k) {
                    const long long o = off_s[k];
                    if (o >= 0) sum += p_s[k] * to_float(kv[o + vplane + i]);
                }
                acc[r] = acc[r] * corr + sum;
            }
        }
    }
    TS* orow = (TS*)a.out + ((size_t)t * a.nq + h) * d;
    float shrink = 1.0f;
    if (a.sinks) {              // the sink counts once: exp(sink - m) in the denominator, against the larger of the two
        const float sink = a.sinks[h];
        if (sink > m_run) {
            shrink = expf(m_run - sink);
            l_run = l_run * shrink + 1.0f;
        } else {
            l_run += expf(sink - m_run);
        }
    }
    const float inv_l = shrink / l_run;
#pragma unroll
    for (int r = 0; r < DPT; ++r) {
        const int i = threadIdx.x + r * ATT_THREADS;
        if (i < d) orow[i] = from_float<TS>(acc[r] * inv_l);
    }
}

// float32 rows of up to 256 elements, a multiple of 4.  One CTA serves up to R query rows that read the same keys: the
// heads of one key head times the neighbouring tokens of one request (a group: positions of the same multiple of
// `tokens`; the group's first token leads, the CTAs of the others end at once, so a row of a decode step is a CTA of
// its own).  Key tiles of 64 at absolute positions come into shared memory by cp.async, the next keys while the values are
// weighted, the next values while the scores are formed; where a tile's keys lie is looked up a tile ahead, a key a thread.
// A thread forms R / 8 rows x 4 keys of the scores (two chains over even and odd elements: one paired instruction) and R / 8
// rows x 4 JJ elements of the sums (neighbouring elements paired).  Every number is formed by the same operations for both
// R, so a row's bits do not depend on the launch.  What a row must not see does not reach it, finite or not: keys that no row
// of the group sees are not loaded (zeros in their place), and in tiles that some of its rows see and others do not a
// hidden value is left out of the sum (zero times a NaN would be NaN); a hidden probability is minus zero there, which no
// exponential is.  Bound by the multiply-adds and the barriers between a tile's parts.
//   SPLIT: where the CTAs are few, a cluster of `ctas` of them shares the key tiles, tile it in CTA it % ctas.  What follows from tile to
// tile (the running maximum, the factors, the sums) is then a chain over numbers that the CTAs leave in shared memory: every CTA's
// maxima first, then, with them, its probabilities and sums, which all CTAs add up in the tiles' order, each for its share of the
// elements.  The operations and their order are those of one CTA.  4 decode rows at 300 keys: 47 us with a CTA a row and key
// head, 15.5 us so; at 4000 keys 555 and 103 us.
// 980 rows of 4 requests, 8 heads on 2, head size 128: 556 -> 95 us (before: a block a row and head, one key a thread read
// element by element).
constexpr int AR_BK = 64, AR_THREADS = 128, AR_MAX_D = 256;

typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    return (f32x2)__float_as_uint(lo) | ((f32x2)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float lo2(f32x2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(f32x2 v) { return __uint_as_float((unsigned)(v >> 32)); }

// In place of a hidden score: a NaN that no operation makes, so that a score of minus infinity remains one.
constexpr unsigned AR_HIDDEN = 0x7fa51dedu;

// Floats a row takes in shared memory: an odd number of 16-byte pieces, so that neighbouring rows start in other banks.
__host__ __device__ __forceinline__ int ar_ld(int d) { return (d / 4) % 2 ? d + 8 : d + 4; }

// All threads of the cluster: what one wrote into its shared memory before, the others may read behind it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same place in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t in_cta(const void* p, int rank) {
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mma16::smem_addr(p)), "r"(rank));
    return at;
}
__device__ __forceinline__ float load_cluster(uint32_t at) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ float4 load_cluster4(uint32_t at) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

template <int R, int JJ, bool SPLIT>
__global__ void __launch_bounds__(AR_THREADS) attention_rows_f32_kernel(PagedAttnArgs a, int heads_cta, int tokens) {
    static_assert(!SPLIT || R == 8, "a thread has four neighbouring elements of the cluster's sums at most");
    if (SPLIT) pdl_wait();
    const int rank = SPLIT ? (int)blockIdx.z : 0;
    extern __shared__ __align__(16) float ar_smem[];
    __shared__ long long off_s[2][AR_BK];                // where the keys of two tiles lie, -1: not there
    constexpr int RT = R / 8;                            // rows a thread
    const int d = a.d, ld = ar_ld(d), vec = d / 4;
    float* q_s = ar_smem;                                // [R][ld]
    float* k_s = q_s + R * ld;                           // [64][ld]
    float* v_s = k_s + AR_BK * ld;                       // [64][ld] (keys-only pages: none)
    float* p_s = v_s + (a.kv_planes == 2 ? AR_BK * ld : 0);   // [R][68]: scores, then probabilities
    float* corr_s = p_s + R * (AR_BK + 4);               // [R]
    float* top_s = corr_s + R;                           // SPLIT: [R] a tile's maxima, [R] its probabilities' sums, [R][d] its weighted values
    float* l_s = top_s + R;
    float* sum_s = l_s + R;

    const int t = blockIdx.x, pos0 = a.positions[t], req = a.row_req[t];
    if (t > 0 && pos0 % tokens != 0 && a.row_req[t - 1] == req && a.positions[t - 1] == pos0 - 1) return;
    int n_tok = 1;
    while (n_tok < tokens && t + n_tok < a.T && (pos0 + n_tok) % tokens != 0 && a.row_req[t + n_tok] == req &&
           a.positions[t + n_tok] == pos0 + n_tok)
        ++n_tok;
    const int G = a.nq / a.nkv, chunks = (G + heads_cta - 1) / heads_cta;
    const int kvh = blockIdx.y / chunks, head0 = kvh * G + (blockIdx.y % chunks) * heads_cta;
    const int heads_here = min(heads_cta, kvh * G + G - head0);
    const int n_rows = n_tok * heads_here;               // row r: token r / heads_here, head r % heads_here
    const int p_last = pos0 + n_tok - 1;
    const int* table = a.block_table + (size_t)req * a.max_blocks;
    const size_t plane = (size_t)a.nkv * a.page_size * d;
    const float* kv = (const float*)a.kv_base;

    const int keep = a.mask_kind == SHARPI_MASK_WINDOW ? a.keep_first : 0;
    const int lo_first = visible_lo(pos0, a.mask_kind, a.mask_span), lo_last = visible_lo(p_last, a.mask_kind, a.mask_span);
    const int b_first = lo_first / AR_BK, b_last = p_last / AR_BK;
    const int n_keep = min((keep + AR_BK - 1) / AR_BK, b_first);   // tiles with kept positions below the others
    const int n_iter = n_keep + b_last - b_first + 1;
    // How many CTAs of the cluster share the tiles goes by the tiles that there are (the launch knows the block table's width, which a
    // captured step pads, and no window): the others end here, where none of them has met another one yet.  Together they have four
    // elements of the sums a thread; a single one keeps its sums to itself.  Rows of 30 keys on a table of 1024, without clusters / with
    // all CTAs of eight going along / so: 8 heads on 2 of 128, one row 11.6 / 12.1 / 11.6, 16 rows 12.2 / 15.0 / 13.5; 16 heads on 4
    // of 64, 16 rows 10.3 / 16.8 / 15.1 (what is left is the launch of CTAs that end).
    const int ctas = !SPLIT || n_iter == 1 ? 1 : min((int)gridDim.z, max(n_iter, (d + 63) / 64));
    if (rank >= ctas) return;
    const bool shared = SPLIT && ctas > 1;
    auto key0_of = [&](int it) { return (it < n_keep ? it : b_first + it - n_keep) * AR_BK; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    auto place = [&](int it) -> long long {               // of key tid of a tile
        const int key = key0_of(it) + tid;
        const int page = key <= p_last && (key >= lo_first || key < keep) ? table[key / a.page_size] : -1;
        return page >= 0 ? (long long)page * a.kv_planes * plane + ((long long)kvh * a.page_size + key % a.page_size) * d : -1;
    };
    auto side = [&](int it) { return it / ctas & 1; };    // which of off_s is tile it's
    auto load = [&](float* dst, int it, size_t second) {  // a warp copies every fourth row
#pragma unroll 4
        for (int r = warp; r < AR_BK; r += AR_THREADS / 32) {
            const long long off = off_s[side(it)][r];
            const float* src = kv + (off >= 0 ? off + second : 0);
            for (int c = lane; c < vec; c += 32) mma16::cp_async_16(dst + r * ld + c * 4, src + (off >= 0 ? c * 4 : 0), off >= 0 ? 16 : 0);
        }
        mma16::cp_async_commit();
    };
    if (tid < AR_BK) off_s[0][tid] = SPLIT && rank >= n_iter ? -1 : place(rank);
    __syncthreads();
    load(k_s, rank, 0);
    if (a.kv_planes == 2) load(v_s, rank, plane);
    for (int r = warp; r < R; r += AR_THREADS / 32) {
        const bool ok = r < n_rows;
        const float* src = (const float*)a.q + ((size_t)(t + (ok ? r / heads_here : 0)) * a.nq + head0 + (ok ? r % heads_here : 0)) * d;
        for (int c = lane; c < vec; c += 32)
            *reinterpret_cast<float4*>(q_s + r * ld + c * 4) = ok ? *reinterpret_cast<const float4*>(src + c * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }

    f32x2 acc[RT][JJ][2];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < JJ; ++j) acc[i][j][0] = acc[i][j][1] = 0;
    float m_run = -INFINITY, l_run = 0.0f;               // of row tid / 4 (four threads a row)
    // SPLIT: this thread's four elements of the cluster's sums
    const int unit = rank + ctas * tid, unit_r = unit / vec, unit_c = unit % vec * 4;
    float4 joint = make_float4(0.f, 0.f, 0.f, 0.f);

    for (int it0 = 0; it0 < n_iter; it0 += ctas) {
        const int it = it0 + rank;
        const bool have = !shared || it < n_iter, more = it0 + ctas < n_iter;      // (a CTA without a tile in the last round goes along)
        const int key0 = key0_of(have ? it : 0);
        const long long next = tid < AR_BK && it + ctas < n_iter ? place(it + ctas) : -1;      // arrives while the scores are formed
        if (a.kv_planes == 2) mma16::cp_async_wait<1>(); else mma16::cp_async_wait<0>();
        __syncthreads();                                 // the keys are here (and the queries); p_s is free
        {
            f32x2 s[RT][4];
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = 0;
            const float* kr = k_s + tx * ld;
            const float* qr = q_s + ty * ld;
#pragma unroll 4
            for (int c = 0; c < d; c += 4) {
                ulonglong2 kk[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) kk[j] = *reinterpret_cast<const ulonglong2*>(kr + j * 16 * ld + c);
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(qr + i * 8 * ld + c);
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma2(s[i][j], qq.x, kk[j].x);
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma2(s[i][j], qq.y, kk[j].y);
                }
            }
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int r = ty + i * 8;
                const int pos = pos0 + (r < n_rows ? r / heads_here : 0), h = head0 + (r < n_rows ? r % heads_here : 0);
                const int lo = visible_lo(pos, a.mask_kind, a.mask_span);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = key0 + tx + 16 * j;
                    float v = __uint_as_float(AR_HIDDEN);
                    if (key <= pos && (key >= lo || key < keep) && off_s[side(it)][tx + 16 * j] >= 0) {
                        v = __fmul_rn(__fadd_rn(lo2(s[i][j]), hi2(s[i][j])), a.scale);
                        if (a.softcap > 0.0f) v = a.softcap * tanhf(v / a.softcap);
                        if (a.dist_bias) v += a.dist_bias[(size_t)min(pos - key, a.dist_far) * a.nq + h];
                    }
                    p_s[r * (AR_BK + 4) + tx + 16 * j] = v;
                }
            }
        }
        if (tid < AR_BK) off_s[side(it + ctas)][tid] = next;
        __syncthreads();                                 // the scores are here; keys are free
        if (a.kv_planes == 2 && more) load(k_s, it + ctas, 0);
        if (SPLIT && shared) {
            float* p = p_s + (tid >> 2) * (AR_BK + 4) + (tid & 3) * 4;
            if (tid < 4 * R) {
                float m = -INFINITY;
#pragma unroll
                for (int i = 0; i < AR_BK; i += 16)
#pragma unroll
                    for (int c = 0; c < 4; ++c) m = fmaxf(m, p[i + c]);
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                if ((tid & 3) == 0) top_s[tid >> 2] = have ? m : -INFINITY;
            }
            cluster_sync();
            if (tid < 4 * R) {
                float before = m_run, m = m_run, all = m_run, l = 0.0f;
                for (int q = 0; q < ctas; ++q) {
                    const float top = load_cluster(in_cta(top_s + (tid >> 2), q));
                    all = fmaxf(all, top);
                    if (q < rank) before = all;
                    if (q <= rank) m = all;
                }
                const float corr = before == -INFINITY ? 0.0f : expf(before - m);
                const float base = m == -INFINITY ? 0.0f : m;
                m_run = all;
#pragma unroll
                for (int i = 0; i < AR_BK; i += 16)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float v = p[i + c], e = __float_as_uint(v) == AR_HIDDEN ? -0.0f : expf(v - base);
                        p[i + c] = e;
                        l = __fadd_rn(l, e);
                    }
                l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
                l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 2));
                if ((tid & 3) == 0) { corr_s[tid >> 2] = corr; l_s[tid >> 2] = l; }
            }
        } else if (tid < 4 * R) {
            float* p = p_s + (tid >> 2) * (AR_BK + 4) + (tid & 3) * 4;
            float m = -INFINITY, l = 0.0f;
#pragma unroll
            for (int i = 0; i < AR_BK; i += 16)
#pragma unroll
                for (int c = 0; c < 4; ++c) m = fmaxf(m, p[i + c]);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m_run, fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2)));
            const float corr = m_run == -INFINITY ? 0.0f : expf(m_run - m);
            const float base = m == -INFINITY ? 0.0f : m;         // (a score of minus infinity gives zero also where there is no other)
#pragma unroll
            for (int i = 0; i < AR_BK; i += 16)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float v = p[i + c], e = __float_as_uint(v) == AR_HIDDEN ? -0.0f : expf(v - base);
                    p[i + c] = e;
                    l = __fadd_rn(l, e);
                }
            l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
            l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 2));
            l_run = __fmaf_rn(l_run, corr, l);
            m_run = m;
            if ((tid & 3) == 0) corr_s[tid >> 2] = corr;
        }
        if (a.kv_planes == 2) {
            if (more) mma16::cp_async_wait<1>(); else mma16::cp_async_wait<0>();
        }
        __syncthreads();                                 // values, probabilities and corrections are here
        {
            f32x2 sum[RT][JJ][2];
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < JJ; ++j) sum[i][j][0] = sum[i][j][1] = 0;
            const float* vr = (a.kv_planes == 2 ? v_s : k_s) + tx * 4;
            const float* pr = p_s + ty * (AR_BK + 4);
            // some row of the group sees a key of this tile that another one does not
            const bool mixed = n_tok > 1 && (key0 + AR_BK - 1 > pos0 || (key0 < lo_last && key0 + AR_BK > keep));
            auto weigh = [&](auto guarded) {
#pragma unroll 2
                for (int k = 0; k < AR_BK; k += 4) {
                    float4 pv[RT];
#pragma unroll
                    for (int i = 0; i < RT; ++i) pv[i] = *reinterpret_cast<const float4*>(pr + i * 8 * (AR_BK + 4) + k);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int j = 0; j < JJ; ++j) {
                            // (elements of rows of at most 64 that do not exist: what is read there is not used)
                            if (JJ > 1 && tx * 4 + 64 * j >= d) continue;
                            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vr + (k + c) * ld + 64 * j);
#pragma unroll
                            for (int i = 0; i < RT; ++i) {
                                const float e = c == 0 ? pv[i].x : c == 1 ? pv[i].y : c == 2 ? pv[i].z : pv[i].w;
                                if (guarded && __float_as_uint(e) == 0x80000000u) continue;
                                const f32x2 ee = pack2(e, e);
                                fma2(sum[i][j][0], ee, v.x);
                                fma2(sum[i][j][1], ee, v.y);
                            }
                        }
                }
            };
            // (for 32 rows a loop without the question where it need not be asked: 60 rows behind 340 119 -> 110 us; 8 rows lose by a
            // second loop, 64 -> 70 us)
            if constexpr (R == 8) weigh(mixed);
            else if (mixed) weigh(std::true_type{});
            else weigh(std::false_type{});
            if (SPLIT && shared) {
#pragma unroll
                for (int j = 0; j < JJ; ++j)
                    if (tx * 4 + 64 * j < d)
                        *reinterpret_cast<float4*>(sum_s + ty * d + tx * 4 + 64 * j) =
                            make_float4(lo2(sum[0][j][0]), hi2(sum[0][j][0]), lo2(sum[0][j][1]), hi2(sum[0][j][1]));
                cluster_sync();
                const int tiles = min(ctas, n_iter - it0);
                for (int q = 0; q < tiles; ++q) {
                    if (unit_r < R) {
                        const float corr = load_cluster(in_cta(corr_s + unit_r, q));
                        const float4 v = load_cluster4(in_cta(sum_s + unit_r * d + unit_c, q));
                        joint = make_float4(__fmaf_rn(joint.x, corr, v.x), __fmaf_rn(joint.y, corr, v.y),
                                            __fmaf_rn(joint.z, corr, v.z), __fmaf_rn(joint.w, corr, v.w));
                    }
                    if (tid < 4 * R) l_run = __fmaf_rn(l_run, load_cluster(in_cta(corr_s + (tid >> 2), q)), load_cluster(in_cta(l_s + (tid >> 2), q)));
                }
            } else
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const float corr = corr_s[ty + i * 8];
#pragma unroll
                for (int j = 0; j < JJ; ++j)
#pragma unroll
                    for (int c = 0; c < 2; ++c)
                        acc[i][j][c] = pack2(__fmaf_rn(lo2(acc[i][j][c]), corr, lo2(sum[i][j][c])),
                                             __fmaf_rn(hi2(acc[i][j][c]), corr, hi2(sum[i][j][c])));
            }
        }
        if (more) {
            __syncthreads();                             // the values are free
            if (a.kv_planes == 2) load(v_s, it + ctas, plane); else load(k_s, it + ctas, 0);
        }
    }
    if (SPLIT && shared) cluster_sync();                 // nobody reads this CTA's shared memory any more
    else __syncthreads();
    if (tid < 4 * R && (tid & 3) == 0) {
        float shrink = 1.0f;
        const int r = tid >> 2, h = head0 + (r < n_rows ? r % heads_here : 0);
        if (a.sinks) {          // the sink counts once: exp(sink - m) in the denominator, against the larger of the two
            const float sink = a.sinks[h];
            if (sink > m_run) {
                shrink = expf(m_run - sink);
                l_run = l_run * shrink + 1.0f;
            } else {
                l_run += expf(sink - m_run);
            }
        }
        corr_s[r] = shrink / l_run;
    }
    __syncthreads();
    if (SPLIT && shared) {
        if (unit_r < n_rows) {
            const float f = corr_s[unit_r];
            float* out = (float*)a.out + ((size_t)(t + unit_r / heads_here) * a.nq + head0 + unit_r % heads_here) * d;
            *reinterpret_cast<float4*>(out + unit_c) = make_float4(joint.x * f, joint.y * f, joint.z * f, joint.w * f);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int r = ty + i * 8;
        if (r >= n_rows) continue;
        const float f = corr_s[r];
        float* out = (float*)a.out + ((size_t)(t + r / heads_here) * a.nq + head0 + r % heads_here) * d;
#pragma unroll
        for (int j = 0; j < JJ; ++j) {
            const int c = tx * 4 + 64 * j;
            if (c < d)
                *reinterpret_cast<float4*>(out + c) = make_float4(lo2(acc[i][j][0]) * f, hi2(acc[i][j][0]) * f,
                                                                  lo2(acc[i][j][1]) * f, hi2(acc[i][j][1]) * f);
        }
    }
}

// `ctas`: of a cluster (1: none)
template <int R, int JJ, bool SPLIT>
static int launch_rows_f32(const PagedAttnArgs& a, int ctas, cudaStream_t stream) {
    const int G = a.nq / a.nkv, heads_cta = G < R ? G : R, tokens = R / heads_cta;
    const size_t smem = ((size_t)(R + (a.kv_planes == 2 ? 2 : 1) * AR_BK) * ar_ld(a.d) + R * (AR_BK + 4) + R + (SPLIT ? R * (2 + a.d) : 0)) * sizeof(float);
    auto kern = attention_rows_f32_kernel<R, JJ, SPLIT>;
    // (the same limit whatever the size: another thread's launch, or a captured one, must not find it lowered)
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) return SHARPI_LAUNCH_FAILED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.T, a.nkv * ((G + heads_cta - 1) / heads_cta), ctas);
    cfg.blockDim = AR_THREADS;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = ctas;
    cfg.attrs = attr;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = SPLIT ? 1 + sharpi_pdl_enabled() : 0;
    return cudaLaunchKernelEx(&cfg, kern, a, heads_cta, tokens) == cudaSuccess ? SHARPI_OK : SHARPI_LAUNCH_FAILED;
}

template <int R, bool SPLIT = false>
static int launch_rows_f32(const PagedAttnArgs& a, int ctas, cudaStream_t stream) {
    return a.d <= 64 ? launch_rows_f32<R, 1, SPLIT>(a, ctas, stream) : a.d <= 128 ? launch_rows_f32<R, 2, SPLIT>(a, ctas, stream)
                                                                                   : launch_rows_f32<R, 4, SPLIT>(a, ctas, stream);
}

// Whether CTAs take 32 rows instead of 8.  A CTA of 8 walks its keys in two thirds of the time and three to six of them share an
// SM (of 32 rows: one to three), so 32 only where CTAs of 8 do not fit the SMs at once and 32 rows a CTA leave well fewer of them
// (single rows beside a portion stay a CTA each).  us, 8 / 32 rows a CTA, head size 128, 400 positions: 8 heads on 2: 60 rows
// 66 / 109, 300 rows 80 / 111, 60 rows and 63 single ones 75 / 118, four portions of 250 181 / 128; 32 heads on 8, 2500 positions:
// 100 rows 475 / 645, 150 rows 900 / 647, 16 portions of 16 1372 / 1278, 64 of 3 1386 / 1294, 300 rows and 63 single ones 1840 / 1917.
static int launch_rows_f32(const PagedAttnArgs& a, int B, cudaStream_t stream) {
    const int G = a.nq / a.nkv, first = a.T < B ? a.T : B;       // rows that open a request's portion, at most
    auto ctas = [&](int R) {
        const int heads_cta = G < R ? G : R, tokens = R / heads_cta;
        return (long long)((a.T - first) / tokens + first) * a.nkv * ((G + heads_cta - 1) / heads_cta);
    };
    const int per_sm = a.d <= 64 ? 6 : a.d <= 128 ? 3 : 1;
    if (ctas(8) > 148 * per_sm && 2 * ctas(8) > 5 * ctas(32)) return launch_rows_f32<32>(a, 1, stream);
    // CTAs of 8 rows that leave SMs empty share their tiles in clusters, as long as those fit two thirds of the places at once.  us,
    // without / with clusters, 8 heads on 2, head size 128: one row at 30 keys 11.6 / 11.6, at 100 20.8 / 13.0; 16 rows at 400 65 / 18;
    // 60 rows behind 300 57 / 30; 32 heads on 8, 16 rows at 2000 287 / 205; four portions of 40 rows behind 250 (pairs, three quarters
    // of the places) 65 / 67.
    const long long grid = (long long)a.T * a.nkv * ((G + 7) / 8);
    const int tiles = (int)(((long long)a.max_blocks * a.page_size + AR_BK - 1) / AR_BK);
    for (int n = 8; n > 1; n >>= 1)
        if (ctas(8) * n * 3 <= 148 * per_sm * 2 && tiles >= n && n * 64 >= a.d && grid * n <= 1 << 30) return launch_rows_f32<8, true>(a, n, stream);
    return launch_rows_f32<8>(a, 1, stream);
}

SHARPI_API int sharpi_paged_attention_generic(const void* q, const void* kv_base, const int* block_table,
                                              const int* row_req, const int* positions, void* out, int dtype,
                                              int T, int B, int nq, int nkv, int d, int max_blocks, int page_size,
                                              int mask_kind, int mask_span, float scale, int kv_planes,
                                              int keep_first, const float* dist_bias, int dist_far,
                                              float softcap, const float* sinks, cudaStream_t stream) {
    if (T <= 0) return SHARPI_OK;
    if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || d <= 0 || d > ATT_MAX_D || nq > 65535 || page_size <= 0 ||
        max_blocks <= 0)
        return SHARPI_BAD_ARGUMENT;
    if (mask_kind != SHARPI_MASK_FULL && mask_span <= 0) return SHARPI_BAD_ARGUMENT;
    if ((kv_planes != 1 && kv_planes != 2) || keep_first < 0 || (dist_bias && dist_far < 0)) return SHARPI_BAD_ARGUMENT;
    PagedAttnArgs a;
    a.kv_planes = kv_planes; a.keep_first = keep_first; a.dist_bias = dist_bias; a.dist_far = dist_far;
    a.softcap = softcap; a.sinks = sinks;
    a.q = q; a.kv_base = kv_base; a.block_table = block_table; a.row_req = row_req; a.positions = positions;
    a.out = out; a.T = T; a.nq = nq; a.nkv = nkv; a.d = d; a.max_blocks = max_blocks; a.page_size = page_size;
    a.mask_kind = mask_kind; a.mask_span = mask_span; a.scale = scale;
    // (16 bytes a lane: other row sizes, larger ones and bfloat16 stay with the general kernel)
    const uintptr_t bases = (uintptr_t)q | (uintptr_t)kv_base | (uintptr_t)out;
    if (dtype == SHARPI_F32 && d % 4 == 0 && d <= AR_MAX_D && (bases & 15) == 0)
        return launch_rows_f32(a, B, stream);
    dim3 grid(T, nq);
    if (dtype == SHARPI_F32)
        paged_attention_generic_kernel<float><<<grid, ATT_THREADS, 0, stream>>>(a);
    else if (dtype == SHARPI_BF16)
        paged_attention_generic_kernel<bf16><<<grid, ATT_THREADS, 0, stream>>>(a);
    else
        return SHARPI_BAD_ARGUMENT;
    SHARPI_CHECK_LAUNCH();
    return SHARPI_OK;
}
