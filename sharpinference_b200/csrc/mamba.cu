// The selective state-space scan (Mamba) from per-request state, and the short causal convolution before it.
//
//   sharpi_causal_conv   (optionally the silu of a second block of columns, the scan's gate, in place, and)
//                        x_t[c] = silu(b[c] + sum_j w[c][j] in_{t - (taps - 1 - j)}[c]): the last column of w is
//                        the current token's.  Inputs before a portion's first row come from the request's state
//                        (its last taps - 1 inputs; zeros at a sequence's start), which a second launch then
//                        moves on to the portion's last inputs.
//   sharpi_slice_cols    a block of columns of a float32 matrix as a contiguous matrix in the activation dtype
//                        (the step-size inputs of the scan, cut out of the fused projection).
//   sharpi_selective_scan  per channel c and state n, for the rows of a request in order:
//                            S[c][n] <- exp(dt[c] A[c][n]) S[c][n] + dt[c] x[c] B[n],  A = -exp(A_log)
//                            y[c] = sum_n S[c][n] C[n] + D[c] x[c],  out = y g[c]
//                        with dt the step sizes (after their softplus) and g the gate (after its silu),
//                        all in float32 (exp(dt A) as exp2 of dt A log2(e)); or with dt before bias and softplus and z
//                        before its silu, which the walk's warps then apply to every element once.  A group of lanes owns
//                        one channel, a lane two states in registers; the sum over the states is a fixed tree of exchanges,
//                        and the walk over a request's rows is sequential, so a walked row's result does not depend on how
//                        the prompt was cut or batched.  A portion of many rows may run in chunks instead (further down), whose
//                        sums are rounded in another order: its rows do not depend on the rest of the step either, but they are
//                        not the bits of the same prompt in shorter portions.
#include "common.cuh"
#include "chunk_mma.cuh"

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }

// 2^x for x <= 0 in one special-function instruction (two units in the last place; results below the smallest
// normal number become zero, which is what a decay that small is).
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <typename TO>
__global__ void __launch_bounds__(256)
causal_conv_kernel(const float* in, int ld, const float* __restrict__ w, const float* __restrict__ bias,
                   const float* state, long long state_stride, const int* row_request, const int* row_offsets,
                   const int* state_slots, float* x32, TO* xact, int C, int taps, float* gate) {
    pdl_wait();
    const int t = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= C) return;
    if (gate) gate[(size_t)t * ld + c] = silu_f(gate[(size_t)t * ld + c]);
    const int b = row_request[t];
    const int i = t - row_offsets[b];                 // place within the portion
    const float* st = state + (size_t)state_slots[b] * state_stride;      // [taps - 1][C], oldest first
    float acc = bias ? bias[c] : 0.0f;
    for (int j = 0; j < taps; ++j) {
        const int back = taps - 1 - j;
        const float v = (i - back >= 0) ? in[(size_t)(t - back) * ld + c] : st[(size_t)(taps - 1 + i - back) * C + c];
        acc += w[(size_t)c * taps + j] * v;
    }
    const float y = silu_f(acc);
    x32[(size_t)t * C + c] = y;
    if (xact) xact[(size_t)t * C + c] = from_float<TO>(y);
}

// Four neighbouring channels a thread, CONV_ROWS rows one after the other with the inputs before them in registers: an input is read
// once instead of once a tap, 16 bytes a lane, all rows on their way before the first is used.  A row that opens a portion
// takes the window from its request's state; rows inside one took it over from the row before.  Additions as in the kernel
// above, which serves other numbers of taps, of channels and unaligned rows.  2048 rows of 4096 channels, four taps: 28.4
// us = 2950 GB/s of bytes read and written once; a channel a thread and every tap read from memory: 58.2 us.
constexpr int CONV_ROWS = 8;

template <typename TO, int TAPS>
__global__ void __launch_bounds__(128)
causal_conv_rows_kernel(const float* in, int ld, const float* __restrict__ w, const float* __restrict__ bias,
                        const float* state, long long state_stride, const int* row_request, const int* row_offsets,
                        const int* state_slots, float* x32, TO* xact, int C, int T, float* gate) {
    pdl_wait();
    constexpr int K = TAPS - 1, R = CONV_ROWS;
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4, t0 = blockIdx.x * R;
    if (c >= C) return;
    float4 v[R], win[K > 0 ? K : 1];
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (t0 + r < T) v[r] = *reinterpret_cast<const float4*>(in + (size_t)(t0 + r) * ld + c);
    float wt[4][TAPS];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < TAPS; ++j) wt[q][j] = w[(size_t)(c + q) * TAPS + j];
    const float4 b4 = bias ? make_float4(bias[c], bias[c + 1], bias[c + 2], bias[c + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int t = t0 + r;
        if (t >= T) break;
        const int b = row_request[t], i = t - row_offsets[b];           // place within the portion
        if (r == 0 || i == 0) {                                        // win[j]: the input j - K rows before this one
            const float* st = state + (size_t)state_slots[b] * state_stride + c;
#pragma unroll
            for (int j = 0; j < K; ++j)
                win[j] = i - K + j >= 0 ? *reinterpret_cast<const float4*>(in + (size_t)(t - K + j) * ld + c)
                                        : *reinterpret_cast<const float4*>(st + (size_t)(i + j) * C);
        }
        float4 y = b4;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const float4 u = j < K ? win[j < K ? j : 0] : v[r];
            y.x += wt[0][j] * u.x; y.y += wt[1][j] * u.y; y.z += wt[2][j] * u.z; y.w += wt[3][j] * u.w;
        }
#pragma unroll
        for (int j = 0; j + 1 < K; ++j) win[j] = win[j + 1];
        if (K > 0) win[K > 0 ? K - 1 : 0] = v[r];
        y = make_float4(silu_f(y.x), silu_f(y.y), silu_f(y.z), silu_f(y.w));
        *reinterpret_cast<float4*>(x32 + (size_t)t * C + c) = y;
        if (xact) {
            TO o[4] = {from_float<TO>(y.x), from_float<TO>(y.y), from_float<TO>(y.z), from_float<TO>(y.w)};
            if (sizeof(TO) == 2) *reinterpret_cast<uint2*>(xact + (size_t)t * C + c) = *reinterpret_cast<const uint2*>(o);
        }
        if (gate) {
            float4* g = reinterpret_cast<float4*>(gate + (size_t)t * ld + c);
            *g = make_float4(silu_f(g->x), silu_f(g->y), silu_f(g->z), silu_f(g->w));
        }
    }
}

__global__ void __launch_bounds__(256)
causal_conv_state_kernel(const float* in, int ld, float* state, long long state_stride, const int* row_offsets,
                         const int* state_slots, int C, int taps) {
    pdl_wait();
    const int b = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int first = row_offsets[b], n = row_offsets[b + 1] - first, K = taps - 1;
    float* st = state + (size_t)state_slots[b] * state_stride;
    if (K <= 3) {                                      // read before the first store: a load behind one waits for it
        float v[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int src = n - K + j;
            if (j < K) v[j] = src >= 0 ? in[(size_t)(first + src) * ld + c] : st[(size_t)(j + n) * C + c];
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (j < K) st[(size_t)j * C + c] = v[j];
        return;
    }
    for (int j = 0; j < K; ++j) {                      // ascending: st[j + n] is read before it is overwritten
        const int src = n - K + j;
        st[(size_t)j * C + c] = src >= 0 ? in[(size_t)(first + src) * ld + c] : st[(size_t)(j + n) * C + c];
    }
}

SHARPI_API int sharpi_causal_conv(const float* in, int ld, const float* w, const float* bias, float* state,
                                  long long state_stride, const int* row_request, const int* row_offsets,
                                  const int* state_slots, float* x32, void* xact, int act_dtype, int T, int B, int C,
                                  int taps, int gate_col, cudaStream_t stream) {
    if (T <= 0) return SHARPI_OK;
    if (C <= 0 || taps <= 0 || B <= 0 || gate_col + C > ld || (gate_col >= 0 && gate_col < C)) return SHARPI_BAD_ARGUMENT;
    float* gate = gate_col >= 0 ? const_cast<float*>(in) + gate_col : nullptr;
    const dim3 grid(T, (C + 255) / 256);
    if (act_dtype != SHARPI_F32 && act_dtype != SHARPI_BF16) return SHARPI_BAD_ARGUMENT;
    const uintptr_t bases = (uintptr_t)in | (uintptr_t)state | (uintptr_t)x32 | (uintptr_t)gate | (uintptr_t)(act_dtype == SHARPI_BF16 ? xact : nullptr);
    // from about a block an SM on eight rows a thread are faster (200 rows of 4352 channels: 8.8 against 9.6 us; 300 of 2048:
    // 8.7 against 7.9; 64 of 4096: 6.8 against 5.7)
    if ((long long)T * C >= 800000 && taps <= 4 && C % 4 == 0 && ld % 4 == 0 && state_stride % 4 == 0 && (bases & 15) == 0) {
#define CONV_CASE(TO, TAPS, X)                                                                                            \
    case TAPS:                                                                                                             \
        SHARPI_LAUNCH_PDL((causal_conv_rows_kernel<TO, TAPS>), dim3((T + CONV_ROWS - 1) / CONV_ROWS, (C + 511) / 512), 128, \
                          0, stream, in, ld, w, bias, (const float*)state, state_stride, row_request, row_offsets,          \
                          state_slots, x32, X, C, T, gate);                                                                \
        break;
        if (act_dtype == SHARPI_F32) {
            switch (taps) { CONV_CASE(float, 1, (float*)nullptr) CONV_CASE(float, 2, (float*)nullptr) CONV_CASE(float, 3, (float*)nullptr) CONV_CASE(float, 4, (float*)nullptr) }
        } else {
            switch (taps) { CONV_CASE(bf16, 1, (bf16*)xact) CONV_CASE(bf16, 2, (bf16*)xact) CONV_CASE(bf16, 3, (bf16*)xact) CONV_CASE(bf16, 4, (bf16*)xact) }
        }
#undef CONV_CASE
    } else if (act_dtype == SHARPI_F32)
        SHARPI_LAUNCH_PDL(causal_conv_kernel<float>, grid, 256, 0, stream, in, ld, w, bias, (const float*)state,
                          state_stride, row_request, row_offsets, state_slots, x32, (float*)nullptr, C, taps, gate);
    else if (act_dtype == SHARPI_BF16)
        SHARPI_LAUNCH_PDL(causal_conv_kernel<bf16>, grid, 256, 0, stream, in, ld, w, bias, (const float*)state,
                          state_stride, row_request, row_offsets, state_slots, x32, (bf16*)xact, C, taps, gate);
    if (taps > 1) {
        SHARPI_LAUNCH_PDL(causal_conv_state_kernel, dim3((C + 255) / 256, B), 256, 0, stream, in, ld, state, state_stride, row_offsets,
                          state_slots, C, taps);
    }
    return SHARPI_OK;
}

template <typename TO>
__global__ void __launch_bounds__(256)
slice_cols_kernel(const float* src, int ld, int col0, int ncols, TO* out, long long total) {
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long t = i / ncols;
    const int c = (int)(i % ncols);
    out[i] = from_float<TO>(src[(size_t)t * ld + col0 + c]);
}

SHARPI_API int sharpi_slice_cols(const float* src, int ld, int col0, int ncols, void* out, int out_dtype, int T,
                                 cudaStream_t stream) {
    if (T <= 0 || ncols <= 0) return SHARPI_OK;
    if (col0 < 0 || col0 + ncols > ld) return SHARPI_BAD_ARGUMENT;
    const long long total = (long long)T * ncols;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (out_dtype == SHARPI_F32)
        SHARPI_LAUNCH_PDL(slice_cols_kernel<float>, blocks, 256, 0, stream, src, ld, col0, ncols, (float*)out, total);
    else if (out_dtype == SHARPI_BF16)
        SHARPI_LAUNCH_PDL(slice_cols_kernel<bf16>, blocks, 256, 0, stream, src, ld, col0, ncols, (bf16*)out, total);
    else
        return SHARPI_BAD_ARGUMENT;
    return SHARPI_OK;
}

struct ScanArgs {
    const float* x;          // [T, C] after convolution and silu
    const float* dtraw;      // [T, C]: the step sizes (with dt_bias: before bias and softplus)
    const float* dt_bias;    // [C], or null: dtraw and z are the step sizes and gates themselves
    const float* bc;         // [T, ld_bc]: B at col_b, C at col_c, N columns each
    int ld_bc, col_b, col_c;
    const float* a_log;      // [C, N]
    const float* dskip;      // [C]
    const float* z;          // [T, ld_z]: the gate (with dt_bias: before its silu)
    int ld_z;
    const int* row_offsets;
    const int* state_slots;
    float* state;            // [slots, C * N]
    long long state_stride;
    void* out;               // [T, C]
    int C, N;
    int vec_ch, vec_bc;      // whether the channel arrays / B and C may be fetched 16 bytes at a time
    int ch;                  // rows a chunk (at most SCAN_CH; fewer when no request brings that many)
    int alone;               // a long walk: the next kernel's blocks stay off the SMs until it ends
    int skip;                // requests of this many rows or more are not walked (the chunk kernels serve them)
};

constexpr int SCAN_CH = 16;      // rows a chunk at most
constexpr int SCAN_HELPERS = 1;  // warps that prepare for one that walks
constexpr int SCAN_RB = 8;       // rows whose exponentials and sums are formed side by side

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A block serves CPB = warps * 32 / G channels of one request: G lanes a channel, NPT states a lane.  The rows' inputs arrive
// in shared memory by cp.async, two chunks of SCAN_CH rows on their way while a third is walked: per row the block's
// channels of dtraw, x and z and the row's B and C.  A warp then forms (dt, dt x) and the gate of its own channels, each
// once.  Rows are taken SCAN_RB at a time: the states' chain is one multiply-add a row, everything else of the eight rows is
// independent of it, and the eight rows' sums over the lanes are formed by halving exchanges (7 for 8 rows on 8 lanes), after
// which a lane holds and stores 8 / G of them.
//   The sum over the states: pairs of neighbouring states, then a tree over the pairs that halves their number from the
// top (pair l with pair l + P / 2, and so on).  Lane g holds the pairs g, g + G, ...: the tree's first levels are in its
// registers, the others exchanges, and the additions are the same for every NPT and G.
//   Few states a lane where a prompt is alone (its rows can only be walked, and nothing hides a row's latency but other
// warps: 4096 channels of 16 states are 1024 warps with two states a lane, 256 with eight); eight where there are warps
// enough, because a lane's share of a row (its inputs from shared memory, the exchanges) is the same for two states.
//   SPLIT (few states a lane): half of the block's warps walk, the others fetch and prepare the next chunk meanwhile;
// otherwise a warp prepares its chunk before it walks it.
// One prompt of 2048 rows of 4096 channels x 16 states, softplus, silu and all: 354 + 36 us with eight states a lane, row by row,
// and softplus in a kernel of its own; 230 two states a lane; 177 with walkers and helpers; 152 with the fetching
// in the helpers too (157 with two helpers a walker).  What bounds it is the chain of a chunk (reads, exponentials, sums, barrier)
// at three to four warps a scheduler: 62 % of the issue slots.
template <typename TO, int NPT, int G, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 64 * (1 + SCAN_HELPERS) : 128) selective_scan_kernel(ScanArgs a) {
    constexpr int SCAN_STAGES = SPLIT ? 4 : 3;         // chunks in shared memory: walked, (prepared,) two on their way
    extern __shared__ __align__(16) float sm[];
    if (a.alone) pdl_wait_only(); else pdl_wait();
    if (a.row_offsets[blockIdx.y + 1] - a.row_offsets[blockIdx.y] >= a.skip) return;
    constexpr int CPW = 32 / G, NP = G * NPT;
    const int warps = (blockDim.x >> 5) / (SPLIT ? 1 + SCAN_HELPERS : 1), CPB = warps * CPW;
    const int lane = threadIdx.x & 31;
    const bool helper = SPLIT && (int)(threadIdx.x >> 5) >= warps;
    const int warp = (int)(threadIdx.x >> 5) % warps;          // a helper prepares rows of the same channels as this walker
    const int part = helper ? (int)(threadIdx.x >> 5) / warps - 1 : 0, parts = helper ? SCAN_HELPERS : 1;
    const int sub = lane % G;
    const int cl = warp * CPW + lane / G;              // channel within the block
    const int c0 = blockIdx.x * CPB;
    const bool live = c0 + cl < a.C;
    const int c = live ? c0 + cl : a.C - 1;
    const int b = blockIdx.y;
    const int first = a.row_offsets[b], end = a.row_offsets[b + 1];
    const int N = a.N;
    auto n_of = [&](int i) { return 2 * (sub + (i >> 1) * G) + (i & 1); };      // the state behind register i
    // one buffer: [CH] rows of dt | x | gate [CPB each], (dt, dt x) [CPB pairs], B | C [NP each]
    const int CH = a.ch, stride = 5 * CPB + 2 * NP, buf_floats = CH * stride;
    const bool raw = a.dt_bias != nullptr;
    float* S_g = a.state + (size_t)a.state_slots[b] * a.state_stride + (size_t)c * N;
    float S[NPT], A[NPT];
    const bool vec = NPT % 2 == 0 && N % 2 == 0 && (reinterpret_cast<uintptr_t>(S_g) & 7) == 0;
    if (vec) {
#pragma unroll
        for (int i = 0; i < NPT; i += 2) {
            float2 v = make_float2(0.0f, 0.0f);
            if (n_of(i) < N) v = *reinterpret_cast<const float2*>(S_g + n_of(i));
            S[i] = v.x; S[i + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NPT; ++i) S[i] = n_of(i) < N ? S_g[n_of(i)] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < NPT; ++i)
        A[i] = n_of(i) < N ? -expf(a.a_log[(size_t)c * N + n_of(i)]) * 1.4426950408889634f : 0.0f;
    // states beyond N stay zero in every buffer's B and C
    if (NP != N) for (int i = threadIdx.x; i < SCAN_STAGES * buf_floats; i += blockDim.x) {
        const int part = i % buf_floats % stride;
        if (part >= 5 * CPB && (part - 5 * CPB) % NP >= N) sm[i] = 0.0f;
    }
    const int live_ch = min(CPB, a.C - c0);
    const int fetcher = threadIdx.x - (SPLIT ? warps * 32 : 0), fetchers = blockDim.x - (SPLIT ? warps * 32 : 0);
    auto fetch = [&](int t0, int buf) {
        const int rows = max(0, min(CH, end - t0));           // none: an empty group keeps the count of groups even
        float* base = sm + buf * buf_floats;
        if (a.vec_ch) {
            const int q = live_ch >> 2;
            for (int i = fetcher; i < rows * q; i += fetchers) {
                const int tt = i / q, ch = (i % q) * 4;
                float* row = base + tt * stride;
                const size_t t = (size_t)(t0 + tt);
                cp_async16(row + ch, a.dtraw + t * a.C + c0 + ch);
                cp_async16(row + CPB + ch, a.x + t * a.C + c0 + ch);
                cp_async16(row + 2 * CPB + ch, a.z + t * a.ld_z + c0 + ch);
            }
        } else {
            for (int i = fetcher; i < rows * live_ch; i += fetchers) {
                const int tt = i / live_ch, ch = i % live_ch;
                float* row = base + tt * stride;
                const size_t t = (size_t)(t0 + tt);
                cp_async4(row + ch, a.dtraw + t * a.C + c0 + ch);
                cp_async4(row + CPB + ch, a.x + t * a.C + c0 + ch);
                cp_async4(row + 2 * CPB + ch, a.z + t * a.ld_z + c0 + ch);
            }
        }
        if (a.vec_bc) {
            const int q = N >> 2;
            for (int i = fetcher; i < rows * q; i += fetchers) {
                const int tt = i / q, n = (i % q) * 4;
                float* row = base + tt * stride + 5 * CPB;
                const float* src = a.bc + (size_t)(t0 + tt) * a.ld_bc;
                cp_async16(row + n, src + a.col_b + n);
                cp_async16(row + NP + n, src + a.col_c + n);
            }
        } else {
            for (int i = fetcher; i < rows * N; i += fetchers) {
                const int tt = i / N, n = i % N;
                float* row = base + tt * stride + 5 * CPB;
                const float* src = a.bc + (size_t)(t0 + tt) * a.ld_bc;
                cp_async4(row + n, src + a.col_b + n);
                cp_async4(row + NP + n, src + a.col_c + n);
            }
        }
        cp_async_commit();
    };
    const float dsk = a.dskip[c];
    const int pc = warp * CPW + lane % CPW, ptt = lane / CPW;              // channel and row this lane prepares
    const float bias = raw && c0 + pc < a.C ? a.dt_bias[c0 + pc] : 0.0f;
    auto prepare = [&](int t0, int buf) {                     // the warp's channels of a chunk, an element a lane
        const int rows = min(CH, end - t0);
        float* base = sm + buf * buf_floats;
        for (int tt = ptt + part * G; tt < rows; tt += parts * G) {
            float* row = base + tt * stride;
            float dt = row[pc];
            if (raw) {
                const float v = dt + bias;
                dt = v > 20.0f ? v : log1pf(expf(v));
                row[2 * CPB + pc] = silu_f(row[2 * CPB + pc]);
            }
            *reinterpret_cast<float2*>(row + 3 * CPB + 2 * pc) = make_float2(dt, dt * row[CPB + pc]);
        }
    };
#pragma unroll
    for (int i = 0; i < SCAN_STAGES - 1; ++i)
        if (!SPLIT || helper) fetch(first + i * CH, i);
    if (SPLIT) {
        cp_async_wait<SCAN_STAGES - 2>();
        __syncthreads();
        if (helper) prepare(first, 0);
    }
    int buf = 0;
    for (int t0 = first; t0 < end; t0 += CH, buf = (buf + 1) % SCAN_STAGES) {
        const int rows = min(CH, end - t0);
        cp_async_wait<1>();       // all but the newest group: this chunk (SPLIT: and the next one) is here
        __syncthreads();          // ... for everyone, prepared, and everyone has left the chunk before
        if (!SPLIT || helper)         // into the buffer of the chunk before
            fetch(t0 + (SCAN_STAGES - 1) * CH, (buf + SCAN_STAGES - 1) % SCAN_STAGES);
        if (SPLIT) {
            if (helper) {
                prepare(t0 + CH, (buf + 1) % SCAN_STAGES);
                continue;
            }
        } else {
            prepare(t0, buf);
            __syncwarp();
        }
        const float* base = sm + buf * buf_floats;
        // RB rows: everything that does not hang on the states first, then their chain; acc: the lane's parts of the sums
        auto walk = [&](const float* row, auto& acc) {
            constexpr int RB = sizeof(acc) / sizeof(float);
            float2 d[RB], B[RB][NPT / 2], Cn[RB][NPT / 2];
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                d[r] = *reinterpret_cast<const float2*>(row + r * stride + 3 * CPB + 2 * cl);
                const float* Br = row + r * stride + 5 * CPB + 2 * sub;
#pragma unroll
                for (int i = 0; i < NPT / 2; ++i) {
                    B[r][i] = *reinterpret_cast<const float2*>(Br + 2 * i * G);
                    Cn[r][i] = *reinterpret_cast<const float2*>(Br + NP + 2 * i * G);
                }
            }
            float e[RB][NPT];
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
                for (int i = 0; i < NPT; ++i) e[r][i] = ex2_approx(d[r].x * A[i]);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                float p[NPT / 2];
#pragma unroll
                for (int i = 0; i < NPT / 2; ++i) {
                    S[2 * i] = fmaf(e[r][2 * i], S[2 * i], d[r].y * B[r][i].x);
                    S[2 * i + 1] = fmaf(e[r][2 * i + 1], S[2 * i + 1], d[r].y * B[r][i].y);
                    p[i] = fmaf(S[2 * i + 1], Cn[r][i].y, __fmul_rn(S[2 * i], Cn[r][i].x));
                }
#pragma unroll
                for (int o = NPT / 4; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < o; ++i) p[i] += p[i + o];
                acc[r] = p[0];
            }
        };
        auto store = [&](int tt, float sum) {
            const float* row = base + tt * stride;
            ((TO*)a.out)[(size_t)(t0 + tt) * a.C + c] = from_float<TO>(fmaf(dsk, row[CPB + cl], sum) * row[2 * CPB + cl]);
        };
        int tt = 0;
        if (G <= SCAN_RB) {
            for (; tt + SCAN_RB <= rows; tt += SCAN_RB) {
                float acc[SCAN_RB];
                constexpr int RB = NPT <= 4 ? SCAN_RB : 2;      // (what the registers hold)
#pragma unroll
                for (int r = 0; r < SCAN_RB; r += RB) walk(base + (tt + r) * stride, *reinterpret_cast<float(*)[RB]>(acc + r));
                int held = 0;                                  // the first row this lane still holds
#pragma unroll
                for (int o = G / 2, n = SCAN_RB / 2; o > 0; o >>= 1, n >>= 1) {
                    const bool upper = sub & o;
                    held += upper ? n : 0;
#pragma unroll
                    for (int j = 0; j < n; ++j) {
                        const float send = upper ? acc[j] : acc[j + n], keep = upper ? acc[j + n] : acc[j];
                        acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
                if (live)
#pragma unroll
                    for (int j = 0; j < (G <= SCAN_RB ? SCAN_RB / G : 1); ++j) store(tt + held + j, acc[j]);
            }
        }
        for (; tt < rows; ++tt) {
            float acc[1];
            walk(base + tt * stride, acc);
#pragma unroll
            for (int o = G >> 1; o > 0; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
            if (live && sub == 0) store(tt, acc[0]);
        }
    }
    if (live && !helper) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < NPT; i += 2)
                if (n_of(i) < N) *reinterpret_cast<float2*>(S_g + n_of(i)) = make_float2(S[i], S[i + 1]);
        } else {
#pragma unroll
            for (int i = 0; i < NPT; ++i)
                if (n_of(i) < N) S_g[n_of(i)] = S[i];
        }
    }
}

template <typename TO, int NPT, int G, bool SPLIT = false>
static int launch_scan(ScanArgs a, int B, int most, cudaStream_t stream) {
    // two walking warps a block spread a single prompt's channels evenly over the SMs; otherwise four
    const int warps = SPLIT ? 2 : 4;
    const int cpb = warps * (32 / G);
    const dim3 grid((a.C + cpb - 1) / cpb, B);
    a.ch = most < SCAN_CH ? most : SCAN_CH;
    a.alone = most > SCAN_CH;
    const size_t smem = (size_t)(SPLIT ? 4 : 3) * a.ch * (5 * cpb + 2 * G * NPT) * sizeof(float);
    const uintptr_t chp = reinterpret_cast<uintptr_t>(a.dtraw) | reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.z);
    a.vec_ch = (a.C % 4 == 0 && cpb % 4 == 0 && a.ld_z % 4 == 0 && (chp & 15) == 0) ? 1 : 0;
    a.vec_bc = (a.N % 4 == 0 && cpb % 4 == 0 && a.col_b % 4 == 0 && a.col_c % 4 == 0 && a.ld_bc % 4 == 0 &&
                (reinterpret_cast<uintptr_t>(a.bc) & 15) == 0) ? 1 : 0;
    auto kern = selective_scan_kernel<TO, NPT, G, SPLIT>;
    // (the same limit whatever the size: another thread's launch must not find it lowered)
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess)
        return SHARPI_LAUNCH_FAILED;
    if (a.alone) {
        kern<<<grid, warps * (SPLIT ? 32 * (1 + SCAN_HELPERS) : 32), smem, stream>>>(a);
        SHARPI_CHECK_LAUNCH();
    } else {
        SHARPI_LAUNCH_PDL(kern, grid, warps * (SPLIT ? 32 * (1 + SCAN_HELPERS) : 32), smem, stream, a);
    }
    return SHARPI_OK;
}

// `T`: the rows to walk; `most`: a request's at most
template <typename TO>
static int launch_scan(const ScanArgs& a, int B, int T, int longest, int most, cudaStream_t stream) {
    const int NP = a.N <= 4 ? 4 : a.N <= 8 ? 8 : a.N <= 16 ? 16 : a.N <= 32 ? 32 : a.N <= 64 ? 64 : a.N <= 128 ? 128 : 256;
    // Rows to walk and fewer warps (of eight states a lane) than schedulers: two states a lane.  us, two split / four / eight
    // states a lane, 4096 channels of 16 states: one prompt of 2048 rows 152 / 296 / 455; two of 1024 133 / 165 / 230; three of
    // 683 140 / 126 / 173; eight of 2048 909 / 765 / 1015.  Single rows (the state streams through; of 16 states
    // they have a kernel of their own where the strides allow 16-byte loads): 200 requests 240 / 63 / 45.
    // More than 16 states are more than 8 lanes of two, whose rows are walked and summed one by one: one prompt of 2048 rows, two /
    // eight states a lane, 2048 channels of 64 states 915 / 357, 1024 of 128 948 / 510, 4096 of 32 490 / 405.
    // Requests count as walks by their rows over those of the longest.  Every request, a single row too, costs a set of blocks
    // with their set-up, 1.2 us with two states a lane and 0.25 with four at 4096 channels, and a row of the longest 0.08 us less
    // with two: hence the last condition.  One prompt beside 63 single rows, two / four states a lane: 1985 rows 174 / 332,
    // 300 rows 94 / 56, 60 rows 83 / 27; 1800 rows beside 200 337 / 311; of 2048 channels 1985 rows 137 / 300, 300 rows 48 / 50.
    const bool walk = (longest ? longest : most) > SCAN_CH;
    const double walks = longest ? (double)T / longest : B;
    const bool few = walk && NP <= 16 && walks * a.C * NP / (8 * 32) < 4 * 148 &&
                     (long long)(longest ? longest : most) * 340 > (long long)a.C * B;
    switch (NP) {
        case 4: return few ? launch_scan<TO, 2, 2, true>(a, B, most, stream) : launch_scan<TO, 4, 1>(a, B, most, stream);
        case 8: return few ? launch_scan<TO, 2, 4, true>(a, B, most, stream) : launch_scan<TO, 8, 1>(a, B, most, stream);
        case 16: return few ? launch_scan<TO, 2, 8, true>(a, B, most, stream) : walk ? launch_scan<TO, 4, 4>(a, B, most, stream) : launch_scan<TO, 8, 2>(a, B, most, stream);
        case 32: return launch_scan<TO, 8, 4>(a, B, most, stream);
        case 64: return launch_scan<TO, 8, 8>(a, B, most, stream);
        case 128: return launch_scan<TO, 8, 16>(a, B, most, stream);
        default: return launch_scan<TO, 8, 32>(a, B, most, stream);
    }
}

// -------------------------------------------------------------------------------------------------------------
// The scan in chunks of 64 rows that work side by side, for up to 16 states:
//   scan_sums_kernel   per chunk and channel: the step sizes (softplus), the state that the chunk's own inputs leave behind it, and the
//                      sum of its step sizes, of which exp(A sum) is the decay over the chunk
//   scan_carry_kernel  over the chunks of a request: the state before each chunk in the place of what it leaves
//   scan_outs_kernel   per chunk and channel: the rows from the state before the chunk, as the walk forms them
// A lane is a channel with all its states, two of them an instruction (f32x2); nothing is exchanged between lanes, a row's B and C are
// read by all lanes of a warp at once, and a lane's own numbers of the next rows are on their way into shared memory, where it alone
// reads them.  The exponentials are formed twice, and still the walk, whose rows follow one another, is the slower form for one long
// prompt (us, walked / in chunks, 16 states: 2048 rows of 4096 channels 154 / 112, of 2048 channels 120 / 79; 400 rows of 4096
// channels 35 / 41).  Bound by the special-function unit (two thirds busy: 36 operations a row and channel) and the last wave;
// an eighth to a half of the exponentials as polynomials on the multiply-add pipe instead were slower (115 to 135 us).
// -------------------------------------------------------------------------------------------------------------
constexpr int SC_THREADS = 128, SC_ROWS = 64, SC_AHEAD = 8;

struct ScanChunks {
    ScanArgs s;
    int B, least;
    float* dt;               // [T, C]: the step sizes
    float* sums;             // [chunks][C][N]
    float* total;            // [chunks][C]
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair2(float lo, float hi) { return (f32x2)__float_as_uint(lo) | ((f32x2)__float_as_uint(hi) << 32); }
__device__ __forceinline__ float low2(f32x2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float high2(f32x2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 ex2_pair(f32x2 v) { return pair2(ex2_approx(low2(v)), ex2_approx(high2(v))); }

// A thread's own numbers of the rows ahead, in shared memory: V floats a row, SC_AHEAD rows a group, two groups on their way
template <int V>
struct ScanRing {
    static constexpr int GROUP = SC_AHEAD * V * SC_THREADS;
    float* mine;                                           // [2][SC_AHEAD][V] of this thread, SC_THREADS floats apart
    __device__ __forceinline__ float at(int group, int j, int v) const { return mine[group * GROUP + (j * V + v) * SC_THREADS]; }
    // rows r0 .. of a chunk of `rows`: source[v] + row * ld[v]
    __device__ __forceinline__ void fetch(int group, int r0, int rows, const float* const (&source)[V], const unsigned (&ld)[V]) const {
        unsigned off[V];
#pragma unroll
        for (int v = 0; v < V; ++v) off[v] = r0 * ld[v];
#pragma unroll
        for (int j = 0; j < SC_AHEAD; ++j)
            if (r0 + j < rows)
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    cp_async4(mine + group * GROUP + (j * V + v) * SC_THREADS, source[v] + off[v]);
                    off[v] += ld[v];
                }
        cp_async_commit();
    }
};

// softplus(v) = max(v, 0) + log(1 + w), w = exp(-|v|) in [0, 1]; log(1 + w) = w + w q, q = w Q(w), Q of degree 8 fitted by reweighted
// least squares (Lawson's method), its coefficients rounded one after the other: 5e-9 of the value.  The large term joins in the last,
// rounded once operation: w where v < 0, v where not.  Two at a time.  Error against 64 bits, here / log1pf(expf(v)) as the walk has
// it: v in [-30, 0] 1.9e-7 / 1.8e-7 at most and the same root mean square (4e-8 to 5e-8 by range), v in [0, 1] 1.4e-7 / 1.3e-7 and 3.5e-8 /
// 3.7e-8, above less than there.  2048 rows of 4096 channels: the chunks 111 us so, 116 with log1pf(expf(v)), 110 with ex2.approx of
// v log2(e), whose argument is rounded once: 9e-7 off near v = -10.
__device__ __forceinline__ f32x2 softplus2(float v0, float v1) {
    constexpr float Q[9] = {-0.4999993145465851f, 0.333304762840271f, -0.24958248436450958f, 0.19693760573863983f, -0.15350909531116486f,
                            0.10673291236162186f, -0.057595446705818176f, 0.020169047638773918f, -0.0033108105417340994f};
    const f32x2 w = pair2(expf(-fabsf(v0)), expf(-fabsf(v1)));
    f32x2 q = pair2(Q[8], Q[8]);
#pragma unroll
    for (int i = 7; i >= 0; --i) q = fma2(q, w, pair2(Q[i], Q[i]));
    q = mul2(q, w);
    const float q0 = low2(q), q1 = high2(q);
    return fma2(w, pair2(v0 < 0.0f ? q0 : 1.0f + q0, v1 < 0.0f ? q1 : 1.0f + q1), pair2(v0 < 0.0f ? low2(w) : v0, v1 < 0.0f ? high2(w) : v1));
}

// Columns col .. col + N - 1 of the chunk's rows of B or C, zeros behind N
template <int NP>
__device__ __forceinline__ void scan_stage(const ScanArgs& a, const chunked::Place& p, int col, float* dst) {
    for (int i = threadIdx.x; i < p.rows * NP; i += SC_THREADS) {
        const int r = i / NP, n = i % NP;
        dst[i] = n < a.N ? a.bc[(size_t)(p.row0 + r) * a.ld_bc + col + n] : 0.0f;
    }
}

// A log2(e) of a channel's states (0 behind N: what is there stays zero)
template <int NP>
__device__ __forceinline__ void scan_rates(const ScanArgs& a, int c, f32x2 (&A)[NP / 2]) {
#pragma unroll
    for (int i = 0; i < NP / 2; ++i) {
        float v[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) v[e] = 2 * i + e < a.N ? -expf(a.a_log[(size_t)c * a.N + 2 * i + e]) * 1.4426950408889634f : 0.0f;
        A[i] = pair2(v[0], v[1]);
    }
}

template <int NP, bool RAW>
__global__ void __launch_bounds__(SC_THREADS, 5) scan_sums_kernel(ScanChunks q) {
    __shared__ __align__(16) float B_s[SC_ROWS * NP];
    __shared__ float ring_s[2 * SC_AHEAD * 2 * SC_THREADS];
    const ScanArgs& a = q.s;
    pdl_wait();
    chunked::Place p;
    if (!chunked::find_chunk<SC_ROWS>(a.row_offsets, q.B, q.least, blockIdx.y, p)) return;
    scan_stage<NP>(a, p, a.col_b, B_s);
    __syncthreads();
    const int c = blockIdx.x * SC_THREADS + threadIdx.x;
    if (c >= a.C) return;
    f32x2 A[NP / 2], S[NP / 2];
    scan_rates<NP>(a, c, A);
#pragma unroll
    for (int i = 0; i < NP / 2; ++i) S[i] = 0;
    const float bias = RAW ? a.dt_bias[c] : 0.0f;
    const size_t at0 = (size_t)p.row0 * a.C + c;
    const ScanRing<2> ring{ring_s + threadIdx.x};
    const float* const source[2] = {a.dtraw + at0, a.x + at0};
    const unsigned ld[2] = {(unsigned)a.C, (unsigned)a.C};
    ring.fetch(0, 0, p.rows, source, ld);
    ring.fetch(1, SC_AHEAD, p.rows, source, ld);
    float* dt = q.dt + at0;
    float sum = 0.0f;
    auto walk = [&](int g, int r0, int n) {
        float d[SC_AHEAD], dx[SC_AHEAD];
#pragma unroll
        for (int j = 0; j < SC_AHEAD; j += 2) {
            f32x2 v = pair2(ring.at(g, j, 0), ring.at(g, j + 1, 0));
            if (RAW) v = softplus2(low2(v) + bias, high2(v) + bias);
            d[j] = low2(v); d[j + 1] = high2(v);
            dx[j] = d[j] * ring.at(g, j, 1); dx[j + 1] = d[j + 1] * ring.at(g, j + 1, 1);
        }
#pragma unroll
        for (int j = 0; j < SC_AHEAD; ++j) {
            if (j >= n) break;
            dt[(unsigned)(r0 + j) * (unsigned)a.C] = d[j];
            sum += d[j];
            const f32x2 dd = pair2(d[j], d[j]), ee = pair2(dx[j], dx[j]);
            const ulonglong2* B = reinterpret_cast<const ulonglong2*>(B_s + (r0 + j) * NP);
#pragma unroll
            for (int i = 0; i < NP / 4; ++i) {
                const ulonglong2 b = B[i];
                S[2 * i] = fma2(ex2_pair(mul2(dd, A[2 * i])), S[2 * i], mul2(ee, b.x));
                S[2 * i + 1] = fma2(ex2_pair(mul2(dd, A[2 * i + 1])), S[2 * i + 1], mul2(ee, b.y));
            }
        }
    };
    int r0 = 0, g = 0;
    for (; r0 + SC_AHEAD <= p.rows; r0 += SC_AHEAD, g ^= 1) {
        cp_async_wait<1>();
        walk(g, r0, SC_AHEAD);
        ring.fetch(g, r0 + 2 * SC_AHEAD, p.rows, source, ld);
    }
    cp_async_wait<0>();
    if (r0 < p.rows) walk(g, r0, p.rows - r0);
    float* out = q.sums + ((size_t)blockIdx.y * a.C + c) * a.N;
#pragma unroll
    for (int i = 0; i < NP / 2; ++i) {
        if (2 * i < a.N) out[2 * i] = low2(S[i]);
        if (2 * i + 1 < a.N) out[2 * i + 1] = high2(S[i]);
    }
    q.total[(size_t)blockIdx.y * a.C + c] = sum;
}

__global__ void __launch_bounds__(256) scan_carry_kernel(ScanChunks q) {
    const ScanArgs& a = q.s;
    pdl_wait();
    const int b = blockIdx.y, rows = a.row_offsets[b + 1] - a.row_offsets[b];
    if (rows < q.least) return;
    const int base = chunked::chunks_before<SC_ROWS>(a.row_offsets, b, q.least), n = (rows + SC_ROWS - 1) / SC_ROWS;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x, size = (long long)a.C * a.N;
    if (i >= size) return;
    const int c = (int)(i / a.N);
    const float A = -expf(a.a_log[i]) * 1.4426950408889634f;
    float* state = a.state + (size_t)a.state_slots[b] * a.state_stride + i;
    float* u = q.sums + base * size + i;
    const float* total = q.total + (size_t)base * a.C + c;
    float S = *state, own[SC_AHEAD], dt[SC_AHEAD];
    auto fetch = [&](int k) {
#pragma unroll
        for (int j = 0; j < SC_AHEAD; ++j)
            if (k + j < n) { own[j] = u[(k + j) * size]; dt[j] = total[(size_t)(k + j) * a.C]; }
    };
    fetch(0);
    for (int k = 0; k < n; k += SC_AHEAD) {
        float o[SC_AHEAD], e[SC_AHEAD];
#pragma unroll
        for (int j = 0; j < SC_AHEAD; ++j) { o[j] = own[j]; e[j] = ex2_approx(dt[j] * A); }
        fetch(k + SC_AHEAD);
#pragma unroll
        for (int j = 0; j < SC_AHEAD; ++j) {
            if (k + j >= n) break;
            u[(k + j) * size] = S;
            S = fmaf(e[j], S, o[j]);
        }
    }
    *state = S;
}

template <typename TO, int NP, bool RAW>
__global__ void __launch_bounds__(SC_THREADS, 5) scan_outs_kernel(ScanChunks q) {
    __shared__ __align__(16) float B_s[SC_ROWS * NP], C_s[SC_ROWS * NP];
    __shared__ float ring_s[2 * SC_AHEAD * 3 * SC_THREADS];
    const ScanArgs& a = q.s;
    pdl_wait();
    chunked::Place p;
    if (!chunked::find_chunk<SC_ROWS>(a.row_offsets, q.B, q.least, blockIdx.y, p)) return;
    scan_stage<NP>(a, p, a.col_b, B_s);
    scan_stage<NP>(a, p, a.col_c, C_s);
    __syncthreads();
    const int c = blockIdx.x * SC_THREADS + threadIdx.x;
    if (c >= a.C) return;
    f32x2 A[NP / 2], S[NP / 2];
    scan_rates<NP>(a, c, A);
    const float* before = q.sums + ((size_t)blockIdx.y * a.C + c) * a.N;
#pragma unroll
    for (int i = 0; i < NP / 2; ++i) S[i] = pair2(2 * i < a.N ? before[2 * i] : 0.0f, 2 * i + 1 < a.N ? before[2 * i + 1] : 0.0f);
    const float dsk = a.dskip[c];
    const size_t at0 = (size_t)p.row0 * a.C + c;
    const ScanRing<3> ring{ring_s + threadIdx.x};
    const float* const source[3] = {q.dt + at0, a.x + at0, a.z + (size_t)p.row0 * a.ld_z + c};
    const unsigned ld[3] = {(unsigned)a.C, (unsigned)a.C, (unsigned)a.ld_z};
    ring.fetch(0, 0, p.rows, source, ld);
    ring.fetch(1, SC_AHEAD, p.rows, source, ld);
    TO* out = reinterpret_cast<TO*>(a.out) + at0;
    auto walk = [&](int g, int r0, int n) {
#pragma unroll
        for (int j = 0; j < SC_AHEAD; ++j) {
            if (j >= n) break;
            const float d = ring.at(g, j, 0), x = ring.at(g, j, 1), z = ring.at(g, j, 2), dx = d * x;
            const f32x2 dd = pair2(d, d), ee = pair2(dx, dx);
            const ulonglong2* B = reinterpret_cast<const ulonglong2*>(B_s + (r0 + j) * NP);
            const ulonglong2* Cn = reinterpret_cast<const ulonglong2*>(C_s + (r0 + j) * NP);
            f32x2 y0 = 0, y1 = 0;
#pragma unroll
            for (int i = 0; i < NP / 4; ++i) {
                const ulonglong2 b = B[i], cn = Cn[i];
                S[2 * i] = fma2(ex2_pair(mul2(dd, A[2 * i])), S[2 * i], mul2(ee, b.x));
                S[2 * i + 1] = fma2(ex2_pair(mul2(dd, A[2 * i + 1])), S[2 * i + 1], mul2(ee, b.y));
                y0 = fma2(S[2 * i], cn.x, y0);
                y1 = fma2(S[2 * i + 1], cn.y, y1);
            }
            const float y = (low2(y0) + low2(y1)) + (high2(y0) + high2(y1));
            out[(unsigned)(r0 + j) * (unsigned)a.C] = from_float<TO>(fmaf(dsk, x, y) * (RAW ? silu_f(z) : z));
        }
    };
    int r0 = 0, g = 0;
    for (; r0 + SC_AHEAD <= p.rows; r0 += SC_AHEAD, g ^= 1) {
        cp_async_wait<1>();
        walk(g, r0, SC_AHEAD);
        ring.fetch(g, r0 + 2 * SC_AHEAD, p.rows, source, ld);
    }
    cp_async_wait<0>();
    if (r0 < p.rows) walk(g, r0, p.rows - r0);
}

template <typename TO, int NP, bool RAW>
static int launch_scan_chunks(const ScanChunks& q, int chunks, cudaStream_t stream) {
    const dim3 grid((q.s.C + SC_THREADS - 1) / SC_THREADS, chunks);
    SHARPI_LAUNCH_PDL((scan_sums_kernel<NP, RAW>), grid, SC_THREADS, 0, stream, q);
    SHARPI_LAUNCH_PDL(scan_carry_kernel, dim3((unsigned)(((long long)q.s.C * q.s.N + 255) / 256), q.B), 256, 0, stream, q);
    SHARPI_LAUNCH_PDL((scan_outs_kernel<TO, NP, RAW>), grid, SC_THREADS, 0, stream, q);
    return SHARPI_OK;
}

template <typename TO, int NP>
static int launch_scan_chunks(const ScanChunks& q, int chunks, cudaStream_t stream) {
    return q.s.dt_bias ? launch_scan_chunks<TO, NP, true>(q, chunks, stream) : launch_scan_chunks<TO, NP, false>(q, chunks, stream);
}

template <typename TO>
static int launch_scan_chunks(const ScanChunks& q, int chunks, cudaStream_t stream) {
    return q.s.N <= 4 ? launch_scan_chunks<TO, 4>(q, chunks, stream)
                      : q.s.N <= 8 ? launch_scan_chunks<TO, 8>(q, chunks, stream) : launch_scan_chunks<TO, 16>(q, chunks, stream);
}

// Steps that bring about a row a request, 16 states a channel: the states' bytes and little else.  A warp is 32 channels of a
// request; four lanes own four channels, four neighbouring states of each (a warp's load is 512 contiguous bytes), and what a
// channel needs once a row (step size, gate, output) is formed by one of the four.  The operations of a channel and their order
// are the walk's.  4096 channels: 200 requests 48 us with the walk (its blocks stage, prepare and meet for one row), 21 us so
// (31 where every lane formed all of its channels' step sizes); 20 requests 8.4 and 4.1.  Two or four requests a warp, for one
// set of decay rates: 22 us.  Four lanes of four states make 16, the usual count; others stay with the walk.
constexpr int SS_THREADS = 128;

template <typename TO, bool RAW>
__global__ void __launch_bounds__(SS_THREADS) scan_step_kernel(ScanArgs a) {
    constexpr int U = 4;                                   // channels of four lanes: c0, c0 + 8, c0 + 16 and c0 + 24
    const int lane = threadIdx.x & 31, sub = lane % 4, c0 = (blockIdx.x * (SS_THREADS / 32) + (threadIdx.x >> 5)) * 8 * U + lane / 4;
    const int own = c0 + 8 * sub, own_c = min(own, a.C - 1), b = blockIdx.y;
    float4 A[U], S[U];
    auto live = [&](int u) { return c0 + 8 * u < a.C; };
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const float4 l = *reinterpret_cast<const float4*>(a.a_log + (size_t)min(c0 + 8 * u, a.C - 1) * 16 + 4 * sub);
        A[u] = make_float4(-expf(l.x) * 1.4426950408889634f, -expf(l.y) * 1.4426950408889634f, -expf(l.z) * 1.4426950408889634f,
                           -expf(l.w) * 1.4426950408889634f);
    }
    const float bias = RAW ? a.dt_bias[own_c] : 0.0f, dsk = a.dskip[own_c];
    pdl_wait();
    const int first = a.row_offsets[b], end = a.row_offsets[b + 1];
    if (first >= end || end - first >= a.skip) return;
    float* st = a.state + (size_t)a.state_slots[b] * a.state_stride + (size_t)c0 * 16 + 4 * sub;
#pragma unroll
    for (int u = 0; u < U; ++u)
        S[u] = live(u) ? *reinterpret_cast<const float4*>(st + u * 128) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t = first; t < end; ++t) {
        const float4 Bn = *reinterpret_cast<const float4*>(a.bc + (size_t)t * a.ld_bc + a.col_b + 4 * sub);
        const float4 Cn = *reinterpret_cast<const float4*>(a.bc + (size_t)t * a.ld_bc + a.col_c + 4 * sub);
        const float x = a.x[(size_t)t * a.C + own_c], z = a.z[(size_t)t * a.ld_z + own_c];
        float d_own = a.dtraw[(size_t)t * a.C + own_c], y = 0.0f;
        if (RAW) {
            const float v = d_own + bias;
            d_own = v > 20.0f ? v : log1pf(expf(v));
        }
        const float dx_own = d_own * x;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float d = __shfl_sync(0xffffffffu, d_own, u, 4), dx = __shfl_sync(0xffffffffu, dx_own, u, 4);
            S[u].x = fmaf(ex2_approx(d * A[u].x), S[u].x, __fmul_rn(dx, Bn.x));
            S[u].y = fmaf(ex2_approx(d * A[u].y), S[u].y, __fmul_rn(dx, Bn.y));
            S[u].z = fmaf(ex2_approx(d * A[u].z), S[u].z, __fmul_rn(dx, Bn.z));
            S[u].w = fmaf(ex2_approx(d * A[u].w), S[u].w, __fmul_rn(dx, Bn.w));
            // pairs of states, then the tree over the eight pairs (this lane has 2 sub and 2 sub + 1)
            float p0 = fmaf(S[u].y, Cn.y, __fmul_rn(S[u].x, Cn.x)), p1 = fmaf(S[u].w, Cn.w, __fmul_rn(S[u].z, Cn.z));
            p0 += __shfl_xor_sync(0xffffffffu, p0, 2); p1 += __shfl_xor_sync(0xffffffffu, p1, 2);
            p0 += __shfl_xor_sync(0xffffffffu, p0, 1); p1 += __shfl_xor_sync(0xffffffffu, p1, 1);
            if (sub == u) y = p0 + p1;
        }
        if (own < a.C)
            reinterpret_cast<TO*>(a.out)[(size_t)t * a.C + own] = from_float<TO>(fmaf(dsk, x, y) * (RAW ? silu_f(z) : z));
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (live(u)) *reinterpret_cast<float4*>(st + u * 128) = S[u];
}

template <typename TO>
static int launch_scan_step(const ScanArgs& a, int B, cudaStream_t stream) {
    const dim3 grid((a.C + SS_THREADS - 1) / SS_THREADS, B);
    if (a.dt_bias) SHARPI_LAUNCH_PDL((scan_step_kernel<TO, true>), grid, SS_THREADS, 0, stream, a);
    else SHARPI_LAUNCH_PDL((scan_step_kernel<TO, false>), grid, SS_THREADS, 0, stream, a);
    return SHARPI_OK;
}

// `longest`: the rows of the longest request, 0 where it is not known (a choice of kernels, no result depends on it).  `work`
// (nullable; T * C + `chunks` * C * (N + 1) floats): requests of at least `least` rows run in chunks, `chunks` of them at most; the
// others, and without it all, are walked (`walk` = 0: there are no others; `walked` rows, `longest_walked` of one request, 0 where
// that is not known).
SHARPI_API int sharpi_selective_scan(const float* x, const float* dtraw, const float* dt_bias, const float* bc,
                                     int ld_bc, int col_b, int col_c, const float* a_log, const float* dskip,
                                     const float* z, int ld_z, const int* row_offsets, const int* state_slots,
                                     float* state, long long state_stride, void* out, int out_dtype, int T, int B,
                                     int C, int N, int longest, float* work, int chunks, int least, int walk, int walked, int longest_walked,
                                     cudaStream_t stream) {
    if (B <= 0) return SHARPI_OK;
    if (C <= 0 || N <= 0 || N > 256) return SHARPI_BAD_ARGUMENT;
    ScanArgs a;
    a.x = x; a.dtraw = dtraw; a.dt_bias = dt_bias; a.bc = bc; a.ld_bc = ld_bc; a.col_b = col_b; a.col_c = col_c;
    a.a_log = a_log; a.dskip = dskip; a.z = z; a.ld_z = ld_z; a.row_offsets = row_offsets; a.state_slots = state_slots;
    a.state = state; a.state_stride = state_stride; a.out = out; a.C = C; a.N = N; a.skip = 0x7fffffff;
    int most = T - B + 1 < 1 ? 1 : T - B + 1;              // no request brings more rows
    if (work) {
        if (N > 16 || chunks < 1 || chunks > 65535 || B > 65535 || least < 1) return SHARPI_BAD_ARGUMENT;
        ScanChunks q;
        q.s = a; q.B = B; q.least = least; q.dt = work; q.sums = work + (size_t)T * C; q.total = q.sums + (size_t)chunks * C * N;
        int rc = SHARPI_BAD_ARGUMENT;
        if (out_dtype == SHARPI_F32) rc = launch_scan_chunks<float>(q, chunks, stream);
        if (out_dtype == SHARPI_BF16) rc = launch_scan_chunks<bf16>(q, chunks, stream);
        if (rc != SHARPI_OK || !walk) return rc;
        a.skip = least;
        // The kernel for the others goes by their rows, not by the step's.  us, all walked / chunks with a walk chosen by the prompt's
        // rows / so: 60 single rows beside a prompt of 1286, 2048 channels 94 / 98 / 73, 4096 channels 139 / 175 / 106.
        if (walked > 0) { T = walked; longest = most = longest_walked; }
        else if (longest >= least) longest = least - 1;
    }
    const uintptr_t bases = (uintptr_t)state | (uintptr_t)bc | (uintptr_t)a_log;
    if (T <= B && longest <= SCAN_CH && N == 16 && state_stride % 4 == 0 && ld_bc % 4 == 0 && col_b % 4 == 0 && col_c % 4 == 0 && (bases & 15) == 0) {
        if (out_dtype == SHARPI_F32) return launch_scan_step<float>(a, B, stream);
        if (out_dtype == SHARPI_BF16) return launch_scan_step<bf16>(a, B, stream);
    }
    if (out_dtype == SHARPI_F32) return launch_scan<float>(a, B, T, longest, most, stream);
    if (out_dtype == SHARPI_BF16) return launch_scan<bf16>(a, B, T, longest, most, stream);
    return SHARPI_BAD_ARGUMENT;
}
