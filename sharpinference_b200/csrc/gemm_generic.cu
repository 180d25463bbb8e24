// C = A . W^T on the CUDA cores with fp32 accumulation, for any M, N, K: the matrix product
// of the true 32-bit path (no tensor cores, no reduced-precision mode) and the fallback for
// shapes the tensor-core kernels refuse.  Dense and grouped (one weight matrix per expert,
// rows sorted by expert) share the kernel.
//
// Each output element is the same sequence of operations in every kernel of this file: K is cut into segments of 128
// (from k = 0 on), a segment is two chains of fused multiply-adds, one over its even and one over its odd k, and the
// segments' sums (even + odd) are added in order.  So a value depends on its own row and column only: never on M, on
// the other rows of the step, on the tile it fell into or on which kernel formed it.  Two chains, because sm_100 multiplies
// and adds two neighbouring floats in one instruction (fma.rn.f32x2) and neighbours in k lie side by side in memory;
// segments, because they let a few rows be formed by many threads without another order of additions.
//
//   gemm_few_kernel    up to GF_MAX_ROWS rows (decode): a lane is one segment of one weight row, for all rows of the pass
//   gemm_tile_kernel   float32 operands whose rows start on 16 bytes: 128 x 64 or 64 x 64 tiles, operands through cp.async
//   gemm_nt_kernel     everything else (bfloat16 operands, odd inner sizes, unaligned rows)
//
// The reference's counterparts are llm_matvec_f32
// (src/SharpInference.Cuda/CudaTextKernels.cs:1325) and its per-expert matvec loop
// (src/SharpInference.Engine/CudaForwardPass.cs:5554-5578).
#include "common.cuh"
#include "mma_sync.cuh"

constexpr int GB_M = 64, GB_N = 64, GB_K = 16;
constexpr int GB_SEG = 128;          // k of a segment

struct GemmArgs {
    const void* A;              // [rows, K], row r of the product reads A[a_rows ? a_rows[r] : r]
    const void* W;              // [E, N, K]
    float* C;                   // [rows, N], row r writes C[out_rows ? out_rows[r] : r]
    const int* group_offsets;   // [E + 1] first sorted row of every group; null: one group [0, M)
    const int* a_rows;
    const int* out_rows;
    int M, N, K, E;
    int accumulate;             // C += instead of C =
    const float* bias;          // [N] added to every row (nullable)
    const float* row_scale;     // row r of the product is multiplied by row_scale[scale_rows ? scale_rows[r] : r]
    const int* scale_rows;      //   before the bias and before it is stored or added in (both nullable)
};

// What happens to a finished sum: the row's factor, the bias, and the store or add-in.
__device__ __forceinline__ void gemm_store(const GemmArgs& g, int m, int n, float sum) {
    float v = g.row_scale ? __fmul_rn(sum, g.row_scale[g.scale_rows ? g.scale_rows[m] : m]) : sum;
    if (g.bias) v = __fadd_rn(v, g.bias[n]);
    float* c = g.C + (size_t)(g.out_rows ? g.out_rows[m] : m) * g.N + n;
    *c = g.accumulate ? *c + v : v;
}

// The rows [m0, m_end) and the weight matrix `e` of tile number `tile` (tiles of `rows` rows, groups one after the
// other); false: there is no such tile.
__device__ __forceinline__ bool gemm_tile_rows(const GemmArgs& g, int tile, int rows, int& e, int& m0, int& m_end) {
    e = 0;
    if (g.group_offsets) {
        int start = 0;
        for (; e < g.E; ++e) {
            start = g.group_offsets[e];
            const int tiles = (g.group_offsets[e + 1] - start + rows - 1) / rows;
            if (tile < tiles) break;
            tile -= tiles;
        }
        if (e >= g.E) return false;
        m0 = start + tile * rows;
        m_end = g.group_offsets[e + 1];
    } else {
        m0 = tile * rows;
        m_end = g.M;
    }
    return m0 < m_end;
}

typedef unsigned long long f32x2;      // two floats in one 64-bit register: an even k below, an odd k above
__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(f32x2 v) {
    return __fadd_rn(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
}

template <typename TA, typename TW>
__global__ void __launch_bounds__(256) gemm_nt_kernel(GemmArgs g) {
    __shared__ float As[GB_K][GB_M + 4];
    __shared__ float Ws[GB_K][GB_N + 4];

    int m0, m_end, e;
    if (!gemm_tile_rows(g, blockIdx.y, GB_M, e, m0, m_end)) return;
    const int n0 = blockIdx.x * GB_N;
    const TA* A = (const TA*)g.A;
    const TW* W = (const TW*)g.W + (size_t)e * g.N * g.K;

    const int tid = threadIdx.x;
    const int lrow = tid >> 2;        // 0..63: tile row loaded by this thread
    const int lk = (tid & 3) * 4;     // 0,4,8,12: first of its 4 k values
    const int am = m0 + lrow;
    const bool a_ok = am < m_end;
    const TA* a_ptr = a_ok ? A + (size_t)(g.a_rows ? g.a_rows[am] : am) * g.K : nullptr;
    const int wn = n0 + lrow;
    const bool w_ok = wn < g.N;
    const TW* w_ptr = w_ok ? W + (size_t)wn * g.K : nullptr;

    const int tx = tid & 15, ty = tid >> 4;  // thread computes rows ty*4.., cols tx*4..
    float acc[4][4][2], total[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = total[i][j] = 0.0f;

    for (int k0 = 0; k0 < g.K; k0 += GB_K) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            As[lk + i][lrow] = (a_ok && k < g.K) ? to_float(a_ptr[k]) : 0.0f;
            Ws[lk + i][lrow] = (w_ok && k < g.K) ? to_float(w_ptr[k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GB_K; ++k) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j][k & 1] = __fmaf_rn(av[i], wv[j], acc[i][j][k & 1]);
        }
        __syncthreads();
        if ((k0 + GB_K) % GB_SEG == 0 || k0 + GB_K >= g.K) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    total[i][j] = __fadd_rn(total[i][j], __fadd_rn(acc[i][j][0], acc[i][j][1]));
                    acc[i][j][0] = acc[i][j][1] = 0.0f;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= m_end) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n0 + tx * 4 + j < g.N) gemm_store(g, m, n0 + tx * 4 + j, total[i][j]);
    }
}

// float32 operands, rows on 16 bytes.  A thread has rows ty + i BM / 8 and columns tx + 16 j of the tile; a stage is 32 k of
// the tile's rows as they lie in memory (k in front), 4 floats of padding a row, so that neighbouring rows start in other
// banks: 12 reads of 16 bytes serve 64 paired multiply-adds, eight of which in a row take the same weights (an operand that
// the register file need not give again).  A stage is written out in full: the reads of the next k are then under way before
// the products of these (219 registers, so one CTA of 256 threads an SM; two of 128 registers each were no faster: the
// multiply-adds themselves are the bound, 58 TFLOP/s of them alone).  2048 rows of 5120 x 5120: 37.3 -> 41.3 TFLOP/s, 980 rows of
// 8192 x 1024 470 -> 428 us, 300 rows of 8192 x 1024 199 -> 181 us, 64 rows of 1024 x 1024 46 -> 40 us.
constexpr int GT_N = 64, GT_K = 32, GT_LD = GT_K + 4, GT_STAGES = 3;

template <int BM>
__global__ void __launch_bounds__(2 * BM) gemm_tile_kernel(GemmArgs g) {
    extern __shared__ __align__(16) float gt_smem[];
    constexpr int THREADS = 2 * BM, STAGE = (BM + GT_N) * GT_LD;
    int m0, m_end, e;
    if (!gemm_tile_rows(g, blockIdx.y, BM, e, m0, m_end)) return;
    const int n0 = blockIdx.x * GT_N;
    const float* W = (const float*)g.W + (size_t)e * g.N * g.K;
    const int tid = threadIdx.x, piece = (tid & 7) * 4;

    // a thread copies the same 16 bytes of the same rows of every stage
    constexpr int LA = BM / (THREADS / 8), LW = GT_N / (THREADS / 8);
    const float* src[LA + LW];
#pragma unroll
    for (int i = 0; i < LA + LW; ++i) {
        const int r = (tid >> 3) + (i < LA ? i : i - LA) * (THREADS / 8);
        if (i < LA) {
            const int m = m0 + r;
            src[i] = m < m_end ? (const float*)g.A + (size_t)(g.a_rows ? g.a_rows[m] : m) * g.K + piece : nullptr;
        } else {
            src[i] = n0 + r < g.N ? W + (size_t)(n0 + r) * g.K + piece : nullptr;
        }
    }
    const int stages = (g.K + GT_K - 1) / GT_K;
    auto load = [&](int s) {
        float* dst = gt_smem + (s % GT_STAGES) * STAGE + (tid >> 3) * GT_LD + piece;
        const int k = s * GT_K;
#pragma unroll
        for (int i = 0; i < LA + LW; ++i) {
            const bool ok = src[i] != nullptr && k + piece < g.K;
            const int row = i < LA ? i * (THREADS / 8) : BM + (i - LA) * (THREADS / 8);
            mma16::cp_async_16(dst + row * GT_LD, ok ? src[i] + k : (const float*)g.W, ok ? 16 : 0);
        }
    };
#pragma unroll
    for (int s = 0; s < GT_STAGES - 1; ++s) {
        if (s < stages) load(s);
        mma16::cp_async_commit();
    }

    const int tx = tid & 15, ty = tid >> 4;
    f32x2 acc[8][4];
    float total[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0, total[i][j] = 0.0f;

    for (int s = 0; s < stages; ++s) {
        mma16::cp_async_wait<GT_STAGES - 2>();
        __syncthreads();                        // the stage has arrived, and the one read last is free
        if (s + GT_STAGES - 1 < stages) load(s + GT_STAGES - 1);
        mma16::cp_async_commit();
        const float* a_s = gt_smem + (s % GT_STAGES) * STAGE + ty * GT_LD;
        const float* w_s = gt_smem + (s % GT_STAGES) * STAGE + (BM + tx) * GT_LD;
#pragma unroll
        for (int k = 0; k < GT_K; k += 4) {
            ulonglong2 a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(a_s + i * (BM / 8) * GT_LD + k);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(w_s + j * 16 * GT_LD + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].x, w.x);
#pragma unroll
                for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].y, w.y);
            }
        }
        if ((s + 1) % (GB_SEG / GT_K) == 0 || s + 1 == stages) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    total[i][j] = __fadd_rn(total[i][j], sum2(acc[i][j]));
                    acc[i][j] = 0;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty + i * (BM / 8);
        if (m >= m_end) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n0 + tx + 16 * j < g.N) gemm_store(g, m, n0 + tx + 16 * j, total[i][j]);
    }
}

// A few float32 rows: the weights stream through once and every segment is a lane's own.  A warp takes 8 weight rows x 4
// segments (lane = row * 4 + segment), copies them 32 k at a time into buffers of its own (whole 128-byte lines), the same k
// of the pass's MR activation rows beside them; the segments' sums meet in shared memory and are added in order.  Four rows
// of 1024 x 4096: 9 us, 223 us as one tile a 64 columns whose threads walk all of K; 5120 x 5120 at one row 26 us = 4.0 TB/s.
constexpr int GF_N = 8, GF_STAGES = 4, GF_MAX_WARPS = 4, GF_MAX_ROWS = 32, GF_MAX_K = 32768;   // at most 212 KB of buffers

template <int MR>
__global__ void __launch_bounds__(32 * GF_MAX_WARPS) gemm_few_kernel(GemmArgs g, int passes) {
    extern __shared__ __align__(16) float gf_smem[];
    constexpr int STAGE = (32 + 4 * MR) * GT_LD;
    pdl_wait();
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.y / passes;
    const int m0 = (g.group_offsets ? g.group_offsets[e] : 0) + (blockIdx.y % passes) * MR;
    const int m_end = g.group_offsets ? g.group_offsets[e + 1] : g.M;
    if (m0 >= m_end) return;
    const int n0 = blockIdx.x * GF_N;
    const float* W = (const float*)g.W + (size_t)e * g.N * g.K;
    const int segs = (g.K + GB_SEG - 1) / GB_SEG;
    float* buf = gf_smem + warp * GF_STAGES * STAGE;
    float* part = gf_smem + warps * GF_STAGES * STAGE;       // [MR][GF_N][segs]

    const int piece = (lane & 7) * 4;
    const float* a_src[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) {
        const int r = m0 + m;
        a_src[m] = r < m_end ? (const float*)g.A + (size_t)(g.a_rows ? g.a_rows[r] : r) * g.K : nullptr;
    }
    // stage i of this warp: segments 4 (warp + (i / 4) warps) ..., k 32 (i % 4) ... of each
    constexpr int PER = GB_SEG / GT_K;
    const int groups = (segs + 3) / 4;
    const int mine = groups > warp ? (groups - warp + warps - 1) / warps : 0;
    auto load = [&](int i) {
        float* dst = buf + (i % GF_STAGES) * STAGE + piece;
        const int seg0 = 4 * (warp + (i / PER) * warps);
#pragma unroll
        for (int r = 0; r < 8; ++r) {                         // rows 4 r + lane / 8 of the stage: weight row r, segment lane / 8
            const int n = n0 + r, k = (seg0 + (lane >> 3)) * GB_SEG + (i % PER) * GT_K + piece;
            const bool ok = n < g.N && k < g.K;
            mma16::cp_async_16(dst + (4 * r + (lane >> 3)) * GT_LD, ok ? W + (size_t)n * g.K + k : W, ok ? 16 : 0);
        }
#pragma unroll
        for (int m = 0; m < MR; ++m) {
            const int k = (seg0 + (lane >> 3)) * GB_SEG + (i % PER) * GT_K + piece;
            const bool ok = a_src[m] != nullptr && k < g.K;
            mma16::cp_async_16(dst + (32 + 4 * m + (lane >> 3)) * GT_LD, ok ? a_src[m] + k : W, ok ? 16 : 0);
        }
    };
#pragma unroll
    for (int i = 0; i < GF_STAGES - 1; ++i) {
        if (i < mine * PER) load(i);
        mma16::cp_async_commit();
    }
    f32x2 acc[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[m] = 0;
    for (int i = 0; i < mine * PER; ++i) {
        mma16::cp_async_wait<GF_STAGES - 2>();
        __syncwarp();
        if (i + GF_STAGES - 1 < mine * PER) load(i + GF_STAGES - 1);
        mma16::cp_async_commit();
        const float* w_s = buf + (i % GF_STAGES) * STAGE + lane * GT_LD;
        const float* a_s = buf + (i % GF_STAGES) * STAGE + (32 + (lane & 3)) * GT_LD;
#pragma unroll
        for (int k = 0; k < GT_K; k += 4) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(w_s + k);
#pragma unroll
            for (int m = 0; m < MR; ++m) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_s + 4 * m * GT_LD + k);
                fma2(acc[m], a.x, w.x);
                fma2(acc[m], a.y, w.y);
            }
        }
        if ((i + 1) % PER == 0) {
            const int seg = 4 * (warp + (i / PER) * warps) + (lane & 3);
#pragma unroll
            for (int m = 0; m < MR; ++m) {
                if (seg < segs) part[(m * GF_N + (lane >> 2)) * segs + seg] = sum2(acc[m]);
                acc[m] = 0;
            }
        }
    }
    __syncthreads();
    for (int o = threadIdx.x; o < MR * GF_N; o += blockDim.x) {
        const int m = m0 + o / GF_N, n = n0 + o % GF_N;
        if (m >= m_end || n >= g.N) continue;
        float total = 0.0f;
        for (int sg = 0; sg < segs; ++sg) total = __fadd_rn(total, part[o * segs + sg]);
        gemm_store(g, m, n, total);
    }
}

template <int MR>
static int launch_few(const GemmArgs& g, cudaStream_t stream) {
    const int segs = (g.K + GB_SEG - 1) / GB_SEG, groups = (segs + 3) / 4;
    const int warps = groups < GF_MAX_WARPS ? groups : GF_MAX_WARPS, passes = (g.M + MR - 1) / MR;
    const size_t smem = ((size_t)warps * GF_STAGES * (32 + 4 * MR) * GT_LD + (size_t)MR * GF_N * segs) * sizeof(float);
    // (the same limit whatever the size: another thread's launch, or a captured one, must not find it lowered)
    if (cudaFuncSetAttribute(gemm_few_kernel<MR>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess)
        return SHARPI_LAUNCH_FAILED;
    // (its set-up beside the tail of the kernel before it: the float32 decode step is a chain of 20 launches of 3 to 15 us)
    SHARPI_LAUNCH_PDL(gemm_few_kernel<MR>, dim3((unsigned)((g.N + GF_N - 1) / GF_N), (unsigned)(passes * g.E)), 32 * warps, smem, stream, g, passes);
    return SHARPI_OK;
}

template <int BM>
static int launch_tile(const GemmArgs& g, cudaStream_t stream) {
    constexpr size_t smem = (size_t)GT_STAGES * (BM + GT_N) * GT_LD * sizeof(float);
    const long long m_tiles = (g.M + BM - 1) / BM + (g.group_offsets ? g.E : 0), n_tiles = (g.N + GT_N - 1) / GT_N;
    if (m_tiles > 65535) return SHARPI_BAD_ARGUMENT;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(gemm_tile_kernel<BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return SHARPI_LAUNCH_FAILED;
    gemm_tile_kernel<BM><<<dim3((unsigned)n_tiles, (unsigned)m_tiles), 2 * BM, smem, stream>>>(g);
    SHARPI_CHECK_LAUNCH();
    return SHARPI_OK;
}

SHARPI_API int sharpi_gemm_nt(const void* A, int a_dtype, const void* W, int w_dtype, float* C,
                              const int* group_offsets, const int* a_rows, const int* out_rows, int M, int N,
                              int K, int E, int accumulate, const float* bias, const float* row_scale,
                              const int* scale_rows, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return SHARPI_OK;
    if (K <= 0 || E <= 0) return SHARPI_BAD_ARGUMENT;
    if (!group_offsets && E != 1) return SHARPI_BAD_ARGUMENT;
    GemmArgs g;
    g.A = A; g.W = W; g.C = C; g.group_offsets = group_offsets; g.a_rows = a_rows; g.out_rows = out_rows;
    g.M = M; g.N = N; g.K = K; g.E = E; g.accumulate = accumulate;
    g.bias = bias; g.row_scale = row_scale; g.scale_rows = scale_rows;
    long long m_tiles = (M + GB_M - 1) / GB_M + (group_offsets ? E : 0);
    long long n_tiles = (N + GB_N - 1) / GB_N;
    if (m_tiles > 65535 || n_tiles > 2147483647LL) return SHARPI_BAD_ARGUMENT;
    // rows of both operands start on 16 bytes: pieces of four k go straight to shared memory
    const bool aligned = a_dtype == SHARPI_F32 && w_dtype == SHARPI_F32 && K % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    // Few rows: the weights' bytes and the chains' length count.  Measured (us, few-row kernel / tiles): 1024 x 4096 at 4 rows
    // 9 / 154, at 32 rows 43 / 154; 5120 x 5120 at 16 rows 118 / 194, at 32 rows 232 / 194 (every pass of eight rows copies the
    // weights once more): hence 16 rows, and 32 where the tiles leave most SMs empty.
    if (aligned && M <= GF_MAX_ROWS && K <= GF_MAX_K && (long long)M * E <= 65535 && (M <= 16 || N <= 4096)) {
        if (M == 1) return launch_few<1>(g, stream);
        if (M == 2) return launch_few<2>(g, stream);
        if (M <= 4) return launch_few<4>(g, stream);
        return launch_few<8>(g, stream);
    }
    if (aligned) {
        // tiles of 128 rows read the weights half as often, tiles of 64 fill the GPU with fewer rows
        const long long wide = ((M + 127) / 128) * ((N + GT_N - 1) / GT_N);
        return wide >= 148 ? launch_tile<128>(g, stream) : launch_tile<64>(g, stream);
    }
    dim3 grid((unsigned)n_tiles, (unsigned)m_tiles);
    if (a_dtype == SHARPI_F32 && w_dtype == SHARPI_F32)
        gemm_nt_kernel<float, float><<<grid, 256, 0, stream>>>(g);
    else if (a_dtype == SHARPI_BF16 && w_dtype == SHARPI_BF16)
        gemm_nt_kernel<bf16, bf16><<<grid, 256, 0, stream>>>(g);
    else if (a_dtype == SHARPI_F32 && w_dtype == SHARPI_BF16)
        gemm_nt_kernel<float, bf16><<<grid, 256, 0, stream>>>(g);
    else if (a_dtype == SHARPI_BF16 && w_dtype == SHARPI_F32)
        gemm_nt_kernel<bf16, float><<<grid, 256, 0, stream>>>(g);
    else
        return SHARPI_BAD_ARGUMENT;
    SHARPI_CHECK_LAUNCH();
    return SHARPI_OK;
}
