// Plain matrix product C[M][N] = A[M][K] * W[N][K]^T on the CUDA cores.
//
// This is the true 32-bit path of every projection (float32 operands, FFMA
// accumulation, no tensor cores, no reduced-precision mode) and, with bfloat16
// operands, the plain twin the tensor-core kernels are tested against.  The
// reference keeps exact f32 FMA matvecs for the same purpose
// (crates/airun-cuda/kernels/matmul.cu:59-141, switch at
// crates/airun-core/src/runtime.rs:5344-5352).  The tile kernels form every
// output element as one sequential sum over k; the kernel for few float32 rows
// cuts it over the block in a fixed order.
#include "common.cuh"

#define TM 64
#define TN 64
#define TK 16
#define PAD 4

// Two more forms of the same tile loop.  BATCHED: blockIdx.z names one of several products of equal sizes whose
// operands lie `sa`, `sw`, `sc` elements apart (the heads of a per-head product over column slices of one buffer).
// GROUPED: the rows of A are cut into segments, segment e = rows seg[e] .. seg[e + 1] - 1 (device memory), and the
// rows of segment e are multiplied by the matrix W + e * sw; blockIdx.y counts the row tiles of all segments in
// turn, and a block beyond the last tile leaves at once, so one launch of a fixed shape serves any cut.
struct GemmExtra {
    long long sa, sw, sc;          // strides between the products of a batch; sw also between the matrices of segments
    const int32_t* seg;            // [n_seg + 1] row offsets of the segments (GROUPED)
    int n_seg;
};

template <typename TA, typename TW, typename TC, int FORM>      // FORM 0 plain, 1 batched, 2 grouped
__global__ __launch_bounds__(256) void gemm_simt_kernel(
    const TA* A, const TW* __restrict__ W, TC* __restrict__ C,
    int M, int N, int K, long long lda, long long ldw, long long ldc, GemmExtra ex) {
    pdl_trigger();
    pdl_wait();
    __shared__ __align__(16) float As[TK][TM + PAD];
    __shared__ __align__(16) float Ws[TK][TN + PAD];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    int m0 = blockIdx.y * TM;
    const int n0 = blockIdx.x * TN;
    if (FORM == 1) {
        A += (size_t)blockIdx.z * ex.sa;
        W += (size_t)blockIdx.z * ex.sw;
        C += (size_t)blockIdx.z * ex.sc;
    }
    if (FORM == 2) {
        int tile = blockIdx.y, e = 0, found = 0;
        for (; e < ex.n_seg; ++e) {
            const int lo = ex.seg[e], hi = ex.seg[e + 1];
            const int tiles = (hi - lo + TM - 1) / TM;
            if (tile < tiles) { m0 = lo + tile * TM; M = min(M, hi); found = 1; break; }
            tile -= tiles;
        }
        if (!found) return;
        W += (size_t)e * ex.sw;
    }
    const int lr = tid >> 2, lk = (tid & 3) * 4;

    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += TK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lk + j;
            float a = 0.0f, w = 0.0f;
            if (k < K) {
                if (m0 + lr < M) a = to_f32<TA>(A[(size_t)(m0 + lr) * lda + k]);
                if (n0 + lr < N) w = to_f32<TW>(W[(size_t)(n0 + lr) * ldw + k]);
            }
            As[lk + j][lr] = a;
            Ws[lk + j][lr] = w;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            const float4 a4 = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
            const float4 b4 = *reinterpret_cast<const float4*>(&Ws[k][tx * 4]);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w};
            const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) C[(size_t)m * ldc + n] = from_f32<TC>(acc[i][j]);
        }
    }
}

// ------------------------------------------------------------------ float32, 16-byte aligned rows
// The tile kernel above loads element by element and keeps one tile in flight; it stays for bfloat16 operands and for
// rows that are not 16-byte aligned.  Aligned float32 operands (every width in multiples of 4) take one of two kernels:
// few rows are bound by the bytes of W and go to gemv_f32_kernel, more rows are bound by the FMA pipe and go to
// gemm_f32_kernel.  The 39 products of three prompts of 171 to 257 tokens and two decoded tokens of each on a three-layer
// model of width 1,024 took 6,856 us in the tile kernel above and take 2,070 us here (twelve with 642 rows at 35 to 38
// TFLOP/s, about half of 128 FMA a clock and SM; 3 rows x [3072, 1024] 4.9 us, at 2.6 TB/s of weights).

// Sums of NV values over the warp's lanes by halving exchanges: every step a lane hands half of its values to its
// partner and keeps the sums of the other half; the last steps, with one value left, are plain exchanges.  Lane l ends
// with the sum of value index(l); for NV = 64 with two of them, v[0] and v[1], index(l) and index(l) + 1.
template <int NV> __device__ __forceinline__ int halving_sum(float (&v)[NV], int lane) {
    int idx = 0, n = NV;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < NV / 2; ++i) {
                if (i >= n) break;
                const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
            idx += up ? n : 0;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    return idx;
}

#define GV_WARPS 8
// MR rows x NC columns a block; the eight warps share K (a lane takes four neighbouring k of every 1024), so that even
// N = 1024 gives a block to every SM; the first weights are asked for before the kernel in front has finished.  The sums
// are formed in a fixed order (lanes by halving, then warps in turn).
template <int MR, int NC, int FORM>
__global__ __launch_bounds__(32 * GV_WARPS) void gemv_f32_kernel(
    const float* A, const float* __restrict__ W, float* __restrict__ C,
    int M, int N, int K, long long lda, long long ldw, long long ldc, GemmExtra ex) {
    pdl_trigger();
    __shared__ float red[GV_WARPS][MR * NC];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * NC;
    int lo = blockIdx.y * MR, hi = min(M, lo + MR);
    if (FORM == 1) {
        A += (size_t)blockIdx.z * ex.sa;
        W += (size_t)blockIdx.z * ex.sw;
        C += (size_t)blockIdx.z * ex.sc;
    }
    if (FORM == 2) W += (size_t)blockIdx.y * ex.sw;
    const float* wr[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) wr[c] = W + (size_t)min(n0 + c, N - 1) * ldw;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int k_first = (warp * 32 + lane) * 4;
    float4 w0[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) w0[c] = k_first < K ? __ldg(reinterpret_cast<const float4*>(wr[c] + k_first)) : zero;
    pdl_wait();
    if (FORM == 2) { lo = ex.seg[blockIdx.y]; hi = min(M, ex.seg[blockIdx.y + 1]); }
    for (int m0 = lo; m0 < hi; m0 += MR) {                     // more than once in a segment of more than MR rows only
        float acc[MR * NC];
#pragma unroll
        for (int i = 0; i < MR * NC; ++i) acc[i] = 0.0f;
        float4 w[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) w[c] = w0[c];
        for (int k = k_first; k < K; k += GV_WARPS * 128) {
            const int kn = k + GV_WARPS * 128;
            float4 nx[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) nx[c] = kn < K ? __ldg(reinterpret_cast<const float4*>(wr[c] + kn)) : zero;
#pragma unroll
            for (int r = 0; r < MR; ++r) {
                const float4 a = *reinterpret_cast<const float4*>(A + (size_t)min(m0 + r, hi - 1) * lda + k);
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    acc[r * NC + c] = fmaf(a.w, w[c].w, fmaf(a.z, w[c].z, fmaf(a.y, w[c].y, fmaf(a.x, w[c].x, acc[r * NC + c]))));
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) w[c] = nx[c];
        }
        const int idx = halving_sum<MR * NC>(acc, lane);
        constexpr int LEFT = MR * NC > 32 ? MR * NC / 32 : 1;  // sums a lane ends with
        constexpr int SAME = MR * NC < 32 ? 32 / (MR * NC) : 1;   // neighbouring lanes that end with the same one
        if (lane % SAME == 0) {
#pragma unroll
            for (int i = 0; i < LEFT; ++i) red[warp][idx + i] = acc[i];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < MR * NC; i += 32 * GV_WARPS) {
            float t = 0.0f;
#pragma unroll
            for (int q = 0; q < GV_WARPS; ++q) t += red[q][i];
            const int m = m0 + i / NC, n = n0 + i % NC;
            if (m < hi && n < N) C[(size_t)m * ldc + n] = t;
        }
        __syncthreads();
    }
}

// A tile of 64 x 64 by 256 threads in two groups of 128: every thread has 8 x 4 results, each as a packed pair of sums (over
// even and over odd k), and its group takes sixteen of the 32 k-values of a step, so that a few hundred rows still give
// every scheduler several warps.  Rows are staged as they lie in memory by asynchronous 16-byte copies, two steps ahead;
// a thread reads four k-values of a row at once and multiplies pairs of them with pairs, so nothing is transposed or
// packed on the way: 12 reads of shared memory (16 wavefronts a warp) for 64 packed multiply-adds of two clocks, and
// the FMA pipe is the bound.  The four partial sums of a result are added in a fixed order.
#define FT 64
#define FK 32
#define FS (FK + 4)               // floats of a staged row: eight neighbouring rows lie in different banks
#define F_STAGES 3
__device__ __forceinline__ void f32_cp16(float* smem, const float* gmem, bool on) {
    const int bytes = on ? 16 : 0;                             // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes) : "memory");
}
template <int FORM>
__global__ __launch_bounds__(256, 2) void gemm_f32_kernel(
    const float* A, const float* __restrict__ W, float* __restrict__ C,
    int M, int N, int K, long long lda, long long ldw, long long ldc, GemmExtra ex) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float f_tiles[];           // [stage][operand][64][FS]
    const int tid = threadIdx.x, grp = tid >> 7, l = tid & 127, tx = l & 15, ty = l >> 4;
    int m0 = blockIdx.y * FT;
    const int n0 = blockIdx.x * FT;
    if (FORM == 1) {
        A += (size_t)blockIdx.z * ex.sa;
        W += (size_t)blockIdx.z * ex.sw;
        C += (size_t)blockIdx.z * ex.sc;
    }
    if (FORM == 2) {
        int tile = blockIdx.y, e = 0, found = 0;
        for (; e < ex.n_seg; ++e) {
            const int lo = ex.seg[e], hi = ex.seg[e + 1];
            const int n = (hi - lo + FT - 1) / FT;
            if (tile < n) { m0 = lo + tile * FT; M = min(M, hi); found = 1; break; }
            tile -= n;
        }
        if (!found) return;
        W += (size_t)e * ex.sw;
    }
    const int lr = tid >> 3, lk = 4 * (tid & 7);               // this thread copies rows lr and lr + 32, k-values lk .. lk + 3
    const int steps = (K + FK - 1) / FK;
    auto stage = [&](int step) {
        if (step < steps) {
            float* dst = f_tiles + (step % F_STAGES) * (2 * FT * FS);
            const int k = step * FK + lk;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = lr + 32 * i;
                const bool a_on = k < K && m0 + row < M, w_on = k < K && n0 + row < N;
                f32_cp16(dst + row * FS + lk, a_on ? A + (size_t)(m0 + row) * lda + k : A, a_on);
                f32_cp16(dst + (FT + row) * FS + lk, w_on ? W + (size_t)(n0 + row) * ldw + k : W, w_on);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    stage(0);
    stage(1);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                       // the step has landed, and the one before it has been read
        stage(step + 2);
        const float* as = f_tiles + (step % F_STAGES) * (2 * FT * FS) + 16 * grp;
        const float* ws = as + FT * FS;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float4 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const float4*>(ws + (tx + 16 * j) * FS + 4 * q);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(as + (ty + 8 * i) * FS + 4 * q);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = __ffma2_rn(make_float2(a.x, a.y), make_float2(w[j].x, w[j].y), acc[i][j]);
                    acc[i][j] = __ffma2_rn(make_float2(a.z, a.w), make_float2(w[j].z, w[j].w), acc[i][j]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (grp == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) f_tiles[(i * 4 + j) * 128 + l] = acc[i][j].x + acc[i][j].y;
    }
    __syncthreads();
    if (grp == 1) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty + 8 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n < N) C[(size_t)m * ldc + n] = (acc[i][j].x + acc[i][j].y) + f_tiles[(i * 4 + j) * 128 + l];
        }
    }
}

template <int FORM, int MR>
static void launch_gemv(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                        int gy, int gz, const GemmExtra& ex, cudaStream_t stream) {
    // eight columns a block once that still gives every SM several blocks: the rows of A are read half as often
    if (N >= 4096)
        airun_launch(gemv_f32_kernel<MR, 8, FORM>, dim3(ceil_div_i(N, 8), gy, gz), dim3(32 * GV_WARPS), 0, stream, A, W, C, M, N, K, lda, ldw, ldc, ex);
    else
        airun_launch(gemv_f32_kernel<MR, 4, FORM>, dim3(ceil_div_i(N, 4), gy, gz), dim3(32 * GV_WARPS), 0, stream, A, W, C, M, N, K, lda, ldw, ldc, ex);
}

// True when the aligned float32 kernels took the product.  Up to 16 rows (an average of up to four a segment) the bytes
// of W are the bound; from there on a row group's further reading of W from the L2 cache costs more than the tiles.
template <int FORM>
static bool f32_product(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M, int N, int K, long long lda,
                        long long ldw, long long ldc, int batch, const GemmExtra& ex, cudaStream_t stream) {
    if (a_dtype != AIRUN_DT_F32 || w_dtype != AIRUN_DT_F32 || c_dtype != AIRUN_DT_F32) return false;
    if ((K | lda | ldw | ex.sa | ex.sw) & 3 || ((uintptr_t)A | (uintptr_t)W) & 15) return false;
    const float *a = (const float*)A, *w = (const float*)W;
    float* c = (float*)C;
    const int segs = FORM == 2 ? ex.n_seg : 1;
    if (FORM == 2 ? (M <= 4 * segs && segs <= 65535) : M <= 16) {
        const int rows = FORM == 2 ? ceil_div_i(M, segs) : M;
        const int mr = rows <= 1 ? 1 : rows <= 2 ? 2 : rows <= 4 ? 4 : 8;
        const int gy = FORM == 2 ? segs : ceil_div_i(M, mr), gz = FORM == 1 ? batch : 1;
        if (mr == 1) launch_gemv<FORM, 1>(a, w, c, M, N, K, lda, ldw, ldc, gy, gz, ex, stream);
        else if (mr == 2) launch_gemv<FORM, 2>(a, w, c, M, N, K, lda, ldw, ldc, gy, gz, ex, stream);
        else if (mr == 4) launch_gemv<FORM, 4>(a, w, c, M, N, K, lda, ldw, ldc, gy, gz, ex, stream);
        else launch_gemv<FORM, 8>(a, w, c, M, N, K, lda, ldw, ldc, gy, gz, ex, stream);
        return true;
    }
    const dim3 grid(ceil_div_i(N, FT), ceil_div_i(M, FT) + (FORM == 2 ? segs : 0), FORM == 1 ? batch : 1);
    if (grid.y > 65535) return false;
    constexpr int SMEM = F_STAGES * 2 * FT * FS * (int)sizeof(float);
    static unsigned long long configured = 0;
    if (first_on_device(configured) &&
        cudaFuncSetAttribute(gemm_f32_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) {
        cudaGetLastError();
        configured = 0;
        return false;
    }
    airun_launch(gemm_f32_kernel<FORM>, grid, dim3(256), SMEM, stream, a, w, c, M, N, K, lda, ldw, ldc, ex);
    return true;
}

// dtypes: a_dtype == w_dtype in {f32, bf16}; c_dtype in {f32, bf16}.
AIRUN_EXPORT int airun_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype,
                                 void* C, int c_dtype, int M, int N, int K,
                                 long long lda, long long ldw, long long ldc, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N) return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    dim3 grid(ceil_div_i(N, TN), ceil_div_i(M, TM));
    if (grid.y > 65535) return AIRUN_ERR_ARG;
    GemmExtra ex = {};
    if (f32_product<0>(A, a_dtype, W, w_dtype, C, c_dtype, M, N, K, lda, ldw, ldc, 1, ex, stream)) return airun_launch_status();
#define LAUNCH(TA, TW, TC) \
    airun_launch(gemm_simt_kernel<TA, TW, TC, 0>, dim3(grid), dim3(256), 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc, ex)
    if (a_dtype == AIRUN_DT_F32 && w_dtype == AIRUN_DT_F32 && c_dtype == AIRUN_DT_F32) LAUNCH(float, float, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_F32) LAUNCH(__nv_bfloat16, __nv_bfloat16, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
    else return AIRUN_ERR_UNSUPPORTED;
#undef LAUNCH
    return airun_launch_status();
}

// `batch` products of equal sizes, product b on A + b*sa, W + b*sw, C + b*sc (elements).
AIRUN_EXPORT int airun_gemm_simt_batched(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype,
                                         int M, int N, int K, long long lda, long long ldw, long long ldc, int batch,
                                         long long sa, long long sw, long long sc, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N || batch <= 0 || batch > 65535) return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    dim3 grid(ceil_div_i(N, TN), ceil_div_i(M, TM), batch);
    if (grid.y > 65535) return AIRUN_ERR_ARG;
    GemmExtra ex = {};
    ex.sa = sa; ex.sw = sw; ex.sc = sc;
    if (f32_product<1>(A, a_dtype, W, w_dtype, C, c_dtype, M, N, K, lda, ldw, ldc, batch, ex, stream)) return airun_launch_status();
#define LAUNCH(TA, TW, TC) \
    airun_launch(gemm_simt_kernel<TA, TW, TC, 1>, dim3(grid), dim3(256), 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc, ex)
    if (a_dtype == AIRUN_DT_F32 && w_dtype == AIRUN_DT_F32 && c_dtype == AIRUN_DT_F32) LAUNCH(float, float, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_F32) LAUNCH(__nv_bfloat16, __nv_bfloat16, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
    else return AIRUN_ERR_UNSUPPORTED;
#undef LAUNCH
    return airun_launch_status();
}

// The rows of A in `n_seg` segments (`seg`: int32 [n_seg + 1] on the device, rising, seg[n_seg] <= M); rows of
// segment e times W + e*sw.  The launch covers ceil(M / TM) + n_seg row tiles, which is enough for every cut.
AIRUN_EXPORT int airun_gemm_simt_grouped(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype,
                                         int M, int N, int K, long long lda, long long ldw, long long ldc,
                                         const int32_t* seg, int n_seg, long long sw, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N || !seg || n_seg <= 0) return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    dim3 grid(ceil_div_i(N, TN), ceil_div_i(M, TM) + n_seg);
    if (grid.y > 65535) return AIRUN_ERR_ARG;
    GemmExtra ex = {};
    ex.sw = sw; ex.seg = seg; ex.n_seg = n_seg;
    if (f32_product<2>(A, a_dtype, W, w_dtype, C, c_dtype, M, N, K, lda, ldw, ldc, 1, ex, stream)) return airun_launch_status();
#define LAUNCH(TA, TW, TC) \
    airun_launch(gemm_simt_kernel<TA, TW, TC, 2>, dim3(grid), dim3(256), 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc, ex)
    if (a_dtype == AIRUN_DT_F32 && w_dtype == AIRUN_DT_F32 && c_dtype == AIRUN_DT_F32) LAUNCH(float, float, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_F32) LAUNCH(__nv_bfloat16, __nv_bfloat16, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
    else return AIRUN_ERR_UNSUPPORTED;
#undef LAUNCH
    return airun_launch_status();
}
