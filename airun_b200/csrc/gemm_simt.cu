// Plain matrix product C[M][N] = A[M][K] * W[N][K]^T.
//
// This is the true 32-bit path of every projection (float32 operands, no operand rounded, no reduced-precision mode): FFMA
// kernels on the CUDA cores, and for many long rows the tensor cores with each operand in three parts that keep all its bits.
// With bfloat16 operands it is the plain twin the tensor-core kernels are tested against.  The
// reference keeps exact f32 FMA matvecs for the same purpose
// (crates/airun-cuda/kernels/matmul.cu:59-141, switch at
// crates/airun-core/src/runtime.rs:5344-5352).  The tile kernels on the CUDA cores form every
// output element as one sequential sum over k or as a few in a fixed order; the others cut it over the block, steps and slices in a fixed order.
#include "tcgen05.cuh"

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

// ------------------------------------------------------------------ float32 on the tensor cores, without rounding an operand
// More than a few rows of float32 products are bound by the FMA pipe, so they go to the tensor cores with every operand
// cut into three bfloat16 parts whose sum it is: its 8 leading bits (rounded), 8 of what is left (rounded) and the rest, which is the whole
// significand of 24 bits down to 2^-133 (the split of S. Markidis et al., IPDPS Workshops 2018, in bfloat16 and three parts: G. Henry, P. T. P. Tang and
// A. Heinecke, ARITH 2019).  Of the nine products of parts eight are formed; x3 w3, below 2^-35 of x w, is left out.
// The tensor cores add up in float32 but cut off where float32 rounds.  So the leading product x1 w1, whose 16 bits leave room for a sum of many, has a sum
// of its own, over the 64 k-values of a step, and the seven small ones, 2^-8 of it and less, have another over X_LOW_STEPS steps: its cuts, 28 a step, are 2^-8 of
// those of one sum.  Both are added up in registers, rounded; a sum of one product is the rounded product, as an FMA has it.
// Error against 64 bits (2-norm, in 1e-7), this and the FMA kernel, 300 rows: K = 1,024 dense 0.9, 2.9 (operands of one sign 0.9, 1.3); 10 % of x other than zero
// 0.6, 1.0 (0.5, 0.6); 1 % 0.5, 0.5 (0.4, 0.4); one 0.25, 0.25.  K = 4,096 dense 1.8, 5.7 (1.6, 2.5); 10 % 1.4, 1.9 (1.3, 0.8); 1 % 0.9, 0.7 (0.7, 0.5): of many steps
// with a few terms of one sign each, adding up the steps is the larger part.  Six products and one sum had 0.55 for one product.
//
// What the parts cannot hold is found and formed by multiply-adds (f32_plain_results): results that are not finite (an infinite operand
// has no parts, and small products can overflow with the other sign), results below 2^-100, whose small products end at 2^-149, and small results of
// rows and columns with an operand below 2^-110, whose last bits end at 2^-133.
//
// A tile is 128 weight rows by `bn` rows of A (16 .. 128), its K range cut into `ks` slices that run as one cluster and are added up in order
// through distributed shared memory.
//   warps 0-7  : read the sums from tensor memory (a quadrant of lanes each, every other 16 columns) and add them up; they store the tile;
//   warps 8-15 : cut the 64 k-values of a step of every row of both operands.  The parts of W go to tensor memory, those of A to shared memory
//                (128-byte swizzle): with both there, what the products, the cutting and the loads move through shared memory is the bound (390 KB a
//                step of 128 x 112, 3,300 clocks for 1,540 of six products).  They load nothing themselves: their fence would wait for loads under way;
//   warp 16    : issues the 32 tcgen05.mma of a step (in a warp that adds up, no product would run while it does), the small products first: meanwhile
//                the leading sum of the step before is read;
//   warp 17    : issues the TMA loads, two steps ahead.
#define XT 128                    // weight rows of a tile
#define XB 128                    // most rows of A
#define XK 64                     // k-values of a step
#define X_STAGES 2                // steps of parts
#define X_RING 2                  // steps of operands on their way to the threads that cut them
#define X_PRODUCTS 8              // of parts
#define X_SUM_WARPS 8
#define X_CUT_WARPS 8
#define X_THREADS (32 * (X_SUM_WARPS + X_CUT_WARPS + 2))   // 18 warps: 96 registers a thread
#define X_PART (XB * XK * 2)      // bytes of one part of A
#define X_WCOLS (XK / 2)          // columns of tensor memory of one part of W
#define X_WAT (2 * XB)            // their place, behind the sums of the leading and of the small products
static_assert(X_WAT + 3 * X_STAGES * X_WCOLS <= 512, "");
#define X_LOW_STEPS 4             // steps that the small products are added up over
#define X_STAGE (3 * X_PART)
#define X_SUM_SPACE (XT * XB * 4) // the slices' sums take the place of the stages and of the ring
#define X_RING_STEP ((XT + XB) * XK * 4)
#define X_SMEM (X_STAGES * X_STAGE + X_RING * X_RING_STEP + 1024)
static_assert(X_SUM_SPACE <= X_STAGES * X_STAGE + X_RING * X_RING_STEP && X_STAGE % 1024 == 0, "");

// The product with the rows of A (here W) in tensor memory: 8 columns of 32 bits hold 16 k-values of a lane's row.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint2 (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0].x), "r"(v[0].y), "r"(v[1].x),
                 "r"(v[1].y), "r"(v[2].x), "r"(v[2].y), "r"(v[3].x), "r"(v[3].y) : "memory");
}

// One float4's three parts, packed to bfloat16 (8 bytes each).
__device__ __forceinline__ void f32_parts(const float4& v, uint2 (&part)[3]) {
    const float2 minus = make_float2(-1.0f, -1.0f);
    uint32_t b[3][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {                              // packed: what is left is exact, as a multiply-add too
        float2 r = i == 0 ? make_float2(v.x, v.y) : make_float2(v.z, v.w);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(r.x, r.y);
            b[j][i] = *reinterpret_cast<const uint32_t*>(&h);
            if (j < 2) r = __ffma2_rn(make_float2(__uint_as_float(b[j][i] << 16), __uint_as_float(b[j][i] & 0xffff0000u)), minus, r);
        }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) part[j] = make_uint2(b[j][0], b[j][1]);
}
// The smallest of 2 |x| - 1 as whole numbers, where zero is the largest: below X_SMALL for values other than zero below 2^-110.
#define X_SMALL (2u * 0x08800000u - 1u)
__device__ __forceinline__ uint32_t f32_least(uint32_t least, const float4& v) {
    const uint32_t a = 2u * __float_as_uint(v.x) - 1u, b = 2u * __float_as_uint(v.y) - 1u, c = 2u * __float_as_uint(v.z) - 1u, d = 2u * __float_as_uint(v.w) - 1u;
    return min(min(least, min(a, b)), min(c, d));
}
// Not a number for a result that the parts may not hold (see above), else zero (added up, one check answers for many results).
__device__ __forceinline__ float f32_doubt(float v) { return fabsf(v) < 7.888609e-31f && v != 0.0f ? __int_as_float(0x7fffffff) : v * 0.0f; }

// The results of a tile that are in doubt, and the small ones (below 2^-20, whose terms' last bits can count) of marked rows and columns, a warp each: columns
// first, first + step, .. of the tile.  Columns whose row of A holds a NaN are NaN already.  (Rows of padding hold whatever was in their place, so this must not be
// slow: 642 x [3072, 1024], 29 us, with 64 rows of one infinite value 452 us (6,671 with a thread each), of one NaN 39, of one value below 2^-110 38, of nothing else 452.)
__device__ __noinline__ void f32_plain_results(const float* A, const float* W, float* C, int K, long long lda, long long ldw, long long ldc, int m0,
                                               int cols, int n0, int rows, const uint32_t* marks, int first, int step) {
    __shared__ uint32_t nan_cols[4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    if (threadIdx.x < 4) nan_cols[threadIdx.x] = 0;
    __syncthreads();
    if (marks[8]) {
        for (int col = warp; col < cols; col += warps) {
            if (col % step != first) continue;
            const float4* a = reinterpret_cast<const float4*>(A + (size_t)(m0 + col) * lda);
            bool nan = false;
            for (int k = lane; 4 * k < K; k += 32) { const float4 x = a[k]; nan |= isnan(x.x) | isnan(x.y) | isnan(x.z) | isnan(x.w); }
            if (__any_sync(0xffffffffu, nan) && lane == 0) atomicOr(&nan_cols[col >> 5], 1u << (col & 31));
        }
    }
    __syncthreads();
    for (int base = 32 * warp; base < cols * rows; base += 32 * warps) {
        const int i = base + lane, col = i / rows, r = i % rows;
        bool form = false;
        if (i < cols * rows && col % step == first && !((nan_cols[col >> 5] >> (col & 31)) & 1u)) {
            const float v = __ldcg(C + (size_t)(m0 + col) * ldc + n0 + r), doubt = f32_doubt(v);
            form = doubt != doubt || (fabsf(v) < 9.5367432e-7f && (((marks[r >> 5] >> (r & 31)) | (marks[4 + (col >> 5)] >> (col & 31))) & 1u));
        }
        for (uint32_t left = __ballot_sync(0xffffffffu, form); left; left &= left - 1) {
            const int j = base + __ffs(left) - 1, jc = j / rows, jr = j % rows;
            const float4 *a = reinterpret_cast<const float4*>(A + (size_t)(m0 + jc) * lda), *w = reinterpret_cast<const float4*>(W + (size_t)(n0 + jr) * ldw);
            float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
            for (int k = lane; 4 * k < K; k += 32) {           // (rows of a multiple of four values, aligned)
                const float4 x = a[k], y = w[k];
                s.x = fmaf(x.x, y.x, s.x); s.y = fmaf(x.y, y.y, s.y); s.z = fmaf(x.z, y.z, s.z); s.w = fmaf(x.w, y.w, s.w);
            }
            float v = (s.x + s.y) + (s.z + s.w);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) C[(size_t)(m0 + jc) * ldc + n0 + jr] = v;
        }
    }
}

template <int FORM>                                            // 0 plain, 2 grouped
__global__ __launch_bounds__(X_THREADS, 1) void gemm_f32_parts_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* A, const float* __restrict__ W,
    float* __restrict__ C, int M, int N, int K, long long lda, long long ldw, long long ldc, GemmExtra ex, int bn, int ks, int* err) {
    pdl_trigger();
    extern __shared__ uint8_t x_raw[];
    uint8_t* tiles = (uint8_t*)(((uintptr_t)x_raw + 1023) & ~(uintptr_t)1023);
    // full, empty of the stages of parts; full, empty of the leading sum and of the other; landed, read of the ring
    __shared__ __align__(8) uint64_t bars[2 * X_STAGES + 4 + 2 * X_RING];
    __shared__ uint32_t tmem_slot, marks[9], all_marks[9];         // bit r of 0-3: weight row r has an operand that is too small for its parts; 4-7: row of A; 8: a result is in doubt
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int slice = blockIdx.z, n0 = blockIdx.x * XT;
    int m0 = blockIdx.y * bn, m_end = M, set_w = 0;
    if (FORM == 2) {
        pdl_wait();                                            // the segments are the kernel's in front
        int tile = blockIdx.y, e = 0, found = 0;
        for (; e < ex.n_seg; ++e) {
            const int lo = ex.seg[e], hi = ex.seg[e + 1];
            const int n = (hi - lo + bn - 1) / bn;
            if (tile < n) { m0 = lo + tile * bn; m_end = min(M, hi); found = 1; break; }
            tile -= n;
        }
        if (!found) return;
        W += (size_t)e * ex.sw;
        set_w = e;
    }
    const int steps_all = (K + XK - 1) / XK, per = (steps_all + ks - 1) / ks;
    const int step0 = min(slice * per, steps_all), steps = min(step0 + per, steps_all) - step0;
    const uint32_t full = smem_u32(bars), empty = full + 8 * X_STAGES, sfull = empty + 8 * X_STAGES, sempty = sfull + 8, lfull = sempty + 8, lempty = lfull + 8, landed = lempty + 8, taken = landed + 8 * X_RING;
    if (threadIdx.x == 0) {
        for (int s = 0; s < X_STAGES; ++s) { mbar_init(full + 8 * s, X_CUT_WARPS); mbar_init(empty + 8 * s, 1); }
        for (uint32_t b = sfull; b <= lfull; b += 16) { mbar_init(b, 1); mbar_init(b + 8, X_SUM_WARPS); }
        for (int r = 0; r < X_RING; ++r) { mbar_init(landed + 8 * r, 1); mbar_init(taken + 8 * r, X_CUT_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x < 9) marks[threadIdx.x] = all_marks[threadIdx.x] = 0;
    if (warp == X_SUM_WARPS) tmem_alloc(smem_u32(&tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    const int cols = min(bn, m_end - m0);
    float* sums = reinterpret_cast<float*>(tiles);             // of this slice, [column][128], once the products are done
    if (warp < X_SUM_WARPS) {
        const int quad = warp & 3, half = warp >> 2;
        float2 acc[XB / 4];                                    // columns 16 (2 j + half) + 2 i and the next at [8 j + i]
#pragma unroll
        for (int i = 0; i < XB / 4; ++i) acc[i] = make_float2(0.0f, 0.0f);
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        auto add = [&](uint32_t from, uint32_t read) {
#pragma unroll
            for (int j = 0; j < XB / 32; ++j) {
                const int c = 16 * (2 * j + half);
                if (c >= bn) break;
                uint32_t r[16];
                tmem_ld_async(from + c, r);
                tmem_wait(r);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[8 * j + i] = __fadd2_rn(acc[8 * j + i], make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(read) : "memory");
        };
        for (int it = 0, group = 0; it < steps; ++it) {
            if (!mbar_wait(sfull, it & 1)) { atomicOr(err, AIRUN_DEV_TIMEOUT); break; }
            if (it % X_LOW_STEPS == X_LOW_STEPS - 1 || it + 1 == steps) {      // (first, as the next step's products begin with it)
                if (!mbar_wait(lfull, group & 1)) { atomicOr(err, AIRUN_DEV_TIMEOUT); break; }
                ++group;
                tc_fence_after();
                __syncwarp();
                add(lanes + XB, lempty);
            }
            tc_fence_after();
            __syncwarp();
            add(lanes, sempty);
        }
        // the last step's products are done, so the stages may be written over
        const int r = quad * 32 + lane;
        if (ks > 1) {
#pragma unroll
            for (int j = 0; j < XB / 32; ++j) {
                const int c0 = 16 * (2 * j + half);
                if (c0 >= bn) break;
#pragma unroll
                for (int i = 0; i < 16; ++i) sums[(c0 + i) * XT + r] = i & 1 ? acc[8 * j + i / 2].y : acc[8 * j + i / 2].x;
            }
        } else if (n0 + r < N) {
            float* c = C + (size_t)(m0 + 16 * half) * ldc + n0 + r;
            float doubt = 0.0f;
#pragma unroll
            for (int j = 0; j < XB / 32; ++j, c += 32 * ldc) {
                const int n = cols - 16 * (2 * j + half);
                float* o = c;
#pragma unroll
                for (int i = 0; i < 16; ++i, o += ldc) {
                    const float v = i & 1 ? acc[8 * j + i / 2].y : acc[8 * j + i / 2].x;
                    if (i < n) { *o = v; doubt += f32_doubt(v); }
                }
            }
            if (doubt != doubt) atomicOr(&marks[8], 1u);
        }
    } else if (warp < X_SUM_WARPS + X_CUT_WARPS) {
        // W: this thread's row is lane `lane` of its quadrant, 32 of the step's k-values.  A: rows row + 32 i, k-values 4 q .. 4 q + 3 and 32 more on.
        // The ring holds boxes of 32 k-values; 16 bytes j of a row lie at place j ^ (row % 8) (the loads' 128-byte swizzle).
        const int t = threadIdx.x - 32 * X_SUM_WARPS, quad = warp & 3, half = t >> 7;
        const int row = t >> 3, q = t & 7;
        constexpr int RP = X_CUT_WARPS * 4;                    // 32: rows of a pass over A, four passes
        static_assert(RP == 32 && XT == 128 && XB == 128 && XK == 64, "two threads a row of W, four passes over A");
        uint32_t least_w = ~0u, least_a[4] = {~0u, ~0u, ~0u, ~0u};
        const uint32_t w_at = half * (XT * 128) + (quad * 32 + lane) * 128, a_at = 2 * XT * 128 + row * 128 + ((q ^ (row & 7)) << 4);
        for (int it = 0; it < steps; ++it) {
            const int s = it % X_STAGES, g = it % X_RING;
            if (!mbar_wait(landed + 8 * g, (it / X_RING) & 1) || !mbar_wait(empty + 8 * s, ((it / X_STAGES) & 1) ^ 1)) {
                atomicOr(err, AIRUN_DEV_TIMEOUT);
                break;
            }
            tc_fence_after();
            __syncwarp();
            const uint8_t* from = tiles + X_STAGES * X_STAGE + g * X_RING_STEP;
            uint8_t* to = tiles + s * X_STAGE + row * (XK * 2) + ((q & 1) << 3);
            // four values at a time, read, cut and stored: their chains of dependent instructions run side by side
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4 v[4];
                uint2 part[4][3];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4*>(from + w_at + (((4 * h + i) ^ (lane & 7)) << 4));
#pragma unroll
                for (int i = 0; i < 4; ++i) { f32_parts(v[i], part[i]); least_w = f32_least(least_w, v[i]); }
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const uint2 p[4] = {part[0][j], part[1][j], part[2][j], part[3][j]};
                    tmem_st8(tmem + ((uint32_t)(quad * 32) << 16) + X_WAT + (3 * s + j) * X_WCOLS + 16 * half + 8 * h, p);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4 v[4];
                uint2 part[4][3];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4*>(from + a_at + h * (XB * 128) + RP * i * 128);
#pragma unroll
                for (int i = 0; i < 4; ++i) { f32_parts(v[i], part[i]); least_a[i] = f32_least(least_a[i], v[i]); }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (row + RP * i >= bn) continue;
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        *reinterpret_cast<uint2*>(to + j * X_PART + RP * i * (XK * 2) + (((4 * h + (q >> 1)) ^ (row & 7)) << 4)) = part[i][j];
                }
            }
            __syncwarp();
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full + 8 * s) : "memory");
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(taken + 8 * g) : "memory");
            }
        }
        if (least_w < X_SMALL) atomicOr(&marks[quad], 1u << lane);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (row + RP * i < cols && least_a[i] < X_SMALL) atomicOr(&marks[4 + i], 1u << row);
    } else if (warp == X_SUM_WARPS + X_CUT_WARPS) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(XT >> 4) << 24);
        for (int it = 0; it < steps; ++it) {
            const int s = it % X_STAGES, group = it / X_LOW_STEPS;
            const bool first = it % X_LOW_STEPS == 0, last = it % X_LOW_STEPS == X_LOW_STEPS - 1 || it + 1 == steps;
            if ((first && !mbar_wait_warp(lempty, (group & 1) ^ 1)) || !mbar_wait_warp(full + 8 * s, (it / X_STAGES) & 1)) {
                atomicOr(err, AIRUN_DEV_TIMEOUT);
                break;
            }
            tc_fence_after();
            const uint32_t base = smem_u32(tiles) + s * X_STAGE;
            constexpr int WP[X_PRODUCTS] = {2, 1, 2, 0, 1, 1, 0, 0}, AP[X_PRODUCTS] = {1, 2, 0, 2, 1, 0, 1, 0};     // the smallest products first, the leading one last
            auto product = [&](int j, uint32_t sum, bool fresh) {
                const uint32_t tw = tmem + X_WAT + (3 * s + WP[j]) * X_WCOLS;
                const uint64_t da = smem_desc_sw128(base + AP[j] * X_PART);
#pragma unroll
                for (int k = 0; k < XK / 16; ++k) umma_bf16_ts(sum, tw + 8 * k, da + (uint64_t)(k * 2), idesc, fresh && k == 0 ? 0u : 1u);
            };
            if (elect_one()) {
#pragma unroll
                for (int j = 0; j < X_PRODUCTS - 1; ++j) product(j, tmem + XB, first && j == 0);
            }
            __syncwarp();
            if (!mbar_wait_warp(sempty, (it & 1) ^ 1)) { atomicOr(err, AIRUN_DEV_TIMEOUT); break; }
            tc_fence_after();
            if (elect_one()) {
                product(X_PRODUCTS - 1, tmem, true);
                umma_commit(empty + 8 * s);
                umma_commit(sfull);
                if (last) umma_commit(lfull);
            }
            __syncwarp();
        }
    } else {
        const uint32_t ring = smem_u32(tiles) + X_STAGES * X_STAGE;
        auto ask = [&](int it, bool w, bool a) {
            const uint32_t to = ring + (it % X_RING) * X_RING_STEP, bar = landed + 8 * (it % X_RING);
            const int k = (step0 + it) * XK;
            if (elect_one()) {
                if (w) {
                    mbar_expect_tx(bar, (XT + bn) * XK * 4);
                    tma_load_3d(to, &map_w, bar, k, n0, set_w);
                    tma_load_3d(to + XT * 128, &map_w, bar, k + 32, n0, set_w);
                }
                if (a) {
                    tma_load_3d(to + 2 * XT * 128, &map_a, bar, k, m0, 0);
                    tma_load_3d(to + (2 * XT + XB) * 128, &map_a, bar, k + 32, m0, 0);
                }
            }
            __syncwarp();
        };
        const int first = min(steps, X_RING);
        for (int it = 0; it < first; ++it) ask(it, true, false);
        if (FORM != 2) pdl_wait();
        for (int it = 0; it < first; ++it) ask(it, false, true);
        for (int it = X_RING; it < steps; ++it) {
            if (!mbar_wait_warp(taken + 8 * (it % X_RING), ((it / X_RING) & 1) ^ 1)) { atomicOr(err, AIRUN_DEV_TIMEOUT); break; }
            ask(it, true, true);
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();                                           // every step has been added up: no product is under way any more
    if (warp == X_SUM_WARPS) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (ks == 1) {
        uint32_t any = 0;
        for (int i = 0; i < 9; ++i) any |= marks[i];
        if (any) f32_plain_results(A, W, C, K, lda, ldw, ldc, m0, cols, n0, min(XT, N - n0), marks, 0, 1);
        return;
    }
    // the slices of the tile are added up in order, every CTA taking every ks-th column
    cluster_sync_all();
    {
        const int r = threadIdx.x & (XT - 1);
        if (n0 + r < N) {
            for (int col = slice + ks * (threadIdx.x / XT); col < cols && threadIdx.x < 4 * XT; col += ks * 4) {
                const uint32_t mine = smem_u32(sums + col * XT + r);
                float v[8];                                    // all slices are asked for before one is added
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = q < ks ? ld_cluster_f32(map_to_cta(mine, q)) : 0.0f;
                float t = v[0];
#pragma unroll
                for (int q = 1; q < 8; ++q) if (q < ks) t += v[q];
                C[(size_t)(m0 + col) * ldc + n0 + r] = t;
                const float doubt = f32_doubt(t);
                if (doubt != doubt) all_marks[8] = 1;
            }
        }
        if (threadIdx.x < 8) {                                 // the rows noted by all slices
            uint32_t m = 0;
            for (int q = 0; q < ks; ++q) m |= __float_as_uint(ld_cluster_f32(map_to_cta(smem_u32(marks + threadIdx.x), q)));
            all_marks[threadIdx.x] = m;
        }
        __syncthreads();
        uint32_t any = 0;
        for (int i = 0; i < 9; ++i) any |= all_marks[i];
        if (any) f32_plain_results(A, W, C, K, lda, ldw, ldc, m0, cols, n0, min(XT, N - n0), all_marks, slice, ks);
    }
    __syncwarp();
    cluster_sync_all();                                        // nobody leaves while a peer may still read its memory
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

// How many clusters of `ks` CTAs the current device, `dev`, holds at once, one CTA an SM.
static int f32_clusters(int ks, int dev) {
    static int known[64][9];
    int n = 0;
    if (ks < 2 || ks > 8 || dev < 0 || dev >= 64) return 0;
    if ((n = __atomic_load_n(&known[dev][ks], __ATOMIC_RELAXED)) != 0) return n > 0 ? n : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, ks);
    cfg.blockDim = dim3(X_THREADS);
    cfg.dynamicSmemBytes = X_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = ks;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(gemm_f32_parts_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, X_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_f32_parts_kernel<0>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    __atomic_store_n(&known[dev][ks], n > 0 ? n : -1, __ATOMIC_RELAXED);
    return n;
}

// Rows of A in a tile and K slices of the products on the tensor cores, by the time they take (B200, us): a step of 64 k-values 1.13, 0.0006 a row and from 80
// rows on, where the products are the bound, 0.0056 more; bringing the slices together 2 to 7, the more the larger the share of the tile's columns that a CTA
// adds up.  64 rows x [1024, 1024] in 1, 2, 4 and 8 slices 21.8, 15.9, 10.6, 8.7; 642 x [1024, 2048] as 112 tiles of 48 rows 40.8, as 56 of 96 rows in two slices
// 30.0; 642 x [3072, 1024] in tiles of 64, 96, 112 and 128 rows 46.1, 49.8, 28.6, 30.0; 257 x [4096, 4096] in tiles of 64, 80, 96 and 128 rows 153, 80, 88, 103.
// The choice for the sizes of a model's products is kept, by thread (2 us a call otherwise, which a step that is not replayed from a graph would wait for).
struct F32Plan { int bn, ks; };
static F32Plan f32_plan(long long rows, long long sets, int N, int K) {
    struct Kept { long long rows, sets; int N, K, dev; F32Plan plan; };
    static thread_local Kept table[64];                        // rows 0: empty
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); dev = -1; }
    Kept& kept = table[((unsigned)rows * 31u + (unsigned)N * 7u + (unsigned)K / 4u + (unsigned)sets) % 64u];
    if (kept.rows == rows && kept.sets == sets && kept.N == N && kept.K == K && kept.dev == dev) return kept.plan;
    const int sms = airun_sm_count(), steps = ceil_div_i(K, XK);
    const long long nt = (N + XT - 1) / XT * sets;
    F32Plan best = {XB, 1};
    double best_us = 1e30;
    for (int bn = 16; bn <= XB; bn += 16) {
        const long long tiles = nt * ((rows + bn - 1) / bn);
        for (int ks = 1; ks <= 8 && (ks == 1 || 2 * ks <= steps); ++ks) {
            const int per = (steps + ks - 1) / ks;
            if ((steps + per - 1) / per != ks || (ks > 1 && tiles > f32_clusters(ks, dev))) continue;   // an empty slice, or not all resident
            const double step = 1.13 + 0.0006 * bn + 0.0056 * (bn > 80 ? bn - 80 : 0), merge = ks > 1 ? 1.2 + bn * (0.015 + 0.06 / ks) : 0.0;
            const double us = (double)((tiles * ks + sms - 1) / sms) * per * step + merge;
            if (us < best_us) { best_us = us; best = {bn, ks}; }
        }
    }
    kept = {rows, sets, N, K, dev, best};
    return best;
}

// Fewest k-values of a product on the tensor cores.  Error of the FMA kernel against 64 bits (2-norm), K = 128, 512, 1024, 2048, 8192: operands of either
// sign 1.1e-7, 2.1e-7, 2.9e-7, 4.1e-7, 8.1e-7, of one sign 0.5e-7, 0.85e-7, 1.3e-7, 1.8e-7, 3.5e-7.  The parts have 0.9e-7 to 1.1e-7 at 1,024 of either, which the
// cuts within a step make up, so that below 1,024 they would be the less exact ones for one sign.
#define X_MIN_K 1024
// A tensor map of `sets` row-major float32 matrices [rows][K], rows `ld` and matrices `set` elements apart, boxes of box_rows x 32.
static bool f32_map(CUtensorMap* out, const float* ptr, long long K, long long rows, long long sets, long long ld, long long set, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)sets};
    cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)(sets > 1 ? set : ld) * 4};
    cuuint32_t box[3] = {32, (cuuint32_t)box_rows, 1}, estr[3] = {1, 1, 1};
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// True when the aligned float32 kernels took the product.  Up to 16 rows (an average of up to four a segment) the bytes
// of W are the bound; from there on a row group's further reading of W from the L2 cache costs more than the tiles.
// Long ones of those go to the tensor cores where the caller gives the error word that their bounded waits need, the others to the FMA pipe.
template <int FORM>
static bool f32_product(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M, int N, int K, long long lda,
                        long long ldw, long long ldc, int batch, const GemmExtra& ex, int* err, cudaStream_t stream) {
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
    static unsigned long long configured = 0;
    [[maybe_unused]] static unsigned long long configured_x = 0;
    if constexpr (FORM != 1) {
        if (err && K >= X_MIN_K) {
            const F32Plan plan = f32_plan(FORM == 2 ? ceil_div_i(M, segs) : M, segs, N, K);
            const long long gy = (M + plan.bn - 1) / plan.bn + (FORM == 2 ? segs : 0);
            CUtensorMap mw, ma;
            bool ready = gy <= 65535 && f32_map(&mw, w, K, N, segs, ldw, ex.sw, XT) && f32_map(&ma, a, K, M, 1, lda, 0, plan.bn);
            if (ready && first_on_device(configured_x) &&
                cudaFuncSetAttribute(gemm_f32_parts_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, X_SMEM) != cudaSuccess) {
                cudaGetLastError();
                configured_x = 0;
                ready = false;
            }
            if (ready) {
                const dim3 grid(ceil_div_i(N, XT), (unsigned)gy, (unsigned)plan.ks);
                if (plan.ks > 1)
                    airun_launch_cluster(gemm_f32_parts_kernel<FORM>, grid, dim3(X_THREADS), X_SMEM, stream, (unsigned)plan.ks, mw, ma, a, w, c, M, N,
                                         K, lda, ldw, ldc, ex, plan.bn, plan.ks, err);
                else
                    airun_launch(gemm_f32_parts_kernel<FORM>, grid, dim3(X_THREADS), X_SMEM, stream, mw, ma, a, w, c, M, N, K, lda, ldw, ldc, ex,
                                 plan.bn, 1, err);
                return true;
            }
        }
    }
    const dim3 grid(ceil_div_i(N, FT), ceil_div_i(M, FT) + (FORM == 2 ? segs : 0), FORM == 1 ? batch : 1);
    if (grid.y > 65535) return false;
    constexpr int SMEM = F_STAGES * 2 * FT * FS * (int)sizeof(float);
    if (first_on_device(configured) &&
        cudaFuncSetAttribute(gemm_f32_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) {
        cudaGetLastError();
        configured = 0;
        return false;
    }
    airun_launch(gemm_f32_kernel<FORM>, grid, dim3(256), SMEM, stream, a, w, c, M, N, K, lda, ldw, ldc, ex);
    return true;
}

// dtypes: a_dtype == w_dtype in {f32, bf16}; c_dtype in {f32, bf16}.  err: error word of the device, or null (see f32_product).
AIRUN_EXPORT int airun_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype,
                                 void* C, int c_dtype, int M, int N, int K,
                                 long long lda, long long ldw, long long ldc, int* err, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N) return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    dim3 grid(ceil_div_i(N, TN), ceil_div_i(M, TM));
    if (grid.y > 65535) return AIRUN_ERR_ARG;
    GemmExtra ex = {};
    if (f32_product<0>(A, a_dtype, W, w_dtype, C, c_dtype, M, N, K, lda, ldw, ldc, 1, ex, err, stream)) return airun_launch_status();
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
    if (f32_product<1>(A, a_dtype, W, w_dtype, C, c_dtype, M, N, K, lda, ldw, ldc, batch, ex, nullptr, stream)) return airun_launch_status();
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
                                         const int32_t* seg, int n_seg, long long sw, int* err, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N || !seg || n_seg <= 0) return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    dim3 grid(ceil_div_i(N, TN), ceil_div_i(M, TM) + n_seg);
    if (grid.y > 65535) return AIRUN_ERR_ARG;
    GemmExtra ex = {};
    ex.sw = sw; ex.seg = seg; ex.n_seg = n_seg;
    if (f32_product<2>(A, a_dtype, W, w_dtype, C, c_dtype, M, N, K, lda, ldw, ldc, 1, ex, err, stream)) return airun_launch_status();
#define LAUNCH(TA, TW, TC) \
    airun_launch(gemm_simt_kernel<TA, TW, TC, 2>, dim3(grid), dim3(256), 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc, ex)
    if (a_dtype == AIRUN_DT_F32 && w_dtype == AIRUN_DT_F32 && c_dtype == AIRUN_DT_F32) LAUNCH(float, float, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_F32) LAUNCH(__nv_bfloat16, __nv_bfloat16, float);
    else if (a_dtype == AIRUN_DT_BF16 && w_dtype == AIRUN_DT_BF16 && c_dtype == AIRUN_DT_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
    else return AIRUN_ERR_UNSUPPORTED;
#undef LAUNCH
    return airun_launch_status();
}
