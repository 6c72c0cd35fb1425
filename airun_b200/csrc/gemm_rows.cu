// bfloat16 matrix product of few rows, out[M][N] = x[M][K] * W[N][K]^T with M up to 16 (decoded tokens), float32
// accumulation, on mma.sync.
//
// What bounds such a product is reading W once, and at a few megabytes a matrix the time to get that stream going and to
// wind it up: a launch of the tcgen05 kernel first allocates tensor memory and sets up barriers, fills a ring through the
// copy engine, hands tiles from warp to warp, and adds up its K slices through a scratch in global memory with a ticket.
// Here the weights go straight from global memory to the registers of the warps that multiply them.  A block takes 16 or 32
// weight rows and all tokens; its eight warps share K (each takes every eighth run of 64 values, a 128-byte line of
// each weight row) and add up through shared memory in warp order.  The weights of a warp's first two runs are on their way
// before anything else is done.  (The kernel is launched once the one in front is done, see launch_mt: asked for while
// that one still runs, they cost the kernels around it more than they save.)  Both operands are used with one permutation of k, chosen so that a lane's
// operands of two m16n8k16 products are the 16 neighbouring bytes it loads: no shared memory, no shuffles.
//
// Three forms, as in the other product kernels: PLAIN; GROUPED, in which the rows of x lie in segments (device memory) with
// a matrix each (blockIdx.y: the segment; a segment of more than 8 * NT rows reads its matrix again for every further
// group of rows); BATCHED, products of equal sizes over column slices of x (blockIdx.z).
//
// The reference's counterparts are its half-precision matvec kernels (crates/airun-cuda/kernels/matmul.cu:518-636) and
// the fused gate/up/SwiGLU one (matmul.cu:150-214).
#include "common.cuh"

#define ROW_WARPS 8
#define EPI_F32 0
#define EPI_BF16 1
#define EPI_SWIGLU 2

namespace {

struct RowsParams {
    const __nv_bfloat16* x;
    const __nv_bfloat16* w;
    void* out;
    int M, N, K;
    long long ldx, ldw, ldc;
    float glu_limit, glu_slope;       // EPI_SWIGLU: 0, 0 for SwiGLU; a limit > 0 for the clamped gated unit
    int act;                          // EPI_F32 / EPI_BF16: 0 the product, 1 + m an activation of it
    const int32_t* seg;               // GROUPED: int32 [n_seg + 1] on the device
    int n_seg;
    long long sx, sw, so;             // BATCHED: elements between products; GROUPED: sw between the segments' matrices
};

__device__ __forceinline__ float activation(float z, int m) {
    if (m == 0) { const float r = fmaxf(z, 0.0f); return r * r; }
    if (m == 1) return z / (1.0f + __expf(-z));
    if (m == 2) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    if (m == 4) return 0.5f * z * (1.0f + erff(z * 0.7071067811865476f));
    return fmaxf(z, 0.0f);
}
__device__ __forceinline__ float gated_unit(float limit, float slope, float g, float u) {
    if (limit > 0.0f) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return g / (1.0f + __expf(-slope * g)) * (u + 1.0f);
    }
    return g / (1.0f + __expf(-g)) * u;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// weights: read once, so they need not stay in the L1 cache (the tokens' rows, which every block reads, should)
__device__ __forceinline__ uint4 load_weights(const __nv_bfloat16* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

enum { FORM_PLAIN = 0, FORM_GROUPED = 1, FORM_BATCHED = 2 };

template <int MT, int NT, int EPI, int FORM>
__global__ __launch_bounds__(32 * ROW_WARPS, 2) void gemm_rows_kernel(const RowsParams p) {
    constexpr int ROWS = 16 * MT, TOKS = 8 * NT, LDR = ROWS + 4;       // LDR: the lanes' partial sums miss each other's banks
    pdl_trigger();
    __shared__ float red[ROW_WARPS][TOKS * LDR];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = blockIdx.x * ROWS;
    const __nv_bfloat16* x = p.x;
    const __nv_bfloat16* w = p.w;
    size_t out_off = 0;
    if (FORM == FORM_BATCHED) { x += (size_t)blockIdx.z * p.sx; w += (size_t)blockIdx.z * p.sw; out_off = (size_t)blockIdx.z * p.so; }
    if (FORM == FORM_GROUPED) w += (size_t)blockIdx.y * p.sw;
    const __nv_bfloat16* wrow[2 * MT];                                  // this lane's weight rows
#pragma unroll
    for (int i = 0; i < 2 * MT; ++i) wrow[i] = w + (size_t)min(r0 + 8 * i + g, p.N - 1) * p.ldw + 8 * t;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    // run s: k from 64 s; this lane's halves lie at 64 s + 8 t and 64 s + 32 + 8 t
    auto fetch = [&](int s, uint4 (&a)[2 * MT][2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 64 * s + 32 * h;
            const bool on = k + 8 * t < p.K;                            // K is a multiple of 8
#pragma unroll
            for (int i = 0; i < 2 * MT; ++i) a[i][h] = on ? load_weights(wrow[i] + k) : zero;
        }
    };
    const int runs = (p.K + 63) / 64;
    uint4 a0[2 * MT][2], a1[2 * MT][2];
    int lo = FORM == FORM_PLAIN ? blockIdx.y * TOKS : 0, hi = p.M;
    if (FORM == FORM_GROUPED) {
        pdl_wait();                                                     // an expert without rows reads nothing
        lo = p.seg[blockIdx.y];
        hi = min(p.seg[blockIdx.y + 1], p.M);
        if (lo >= hi) return;
        fetch(warp, a0);
        fetch(warp + ROW_WARPS, a1);
    } else {
        fetch(warp, a0);
        fetch(warp + ROW_WARPS, a1);
        pdl_wait();
    }
    for (int m0 = lo; m0 < hi; m0 += TOKS) {
        if (FORM != FORM_PLAIN && m0 > lo) { fetch(warp, a0); fetch(warp + ROW_WARPS, a1); }
        if (FORM == FORM_PLAIN && m0 > lo) break;                       // blockIdx.y has the other groups of rows
        const __nv_bfloat16* xrow[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) xrow[j] = x + (size_t)min(m0 + 8 * j + g, hi - 1) * p.ldx + 8 * t;
        float c[MT][NT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) c[i][j][0] = c[i][j][1] = c[i][j][2] = c[i][j][3] = 0.0f;
        auto tokens = [&](int s, uint4 (&b)[NT][2]) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = 64 * s + 32 * h;
                const bool on = k + 8 * t < p.K;
#pragma unroll
                for (int j = 0; j < NT; ++j) b[j][h] = on ? *reinterpret_cast<const uint4*>(xrow[j] + k) : zero;
            }
        };
        auto multiply = [&](const uint4 (&a)[2 * MT][2], const uint4 (&b)[NT][2]) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        const uint4 u = a[2 * i][h], v = a[2 * i + 1][h];
                        mma_bf16(c[i][j], u.x, v.x, u.y, v.y, b[j][h].x, b[j][h].y);
                        mma_bf16(c[i][j], u.z, v.z, u.w, v.w, b[j][h].z, b[j][h].w);
                    }
        };
        for (int s = warp; s < runs; s += 2 * ROW_WARPS) {
            uint4 b0[NT][2], b1[NT][2];
            tokens(s, b0);
            tokens(s + ROW_WARPS, b1);
            multiply(a0, b0);
            fetch(s + 2 * ROW_WARPS, a0);
            multiply(a1, b1);
            fetch(s + 3 * ROW_WARPS, a1);
        }
        // lane (g, t) holds rows g and g + 8 of tokens 2t and 2t + 1 of every tile
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                float* d = &red[warp][(8 * j + 2 * t) * LDR + 16 * i + g];
                d[0] = c[i][j][0]; d[LDR] = c[i][j][1]; d[8] = c[i][j][2]; d[LDR + 8] = c[i][j][3];
            }
        __syncthreads();
        constexpr int OUTS = EPI == EPI_SWIGLU ? ROWS / 2 : ROWS;
        for (int e = threadIdx.x; e < OUTS * TOKS; e += 32 * ROW_WARPS) {
            const int tok = e / OUTS, n = e % OUTS;
            const int row = EPI == EPI_SWIGLU ? (n / 16) * 32 + n % 16 : n;
            float v = 0.0f, u = 0.0f;
#pragma unroll
            for (int q = 0; q < ROW_WARPS; ++q) {
                v += red[q][tok * LDR + row];
                if (EPI == EPI_SWIGLU) u += red[q][tok * LDR + row + 16];
            }
            if (m0 + tok < hi && r0 + row < p.N) {
                if (EPI == EPI_SWIGLU) {
                    __nv_bfloat16* o = (__nv_bfloat16*)p.out + out_off + (size_t)(m0 + tok) * p.ldc;
                    o[r0 / 2 + n] = __float2bfloat16_rn(gated_unit(p.glu_limit, p.glu_slope, v, u));
                } else {
                    if (p.act) v = activation(v, p.act - 1);
                    const size_t at = out_off + (size_t)(m0 + tok) * p.ldc + r0 + n;
                    if (EPI == EPI_F32) ((float*)p.out)[at] = v;
                    else ((__nv_bfloat16*)p.out)[at] = __float2bfloat16_rn(v);
                }
            }
        }
        __syncthreads();
    }
}

template <int NT, int EPI, int FORM>
void launch_mt(const RowsParams& p, int groups, int batch, cudaStream_t stream) {
    // 32 weight rows a block (every block reads all tokens: half as often as with 16) once that gives every SM a block
    const bool two = EPI == EPI_SWIGLU || (long long)p.N * batch * (FORM == FORM_GROUPED ? groups : 1) >= 32LL * airun_sm_count();
    const int rows = two ? 32 : 16;
    const dim3 grid(ceil_div_i(p.N, rows), groups, batch);
    // The launch waits for the kernel in front: resident early, half of an SM's registers a block, these blocks held up the
    // kernels around them.  A step of Qwen3-8B with eight requests took 5.7 ms with them early and 4.1 without (4.1 by the
    // tcgen05 kernel), one of the routed design of width 2048 0.80 and 0.71 (0.91).
    if (two) airun_launch_after(gemm_rows_kernel<2, NT, EPI, FORM>, grid, dim3(32 * ROW_WARPS), 0, stream, p);
    else if constexpr (EPI != EPI_SWIGLU) airun_launch_after(gemm_rows_kernel<1, NT, EPI, FORM>, grid, dim3(32 * ROW_WARPS), 0, stream, p);
}

template <int FORM>
int launch_rows(const RowsParams& p, int epi, int nt, int groups, int batch, cudaStream_t stream) {
#define BY_NT(EPI) do { if (nt == 1) launch_mt<1, EPI, FORM>(p, groups, batch, stream); else launch_mt<2, EPI, FORM>(p, groups, batch, stream); } while (0)
    if (epi == EPI_F32) BY_NT(EPI_F32);
    else if (epi == EPI_BF16) BY_NT(EPI_BF16);
    else if (epi == EPI_SWIGLU) BY_NT(EPI_SWIGLU);
    else return AIRUN_ERR_UNSUPPORTED;
#undef BY_NT
    return airun_launch_status();
}

bool bad_operands(const void* x, const void* W, int K, long long ldx, long long ldw) {
    return K % 8 != 0 || ldx % 8 != 0 || ldw % 8 != 0 || ((uintptr_t)x & 15) || ((uintptr_t)W & 15);
}

}  // namespace

// out[M][N] = x[M][K] * W[N][K]^T.  x, W bfloat16 (K and row strides multiples of 8, 16-byte aligned).
// epi: 0 float32 out; 1 bfloat16 out; 2 gated unit over rows that alternate between blocks of 16 gate and 16 up rows,
// bfloat16 [M][N/2].  act: 0, or 1 + the activation (epi 0, 1).
AIRUN_EXPORT int airun_gemm_rows(const void* x, const void* W, void* out, int M, int N, int K, long long ldx, long long ldw,
                                 long long ldc, int epi, float glu_limit, float glu_slope, int act, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || bad_operands(x, W, K, ldx, ldw) || (epi == EPI_SWIGLU && N % 32) || act < 0 || act > 5) return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    RowsParams p = {};
    p.x = (const __nv_bfloat16*)x; p.w = (const __nv_bfloat16*)W; p.out = out;
    p.M = M; p.N = N; p.K = K; p.ldx = ldx; p.ldw = ldw; p.ldc = ldc;
    p.glu_limit = glu_limit; p.glu_slope = glu_slope; p.act = act;
    const int nt = M <= 8 ? 1 : 2;
    const int groups = ceil_div_i(M, 8 * nt);
    if (groups > 65535) return AIRUN_ERR_ARG;
    return launch_rows<FORM_PLAIN>(p, epi, nt, groups, 1, stream);
}

// Rows seg[e] .. seg[e + 1] - 1 of x times W[e] ([n_seg][N][K], contiguous) into the same rows of out; the segments are
// int32 [n_seg + 1] on the device; rows from seg[n_seg] on are left as they are.
AIRUN_EXPORT int airun_gemm_rows_grouped(const void* x, const void* W, void* out, int M, int N, int K, long long ldx, long long ldc,
                                         int epi, const int32_t* seg, int n_seg, float glu_limit, float glu_slope, int act,
                                         cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || !seg || n_seg <= 0 || n_seg > 65535 || bad_operands(x, W, K, ldx, 8) ||
        (epi == EPI_SWIGLU && N % 32) || act < 0 || act > 5)
        return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    RowsParams p = {};
    p.x = (const __nv_bfloat16*)x; p.w = (const __nv_bfloat16*)W; p.out = out;
    p.M = M; p.N = N; p.K = K; p.ldx = ldx; p.ldw = K; p.ldc = ldc;
    p.glu_limit = glu_limit; p.glu_slope = glu_slope; p.act = act;
    p.seg = seg; p.n_seg = n_seg; p.sw = (long long)N * K;
    return launch_rows<FORM_GROUPED>(p, epi, M <= 4 * n_seg ? 1 : 2, n_seg, 1, stream);
}

// `batch` products of equal sizes: product b reads the columns b * sx .. of x, has W[b] ([batch][N][K], contiguous) and
// writes so elements further on than product b - 1; bfloat16.
AIRUN_EXPORT int airun_gemm_rows_batched(const void* x, const void* W, void* out, int M, int N, int K, int batch, long long ldx,
                                         long long sx, long long ldc, long long so, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || batch <= 0 || batch > 65535 || bad_operands(x, W, K, ldx, 8) || sx % 8) return AIRUN_ERR_ARG;
    if (M == 0) return AIRUN_OK;
    RowsParams p = {};
    p.x = (const __nv_bfloat16*)x; p.w = (const __nv_bfloat16*)W; p.out = out;
    p.M = M; p.N = N; p.K = K; p.ldx = ldx; p.ldw = K; p.ldc = ldc;
    p.sx = sx; p.sw = (long long)N * K; p.so = so;
    return launch_rows<FORM_BATCHED>(p, EPI_BF16, M <= 8 ? 1 : 2, 1, batch, stream);
}
