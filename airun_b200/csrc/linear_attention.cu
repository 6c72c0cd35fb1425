// Gated linear attention: a matrix-valued state per head that decays channel by channel.
//
// Per head, with key channels d < D and value channels j < Dv, for the tokens of a request in order:
//     S[d][j] <- a_t[d] * S[d][j] + k_t[d] * v_t[j]          o_t[j] = sum_d S[d][j] * q_t[d] * q_scale
// (the output uses the state AFTER the token's own update).  The decay a_t[d] lies in (0, 1):
//     a_t = sigmoid(z_t)^(1/tau),  z_t = W2 (low_t) + bias,   low_t = the low-rank projection of the input,
// computed as  a = exp(logsigmoid(z) / tau)  (decay_kernel).
// Then, per head, o_t is divided by its root mean square over Dv (eps inside the root), multiplied by a
// weight vector shared by the heads and by silu of a gate projection (out_gate_kernel).
//
// State, decays, the recurrence and the norm are float32 whatever the storage of the activations.  The
// state of a request lives in its slot of the state tensor between steps, stored per head as [D][Dv]
// (a row per key channel, the value columns side by side), and is zero when the request starts.  The result
// at a token depends only on the request's tokens up to it; its rounding also depends on the form that the
// step takes: token by token, or, from 256 tokens of all its requests on, a request's tokens in segments of 128
// that run side by side, whose sums are added in another order.
#include "common.cuh"

// a[t][c] = exp(logsigmoid(bias[c] + sum_j low[t][j] * w2[c][j]) / tau) for c < n (= heads * D).
// The same kernel serves every second half of a low-rank pair that ends in a function of its own, in float32:
// with z = bias[c] + sum_j f(low[t][j]) * w2[c][j] (f the identity, or tanh when `in_tanh`),
//   LOWRANK_POW_SIGMOID   sigmoid(z)^(1/tau)
//   LOWRANK_EXP_SOFTPLUS  exp(-exp(p[c / group]) * softplus(z))     (p: one number per group of channels)
//   LOWRANK_SIGMOID       sigmoid(z)
//   LOWRANK_EXP_NEG_EXP   exp(-exp(z))
#define LOWRANK_POW_SIGMOID 0
#define LOWRANK_EXP_SOFTPLUS 1
#define LOWRANK_SIGMOID 2
#define LOWRANK_EXP_NEG_EXP 3
// A thread takes a channel of eight tokens.  With VEC its row of w2 (a multiple of eight numbers on a 16-byte boundary) comes in pieces of eight, all asked for ahead
// of the wait up to a rank of 32: one number at a time, each load waited for the one before.  Only the functions that need log(1 + exp(-|z|)) form it.  Three prompts
// through Pogarax, 14 launches of rank 16 over 1,024 and 2,048 channels: 3,130 -> 3,097 us.
#define DECAY_TOKENS 8        // tokens of one block: a row of w2 is read once for all of them
__device__ __forceinline__ void decay_row8(const float* p, float (&w)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}
__device__ __forceinline__ void decay_row8(const __nv_bfloat16* p, float (&w)[8]) {
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    const uint32_t u[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { w[2 * i] = __uint_as_float(u[i] << 16); w[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
}
template <typename TW, bool VEC>
__global__ __launch_bounds__(128) void decay_kernel(const float* low, long long low_stride, const TW* __restrict__ w2,
                                                    const float* __restrict__ bias, float* __restrict__ out, int T, int n, int rank,
                                                    float inv_tau, const int32_t* __restrict__ req_of_token,
                                                    int mode, int in_tanh, const float* __restrict__ group_param, int group) {
    pdl_trigger();
    extern __shared__ float s_low[];                       // [DECAY_TOKENS][rank]
    const int t0 = blockIdx.x * DECAY_TOKENS, nt = min(DECAY_TOKENS, T - t0);
    const int c = blockIdx.y * blockDim.x + threadIdx.x;       // a channel a thread
    const TW* wr = w2 + (size_t)min(c, n - 1) * rank;
    float w[4][8];
    if (VEC) {
#pragma unroll
        for (int i = 0; i < 4; ++i) if (8 * i < rank) decay_row8(wr + 8 * i, w[i]);
    }
    const float b = bias && c < n ? bias[c] : 0.0f;
    pdl_wait();
    for (int e = threadIdx.x; e < nt * rank; e += blockDim.x) {
        const int tk = e / rank, j = e - tk * rank;
        const float lv = low[(size_t)(t0 + tk) * low_stride + j];
        s_low[e] = in_tanh ? tanhf(lv) : lv;
    }
    for (int e = nt * rank + threadIdx.x; e < DECAY_TOKENS * rank; e += blockDim.x) s_low[e] = 0.0f;
    __syncthreads();
    if (c < n) {
        float z[DECAY_TOKENS];
#pragma unroll
        for (int tk = 0; tk < DECAY_TOKENS; ++tk) z[tk] = b;
        if (VEC) {
            auto eight = [&](int j, const float (&v)[8]) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int tk = 0; tk < DECAY_TOKENS; ++tk) z[tk] = fmaf(s_low[tk * rank + j + i], v[i], z[tk]);
            };
#pragma unroll
            for (int i = 0; i < 4; ++i) if (8 * i < rank) eight(8 * i, w[i]);
            for (int j = 32; j < rank; j += 8) {
                decay_row8(wr + j, w[0]);
                eight(j, w[0]);
            }
        } else {
            for (int j = 0; j < rank; ++j) {
                const float v = to_f32<TW>(wr[j]);
#pragma unroll
                for (int tk = 0; tk < DECAY_TOKENS; ++tk) z[tk] = fmaf(s_low[tk * rank + j], v, z[tk]);
            }
        }
        const float p = mode == LOWRANK_EXP_SOFTPLUS ? -expf(group_param[c / group]) : 0.0f;
#pragma unroll
        for (int tk = 0; tk < DECAY_TOKENS; ++tk) {
            if (tk >= nt || req_of_token[t0 + tk] < 0) continue;
            const float zz = z[tk];
            float r;
            if (mode == LOWRANK_POW_SIGMOID) r = expf((fminf(zz, 0.0f) - log1pf(expf(-fabsf(zz)))) * inv_tau);      // logsigmoid(z) = min(z, 0) - log(1 + exp(-|z|))
            else if (mode == LOWRANK_EXP_SOFTPLUS) r = expf(p * (fmaxf(zz, 0.0f) + log1pf(expf(-fabsf(zz)))));
            else if (mode == LOWRANK_SIGMOID) r = 1.0f / (1.0f + expf(-zz));
            else r = expf(-expf(zz));
            out[(size_t)(t0 + tk) * n + c] = r;
        }
    }
}

AIRUN_EXPORT int airun_lowrank_act(const float* low, long long low_stride, const void* w2, int w_dtype, const float* bias,
                                   float* out, int T, int n, int rank, float tau, const int32_t* req_of_token,
                                   int mode, int in_tanh, const float* group_param, int group, cudaStream_t stream) {
    if (T < 0 || n <= 0 || n > 65535 * 128 || rank <= 0 || rank > 1024 || !(tau > 0.0f) || !req_of_token || mode < 0 || mode > 3)
        return AIRUN_ERR_ARG;
    if (mode == LOWRANK_EXP_SOFTPLUS && (!group_param || group <= 0)) return AIRUN_ERR_ARG;
    if (T == 0) return AIRUN_OK;
    const bool vec = rank % 8 == 0 && ((uintptr_t)w2 & 15) == 0;
#define DECAY_ARGS(TW) dim3(blocks, ceil_div_i(n, 128)), dim3(128), smem, stream, low, low_stride, (const TW*)w2, bias, out, T, n, rank, 1.0f / tau, \
        req_of_token, mode, in_tanh, group_param, group
#define DECAY_LAUNCH(TW) do { if (vec) airun_launch(decay_kernel<TW, true>, DECAY_ARGS(TW)); else airun_launch(decay_kernel<TW, false>, DECAY_ARGS(TW)); } while (0)
    const size_t smem = (size_t)DECAY_TOKENS * rank * sizeof(float);
    const int blocks = ceil_div_i(T, DECAY_TOKENS);
    if (w_dtype == AIRUN_DT_F32)
        DECAY_LAUNCH(float);
    else if (w_dtype == AIRUN_DT_BF16)
        DECAY_LAUNCH(__nv_bfloat16);
    else
        return AIRUN_ERR_UNSUPPORTED;
    return airun_launch_status();
}

AIRUN_EXPORT int airun_gla_decay(const float* low, long long low_stride, const void* w2, int w_dtype, const float* bias,
                                 float* out, int T, int n, int rank, float tau, const int32_t* req_of_token,
                                 cudaStream_t stream) {
    return airun_lowrank_act(low, low_stride, w2, w_dtype, bias, out, T, n, rank, tau, req_of_token, LOWRANK_POW_SIGMOID, 0,
                             nullptr, 0, stream);
}

// The recurrence.  One block per (request, head, 32 value columns), 256 threads: a lane owns a column
// and a warp owns NS key channels d = warp * NS + i, so a thread keeps NS elements of the state in
// registers for the whole step, and q, k and the decay of a token are the same for all lanes of a warp:
// they come from shared memory as float4 that every lane reads at one address (one access for the warp).
// The tokens of the request are staged through shared memory a few at a time by asynchronous copies
// (16 bytes each where the rows allow it) into one of two stages, so that the next tokens are on their way
// while these are used.  Each warp leaves its partial sums over its key channels in shared
// memory, and the eight partial sums of every (token, column) of the stage are added together, in warp
// order, once the stage's tokens are through: nothing but the state itself chains one token to the next.
#define GLA_COLS 32
#define GLA_WARPS 8
__device__ __forceinline__ void gla_cp4(float* smem, const float* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void gla_cp16(float* smem, const float* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
// With CONST the decay is one number per head (`head_decay`), the same for every token and key channel, and nothing is
// staged for it; `in_silu` applies z * sigmoid(z) to the staged q, k and v (projections that carry their activation).
//
// SEG: a request's tokens are cut into segments of GLA_SEG that run side by side (blockIdx.x counts the segments of all
// requests in turn): the first starts from the request's state, the others from zero, and each leaves its last state and, per
// key channel, the product of its decays; gla_segment_kernel then adds what the state in front of a segment gives to its
// tokens.  One request's prompt is otherwise a chain of its tokens on heads x Dv / 32 blocks: 2,048 tokens at 16 heads took
// 250 us on 64 blocks and take 123 us in 16 segments (76 us here, 47 in gla_segment_kernel), at 8 heads with one decay a
// head 330 and 85.
#define GLA_SEG 128
struct GlaSegments {
    float* ends;                  // [segments][heads][D][Dv]: a segment's last state, begun from zero but for a request's first
    float* prods;                 // [segments][heads][D]: products of a segment's decays
};
// The request and the place within it of segment g; false: there are not so many segments.
__device__ __forceinline__ bool gla_find_segment(const int32_t* cu_tokens, int num_reqs, int g, int& r, int& s, int& count) {
    for (r = 0; r < num_reqs; ++r) {
        count = (cu_tokens[r + 1] - cu_tokens[r] + GLA_SEG - 1) / GLA_SEG;
        if (g < count) { s = g; return true; }
        g -= max(count, 0);
    }
    return false;
}
template <int NS, bool CONST, bool SEG>
__global__ __launch_bounds__(256) void gla_recurrent_kernel(
    const float* q, const float* k, const float* v, long long row_stride,
    const float* decay, float* state, long long slot_stride,
    const int32_t* __restrict__ cu_tokens, const int32_t* __restrict__ state_slots, int max_slots,
    float* __restrict__ out, int heads, int D, int Dv, float q_scale, int* __restrict__ err,
    const float* __restrict__ head_decay, int in_silu, int num_reqs, GlaSegments segs) {
    pdl_trigger();
    pdl_wait();
    constexpr int DP = NS * GLA_WARPS;
    constexpr int GLA_TT = NS >= 32 ? 4 : NS >= 16 ? 8 : 16;     // tokens of a stage (static shared memory stays under 48 KB)
    __shared__ __align__(16) float s_q[2][GLA_TT][DP], s_k[2][GLA_TT][DP], s_a[2][GLA_TT][DP], s_v[2][GLA_TT][GLA_COLS];
    __shared__ float s_p[GLA_WARPS][GLA_TT][GLA_COLS];
    int r = blockIdx.x, part = 0, parts = 1;
    const int head = blockIdx.y, col0 = blockIdx.z * GLA_COLS;
    if (SEG) {
        const bool there = gla_find_segment(cu_tokens, num_reqs, blockIdx.x, r, part, parts);
        int r2, part2, parts2;                             // a segment that no block has: said by one of the last segment's
        if (blockIdx.x == gridDim.x - 1 && head == 0 && col0 == 0 && threadIdx.x == 0 &&
            gla_find_segment(cu_tokens, num_reqs, gridDim.x, r2, part2, parts2))
            atomicOr(err, AIRUN_DEV_BAD_ROW);
        if (!there) return;
    }
    int t0 = cu_tokens[r], n = cu_tokens[r + 1] - t0;
    if (n <= 0) return;
    if (SEG) { t0 += part * GLA_SEG; n = min(GLA_SEG, n - part * GLA_SEG); }
    const int slot = state_slots[r];
    if (slot < 0 || slot >= max_slots) {
        if (threadIdx.x == 0) atomicOr(err, AIRUN_DEV_BAD_REQ);
        return;
    }
    const bool from_state = !SEG || part == 0, to_state = !SEG || parts == 1;
    float prod = 1.0f;                                     // SEG: of key channel threadIdx.x, by the blocks of the first columns
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col = col0 + lane, d0 = warp * NS;
    const bool col_ok = col < Dv;
    // the padding beyond D and Dv is zero in both stages and is never copied into
    for (int e = threadIdx.x; e < 2 * GLA_TT * DP; e += 256) {
        (&s_q[0][0][0])[e] = 0.0f; (&s_k[0][0][0])[e] = 0.0f; (&s_a[0][0][0])[e] = 0.0f;
    }
    for (int e = threadIdx.x; e < 2 * GLA_TT * GLA_COLS; e += 256) (&s_v[0][0][0])[e] = 0.0f;
    __syncthreads();
    // 16-byte copies when every row begins on a 16-byte boundary
    const bool vec = (D % 4 == 0) && (Dv % 4 == 0) && (row_stride % 4 == 0) &&
                     ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)decay) & 15) == 0);
    const float dec = CONST ? head_decay[blockIdx.y] : 0.0f;
    auto stage = [&](int base, int buf) {
        const int nt = min(GLA_TT, n - base);
        if (vec) {
            const int per = D / 4, nc4 = min(GLA_COLS, Dv - col0) / 4;
            for (int e = threadIdx.x; e < nt * per; e += 256) {
                const int tt = e / per, d = (e - tt * per) * 4;
                const size_t row = (size_t)(t0 + base + tt);
                gla_cp16(&s_q[buf][tt][d], q + row * row_stride + (size_t)head * D + d);
                gla_cp16(&s_k[buf][tt][d], k + row * row_stride + (size_t)head * D + d);
                if (!CONST) gla_cp16(&s_a[buf][tt][d], decay + row * ((size_t)heads * D) + (size_t)head * D + d);
            }
            for (int e = threadIdx.x; e < nt * nc4; e += 256) {
                const int tt = e / nc4, c = (e - tt * nc4) * 4;
                gla_cp16(&s_v[buf][tt][c], v + (size_t)(t0 + base + tt) * row_stride + (size_t)head * Dv + col0 + c);
            }
        } else {
            for (int e = threadIdx.x; e < nt * D; e += 256) {
                const int tt = e / D, d = e - tt * D;
                const size_t row = (size_t)(t0 + base + tt);
                gla_cp4(&s_q[buf][tt][d], q + row * row_stride + (size_t)head * D + d);
                gla_cp4(&s_k[buf][tt][d], k + row * row_stride + (size_t)head * D + d);
                if (!CONST) gla_cp4(&s_a[buf][tt][d], decay + row * ((size_t)heads * D) + (size_t)head * D + d);
            }
            const int nc = min(GLA_COLS, Dv - col0);
            for (int e = threadIdx.x; e < nt * nc; e += 256) {
                const int tt = e / nc, c = e - tt * nc;
                gla_cp4(&s_v[buf][tt][c], v + (size_t)(t0 + base + tt) * row_stride + (size_t)head * Dv + col0 + c);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, 0);
    // the state of this head, [D][Dv]: the lanes of a warp read one row of it side by side
    float* sbase = state + (size_t)slot * slot_stride + (size_t)head * D * Dv + (col_ok ? col : 0);
    float S[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) S[i] = (from_state && col_ok && d0 + i < D) ? sbase[(size_t)(d0 + i) * Dv] : 0.0f;
    int it = 0;
    for (int base = 0; base < n; base += GLA_TT, ++it) {
        const int buf = it & 1, nt = min(GLA_TT, n - base);
        if (base + GLA_TT < n) {
            stage(base + GLA_TT, buf ^ 1);          // that stage was last read before the barrier that ended the round before
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (in_silu) {
            for (int e = threadIdx.x; e < nt * DP; e += 256) {
                const float a = (&s_q[buf][0][0])[e], b = (&s_k[buf][0][0])[e];
                (&s_q[buf][0][0])[e] = a / (1.0f + expf(-a));
                (&s_k[buf][0][0])[e] = b / (1.0f + expf(-b));
            }
            for (int e = threadIdx.x; e < nt * GLA_COLS; e += 256) {
                const float a = (&s_v[buf][0][0])[e];
                (&s_v[buf][0][0])[e] = a / (1.0f + expf(-a));
            }
            __syncthreads();
        }
        if (SEG && !CONST && blockIdx.z == 0 && threadIdx.x < D)
            for (int tt = 0; tt < nt; ++tt) prod *= s_a[buf][tt][threadIdx.x];
#pragma unroll 4
        for (int tt = 0; tt < nt; ++tt) {
            const float vj = s_v[buf][tt][lane];
            float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
            for (int i4 = 0; i4 < NS / 4; ++i4) {
                const float4 a4 = CONST ? make_float4(dec, dec, dec, dec) : *reinterpret_cast<const float4*>(&s_a[buf][tt][d0 + 4 * i4]);
                const float4 k4 = *reinterpret_cast<const float4*>(&s_k[buf][tt][d0 + 4 * i4]);
                const float4 q4 = *reinterpret_cast<const float4*>(&s_q[buf][tt][d0 + 4 * i4]);
                S[4 * i4 + 0] = fmaf(a4.x, S[4 * i4 + 0], k4.x * vj); acc0 = fmaf(S[4 * i4 + 0], q4.x, acc0);
                S[4 * i4 + 1] = fmaf(a4.y, S[4 * i4 + 1], k4.y * vj); acc1 = fmaf(S[4 * i4 + 1], q4.y, acc1);
                S[4 * i4 + 2] = fmaf(a4.z, S[4 * i4 + 2], k4.z * vj); acc0 = fmaf(S[4 * i4 + 2], q4.z, acc0);
                S[4 * i4 + 3] = fmaf(a4.w, S[4 * i4 + 3], k4.w * vj); acc1 = fmaf(S[4 * i4 + 3], q4.w, acc1);
            }
            s_p[warp][tt][lane] = acc0 + acc1;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nt * GLA_COLS; e += 256) {
            const int tt = e / GLA_COLS, c = e - tt * GLA_COLS;
            float o = 0.0f;
#pragma unroll
            for (int w = 0; w < GLA_WARPS; ++w) o += s_p[w][tt][c];
            if (col0 + c < Dv) out[(size_t)(t0 + base + tt) * ((size_t)heads * Dv) + (size_t)head * Dv + col0 + c] = o * q_scale;
        }
        __syncthreads();
    }
    float* const end = to_state ? sbase : segs.ends + ((size_t)blockIdx.x * heads + head) * D * Dv + (col_ok ? col : 0);
    if (col_ok) {
#pragma unroll
        for (int i = 0; i < NS; ++i)
            if (d0 + i < D) end[(size_t)(d0 + i) * Dv] = S[i];
    }
    if (SEG && !CONST && blockIdx.z == 0 && threadIdx.x < D) segs.prods[((size_t)blockIdx.x * heads + head) * D + threadIdx.x] = prod;
}

// What the state in front of a segment gives to the segment's tokens, o_t += (q_t * a_first * .. * a_t) . S_in, and the
// request's last state.  One block per (segment, head, 64 value columns): the states the earlier segments of the request
// ended with are brought together in their order (S <- product of a segment's decays * S + its end), the decayed queries are
// formed in shared memory (four runs of 32 tokens a channel side by side), and the product of the two is added to the
// output, 8 tokens x 4 columns a thread.  Only products of decays occur, never quotients, so a decay near zero only wipes.
template <bool CONST>
__global__ __launch_bounds__(256) void gla_segment_kernel(
    const float* q, long long row_stride, const float* decay, float* state, long long slot_stride,
    const int32_t* __restrict__ cu_tokens, const int32_t* __restrict__ state_slots, int max_slots, float* out, int heads,
    int D, int Dv, float q_scale, const float* __restrict__ head_decay, int in_silu, int num_reqs, GlaSegments segs) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float s_seg[];
    const int QS = D + 4;
    float* const s_qt = s_seg;                             // [GLA_SEG][D + 4]
    float* const s_S = s_seg + GLA_SEG * QS;               // [D][64]
    __shared__ float s_run[4][128];
    int r, part, parts;
    if (!gla_find_segment(cu_tokens, num_reqs, blockIdx.x, r, part, parts) || part == 0) return;
    const int slot = state_slots[r];
    if (slot < 0 || slot >= max_slots) return;             // the kernel in front has said so
    const int head = blockIdx.y, c0 = blockIdx.z * 64, tid = threadIdx.x;
    const int t0 = cu_tokens[r] + part * GLA_SEG, n = min(GLA_SEG, cu_tokens[r + 1] - t0);
    const size_t first = (size_t)blockIdx.x - part;        // the request's first segment
    const float dec = CONST ? head_decay[head] : 0.0f, dec_seg = CONST ? powf(dec, (float)GLA_SEG) : 0.0f;
    float* const srow = state + (size_t)slot * slot_stride + (size_t)head * D * Dv;
    for (int e = tid * 4; e < D * 64; e += 1024) {
        const int d = e / 64, c = c0 + e % 64;
        float4 S = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (c < Dv) {
#pragma unroll 4
            for (int j = 0; j <= part; ++j) {
                const size_t at = (first + j) * heads + head;
                const float4 E = *reinterpret_cast<const float4*>(segs.ends + at * D * Dv + (size_t)d * Dv + c);
                const int len = j < part ? GLA_SEG : n;
                const float a = CONST ? (j < part ? dec_seg : powf(dec, (float)len)) : segs.prods[at * D + d];
                if (j == part) {
                    *reinterpret_cast<float4*>(&s_S[d * 64 + e % 64]) = S;
                    if (part != parts - 1) break;
                }
                S.x = fmaf(a, S.x, E.x); S.y = fmaf(a, S.y, E.y); S.z = fmaf(a, S.z, E.z); S.w = fmaf(a, S.w, E.w);
            }
            if (part == parts - 1) *reinterpret_cast<float4*>(srow + (size_t)d * Dv + c) = S;
        } else {
            *reinterpret_cast<float4*>(&s_S[d * 64 + e % 64]) = S;
        }
    }
    // the decayed queries: run k of a channel has tokens 32 k .. 32 k + 31
    for (int e = tid; e < 4 * D; e += 256) {
        const int run = e / D, d = e - run * D;
        const float* a = decay + (size_t)t0 * heads * D + (size_t)head * D + d;
        float p = 1.0f;
        for (int t = 32 * run; t < min(32 * run + 32, n); ++t) {
            p *= CONST ? dec : a[(size_t)t * heads * D];
            float qv = q[(size_t)(t0 + t) * row_stride + (size_t)head * D + d];
            if (in_silu) qv = qv / (1.0f + expf(-qv));
            s_qt[t * QS + d] = qv * p;
        }
        s_run[run][d] = p;
    }
    __syncthreads();
    for (int e = tid; e < 3 * D; e += 256) {
        const int run = 1 + e / D, d = e % D;
        float p = s_run[0][d];
        for (int k = 1; k < run; ++k) p *= s_run[k][d];
        for (int t = 32 * run; t < min(32 * run + 32, n); ++t) s_qt[t * QS + d] *= p;
    }
    __syncthreads();
    const int cg = (tid & 15) * 4, tg = (tid >> 4) * 8;
    if (tg >= n || c0 + cg >= Dv) return;
    float4 acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int d = 0; d < D; d += 4) {
        float4 S4[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) S4[k] = *reinterpret_cast<const float4*>(&s_S[(d + k) * 64 + cg]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(&s_qt[(tg + i) * QS + d]);       // rows from n on are not stored
            const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[i].x = fmaf(xs[k], S4[k].x, acc[i].x); acc[i].y = fmaf(xs[k], S4[k].y, acc[i].y);
                acc[i].z = fmaf(xs[k], S4[k].z, acc[i].z); acc[i].w = fmaf(xs[k], S4[k].w, acc[i].w);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (tg + i >= n) break;
        float4* o = reinterpret_cast<float4*>(out + (size_t)(t0 + tg + i) * ((size_t)heads * Dv) + (size_t)head * Dv + c0 + cg);
        float4 v = *o;
        v.x = fmaf(q_scale, acc[i].x, v.x); v.y = fmaf(q_scale, acc[i].y, v.y);
        v.z = fmaf(q_scale, acc[i].z, v.z); v.w = fmaf(q_scale, acc[i].w, v.w);
        *o = v;
    }
}

static int gla_recurrent_launch(const float* q, const float* k, const float* v, long long row_stride,
                                const float* decay, const float* head_decay, int in_silu, float* state, long long slot_stride,
                                int max_slots, const int32_t* cu_tokens, const int32_t* state_slots, int num_reqs,
                                float* out, int heads, int D, int Dv, float q_scale, float* work, int max_segments, int* err,
                                cudaStream_t stream) {
    if (num_reqs < 0 || heads <= 0 || D <= 0 || D > 256 || Dv <= 0 || !state || !cu_tokens || !state_slots || !err ||
        slot_stride < (long long)heads * D * Dv || heads > 65535 || (!decay && !head_decay))
        return AIRUN_ERR_ARG;
    if (num_reqs == 0) return AIRUN_OK;
    const int tiles = ceil_div_i(Dv, GLA_COLS);
    if (tiles > 65535) return AIRUN_ERR_ARG;
    GlaSegments segs = {};
#define GLA_LAUNCH_BY(BY, NS, C, SEG) BY(gla_recurrent_kernel<NS, C, SEG>, grid, dim3(256), 0, stream, q, k, v, row_stride, decay, state, \
        slot_stride, cu_tokens, state_slots, max_slots, out, heads, D, Dv, q_scale, err, head_decay, in_silu, num_reqs, segs)
    // segments run long, with fewer blocks than the chip holds: they wait for the kernel in front (airun_launch_after).  A step
    // of 2048 tokens with three layers of one decay per head took 3.38 ms instead of 3.24 with them packed where it leaves room.
#define GLA_LAUNCH(NS, C, SEG) do { if (SEG) GLA_LAUNCH_BY(airun_launch_after, NS, C, SEG); else GLA_LAUNCH_BY(airun_launch, NS, C, SEG); } while (0)
    if (work) {
        if (max_segments <= 0 || D > 128 || D % 4 || Dv % 4 || slot_stride % 4 || (((uintptr_t)state | (uintptr_t)out | (uintptr_t)work) & 15))
            return AIRUN_ERR_ARG;
        segs.ends = work;
        segs.prods = work + (size_t)max_segments * heads * D * Dv;
        const dim3 grid(max_segments, heads, tiles);
#define GLA_PICK(C) do { if (D <= 32) GLA_LAUNCH(4, C, true); else if (D <= 64) GLA_LAUNCH(8, C, true); else GLA_LAUNCH(16, C, true); } while (0)
        if (head_decay) GLA_PICK(true);
        else GLA_PICK(false);
#undef GLA_PICK
        const int smem = (GLA_SEG * (D + 4) + D * 64) * (int)sizeof(float);
        static unsigned long long configured[2];
        auto add = [&](auto kern, int i) -> int {
            if (first_on_device(configured[i])) {
                const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (GLA_SEG * 132 + 128 * 64) * (int)sizeof(float));
                if (e != cudaSuccess) return (int)e;
            }
            airun_launch_after(kern, dim3(max_segments, heads, ceil_div_i(Dv, 64)), dim3(256), smem, stream, q, row_stride, decay, state, slot_stride,
                         cu_tokens, state_slots, max_slots, out, heads, D, Dv, q_scale, head_decay, in_silu, num_reqs, segs);
            return airun_launch_status();
        };
        return head_decay ? add(gla_segment_kernel<true>, 0) : add(gla_segment_kernel<false>, 1);
    }
    const dim3 grid(num_reqs, heads, tiles);
#define GLA_PICK(C) do { if (D <= 32) GLA_LAUNCH(4, C, false); else if (D <= 64) GLA_LAUNCH(8, C, false); \
        else if (D <= 128) GLA_LAUNCH(16, C, false); else GLA_LAUNCH(32, C, false); } while (0)
    if (head_decay) GLA_PICK(true);
    else GLA_PICK(false);
#undef GLA_PICK
#undef GLA_LAUNCH
#undef GLA_LAUNCH_BY
    return airun_launch_status();
}

// `work`: null, or max_segments * heads * (D * Dv + D) floats for the segments (D up to 128, D and Dv in multiples of 4);
// max_segments: at least the sum over the requests of ceil(tokens / GLA_SEG); with fewer the error word says so.
AIRUN_EXPORT int airun_gla_segment_tokens() { return GLA_SEG; }

AIRUN_EXPORT int airun_gla_recurrent(const float* q, const float* k, const float* v, long long row_stride,
                                     const float* decay, float* state, long long slot_stride, int max_slots,
                                     const int32_t* cu_tokens, const int32_t* state_slots, int num_reqs,
                                     float* out, int heads, int D, int Dv, float q_scale, float* work, int max_segments, int* err,
                                     cudaStream_t stream) {
    if (!decay) return AIRUN_ERR_ARG;
    return gla_recurrent_launch(q, k, v, row_stride, decay, nullptr, 0, state, slot_stride, max_slots, cu_tokens, state_slots,
                                num_reqs, out, heads, D, Dv, q_scale, work, max_segments, err, stream);
}

// The same recurrence with ONE decay per head, S <- d_h S + k v^T, o = S^T q (times q_scale); `in_silu`: q, k and v
// arrive without their activation z * sigmoid(z), which is applied as they are staged.
AIRUN_EXPORT int airun_decay_recurrent(const float* q, const float* k, const float* v, long long row_stride,
                                       const float* head_decay, int in_silu, float* state, long long slot_stride, int max_slots,
                                       const int32_t* cu_tokens, const int32_t* state_slots, int num_reqs,
                                       float* out, int heads, int D, int Dv, float q_scale, float* work, int max_segments, int* err,
                                       cudaStream_t stream) {
    if (!head_decay) return AIRUN_ERR_ARG;
    return gla_recurrent_launch(q, k, v, row_stride, nullptr, head_decay, in_silu, state, slot_stride, max_slots, cu_tokens,
                                state_slots, num_reqs, out, heads, D, Dv, q_scale, work, max_segments, err, stream);
}

// out[t][c] = scale * o[t][c] / sqrt(mean_c o[t]^2 + eps) * w[c] * sigmoid(gate[t][c]) over a token's whole row of n
// numbers (all heads at once); one block per token.  o is float32 [T][n], gate float32 rows of `gate_stride`.
template <typename TOut>
__global__ __launch_bounds__(256) void rownorm_gate_kernel(const float* o, const float* gate,
                                                           long long gate_stride, const float* __restrict__ w,
                                                           TOut* __restrict__ out, long long out_stride, int n, float eps,
                                                           float scale, const int32_t* __restrict__ req_of_token) {
    pdl_trigger();
    pdl_wait();
    __shared__ float red[33];
    const int t = blockIdx.x;
    if (req_of_token[t] < 0) return;
    const float* orow = o + (size_t)t * n;
    float ss = 0.0f;
    for (int c = threadIdx.x; c < n; c += blockDim.x) ss = fmaf(orow[c], orow[c], ss);
    ss = block_sum(ss, red);
    const float inv = scale / sqrtf(ss / (float)n + eps);
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        const float g = gate ? 1.0f / (1.0f + expf(-gate[(size_t)t * gate_stride + c])) : 1.0f;
        out[(size_t)t * out_stride + c] = from_f32<TOut>(orow[c] * inv * (w ? w[c] : 1.0f) * g);
    }
}

AIRUN_EXPORT int airun_rownorm_gate(const float* o, const float* gate, long long gate_stride, const float* w, void* out,
                                    int out_dtype, long long out_stride, int T, int n, float eps, float scale,
                                    const int32_t* req_of_token, cudaStream_t stream) {
    if (T < 0 || n <= 0 || !o || !out || !req_of_token || out_stride < n || (gate && gate_stride < n)) return AIRUN_ERR_ARG;
    if (T == 0) return AIRUN_OK;
    if (out_dtype == AIRUN_DT_F32)
        airun_launch(rownorm_gate_kernel<float>, dim3(T), dim3(256), 0, stream, o, gate, gate_stride, w, (float*)out, out_stride, n, eps, scale, req_of_token);
    else if (out_dtype == AIRUN_DT_BF16)
        airun_launch(rownorm_gate_kernel<__nv_bfloat16>, dim3(T), dim3(256), 0, stream, o, gate, gate_stride, w, (__nv_bfloat16*)out, out_stride, n, eps, scale, req_of_token);
    else
        return AIRUN_ERR_UNSUPPORTED;
    return airun_launch_status();
}

// out[t][h][j] = o[t][h][j] / sqrt(mean_j o^2 + eps) * w[j] * silu(gate[t][h][j]); one warp per (token, head).
template <typename TOut>
__global__ __launch_bounds__(128) void out_gate_kernel(const float* o, const float* gate,
                                                       long long gate_stride, const float* __restrict__ w,
                                                       TOut* __restrict__ out, long long out_stride, int T, int heads,
                                                       int Dv, float eps, const int32_t* __restrict__ req_of_token,
                                                       int gate_act, int w_per_head) {
    pdl_trigger();
    pdl_wait();
    const int unit = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (unit >= T * heads) return;
    const int t = unit / heads, h = unit - t * heads;
    if (req_of_token[t] < 0) return;
    if (w && w_per_head) w += (size_t)h * Dv;
    // the gate: silu(g) (0), sigmoid(g) (1), or g as it is (2: the caller has applied its function already)
    auto gf = [&](float g) { return gate_act == 0 ? g / (1.0f + expf(-g)) : gate_act == 1 ? 1.0f / (1.0f + expf(-g)) : g; };
    const float* orow = o + ((size_t)t * heads + h) * Dv;
    const float* grow = gate + (size_t)t * gate_stride + (size_t)h * Dv;
    TOut* dst = out + (size_t)t * out_stride + (size_t)h * Dv;
    if (Dv <= 128 && Dv % 4 == 0 && ((((uintptr_t)orow | (uintptr_t)grow) & 15) == 0)) {
        // a lane takes four values: both loads are issued before anything is used
        const bool on = lane * 4 < Dv;
        float4 ov = make_float4(0.0f, 0.0f, 0.0f, 0.0f), gv = ov, wv = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        if (on) {
            ov = *reinterpret_cast<const float4*>(orow + lane * 4);
            gv = *reinterpret_cast<const float4*>(grow + lane * 4);
            if (w) wv = make_float4(w[lane * 4], w[lane * 4 + 1], w[lane * 4 + 2], w[lane * 4 + 3]);
        }
        const float ss4 = warp_sum(ov.x * ov.x + ov.y * ov.y + ov.z * ov.z + ov.w * ov.w);
        const float inv4 = 1.0f / sqrtf(ss4 / (float)Dv + eps);
        if (on) {
            dst[lane * 4 + 0] = from_f32<TOut>(ov.x * inv4 * wv.x * gf(gv.x));
            dst[lane * 4 + 1] = from_f32<TOut>(ov.y * inv4 * wv.y * gf(gv.y));
            dst[lane * 4 + 2] = from_f32<TOut>(ov.z * inv4 * wv.z * gf(gv.z));
            dst[lane * 4 + 3] = from_f32<TOut>(ov.w * inv4 * wv.w * gf(gv.w));
        }
        return;
    }
    float ss = 0.0f;
    for (int j = lane; j < Dv; j += 32) ss = fmaf(orow[j], orow[j], ss);
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)Dv + eps);
    for (int j = lane; j < Dv; j += 32) {
        const float g = grow[j];
        dst[j] = from_f32<TOut>(orow[j] * inv * (w ? w[j] : 1.0f) * gf(g));
    }
}

AIRUN_EXPORT int airun_gla_out_gate(const float* o, const float* gate, long long gate_stride, const float* w, void* out,
                                    int out_dtype, long long out_stride, int T, int heads, int Dv, float eps,
                                    const int32_t* req_of_token, int gate_act, int w_per_head, cudaStream_t stream) {
    if (T < 0 || heads <= 0 || Dv <= 0 || !req_of_token || out_stride < (long long)heads * Dv) return AIRUN_ERR_ARG;
    if (T == 0) return AIRUN_OK;
    const int blocks = ceil_div_i((long long)T * heads, 4);
    if (out_dtype == AIRUN_DT_F32)
        airun_launch(out_gate_kernel<float>, dim3(blocks), dim3(128), 0, stream, o, gate, gate_stride, w, (float*)out, out_stride, T, heads, Dv, eps, req_of_token, gate_act, w_per_head);
    else if (out_dtype == AIRUN_DT_BF16)
        airun_launch(out_gate_kernel<__nv_bfloat16>, dim3(blocks), dim3(128), 0, stream, o, gate, gate_stride, w, (__nv_bfloat16*)out, out_stride, T, heads, Dv, eps, req_of_token, gate_act, w_per_head);
    else
        return AIRUN_ERR_UNSUPPORTED;
    return airun_launch_status();
}
