// Causal attention over cache pages, any sizes, float32 arithmetic.
//
// One block per (token, query head).  Each warp walks every ATTN_WARPS-th
// visible key with a running maximum and sum (online softmax), lanes hold the
// head dimensions; the warps' partial results are merged at the end.  This is
// the shape of the reference's generic streaming kernel
// (crates/airun-cuda/kernels/ops.cu:524-645): head h reads KV head
// h / (n_heads / n_kv_heads); s_j = scale * (q . K_j); key j is visible iff
// j <= pos and, with a window w > 0, pos - j < w (ops.cu:573-576); a row that
// sees nothing yields 0 (ops.cu:626).  The accurate expf is used.
//
// It is the attention of the true 32-bit path (float32 q and pages) and, with
// bfloat16 storage, the plain twin of the tensor-core kernels.  The result for
// a token depends only on its own q, position and the keys it sees, not on the
// batch around it.
#include "common.cuh"

#define ATTN_WARPS 4
#define MAX_PER_LANE 8   // head_dim <= 256

template <typename TQ, typename TKV>
__global__ __launch_bounds__(32 * ATTN_WARPS) void attention_generic_kernel(
    const TQ* q, TQ* __restrict__ out,
    const TKV* pool, const int32_t* __restrict__ block_table, int max_blocks,
    const int32_t* __restrict__ positions, const int32_t* __restrict__ req_of_token,
    int num_reqs, int num_pages, int page_size, int nh, int nkv, int hd,
    float scale, int window, int* __restrict__ err) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float smem[];
    float* s_max = smem;
    float* s_sum = smem + ATTN_WARPS;
    float* s_acc = smem + 2 * ATTN_WARPS;

    const int t = blockIdx.x, head = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = positions[t];
    const int req = req_of_token[t];
    TQ* dst = out + ((size_t)t * nh + head) * hd;
    if (req < 0 || pos < 0 || req >= num_reqs) {     // a padding row
        if (req >= num_reqs && threadIdx.x == 0) atomicOr(err, AIRUN_DEV_BAD_REQ);
        for (int d = threadIdx.x; d < hd; d += blockDim.x) dst[d] = from_f32<TQ>(0.0f);
        return;
    }
    const int kvh = head / (nh / nkv);
    const TQ* qv = q + ((size_t)t * nh + head) * hd;
    float qreg[MAX_PER_LANE], acc[MAX_PER_LANE];
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
        const int d = lane + i * 32;
        qreg[i] = d < hd ? to_f32<TQ>(qv[d]) : 0.0f;
        acc[i] = 0.0f;
    }
    float run_max = -INFINITY, run_sum = 0.0f;
    const int32_t* bt = block_table + (size_t)req * max_blocks;
    const int begin = window > 0 ? max(0, pos - window + 1) : 0;
    bool bad = false;
    for (int j = begin + warp; j <= pos; j += ATTN_WARPS) {
        const int blk = j / page_size;
        const int page = blk < max_blocks ? bt[blk] : -1;
        if (page < 0 || page >= num_pages) { bad = true; continue; }
        const TKV* kj = pool + (((size_t)page * 2 * nkv + kvh) * page_size + (j % page_size)) * hd;
        const TKV* vj = kj + (size_t)nkv * page_size * hd;
        float dot = 0.0f;
#pragma unroll
        for (int i = 0; i < MAX_PER_LANE; ++i) {
            const int d = lane + i * 32;
            if (d < hd) dot = fmaf(qreg[i], to_f32<TKV>(kj[d]), dot);
        }
        dot = warp_sum(dot) * scale;
        const float new_max = fmaxf(run_max, dot);
        const float corr = expf(run_max - new_max);    // exactly 0 on the first key
        const float p = expf(dot - new_max);
        run_sum = run_sum * corr + p;
#pragma unroll
        for (int i = 0; i < MAX_PER_LANE; ++i) {
            const int d = lane + i * 32;
            if (d < hd) acc[i] = fmaf(p, to_f32<TKV>(vj[d]), acc[i] * corr);
        }
        run_max = new_max;
    }
    if (bad && lane == 0) atomicOr(err, AIRUN_DEV_BAD_PAGE);
    if (lane == 0) { s_max[warp] = run_max; s_sum[warp] = run_sum; }
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
        const int d = lane + i * 32;
        if (d < hd) s_acc[(size_t)warp * hd + d] = acc[i];
    }
    __syncthreads();
    if (warp != 0) return;
    float gmax = -INFINITY;
#pragma unroll
    for (int w = 0; w < ATTN_WARPS; ++w) gmax = fmaxf(gmax, s_max[w]);
    float weight[ATTN_WARPS], gsum = 0.0f;
#pragma unroll
    for (int w = 0; w < ATTN_WARPS; ++w) {
        weight[w] = s_sum[w] > 0.0f ? expf(s_max[w] - gmax) : 0.0f;
        gsum += s_sum[w] * weight[w];
    }
    const float inv = gsum > 0.0f ? 1.0f / gsum : 0.0f;
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
        const int d = lane + i * 32;
        if (d >= hd) continue;
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < ATTN_WARPS; ++w) v = fmaf(s_acc[(size_t)w * hd + d], weight[w], v);
        dst[d] = from_f32<TQ>(v * inv);
    }
}

// float32, head sizes 32, 64 and 128: a block per (token, KV head, up to four of its query heads), so a key or value row
// that is loaded serves them all (the kernel above reads it once per query head, and at 642 tokens x 16 heads that, with
// one key at a time a warp, is what bounds it: nine launches, three of them for 642 tokens of three prompts, took 1,475 us
// and take 324 us here).  A warp takes
// KEYS neighbouring keys at a time: the GH x KEYS dot products are reduced together by halving exchanges, every lane forms the
// exponential of the one it ends with, and the weights are handed round.
#define ROWS_WARPS 8
template <int PL> struct LaneVec { float v[PL]; };
template <int PL> __device__ __forceinline__ LaneVec<PL> lane_load(const float* p) {
    LaneVec<PL> r;
    if constexpr (PL == 4) { const float4 t = *reinterpret_cast<const float4*>(p); r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w; }
    else if constexpr (PL == 2) { const float2 t = *reinterpret_cast<const float2*>(p); r.v[0] = t.x; r.v[1] = t.y; }
    else r.v[0] = *p;
    return r;
}

template <int PL, int GH>
__global__ __launch_bounds__(32 * ROWS_WARPS) void attention_rows_f32_kernel(
    const float* q, float* __restrict__ out, const float* pool,
    const int32_t* __restrict__ block_table, int max_blocks, const int32_t* __restrict__ positions,
    const int32_t* __restrict__ req_of_token, int num_reqs, int num_pages, int page_size, int nh, int nkv,
    float scale, int window, int* __restrict__ err) {
    constexpr int HD = PL * 32, KEYS = GH == 4 ? 2 : 4, NV = GH * KEYS;      // NV scores at a time: 8, 8 or 4
    pdl_trigger();
    pdl_wait();
    __shared__ float s_max[ROWS_WARPS][GH], s_sum[ROWS_WARPS][GH];
    __shared__ float s_acc[ROWS_WARPS][GH][HD];
    const int t = blockIdx.x, G = nh / nkv, kvh = blockIdx.y % nkv;
    const int head0 = kvh * G + blockIdx.y / nkv * GH, heads = min(GH, kvh * G + G - head0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = positions[t], req = req_of_token[t];
    float* dst = out + ((size_t)t * nh + head0) * HD;
    if (req < 0 || pos < 0 || req >= num_reqs) {               // a padding row
        if (req >= num_reqs && threadIdx.x == 0) atomicOr(err, AIRUN_DEV_BAD_REQ);
        for (int d = threadIdx.x; d < heads * HD; d += blockDim.x) dst[d] = 0.0f;
        return;
    }
    float qr[GH][PL], acc[GH][PL];
#pragma unroll
    for (int h = 0; h < GH; ++h) {
        const LaneVec<PL> v = lane_load<PL>(q + ((size_t)t * nh + head0 + min(h, heads - 1)) * HD + lane * PL);
#pragma unroll
        for (int i = 0; i < PL; ++i) { qr[h][i] = v.v[i] * scale; acc[h][i] = 0.0f; }
    }
    // lane l keeps the maximum and the sum of the head whose score it ends with: score h * KEYS + u, neighbouring lanes alike
    constexpr int SAME = 32 / NV;
    const int mine = lane / SAME, my_head = mine / KEYS;
    float run_max = -INFINITY, run_sum = 0.0f;
    const int32_t* bt = block_table + (size_t)req * max_blocks;
    const int begin = window > 0 ? max(0, pos - window + 1) : 0;
    bool bad = false;
    for (int j0 = begin + warp * KEYS; j0 <= pos; j0 += ROWS_WARPS * KEYS) {
        LaneVec<PL> kv[KEYS], vv[KEYS];
        unsigned on = 0;
#pragma unroll
        for (int u = 0; u < KEYS; ++u) {
            const int j = j0 + u, blk = j / page_size;
            const int page = j <= pos && blk < max_blocks ? bt[blk] : -1;
            const bool ok = page >= 0 && page < num_pages;
            if (j <= pos && !ok) bad = true;
            on |= ok ? 1u << u : 0u;
            // (a key that is not there is not read: its weight of zero would not make a NaN of another request harmless)
#pragma unroll
            for (int i = 0; i < PL; ++i) kv[u].v[i] = vv[u].v[i] = 0.0f;
            if (ok) {
                const float* kj = pool + (((size_t)page * 2 * nkv + kvh) * page_size + j % page_size) * HD + lane * PL;
                kv[u] = lane_load<PL>(kj);
                vv[u] = lane_load<PL>(kj + (size_t)nkv * page_size * HD);
            }
        }
        float s[NV];
#pragma unroll
        for (int h = 0; h < GH; ++h)
#pragma unroll
            for (int u = 0; u < KEYS; ++u) {
                float dot = 0.0f;
#pragma unroll
                for (int i = 0; i < PL; ++i) dot = fmaf(qr[h][i], kv[u].v[i], dot);
                s[h * KEYS + u] = dot;
            }
        int n = NV;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            if (n > 1) {
                n >>= 1;
                const bool up = lane & o;
#pragma unroll
                for (int i = 0; i < NV / 2; ++i) {
                    if (i >= n) break;
                    const float send = up ? s[i] : s[i + n], keep = up ? s[i + n] : s[i];
                    s[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            } else {
                s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
            }
        }
        const float score = (on >> (mine % KEYS)) & 1u ? s[0] : -INFINITY;
        float top = score;
#pragma unroll
        for (int o = SAME; o < SAME * KEYS; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float new_max = fmaxf(run_max, top);
        const float p = score == -INFINITY ? 0.0f : expf(score - new_max);
        if (__any_sync(0xffffffffu, new_max > run_max)) {
            const float corr = run_max == -INFINITY ? 0.0f : expf(run_max - new_max);
            run_sum *= corr;
#pragma unroll
            for (int h = 0; h < GH; ++h) {
                const float c = __shfl_sync(0xffffffffu, corr, h * KEYS * SAME);
#pragma unroll
                for (int i = 0; i < PL; ++i) acc[h][i] *= c;
            }
            run_max = new_max;
        }
        run_sum += p;
#pragma unroll
        for (int h = 0; h < GH; ++h)
#pragma unroll
            for (int u = 0; u < KEYS; ++u) {
                const float w = __shfl_sync(0xffffffffu, p, (h * KEYS + u) * SAME);
#pragma unroll
                for (int i = 0; i < PL; ++i) acc[h][i] = fmaf(w, vv[u].v[i], acc[h][i]);
            }
    }
    if (bad && lane == 0) atomicOr(err, AIRUN_DEV_BAD_PAGE);
    // a lane's sum is over its own one of KEYS keys: the others' lie SAME lanes apart
#pragma unroll
    for (int o = SAME; o < SAME * KEYS; o <<= 1) run_sum += __shfl_xor_sync(0xffffffffu, run_sum, o);
    if (lane % (SAME * KEYS) == 0) { s_max[warp][my_head] = run_max; s_sum[warp][my_head] = run_sum; }
#pragma unroll
    for (int h = 0; h < GH; ++h)
#pragma unroll
        for (int i = 0; i < PL; ++i) s_acc[warp][h][lane * PL + i] = acc[h][i];
    __syncthreads();
    for (int e = threadIdx.x; e < heads * HD; e += 32 * ROWS_WARPS) {
        const int h = e / HD, d = e % HD;
        float gmax = -INFINITY, gsum = 0.0f, v = 0.0f;
#pragma unroll
        for (int w = 0; w < ROWS_WARPS; ++w) gmax = fmaxf(gmax, s_max[w][h]);
#pragma unroll
        for (int w = 0; w < ROWS_WARPS; ++w) {
            const float weight = s_sum[w][h] > 0.0f ? expf(s_max[w][h] - gmax) : 0.0f;
            gsum += s_sum[w][h] * weight;
            v = fmaf(s_acc[w][h][d], weight, v);
        }
        dst[e] = v * (gsum > 0.0f ? 1.0f / gsum : 0.0f);           // (a NaN in the sums stays one)
    }
}

// True when the kernel above took the call: float32, head sizes 32, 64, 128, 16-byte aligned q and pages.
static bool rows_f32(const void* q, void* out, int q_dtype, const void* pool, const int32_t* block_table, int max_blocks,
                     const int32_t* positions, const int32_t* req_of_token, int T, int num_reqs, int num_pages, int page_size,
                     int nh, int nkv, int hd, float scale, int window, int* err, cudaStream_t stream) {
    if (q_dtype != AIRUN_DT_F32 || (hd != 32 && hd != 64 && hd != 128) || (((uintptr_t)q | (uintptr_t)pool) & 15)) return false;
    const int G = nh / nkv, gh = G >= 3 ? 4 : G;
    const dim3 grid(T, nkv * ceil_div_i(G, gh));
    if (grid.y > 65535) return false;
#define ROWS(PL, GH) \
    airun_launch(attention_rows_f32_kernel<PL, GH>, grid, dim3(32 * ROWS_WARPS), 0, stream, (const float*)q, (float*)out, (const float*)pool, \
        block_table, max_blocks, positions, req_of_token, num_reqs, num_pages, page_size, nh, nkv, scale, window, err)
#define ROWS_GH(PL) do { if (gh == 1) ROWS(PL, 1); else if (gh == 2) ROWS(PL, 2); else ROWS(PL, 4); } while (0)
    if (hd == 32) ROWS_GH(1);
    else if (hd == 64) ROWS_GH(2);
    else ROWS_GH(4);
#undef ROWS_GH
#undef ROWS
    return true;
}

AIRUN_EXPORT int airun_attention_generic(
    const void* q, void* out, int q_dtype, const void* pool, int kv_dtype,
    const int32_t* block_table, int max_blocks,
    const int32_t* positions, const int32_t* req_of_token, int T, int num_reqs,
    int num_pages, int page_size, int nh, int nkv, int hd, float scale, int window,
    int* err, cudaStream_t stream) {
    if (T < 0 || nh <= 0 || nkv <= 0 || nh % nkv != 0 || hd <= 0 || hd > 32 * MAX_PER_LANE ||
        page_size <= 0 || num_pages <= 0 || max_blocks <= 0 || window < 0 || !err)
        return AIRUN_ERR_ARG;
    if (q_dtype != kv_dtype) return AIRUN_ERR_UNSUPPORTED;
    if (T == 0) return AIRUN_OK;
    if (nh > 65535) return AIRUN_ERR_ARG;
    if (rows_f32(q, out, q_dtype, pool, block_table, max_blocks, positions, req_of_token, T, num_reqs, num_pages, page_size, nh, nkv, hd,
                 scale, window, err, stream))
        return airun_launch_status();
    dim3 grid(T, nh);
    const size_t smem = (size_t)ATTN_WARPS * (2 + hd) * sizeof(float);
#define LAUNCH(TQ, TKV) \
    airun_launch(attention_generic_kernel<TQ, TKV>, dim3(grid), dim3(32 * ATTN_WARPS), smem, stream, (const TQ*)q, (TQ*)out, (const TKV*)pool, \
        block_table, max_blocks, positions, req_of_token, num_reqs, num_pages, page_size, nh, nkv, hd, scale, window, err)
    if (q_dtype == AIRUN_DT_F32) LAUNCH(float, float);
    else if (q_dtype == AIRUN_DT_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16);
    else return AIRUN_ERR_UNSUPPORTED;
#undef LAUNCH
    return airun_launch_status();
}
