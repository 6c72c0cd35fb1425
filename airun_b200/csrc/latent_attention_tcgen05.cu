// Attention over a cached latent on the 5th-generation tensor cores, for prompt portions.  The formulas are those of
// latent_attention.cu, the plain twin: every token caches ONE row of R + rd elements that all heads share; the score of a
// query row and a cached row is their product over all R + rd elements, the value is the row's first R.
//
// A CTA takes up to 128 (token, head) rows of one request and up to four blocks of 64 output columns (two CTAs share a tile
// of rows when R is above 256: the scores are formed twice, since S and 512 columns of O do not fit the 512 columns of
// tensor memory).  The query rows stay in shared memory (144 KB at R + rd = 576), cached rows come in tiles of 64:
//   warp 0   : one elected thread issues TMA loads (64 elements x 16 rows a box, 128-byte swizzle), the blocks this CTA does not
//              need as values first;
//   warp 1   : one elected thread issues tcgen05.mma: S = Q K^T over all blocks into one of two S buffers, O += P V with P from tensor
//              memory and V the first blocks of the SAME shared-memory tile as an MN-major operand.  The blocks that are no
//              values are free as soon as S has read them, so the next tile's arrive, and its S is begun, while the softmax
//              works; the value blocks are free after O;
//   warps 2-5: a thread a row: running maximum and sum in float32 (exp2), P as bfloat16 over S, O rescaled lazily.
// The mma.sync kernel reads the whole tile of cached rows from shared memory once per warp, for 16 rows: 509 us for one
// 1,536-token prompt of 16 heads (R = 512, rd = 64), 323 for three of 811 to 540; here 168 and 122 us.  What bounds it now is bringing 72 KB of cached rows into
// an SM for 128 rows of queries.
//
// Every mbarrier wait is bounded (about two seconds); on a time-out the kernel sets an error bit, stops working, frees its
// tensor memory and returns.  No cluster, no multicast.
#include "tcgen05.cuh"
#include <mutex>
#include <unordered_map>

#define LT_ROWS 128
#define LT_KEYS 64
#define LT_THREADS 192
#define LT_QBLK (LT_ROWS * 128)   // bytes of a block of 64 elements of 128 query rows
#define LT_KBLK (LT_KEYS * 128)   // and of 64 cached rows
#define LT_MAX_BLOCKS 9
#define NEG_BIG (-1.0e30f)
#define LOG2E 1.4426950408889634f

namespace {

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// descriptors as (low word, high word): an offset is one add on the low word (units of 16 bytes)
__device__ __forceinline__ void umma_ss(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
        ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(d), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr),
          "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// K-major operand, rows of 128 bytes with the 128-byte swizzle: 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// MN-major operand: 64 columns are contiguous, the next 64 a block of LT_KBLK bytes further on; along K rows of 128 bytes
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)(LT_KBLK >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

struct LatParams {
    __nv_bfloat16* out;            // [T][H][R]
    const int32_t* block_table;    // [requests][max_blocks]
    const int32_t* positions;      // [T]
    int max_blocks, num_pages, page_size, page_shift, H, R, blocks, vblocks, stages;      // blocks: (R + rd) / 64; vblocks: R / 64
    float scale_log2;
    int window;
    const float* sink;             // [H] or null
    const float* gate;             // [T][gate_stride] or null: head h's result is times sigmoid(gate[t][h])
    long long gate_stride;
    int* err;
};

enum { L_QFULL = 0, L_NFULL = 1, L_NEMPTY = 3, L_VFULL = 5, L_VEMPTY = 7, L_SFULL = 9, L_PFULL = 11, L_FINAL = 12, L_BARS = 13 };

__global__ __launch_bounds__(LT_THREADS, 1) void latent_prefill_kernel(
    const LatParams p, const int4* tiles, const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
    const int* n_tiles_dev) {
    pdl_trigger();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* const smem_k = smem + p.blocks * LT_QBLK;
    __shared__ uint64_t bars[L_BARS];
    __shared__ uint32_t tmem_slot;
    const uint32_t bar0 = smem_u32(bars);
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < L_BARS; ++i) mbar_init(BAR(i), i == L_PFULL ? 4 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    const uint32_t tmem_o = tmem_base + 2 * LT_KEYS;
    pdl_wait();
    // the halves of a tile before the next tile: the tiles with the most keys start first
    const int lin = (int)(blockIdx.y * gridDim.x + blockIdx.x);
    const int tile_idx = lin / (int)gridDim.y, half = lin % (int)gridDim.y;
    if (tile_idx < load_fresh(n_tiles_dev)) {
        const int4 t4 = load_fresh(tiles + tile_idx);
        const int req = t4.x, tok0 = t4.y, n_rows = t4.z * p.H;
        const int pos_lo = p.positions[tok0], pos_hi = p.positions[tok0 + t4.z - 1];
        const int k_first = p.window > 0 ? max(0, pos_lo - p.window + 1) : 0;
        const int tile_first = k_first / LT_KEYS;
        const int n_tiles = pos_hi >= 0 ? pos_hi / LT_KEYS - tile_first + 1 : 0;
        // this CTA's value blocks [v0, v0 + nv); they take the first places of a tile's stage, the other blocks the rest
        const int per = (p.vblocks + (int)gridDim.y - 1) / (int)gridDim.y, v0 = half * per, nv = min(per, p.vblocks - v0), nn = p.blocks - nv;
        auto other = [&](int i) { return i < v0 ? i : i + nv; };       // the i-th block that is no value here

        if (warp == 0) {
            {
                if (elect_one()) {
                    mbar_expect_tx(BAR(L_QFULL), (uint32_t)(p.blocks * LT_QBLK));
                    for (int b = 0; b < p.blocks; ++b) tma_load_2d(smem_u32(smem + b * LT_QBLK), &q_map, BAR(L_QFULL), b * 64, tok0 * p.H);
                }
                __syncwarp();
                const int32_t* bt = p.block_table + (size_t)req * p.max_blocks;
                for (int it = 0; it < n_tiles; ++it) {
                    const int s = it % p.stages;
                    const uint32_t ph = (uint32_t)(it / p.stages) & 1u;
                    const uint32_t dst = smem_u32(smem_k + s * p.blocks * LT_KBLK);
                    int rows[LT_KEYS / 16];
#pragma unroll
                    for (int g = 0; g < LT_KEYS / 16; ++g) {
                        const int j = (tile_first + it) * LT_KEYS + g * 16, blk = j >> p.page_shift;
                        int page = (j <= pos_hi && blk < p.max_blocks) ? __ldg(bt + blk) : 0;
                        if (page < 0 || page >= p.num_pages) {
                            if (j + 15 >= k_first && lane == 0) atomicOr(p.err, AIRUN_DEV_BAD_PAGE);      // a page the window has passed may be gone
                            page = 0;
                        }
                        rows[g] = (page << p.page_shift) + (j & (p.page_size - 1));
                    }
                    if (nn) {
                        if (!mbar_wait_warp(BAR(L_NEMPTY + s), ph ^ 1)) { if (lane == 0) atomicOr(p.err, AIRUN_DEV_TIMEOUT); break; }
                        if (elect_one()) {
                            mbar_expect_tx(BAR(L_NFULL + s), (uint32_t)(nn * LT_KBLK));
                            for (int i = 0; i < nn; ++i)
#pragma unroll
                                for (int g = 0; g < LT_KEYS / 16; ++g)
                                    tma_load_2d(dst + (nv + i) * LT_KBLK + g * 2048, &k_map, BAR(L_NFULL + s), other(i) * 64, rows[g]);
                        }
                        __syncwarp();
                    }
                    if (!mbar_wait_warp(BAR(L_VEMPTY + s), ph ^ 1)) { if (lane == 0) atomicOr(p.err, AIRUN_DEV_TIMEOUT); break; }
                    if (elect_one()) {
                        mbar_expect_tx(BAR(L_VFULL + s), (uint32_t)(nv * LT_KBLK));
                        for (int i = 0; i < nv; ++i)
#pragma unroll
                            for (int g = 0; g < LT_KEYS / 16; ++g)
                                tma_load_2d(dst + i * LT_KBLK + g * 2048, &k_map, BAR(L_VFULL + s), (v0 + i) * 64, rows[g]);
                    }
                    __syncwarp();
                }
            }
        } else if (warp == 1) {
            {
                constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_KEYS >> 3) << 17) | ((uint32_t)(LT_ROWS >> 4) << 24);
                const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(nv * 64 >> 3) << 17) | ((uint32_t)(LT_ROWS >> 4) << 24);
                const uint64_t qd = desc_kmajor(smem_u32(smem)), kd = desc_kmajor(smem_u32(smem_k)), vd = desc_mnmajor(smem_u32(smem_k));
                const uint32_t q_lo = (uint32_t)qd, k_lo = (uint32_t)kd, k_hi = (uint32_t)(kd >> 32), v_lo = (uint32_t)vd, v_hi = (uint32_t)(vd >> 32);
                auto issue_block = [&](int it, int block, int place, bool first) {          // S += Q block * K block
                    const uint32_t a = q_lo + (uint32_t)(block * (LT_QBLK >> 4));
                    const uint32_t b = k_lo + (uint32_t)(((it % p.stages) * p.blocks + place) * (LT_KBLK >> 4));
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_ss(tmem_base + (it & 1) * LT_KEYS, a + 2 * k, b + 2 * k, k_hi, idesc_s, first && k == 0 ? 0u : 1u);
                };
                auto issue_n = [&](int it) -> bool {
                    if (!nn) return true;
                    const int s = it % p.stages;
                    if (!mbar_wait_warp(BAR(L_NFULL + s), (uint32_t)(it / p.stages) & 1u)) return false;
                    tc_fence_after();
                    if (elect_one()) {
                        for (int i = 0; i < nn; ++i) issue_block(it, other(i), nv + i, i == 0);
                        umma_commit(BAR(L_NEMPTY + s));
                    }
                    __syncwarp();
                    return true;
                };
                auto issue_v = [&](int it) -> bool {
                    const int s = it % p.stages;
                    if (!mbar_wait_warp(BAR(L_VFULL + s), (uint32_t)(it / p.stages) & 1u)) return false;
                    tc_fence_after();
                    if (elect_one()) {
                        for (int i = 0; i < nv; ++i) issue_block(it, v0 + i, i, nn == 0 && i == 0);
                        umma_commit(BAR(L_SFULL + (it & 1)));
                    }
                    __syncwarp();
                    return true;
                };
                bool ok = mbar_wait_warp(BAR(L_QFULL), 0);
                if (ok && n_tiles > 0) ok = issue_n(0) && issue_v(0);
                for (int it = 0; it < n_tiles && ok; ++it) {
                    if (it + 1 < n_tiles) ok = issue_n(it + 1);
                    if (!ok || !mbar_wait_warp(BAR(L_PFULL), it & 1)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t v = v_lo + (uint32_t)((it % p.stages) * p.blocks * (LT_KBLK >> 4));
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < LT_KEYS / 16; ++k)        // 16 keys of P are 8 columns of packed pairs
                            umma_ts(tmem_o, tmem_base + (it & 1) * LT_KEYS + 8 * k, v + k * (2048 >> 4), v_hi, idesc_o, it > 0 || k > 0 ? 1u : 0u);
                        umma_commit(BAR(L_VEMPTY + it % p.stages));
                    }
                    __syncwarp();
                    if (it + 1 < n_tiles) ok = issue_v(it + 1);
                }
                if (elect_one()) {
                    if (ok) umma_commit(BAR(L_FINAL));
                    else atomicOr(p.err, AIRUN_DEV_TIMEOUT);
                }
                __syncwarp();
            }
        } else {
            const int quad = warp & 3, r = quad * 32 + lane;
            const bool row_ok = r < n_rows;
            const int tok = tok0 + (row_ok ? r / p.H : 0), head = row_ok ? r % p.H : 0;
            const int pos = row_ok ? p.positions[tok] : -1;
            const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
            const uint32_t o_addr = tmem_o + lane_off;
            float m = NEG_BIG, l = 0.0f;
            bool ok = true;
            const float sc = p.scale_log2;
            for (int it = 0; it < n_tiles; ++it) {
                if (!mbar_wait(BAR(L_SFULL + (it & 1)), (uint32_t)(it >> 1) & 1u)) { ok = false; break; }
                tc_fence_after();
                const uint32_t s_addr = tmem_base + lane_off + (it & 1) * LT_KEYS;
                uint32_t raw[LT_KEYS];
                tmem_ld32_async(s_addr, raw);
                tmem_ld32_async(s_addr + 32, raw + 32);
                tmem_wait32(raw);
                tmem_wait32(raw + 32);
                const int j0 = (tile_first + it) * LT_KEYS;
                if (r < LT_KEYS && (j0 + r < k_first || j0 + r > pos_hi)) {
                    // A cached row that no token of the tile sees may be another request's or left over: as zeros its values add
                    // nothing, as NaN times a weight of zero they would be NaN.  S has been formed, so all blocks have landed.
                    uint8_t* const row = smem_k + (it % p.stages) * p.blocks * LT_KBLK + r * 128;
                    for (int b = 0; b < nv; ++b)
#pragma unroll
                        for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(row + b * LT_KBLK + c * 16) = make_uint4(0, 0, 0, 0);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                __syncwarp();
                float v[LT_KEYS];
                const bool full = p.window == 0 && j0 + LT_KEYS - 1 <= pos_lo;      // every key visible to every row
#pragma unroll
                for (int i = 0; i < LT_KEYS; ++i) {
                    v[i] = __uint_as_float(raw[i]);
                    if (!full) {
                        const int j = j0 + i;
                        if (!(j <= pos && (p.window == 0 || pos - j < p.window))) v[i] = -INFINITY;      // hidden under every scale above 0
                    }
                }
                float r0 = NEG_BIG, r1 = NEG_BIG, r2 = NEG_BIG, r3 = NEG_BIG;
#pragma unroll
                for (int i = 0; i < LT_KEYS; i += 4) {
                    r0 = fmaxf(r0, v[i]); r1 = fmaxf(r1, v[i + 1]); r2 = fmaxf(r2, v[i + 2]); r3 = fmaxf(r3, v[i + 3]);
                }
                const float top = fmaxf(fmaxf(r0, r1), fmaxf(r2, r3));
                const float mx = top > 0.5f * NEG_BIG ? top * sc : NEG_BIG;
                const bool raise = mx > m + 8.0f;
                if (it == 0) {
                    m = mx;                                              // nothing accumulated yet
                } else if (__any_sync(0xffffffffu, raise)) {
                    const float f = raise ? exp2f(m - mx) : 1.0f;          // rescale this warp's rows of O
                    for (int c = 0; c < nv * 64; c += 32) {
                        uint32_t t[32];
                        tmem_ld32_async(o_addr + c, t);
                        tmem_wait32(t);
#pragma unroll
                        for (int i = 0; i < 32; ++i) t[i] = __float_as_uint(__uint_as_float(t[i]) * f);
                        tmem_st32(o_addr + c, t);
                    }
                    l *= f;
                    if (raise) m = mx;
                }
                // hidden keys are minus infinity and come out as 0; a row that has seen no key at all must not add its -m
                const float nm = m > 0.5f * NEG_BIG ? -m : 0.0f;
                const float2 sc2 = make_float2(sc, sc), nm2 = make_float2(nm, nm);
                float2 rs2 = make_float2(0.0f, 0.0f);
                uint32_t pw[LT_KEYS / 2];
#pragma unroll
                for (int i = 0; i < LT_KEYS / 2; ++i) {
                    const float2 e = __ffma2_rn(make_float2(v[2 * i], v[2 * i + 1]), sc2, nm2);
                    const float2 pp = make_float2(exp2f(e.x), exp2f(e.y));
                    rs2 = __fadd2_rn(rs2, pp);
                    __nv_bfloat162 h2 = __floats2bfloat162_rn(pp.x, pp.y);
                    pw[i] = *reinterpret_cast<uint32_t*>(&h2);
                }
                tmem_st32(s_addr, pw);
                tmem_st_wait();
                l += rs2.x + rs2.y;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(L_PFULL));
            }
            if (ok && n_tiles > 0 && !mbar_wait(BAR(L_FINAL), 0)) ok = false;
            if (!ok) atomicOr(p.err, AIRUN_DEV_TIMEOUT);
            tc_fence_after();
            // the sink joins the denominator; if it is above every score the sums are scaled down to it
            const float sink2 = p.sink ? __ldg(p.sink + head) * LOG2E : NEG_BIG;
            const float top = fmaxf(m, sink2), f = m > 0.5f * NEG_BIG ? exp2f(m - top) : 0.0f;
            const float den = l * f + (p.sink ? exp2f(sink2 - top) : 0.0f);
            float inv = den > 0.0f ? f / den : 0.0f;
            if (p.gate && row_ok) inv /= 1.0f + __expf(-p.gate[(size_t)tok * p.gate_stride + head]);
            uint4* dst = reinterpret_cast<uint4*>(p.out + ((size_t)tok * p.H + head) * p.R + v0 * 64);
            for (int c = 0; c < nv * 64; c += 32) {
                uint32_t o[32];
                __syncwarp();
                if (ok && n_tiles > 0) {
                    tmem_ld32_async(o_addr + c, o);
                    tmem_wait32(o);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = 0u;
                }
                if (row_ok && ok) {
#pragma unroll
                    for (int q8 = 0; q8 < 4; ++q8) {
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(o[q8 * 8 + 2 * i]) * inv, __uint_as_float(o[q8 * 8 + 2 * i + 1]) * inv);
                            w[i] = *reinterpret_cast<uint32_t*>(&h2);
                        }
                        dst[c / 8 + q8] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// [rows][width] bfloat16, boxes of 64 elements x box_rows rows
int row_map(CUtensorMap* out, const void* ptr, long long rows, int width, int box_rows) {
    const EncodeTiledFn fn = encode_fn();
    if (!fn) return AIRUN_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)width * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? AIRUN_OK : AIRUN_ERR_ARG;
}

}  // namespace

// qlat [T][H][R + rd] and out [T][H][R] bfloat16, contiguous, 16-byte aligned; pool [pages][page_size][R + rd]; R and R + rd in
// multiples of 64, R up to 512, R + rd up to 576; H up to 128; pages of a power of two >= 16 tokens.  tiles: {request, first
// token, tokens (up to 128 / H), -}, of which *n_tiles_dev are in use.  scale > 0: the largest score of a row is taken ahead of
// the scaling.
AIRUN_EXPORT int airun_latent_prefill(const void* qlat, void* out, const void* pool, const int32_t* block_table, int max_blocks,
                                      const int32_t* positions, int T, int num_pages, int page_size, int H, int R, int rd, float scale,
                                      int window, const float* sink, const float* gate, long long gate_stride, const void* tiles,
                                      int n_tiles, const int32_t* n_tiles_dev, int* err, cudaStream_t stream) {
    const int KD = R + rd;
    if (T < 0 || n_tiles < 0 || H <= 0 || H > LT_ROWS || R <= 0 || rd < 0 || R % 64 || KD % 64 || R > 512 || KD > 64 * LT_MAX_BLOCKS || !err ||
        !n_tiles_dev || !(scale > 0.0f) || (gate && gate_stride < H) || (((uintptr_t)qlat | (uintptr_t)out | (uintptr_t)pool) & 15))
        return AIRUN_ERR_ARG;
    int shift = -1;
    for (int s = 4; s < 20; ++s) if ((1 << s) == page_size) shift = s;
    if (shift < 0) return AIRUN_ERR_UNSUPPORTED;
    if (T == 0 || n_tiles == 0) return AIRUN_OK;
    LatParams p;
    p.out = (__nv_bfloat16*)out; p.block_table = block_table; p.positions = positions; p.max_blocks = max_blocks; p.num_pages = num_pages;
    p.page_size = page_size; p.page_shift = shift; p.H = H; p.R = R; p.blocks = KD / 64; p.vblocks = R / 64;
    p.scale_log2 = scale * LOG2E; p.window = window; p.sink = sink; p.gate = gate; p.gate_stride = gate_stride; p.err = err;
    // two stages of cached rows where they fit; never less shared memory than keeps a second CTA, which would wait for the
    // same tensor memory, off the SM
    const int q_bytes = p.blocks * LT_QBLK, k_bytes = p.blocks * LT_KBLK;
    p.stages = q_bytes + 2 * k_bytes + 1024 <= 226 * 1024 ? 2 : 1;
    int smem = q_bytes + p.stages * k_bytes + 1024;
    if (smem < 120 * 1024) smem = 120 * 1024;
    CUtensorMap qm, km;
    int r = row_map(&qm, qlat, (long long)T * H, KD, LT_ROWS);
    if (r == AIRUN_OK) r = row_map(&km, pool, (long long)num_pages * page_size, KD, 16);
    if (r != AIRUN_OK) return r;
    static unsigned long long configured = 0;
    if (first_on_device(configured)) {
        const cudaError_t e = cudaFuncSetAttribute(latent_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
        if (e != cudaSuccess) return (int)e;
    }
    airun_launch(latent_prefill_kernel, dim3(n_tiles, (p.vblocks + 3) / 4), dim3(LT_THREADS), smem, stream, p, (const int4*)tiles, qm, km, n_tiles_dev);
    return airun_launch_status();
}
