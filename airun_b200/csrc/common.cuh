// Shared helpers of the sm_100a kernels: status codes, typed loads and stores,
// warp and block reductions.  Every entry point is extern "C", takes raw device
// pointers plus sizes and a stream, checks its arguments on the host and returns
// a status the Python side turns into an exception; it never allocates.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <math.h>
#include <stdlib.h>

#define AIRUN_OK 0
#define AIRUN_ERR_ARG 1000        // a size or pointer the kernel refuses
#define AIRUN_ERR_UNSUPPORTED 1001

// Bits of the device-side error word kernels set instead of trapping.
#define AIRUN_DEV_BAD_PAGE 1      // a block-table entry outside [0, num_pages)
#define AIRUN_DEV_BAD_REQ 2       // a token naming a request outside the batch
#define AIRUN_DEV_BAD_TOKEN 4     // a token id outside the vocabulary
#define AIRUN_DEV_TIMEOUT 8       // a bounded wait ran out
#define AIRUN_DEV_BAD_ROW 16      // a row of an expert, or a segment of a prompt, outside its buffer

#define AIRUN_DT_F32 0
#define AIRUN_DT_BF16 1

#define AIRUN_EXPORT extern "C" __attribute__((visibility("default")))

// Programmatic dependent launch: a kernel launched with the attribute may become resident while
// the kernel before it in the stream is still running; it must call pdl_wait() before it touches
// global memory that an earlier kernel writes or reads (the wait returns when the earlier kernels
// have finished and their writes are visible).  Every kernel calls pdl_trigger() first, which lets
// the kernel after it become resident as soon as room is free.  What a kernel does before
// pdl_wait() (shared-memory barriers, tensor-memory allocation, loads of WEIGHTS and of the batch's
// layout, which no kernel of a step writes) overlaps the tail of the kernel before it.  AIRUN_PDL=0 in
// the environment turns it off.
//
// const __restrict__ is for weights and the batch's layout only: it says that nothing writes there while the kernel
// lives, and a kernel lives from ahead of its wait on, so such loads may be moved ahead of the wait or answered from a
// line that the L1 cache has kept.  What the kernels of a step write (activations, cache pages, states, lists, counters)
// is read through plain pointers; results that a kernel does not read may be __restrict__.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Lists and counters of the kernel in front, which say where a kernel reads and writes, are read through volatile as well.
__device__ __forceinline__ int load_fresh(const int* p) { return *(const volatile int*)p; }
__device__ __forceinline__ int4 load_fresh(const int4* p) {
    const volatile int* v = (const volatile int*)p;
    return make_int4(v[0], v[1], v[2], v[3]);
}

// A weight that no kernel writes: on its way to the L2 cache while the kernel in front still runs.
__device__ __forceinline__ void prefetch_l2(const float* p, int n) {
    for (int i = threadIdx.x * 32; i < n; i += blockDim.x * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
}

// The warp's number, the same register for all lanes as the compiler sees it.
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
// True in one lane of a converged warp, the same one every time.  What issues tcgen05 and TMA instructions is a whole warp that loops and waits together, with
// elect_one() around the instructions alone: their operands (addresses, descriptors) are then uniform registers.  Behind `lane == 0` they have to be
// moved there one by one, 64 clocks a product and 250 a commit (B200: a step of four products 585 clocks, 280 with this).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}

static thread_local int airun_launch_rc = 0;

static inline bool airun_pdl_enabled() {
    static int on = -1;
    if (on < 0) {
        const char* e = getenv("AIRUN_PDL");
        on = (e && e[0] == '0') ? 0 : 1;
    }
    return on == 1;
}

template <typename... KArgs, typename... Args>
static inline void airun_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (airun_pdl_enabled()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
    if (e != cudaSuccess && airun_launch_rc == 0) airun_launch_rc = (int)e;
}

// The same once everything before it in the stream is done.  For kernels of fewer blocks than the chip holds at once whose
// blocks run long: blocks that become resident while the kernel in front still runs go where it leaves room, several to an
// SM while others stay empty, and stay there.
template <typename... KArgs, typename... Args>
static inline void airun_launch_after(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                      Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
    if (e != cudaSuccess && airun_launch_rc == 0) airun_launch_rc = (int)e;
}

// The same with thread-block clusters (the grid must be a multiple of them).
template <typename... KArgs, typename... Args>
static inline void airun_launch_clusters(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                         dim3 cluster, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster.x;
    attr[n].val.clusterDim.y = cluster.y;
    attr[n].val.clusterDim.z = cluster.z;
    ++n;
    if (airun_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
    if (e != cudaSuccess && airun_launch_rc == 0) airun_launch_rc = (int)e;
}

// Clusters of (1, 1, cluster_z) CTAs.
template <typename... KArgs, typename... Args>
static inline void airun_launch_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                        unsigned cluster_z, Args&&... args) {
    airun_launch_clusters(kernel, grid, block, smem, stream, dim3(1, 1, cluster_z), static_cast<KArgs>(args)...);
}

static inline int airun_launch_status() {
    cudaError_t e = cudaGetLastError();
    int rc = airun_launch_rc;
    airun_launch_rc = 0;
    if (rc) return rc;
    return e == cudaSuccess ? AIRUN_OK : (int)e;
}

// Thread-block clusters: the CTA's place, a barrier of all threads, and another CTA's shared memory.
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// a / b for b >= 1, infinity included: a reciprocal's quotient corrected by its remainder, which one multiply-add gives exactly
// (the correction step of P. Markstein, IBM Journal of Research and Development 34, 1990).  Divisors beyond 2^64 are scaled down
// first, so that their reciprocals stay normal.  Without branches or a call, so an unrolled epilogue may hold many of them: the
// gate/up product of 512 tokens in a step of Qwen3-1.7B takes 57.5 us with it, 67.7 with a / b, 53.5 with the fast division
// (which is off by two units and gives 0 for divisors beyond 2^126).  Over 1.2e9 pairs of all magnitudes it differs from a / b in
// 2 of 100,000 by one unit, numerators near 2^-126, and in subnormal results by one unit; for b = 1 + e^-z in 5.
__device__ __forceinline__ float quotient(float a, float b) {
    const float s = b > 1.8446744e19f ? 5.4210109e-20f : 1.0f, d = b * s;      // 2^64, 2^-64
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = a * r, p = fmaf(fmaf(-q, d, a), r, q);
    return (fabsf(p) <= 3.4028235e38f ? p : q) * s;                            // infinite or NaN a, infinite b: q is the answer
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over the block; every thread gets the result.  `red` holds 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarp = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();               // `red` may still be read from an earlier call
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nwarp ? red[lane] : 0.0f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

static inline int ceil_div_i(long long a, long long b) { return (int)((a + b - 1) / b); }

// Multiprocessors of the current device.  (Threads that ask for the first time at once all store the same number.)
static inline int airun_sm_count() {
    static int known[64];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    if (dev >= 0 && dev < 64 && (n = __atomic_load_n(&known[dev], __ATOMIC_RELAXED)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 1;
    if (dev >= 0 && dev < 64) __atomic_store_n(&known[dev], n, __ATOMIC_RELAXED);
    return n;
}

// True the first time it is asked on the current device (``mask``: one bit per device, of one kernel).
// cudaFuncSetAttribute holds for one device only, so each kernel is configured once on each.
static inline bool first_on_device(unsigned long long& mask) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;
    if ((mask >> dev) & 1ull) return false;
    mask |= 1ull << dev;
    return true;
}
