// common.cuh -- shared device helpers for the femstep kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fs {

constexpr int kBlock = 256;  // threads per block for the element and node kernels

inline int blocks_for(long long n, int block) { return (int)((n + block - 1) / block); }

// SMs of the current device.
inline int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// A step's kernels follow one another with no gap: each is launched as its predecessor's
// programmatic dependent, so its blocks come up, and load what no step changes, while the
// predecessor drains.  Every such kernel calls pdl_wait() in every block before it reads
// or writes anything a step changes (the wait returns once the predecessor has completed
// and its writes are visible), and pdl_next() only after it, so that no kernel starts
// before its predecessor's predecessor is complete.  Used where every block takes one
// run of work: 960 tets 5.8 -> 4.7 us a step, 480,000 tets 29.0 -> 27.4 us, a bay of
// 28,600 shell elements 48.0 -> 45.0 us.  The pool's passes keep plain launches: the
// blocks of its persistent element grids take tiles by a fixed stride and must come up
// evenly (among the node pass's blocks the 256-mesh batch's step took 772 us for 563), and
// node blocks that come up beside an element pass run with its shared-memory carve-out
// and little L1 (the staged schedule on 12 meshes: 98 us for 58).
//
// launch_kernel: `early`, or else as an ordinary launch, which starts once all before it in the
// stream is complete.
template <class... Params, class... Args>
inline void launch_kernel(bool early, void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream,
                        Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}
template <class... Params, class... Args>
inline void launch_pdl(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream, Args... args) {
    launch_kernel(true, kernel, grid, block, smem, stream, args...);
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- runs of a small mesh in one cluster of blocks ----
//
// A mesh of up to kClusterMost tets and nodes fits on one cluster of up to sixteen blocks,
// one tet and one node a thread, and a run of many steps is then one launch: the blocks
// meet at the cluster's hardware barrier twice a step where the two kernels of a step
// would follow one another, and what no step changes stays in registers.  Forces and
// displacements go from block to block through L2 (read with __ldcg), ordered by the
// barrier's release and acquire.  Two kernels a step against one cluster, us a step: REF32
// 960 tets 4.8 -> 3.0, 4,830 tets 5.1 -> 4.6, 8,160 tets 5.2 -> 5.0; FP32-K 960 tets
// 6.2 -> 3.8, 4,830 tets 6.4 -> 4.9, 8,160 tets 6.6 -> 5.7.  8,192 is sixteen blocks of the 512
// threads that the element's registers allow, where the two meet.  FP64 to 2,048 tets, one
// group of 128 an SM: 16.0 -> 12.0; from there to 4,096 (kCluster64Most, two groups, which
// take turns at the FP64 pipe) the two are within 4 %: 2,448 tets 16.4 -> 16.9 us a step,
// 3,840 tets 17.1 -> 17.1, and a fresh solver's first 400 steps 17.6 -> 16.9.
constexpr int kClusterBlocks = 16, kClusterMost = 8192;
constexpr int kClusterSmem = 96 * 1024;  // the most dynamic shared memory a block of one may ask for

__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The 128-node group of the thread's 128-thread group: dealt round the blocks, for a mesh
// has a quarter as many nodes as tets and they would fill the first blocks alone.
__device__ __forceinline__ int cluster_node_group() { return blockIdx.x + gridDim.x * (threadIdx.x >> 7); }

// Blocks (a power of two) and threads a block (a multiple of 128) for `items` tets or
// nodes: as many blocks as 128 threads each allow, then more threads.
inline void cluster_shape(long long items, int& blocks, int& threads) {
    blocks = 1;
    while (blocks < kClusterBlocks && (long long)blocks * 128 < items) blocks *= 2;
    threads = (int)((items + (long long)blocks * 128 - 1) / ((long long)blocks * 128)) * 128;
}

// `kernel` as one cluster; whether the device takes that shape (else nothing is queued).
template <class... Params, class... Args>
inline bool launch_cluster(void (*kernel)(Params...), int blocks, int threads, size_t smem, cudaStream_t stream,
                           Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmem) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0 &&
        cudaLaunchKernelEx(&cfg, kernel, Params(args)...) == cudaSuccess)
        return true;
    cudaGetLastError();  // the caller takes another way: no error is left for its checks
    return false;
}

// Deterministic block sum in double: shuffle tree inside each warp, then warp 0 adds
// the per-warp partials in warp order.  The association order depends only on the
// block size, never on scheduling, so the same launch always produces the same bits.
__device__ __forceinline__ double block_sum(double v, double* scratch /* >= 32 */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    double total = 0.0;
    if (threadIdx.x == 0) {
        const int warps = (blockDim.x + 31) >> 5;
        for (int w = 0; w < warps; ++w) total += scratch[w];
    }
    __syncthreads();
    return total;  // valid in thread 0 only
}

// The warp part of block_sum2: each of a and b summed over the warp into lane 0.
__device__ __forceinline__ void warp_sum2(double& a, double& b) {
    // a warp whose `a` values are all zero (no tet yielded) has the sum zero already
    if (__any_sync(0xffffffffu, a != 0.0)) {
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    }
    for (int o = 16; o > 0; o >>= 1) b += __shfl_down_sync(0xffffffffu, b, o);
}

// Two deterministic block sums in one pass (one pair of barriers): the same order as
// block_sum for each.  scratch >= 64 doubles.
__device__ __forceinline__ void block_sum2(double& a, double& b, double* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    warp_sum2(a, b);
    if (lane == 0) {
        scratch[warp] = a;
        scratch[32 + warp] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int warps = (blockDim.x + 31) >> 5;
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < warps; ++w) {
            ta += scratch[w];
            tb += scratch[32 + w];
        }
        a = ta;
        b = tb;
    }
    __syncthreads();
}

// Per-thread asynchronous copies global -> shared (16, 8 or 4 bytes, aligned to their
// size), completed by group.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Running sums of a cluster run's 128-thread groups, each the sums block_sum2 would give a
// block of 128: put() leaves the warps' sums, and after a barrier get() gives the sum
// of the thread's group, added up in warp order.
struct GroupSums {
    double2 warp[32];
    __device__ __forceinline__ void put(double a, double b) {
        warp_sum2(a, b);
        if ((threadIdx.x & 31) == 0) warp[threadIdx.x >> 5] = make_double2(a, b);
    }
    __device__ __forceinline__ double2 get() const {  // of the thread's group
        const int w = (threadIdx.x >> 7) * 4;
        double2 s = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            s.x += warp[w + k].x;
            s.y += warp[w + k].y;
        }
        return s;
    }
};

// A global load that bypasses L1 when CG: needed where another SM wrote the data
// earlier in the same (persistent) launch.
template <bool CG>
__device__ __forceinline__ float ldg_coherent(const float* p) {
    if (CG) return __ldcg(p);
    return *p;
}

template <bool CG>
__device__ __forceinline__ float4 ldg_coherent4(const float4* p) {
    if (CG) return __ldcg(p);
    return *p;
}

// sum += v for a slot of the energy account.  A slot has one writer a launch, so the order
// of its additions is fixed; as a reduction at L2 the addition is the same and its block
// does not end on waiting for the old sum (a 2,048-element zone 20.0 -> 18.1 us a step,
// 480,000 tets 25.3 -> 24.2, 24 small meshes 18.0 -> 17.1).
__device__ __forceinline__ void account_add(double* sum, double v) {
    if (v != 0.0) atomicAdd(sum, v);
}

// Column-major 3x3, the layout engine/sim/fem.cpp uses for its M3.
template <typename T>
struct M3 {
    T m[9];
    __device__ __forceinline__ T& operator()(int r, int c) { return m[c * 3 + r]; }
    __device__ __forceinline__ T operator()(int r, int c) const { return m[c * 3 + r]; }
};

template <typename T>
__device__ __forceinline__ M3<T> mul(const M3<T>& a, const M3<T>& b) {
    M3<T> r;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            T s = T(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) s += a(i, k) * b(k, c);
            r(i, c) = s;
        }
    return r;
}

template <typename T>
__device__ __forceinline__ M3<T> transpose(const M3<T>& a) {
    M3<T> r;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) r(i, j) = a(j, i);
    return r;
}

template <typename T>
__device__ __forceinline__ T det3(const M3<T>& a) {
    return a(0, 0) * (a(1, 1) * a(2, 2) - a(1, 2) * a(2, 1)) -
           a(0, 1) * (a(1, 0) * a(2, 2) - a(1, 2) * a(2, 0)) +
           a(0, 2) * (a(1, 0) * a(2, 1) - a(1, 1) * a(2, 0));
}

// Adjugate over the determinant, with the reference's singular guard
// (engine/sim/fem.cpp:42-56): a determinant at or below `tiny` gives the zero matrix.
template <typename T>
__device__ __forceinline__ M3<T> inverse(const M3<T>& a, T tiny) {
    const T det = det3(a);
    const T id = fabs(det) > tiny ? T(1) / det : T(0);
    M3<T> r;
    r(0, 0) = (a(1, 1) * a(2, 2) - a(1, 2) * a(2, 1)) * id;
    r(0, 1) = (a(0, 2) * a(2, 1) - a(0, 1) * a(2, 2)) * id;
    r(0, 2) = (a(0, 1) * a(1, 2) - a(0, 2) * a(1, 1)) * id;
    r(1, 0) = (a(1, 2) * a(2, 0) - a(1, 0) * a(2, 2)) * id;
    r(1, 1) = (a(0, 0) * a(2, 2) - a(0, 2) * a(2, 0)) * id;
    r(1, 2) = (a(0, 2) * a(1, 0) - a(0, 0) * a(1, 2)) * id;
    r(2, 0) = (a(1, 0) * a(2, 1) - a(1, 1) * a(2, 0)) * id;
    r(2, 1) = (a(0, 1) * a(2, 0) - a(0, 0) * a(2, 1)) * id;
    r(2, 2) = (a(0, 0) * a(1, 1) - a(0, 1) * a(1, 0)) * id;
    return r;
}

// Load factor of a linear ramp over `ramp` steps, evaluated for the step that is
// about to be taken: min((step + 1) / ramp, 1).
__device__ __forceinline__ double ramp_factor(long long step, int ramp) {
    if (ramp <= 0) return 1.0;
    const double f = (double)(step + 1) / (double)ramp;
    return f < 1.0 ? f : 1.0;
}

}  // namespace fs
