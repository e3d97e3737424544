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
template <class... Params, class... Args>
inline void launch_pdl(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

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

// Two deterministic block sums in one pass (one pair of barriers): the same order as
// block_sum for each.  scratch >= 64 doubles.
// The warp part of block_sum2: each of a and b summed over the warp into lane 0.
__device__ __forceinline__ void warp_sum2(double& a, double& b) {
    // a warp whose `a` values are all zero (no tet yielded) has the sum zero already
    if (__any_sync(0xffffffffu, a != 0.0)) {
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    }
    for (int o = 16; o > 0; o >>= 1) b += __shfl_down_sync(0xffffffffu, b, o);
}

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
