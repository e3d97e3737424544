// tet.hpp -- device-side layout of a tet mesh and the kernel launchers.
//
// Device layout (built by api.cu from the reference's host TetMesh, fem.hpp:38-68):
//
//   per tet, structure-of-arrays so a warp's loads are contiguous:
//     index      uint4   [T]      the four node ids
//     slot       uint4   [T]      where each corner's force goes in the slot array:
//                                 slot[t].c = the place of entry t*4+c of the CSR
//                                 (adjacencyEntry) in its node's run of slots
//     rest_inv   Real    [9][T]   Dm^-1, column-major per tet
//     rest_vol   Real    [T]
//     plastic    Real    [7][T]   plastic strain (6, engineering shears), eq. plastic strain
//     plastic_c  float   [7][T]   Kahan compensation (FP32-compensated mode only)
//   per node:
//     position / rest   Real  [3N]   (reference AoS x,y,z)
//     disp, disp_c      float [4N]   displacement and its compensation (FP32 modes),
//                                    one (x, y, z, 0) float4 per node
//     velocity          Real  [3N]
//     mass, inv_mass    Real  [N]
//     fixed             uint8 [N]
//     run               uint2 [N]    the node's run of slots: its first, and its length
//                                    (top bit: the slots lie 32 apart, else side by side)
//     ext               Real  [3N]   full-load external force (optional)
//   per CSR entry (each node's in the reference's gather order):
//     slots             float4 (REF32, FP32 J2 modes); FP64: a plane of (x, y) double2, then
//                       a plane of z
//
// The element kernel writes each corner force straight to its slot, and the node kernel
// sums a node's run in exactly the reference's CSR order.  The k-th slots of 32
// consecutive nodes lie side by side, so a warp of the node kernel, one node a lane,
// reads each k as one contiguous piece (a group whose runs differ so much that this
// would more than double its slots keeps each run contiguous instead).  Contiguous runs
// made every load of the node pass 32 lines: 19.5 us for the 491,520-tet REF32 mesh
// (step 39.7 us, L1 72 % busy), with the strided ones the step takes 18.9 us; the
// 480,000-tet beam 35.6 -> 29.0 us (FP32), 113 -> 94.6 us (FP64); 960 tets 8.3 -> 5.8 us.
// No force goes through an atomic, and each slot of the energy account has one writer a
// launch (account_add): the result does not depend on scheduling.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fs {

template <typename Real>
struct TetDevice {
    long long nodes = 0, tets = 0;
    // elements
    const uint4* index = nullptr;
    const uint4* slot = nullptr;
    const Real* rest_inv = nullptr;
    const Real* rest_vol = nullptr;
    Real* plastic = nullptr;
    float* plastic_c = nullptr;
    // nodes
    Real* position = nullptr;   // REF32 / F64: current positions
    const float* rest = nullptr;  // FP32 J2 modes: rest positions
    float* disp = nullptr;        // FP32 J2 modes
    float* disp_c = nullptr;      // FP32 compensated
    Real* velocity = nullptr;
    const Real* mass = nullptr;
    const Real* inv_mass = nullptr;
    const uint8_t* fixed = nullptr;
    const uint2* run = nullptr;
    const Real* ext = nullptr;
    Real* slots = nullptr;
    long long slot_count = 0;
    // step bookkeeping: counter[0] = steps taken, counter[1] = step the node kernel of
    // the current step uses (written by the element kernel's first thread)
    long long* counter = nullptr;
    // FP64 energy partials, one entry per block, fixed block->data mapping:
    //   e_diss (+=), e_strain (=) per element block;
    //   n_work (+=), n_kin (=), n_grav (+=) per node block
    double* e_diss = nullptr;
    double* e_strain = nullptr;
    double* n_work = nullptr;
    double* n_kin = nullptr;
    double* n_grav = nullptr;
};

struct TetParams {
    double lambda, mu, bulk;      // Lame constants and bulk modulus
    double inv_2mu, inv_3bulk;    // 1 / (2 mu), 1 / (3 bulk): the energy account
    double yield, hardening;      // J2 linear isotropic hardening
    double dt, gravity, damping;
    int ramp;
};

// Launchers.  `stream` is the caller's stream; every launch is asynchronous.
// `parts`: kElementPart | kNodePart (a whole step), or one of them alone (profiling).
constexpr uint32_t kRunStrided = 0x80000000u;  // in TetDevice::run's length

// Whether the runs of a group of 32 consecutive nodes lie strided, 32 x `longest` slots, or
// one after the other, `sum` slots.  `allow`: fewer corners than kRunStridedMost, of which
// runs padded to at most twice the slots still have 32-bit ids.
constexpr long long kRunStridedMost = 1ll << 30;
__host__ __device__ __forceinline__ bool run_strided(uint32_t longest, uint32_t sum, bool allow) {
    return allow && (unsigned long long)longest * 32 <= 2ull * sum;
}

// A node's run of slots: slot k at start + k * step.
struct SlotRun {
    uint32_t start, count, step;
};
__device__ __forceinline__ SlotRun slot_run(uint2 r) {
    return SlotRun{r.x, r.y & ~kRunStrided, r.y & kRunStrided ? 32u : 1u};
}

// add(value of slot k), k ascending, over a run: the loads of BATCH slots go out together,
// a remainder's too (one at a time, each would wait for the one before it).
template <int BATCH, class Load, class Add>
__device__ __forceinline__ void for_run(const SlotRun& r, Load load, Add add) {
    for (uint32_t k = 0; k < r.count; k += BATCH) {
        decltype(load(r.start)) v[BATCH];
#pragma unroll
        for (uint32_t j = 0; j < BATCH; ++j)
            if (k + j < r.count) v[j] = load(r.start + (k + j) * r.step);
#pragma unroll
        for (uint32_t j = 0; j < BATCH; ++j)
            if (k + j < r.count) add(v[j]);
    }
}

// The runs of a CSR (adjacency offsets and entries): run [nodes], slot [total] and the
// number of slots, all on the device (queued on `stream`, not waited for).
cudaError_t build_runs_device(const uint32_t* offset, const uint32_t* entry, long long total, long long nodes, uint2* run,
                              uint32_t* slot, uint32_t* slots, cudaStream_t stream);

// Threads per block of the single-mesh node kernels: few, so that a small mesh's nodes
// spread over the SMs.
constexpr int kTetNodeBlock = 128;
constexpr int kTet64Block = 128;   // threads per block of the FP64 element kernel,
constexpr int kTetF32Block = 128;  // and of the FP32 J2 modes'
constexpr int kElementPart = 1, kNodePart = 2, kWholeStep = 3;
void launch_ref32_step(const TetDevice<float>& d, const TetParams& p, cudaStream_t stream,
                       int parts = kWholeStep);
void launch_f64_step(const TetDevice<double>& d, const TetParams& p, cudaStream_t stream,
                     int parts = kWholeStep);
void launch_f32_step(const TetDevice<float>& d, const TetParams& p, bool compensated,
                     cudaStream_t stream, int parts = kWholeStep);
// `steps` whole steps of a mesh of at most kClusterMost tets and nodes in one launch
// (kCluster64Most for FP64); false, with nothing queued, where the device does not take it.
// The state it leaves is the steps' to the bit.
constexpr int kCluster64Most = 4096;
bool launch_ref32_cluster(const TetDevice<float>& d, const TetParams& p, int steps, cudaStream_t stream);
bool launch_f64_cluster(const TetDevice<double>& d, const TetParams& p, int steps, cudaStream_t stream);
bool launch_f32_cluster(const TetDevice<float>& d, const TetParams& p, bool compensated, int steps, cudaStream_t stream);
// FP64 element eigenvalue bound: omega^2 per tet, reduced to the maximum on device.
void launch_tet_omega2(long long tets, const double* rest_inv, double E, double nu, double rho,
                       double* per_block_max, int blocks, cudaStream_t stream);
// The same bound from an FP32 Dm^-1 (SoA with stride `stride`, `rest_inv` pointing at
// the first tet), promoted to double: the matrix the FP32 element kernels use.
void launch_tet_omega2_f32(long long tets, const float* rest_inv, long long stride, double E, double nu, double rho,
                           double* per_block_max, int blocks, cudaStream_t stream);
// The single mesh's rest state on the device, bit-identical to tet_rest_state64:
// per tet Dm^-1 (SoA, `tets` per row), volume and quarter mass; per node the lumped
// mass summed over the node's CSR run (`entry`: corner ids, ascending per node).
void launch_tet_rest64(const float* position, const uint32_t* index, long long tets, double density, double* inv,
                       double* vol, double* quarter, cudaStream_t stream);
void launch_tet_mass64(const uint32_t* offset, const uint32_t* entry, long long nodes, const double* quarter,
                       double* mass, cudaStream_t stream);
// The FP32 modes' rest state from it: Dm^-1, volume, mass and 1 / mass, rounded once.
void launch_tet_rest_f32(const double* inv, const double* vol, long long tets, const double* mass, long long nodes,
                         float* inv32, float* vol32, float* mass32, float* inv_mass32, cudaStream_t stream);
// out[i] = (double)in[i].
void launch_widen(const float* in, long long n, double* out, cudaStream_t stream);
// Fixed-order FP64 sum / max of `n` doubles into out[0] (one block).
void launch_reduce_sum(const double* in, long long n, double* out, cudaStream_t stream);
void launch_reduce_max(const double* in, long long n, double* out, cudaStream_t stream);

}  // namespace fs
