// tet_fast.cu -- the single-mesh FP32 J2 tet step, plain and Kahan-compensated.
//
// The element and node updates are in tet_f32.cuh (shared with the batched pool);
// this file maps them one thread per tet / per node and keeps the energy account as
// FP64 per-block partials, which the host reduces on the device in fixed order.
#include <algorithm>

#include "common.cuh"
#include "tet.hpp"
#include "tet_f32.cuh"

namespace fs {
namespace {

// The FP32 modes keep disp / disp_c as float4 per node and slots as float4 per corner.
__device__ __forceinline__ TetElementRefs refs(const TetDevice<float>& d) {
    return TetElementRefs{d.index,
                          d.slot,
                          d.rest_inv,
                          d.rest_vol,
                          d.plastic,
                          d.plastic_c,
                          reinterpret_cast<const float4*>(d.disp),
                          reinterpret_cast<const float4*>(d.disp_c),
                          reinterpret_cast<float4*>(d.slots),
                          d.tets};
}

// 1024 / kTetF32Block blocks per SM: 64 registers, 32 resident warps per SM
template <bool KAHAN>
__global__ void __launch_bounds__(kTetF32Block, 1024 / kTetF32Block) f32_forces(TetDevice<float> d, J2f m, int wave) {
    __shared__ double scratch[64];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    {
        // the rows of the block one wave later, into L2
        const long long nb = (long long)(blockIdx.x + wave) * blockDim.x;
        const long long ne = nb + blockDim.x < d.tets ? nb + blockDim.x : d.tets;
        prefetch_tet_rows(refs(d), nb, ne);
    }
    const TetElementRefs r = refs(d);
    const LoadedRows rows(r, t < d.tets ? t : d.tets - 1);
    pdl_wait();
    pdl_next();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const long long s = d.counter[0];
        d.counter[1] = s;
        d.counter[0] = s + 1;
    }
    double diss = 0.0, energy = 0.0;
    if (t < d.tets) tet_element_f32<KAHAN, false, LoadedRows>(r, rows, t, m, diss, energy);
    block_sum2(diss, energy, scratch);  // valid in thread 0
    if (threadIdx.x == 0) {
        account_add(&d.e_diss[blockIdx.x], diss);
        d.e_strain[blockIdx.x] = energy;
    }
}

template <bool KAHAN>
__global__ void __launch_bounds__(kTetNodeBlock) f32_nodes(TetDevice<float> d, float dt, float gravity, float damping,
                                                           int ramp) {
    __shared__ double scratch[64];
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double work = 0.0, kin = 0.0, gwork = 0.0;
    const SlotRun run = slot_run(d.run[n < d.nodes ? n : d.nodes - 1]);
    pdl_wait();
    pdl_next();
    if (n < d.nodes) {
        const TetNodeRefs r{reinterpret_cast<const float4*>(d.slots), d.fixed,
                            d.mass,     d.inv_mass,
                            d.ext,      d.velocity,
                            reinterpret_cast<float4*>(d.disp), reinterpret_cast<float4*>(d.disp_c)};
        const float lf = (float)ramp_factor(d.counter[1], ramp);
        const auto gather = [&](float(&force)[3]) {
            for_run<8>(
                run, [&](uint32_t k) { return r.slots[k]; },
                [&](const float4& f) {
                    force[0] += f.x;
                    force[1] += f.y;
                    force[2] += f.z;
                });
        };
        tet_node_f32<KAHAN>(r, gather, n, lf, dt, gravity, damping, work, kin, gwork);
    }
    block_sum2(work, kin, scratch);  // valid in thread 0
    if (threadIdx.x == 0) {
        account_add(&d.n_work[blockIdx.x], work);
        d.n_kin[blockIdx.x] = kin;
    }
    if (gravity != 0.0f) {
        gwork = block_sum(gwork, scratch);
        if (threadIdx.x == 0) account_add(&d.n_grav[blockIdx.x], gwork);
    }
}

// `steps` steps of a small mesh in one cluster (common.cuh), with the two kernels'
// arithmetic and sums.
template <bool KAHAN>
__global__ void __launch_bounds__(512) f32_cluster(TetDevice<float> d, J2f m, float dt, float gravity, float damping, int ramp,
                                                   int steps) {
    __shared__ GroupSums esum, nsum, gsum;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, group = i >> 7;
    const int node_group = cluster_node_group(), ni = node_group * 128 + (threadIdx.x & 127);
    const bool leader = (threadIdx.x & 127) == 0;
    const bool tet = i < d.tets, node = ni < d.nodes;
    const TetElementRefs r = refs(d);
    const LoadedRows rows(r, tet ? i : d.tets - 1);
    // this node's: what no step changes, and its state
    const int n = node ? ni : 0;
    const SlotRun run = slot_run(d.run[n]);
    const bool held = !node || d.fixed[n] != 0;
    const float mass = d.mass[n], im = d.inv_mass[n];
    float load[3] = {0.0f, 0.0f, 0.0f}, vel[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (d.ext) load[k] = d.ext[(size_t)n * 3 + k];
        vel[k] = held ? 0.0f : d.velocity[(size_t)n * 3 + k];
    }
    float4* disp = reinterpret_cast<float4*>(d.disp);
    float4* disp_c = reinterpret_cast<float4*>(d.disp_c);
    float4 u = disp[n], c = KAHAN ? disp_c[n] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4* slots = reinterpret_cast<const float4*>(d.slots);
    const bool eg = leader && (long long)group * 128 < d.tets, ng = leader && (long long)node_group * 128 < d.nodes;
    double dissipated = eg ? d.e_diss[group] : 0.0, strain = 0.0;
    double worked = ng ? d.n_work[node_group] : 0.0, kinetic = 0.0, fallen = ng ? d.n_grav[node_group] : 0.0;
    const long long first = d.counter[0];
    for (int s = 0; s < steps; ++s) {
        double diss = 0.0, energy = 0.0;
        if (tet) tet_element_f32<KAHAN, true, LoadedRows>(r, rows, i, m, diss, energy);
        esum.put(diss, energy);
        cluster_barrier();
        if (leader) {
            const double2 e = esum.get();
            if (e.x != 0.0) dissipated += e.x;
            strain = e.y;
        }
        double work = 0.0, kin = 0.0, gwork = 0.0;
        if (!held) {
            const float lf = (float)ramp_factor(first + s, ramp);
            float force[3] = {0.0f, 0.0f, -gravity * mass};
            for_run<12>(
                run, [&](uint32_t k) { return __ldcg(slots + k); },
                [&](const float4& f) {
                    force[0] += f.x;
                    force[1] += f.y;
                    force[2] += f.z;
                });
            float ext[3] = {0.0f, 0.0f, 0.0f};
            if (d.ext) {
#pragma unroll
                for (int k = 0; k < 3; ++k) ext[k] = lf * load[k];
            }
            tet_node_update<KAHAN>(mass, im, force, ext, dt, damping, vel, u, c, work, kin);
            disp[n] = u;
            if (KAHAN) disp_c[n] = c;
            gwork = -(double)gravity * (double)mass * (double)vel[2] * (double)dt;
        }
        nsum.put(work, kin);
        if (gravity != 0.0f) gsum.put(gwork, 0.0);
        cluster_barrier();
        if (leader) {
            const double2 w = nsum.get();
            worked += w.x;
            kinetic = w.y;
            if (gravity != 0.0f) fallen += gsum.get().x;
        }
    }
    if (node) {
#pragma unroll
        for (int k = 0; k < 3; ++k) d.velocity[(size_t)n * 3 + k] = vel[k];
    }
    if (eg) {
        d.e_diss[group] = dissipated;
        d.e_strain[group] = strain;
    }
    if (ng) {
        d.n_work[node_group] = worked;
        d.n_kin[node_group] = kinetic;
        if (gravity != 0.0f) d.n_grav[node_group] = fallen;
    }
    if (i == 0) {
        d.counter[0] = first + steps;
        d.counter[1] = first + steps - 1;
    }
}

}  // namespace

bool launch_f32_cluster(const TetDevice<float>& d, const TetParams& p, bool compensated, int steps, cudaStream_t stream) {
    int blocks, threads;
    cluster_shape(std::max(d.tets, d.nodes), blocks, threads);
    const J2f m = make_j2f(p.mu, p.bulk, p.yield, p.hardening);
    return launch_cluster(compensated ? f32_cluster<true> : f32_cluster<false>, blocks, threads, 0, stream, d, m, (float)p.dt,
                          (float)p.gravity, (float)p.damping, p.ramp, steps);
}

void launch_f32_step(const TetDevice<float>& d, const TetParams& p, bool compensated, cudaStream_t stream,
                     int parts) {
    const int eb = blocks_for(d.tets, kTetF32Block), nb = blocks_for(d.nodes, kTetNodeBlock);
    const J2f m = make_j2f(p.mu, p.bulk, p.yield, p.hardening);
    const int wave = sm_count() * (1024 / kTetF32Block);
    if (compensated) {
        if (parts & kElementPart) launch_pdl(f32_forces<true>, eb, kTetF32Block, 0, stream, d, m, wave);
        if (parts & kNodePart)
            launch_pdl(f32_nodes<true>, nb, kTetNodeBlock, 0, stream, d, (float)p.dt, (float)p.gravity, (float)p.damping,
                       p.ramp);
    } else {
        if (parts & kElementPart) launch_pdl(f32_forces<false>, eb, kTetF32Block, 0, stream, d, m, wave);
        if (parts & kNodePart)
            launch_pdl(f32_nodes<false>, nb, kTetNodeBlock, 0, stream, d, (float)p.dt, (float)p.gravity,
                       (float)p.damping, p.ramp);
    }
}

}  // namespace fs
