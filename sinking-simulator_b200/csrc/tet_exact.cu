// tet_exact.cu -- the two tet steps that reproduce a CPU path bit for bit.
//
// This translation unit is compiled with -fmad=false: every multiply and add is a
// separately rounded IEEE operation, division and square root are correctly rounded,
// and each expression is written in the order of the CPU code it reproduces.  That is
// what makes these kernels bit-identical to their CPU counterparts:
//
//   REF32  elastic co-rotational tet in float, the arithmetic of fem::tetForces and
//          fem::stepCpu (engine/sim/fem.cpp:73-117, 187-215), i.e. what
//          gpu::FemGpuSolver::run dispatches (engine/gpu/shaders/tet_forces.comp,
//          node_integrate.comp).  Drop-in for the reference's GPU tet back-end.
//   F64    the J2 tet in double: fem.cpp's kinematics with the radial return of
//          plasticity::update (engine/sim/plasticity.cpp:319-505) at the single point,
//          linear isotropic hardening, failure off, and the fem.cpp node update with a
//          ramped external load.  This is the plain FP64 single-mesh step.
//
// Memory-bound kernels (algorithmic bytes: ~240 B per update for REF32, ~435 B for
// F64): one thread per tet / per node, SoA element arrays so each warp load is one
// contiguous 128 B line, node-major force slots so each node's gather is contiguous.
#include <algorithm>

#include "common.cuh"
#include "omega.cuh"
#include "tet.hpp"

namespace fs {
namespace {

// Higham polar iteration.  REF32: four fixed iterations (fem.cpp:62-69).  F64: run to
// convergence, step below 1e-16, at most 64 iterations (solid_shell.cpp:473-487).
__device__ __forceinline__ M3<float> polar_fixed4(const M3<float>& f) {
    M3<float> r = f;
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const M3<float> rit = transpose(inverse(r, 1e-30f));
#pragma unroll
        for (int k = 0; k < 9; ++k) r.m[k] = 0.5f * (r.m[k] + rit.m[k]);
    }
    return r;
}

// One step of it; true once the iteration ends there (converged, or singular).
__device__ __forceinline__ bool polar_step(M3<double>& r) {
    if (det3(r) == 0.0) return true;
    const M3<double> rit = transpose(inverse(r, 1e-300));
    double worst = 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const double next = 0.5 * (r.m[k] + rit.m[k]);
        const double d = fabs(next - r.m[k]);
        worst = worst > d ? worst : d;
        r.m[k] = next;
    }
    return worst < 1e-16;
}

// The same step where det x is 1 to within 2^-30, as it is from the third step on for
// any moderate strain; returns det x, for the caller to check.  A step is a chain of
// dependent FP64 operations, and there it can be shortened without changing a bit:
//   * 1 / det is 2 - det rounded up.  With det = 1 + m 2^-52 (0 < m <= 2^22), 1 / det is
//     2 - det, which is a double, plus at most m^2 2^-104, far under half its ulp; with
//     det = 1 - m 2^-53 it is 1 + m 2^-53 plus a little over m^2 2^-106, so it rounds to
//     2 - det where that is a double (m even) and up from the midpoint where it is not.
//   * 0.5 (r + c / det) is fma(0.5, r, c (0.5 / det)): halving is exact (the cofactors of
//     positions' differences are zero or far above the subnormals).
// Eight operations deep instead of the divide and ten.
__device__ __forceinline__ double polar_near(const M3<double>& r, M3<double>& y) {
    const double c00 = r(1, 1) * r(2, 2) - r(1, 2) * r(2, 1), c01 = r(1, 0) * r(2, 2) - r(1, 2) * r(2, 0),
                 c02 = r(1, 0) * r(2, 1) - r(1, 1) * r(2, 0);
    const double det = r(0, 0) * c00 - r(0, 1) * c01 + r(0, 2) * c02;
    // the transposed inverse's numerators, in inverse()'s own order of terms
    const double c[9] = {c00,
                         r(0, 2) * r(2, 1) - r(0, 1) * r(2, 2),
                         r(0, 1) * r(1, 2) - r(0, 2) * r(1, 1),
                         r(1, 2) * r(2, 0) - r(1, 0) * r(2, 2),
                         r(0, 0) * r(2, 2) - r(0, 2) * r(2, 0),
                         r(0, 2) * r(1, 0) - r(0, 0) * r(1, 2),
                         c02,
                         r(0, 1) * r(2, 0) - r(0, 0) * r(2, 1),
                         r(0, 0) * r(1, 1) - r(0, 1) * r(1, 0)};
    const double half = __fma_ru(-0.5, det, 1.0);
#pragma unroll
    for (int k = 0; k < 9; ++k) y.m[k] = __fma_rn(0.5, r.m[k], c[k] * half);
    return det;
}

// Negative where |y_k - x_k| is under 1e-16 (all finite) for every k in `from`, `from` +
// `by`, ...: the signs of the bit patterns' differences, ANDed.
template <int FROM, int BY>
__device__ __forceinline__ int polar_still(const M3<double>& x, const M3<double>& y) {
    int all = -1;
#pragma unroll
    for (int k = FROM; k < 9; k += BY) {
        const long long bits = __double_as_longlong(fabs(y.m[k] - x.m[k])) - __double_as_longlong(1e-16);
        all &= (int)(bits >> 32);
    }
    return all;
}

// Two steps; true once the iteration has ended (x is then its result).  Almost every
// step that goes on shows it on the diagonal alone (an ulp there is more than 1e-16), so
// the three diagonal entries are tested first, and the two steps' tests are decided
// together beside the second step's arithmetic.
__device__ __forceinline__ bool polar_pair(M3<double>& x) {
    M3<double> y, z;
    const double d0 = polar_near(x, y), d1 = polar_near(y, z);
    const bool near = fabs(d0 - 1.0) <= 0x1p-30 && fabs(d1 - 1.0) <= 0x1p-30;
    if (near && (polar_still<0, 4>(x, y) | polar_still<0, 4>(y, z)) >= 0) {
        x = z;
        return false;
    }
    if (near) {
        if (polar_still<0, 1>(x, y) < 0) {
            x = y;
            return true;
        }
        const bool end = polar_still<0, 1>(y, z) < 0;
        x = z;
        return end;
    }
    return polar_step(x) || polar_step(x);
}

// The iteration for a block's tets together.  Two thirds of moving tets end within six
// steps; the others never meet the test, because the last bits go round (a period of 2
// or 3) or drift, and take all 64 steps.  One tet a lane, nearly every warp would run 64
// steps for a third of its lanes.  So the block packs the unfinished tets into its first
// warps after six steps and again after sixteen, and there leaves out those that are
// where they were six steps before: 48 more steps bring them back to the same bits.
// Every tet ends with the bits of its own 64-step loop.  F and the tet's rows wait in
// shared memory too, so that a block holds few registers while most of its warps wait
// for the packed ones: five blocks an SM (96 registers) where four measured 128 us a
// step, on the 480,000-tet beam in motion, and five 113 us.  One tet a lane with the
// divide in every step took 218 us there, and 34.4 us a step (now 22.6 us) on the
// 3,840-tet cantilever, where the 64 steps of one warp are the pass: 207 cycles each,
// 122 of them issuing its FP64 operations at two cycles each.
struct PolarPark {
    double rows[17][kTet64Block];  // Dm^-1, volume, plastic state: copied in while F is formed
    double f[9][kTet64Block];
    double r[9][kTet64Block];
    uint16_t list[2][kTet64Block];
    int count[2];
};

// The 128 threads of a park meet: a group of a larger block (GROUP), or the whole block --
// with the one barrier, since a block that names barriers by number reserves all sixteen,
// and an SM has enough of them for four such blocks only.
template <bool GROUP>
__device__ __forceinline__ void park_barrier() {
    if (GROUP)
        asm volatile("bar.sync %0, 128;" ::"r"((int)threadIdx.x >> 7) : "memory");
    else
        __syncthreads();
}

template <bool GROUP>
__device__ __forceinline__ M3<double> polar_block(M3<double> r, bool live, PolarPark& park) {
    static_assert(kTet64Block == 128, "a park serves one group of 128 threads");
    constexpr int kFirst = 6, kSnapshot = 10, kSecond = 16, kLast = 64;
    static_assert((kLast - kSecond) % (kSecond - kSnapshot) == 0, "whole periods remain");
    static_assert(kFirst % 2 == 0 && kSnapshot % 2 == 0 && kSecond % 2 == 0 && kLast % 2 == 0, "steps go in pairs");
    const int tid = threadIdx.x & 127;
    if (tid < 2) park.count[tid] = 0;
    park_barrier<GROUP>();
    bool done = !live || polar_step(r) || polar_step(r);
#pragma unroll 1
    for (int it = 2; it < kFirst && !done; it += 2) done = polar_pair(r);
#pragma unroll
    for (int k = 0; k < 9; ++k) park.r[k][tid] = r.m[k];
    if (!done) park.list[0][atomicAdd(&park.count[0], 1)] = (uint16_t)tid;
#pragma unroll 1
    for (int round = 0; round < 2; ++round) {
        park_barrier<GROUP>();
        const int n = park.count[round];
        if (n == 0) break;  // the same for the whole block
        if (tid < n) {
            const int at = park.list[round][tid];
            M3<double> x;
#pragma unroll
            for (int k = 0; k < 9; ++k) x.m[k] = park.r[k][at];
            bool end = false;
            const int last = round ? kLast : kSecond;
#pragma unroll 1
            for (int it = round ? kSecond : kFirst; it < last && !end; it += 2) {
                if (it == kSnapshot) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) park.r[k][at] = x.m[k];
                }
                end = polar_pair(x);
            }
            if (!end && !round) {
                bool same = true;
#pragma unroll
                for (int k = 0; k < 9; ++k)
                    same = same && __double_as_longlong(x.m[k]) == __double_as_longlong(park.r[k][at]);
                if (!same) park.list[1][atomicAdd(&park.count[1], 1)] = (uint16_t)at;
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) park.r[k][at] = x.m[k];
        }
    }
    park_barrier<GROUP>();
#pragma unroll
    for (int k = 0; k < 9; ++k) r.m[k] = park.r[k][tid];
    return r;
}

// ---------------------------------------------------------------------------------
// REF32: fem::tetForces (fem.cpp:73-117), the corner forces written to their slots.  CG: the
// positions were written by other SMs in this launch.
template <bool CG>
__device__ __forceinline__ void ref32_element(const float* p, const uint4& idx, const uint4& sl, const M3<float>& dm_inv,
                                              float scale, float lambda, float mu, float* slot_array) {
    const unsigned nid[4] = {idx.x, idx.y, idx.z, idx.w};
    M3<float> ds;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int a = 0; a < 3; ++a) ds(a, c) = ldg_coherent<CG>(p + (size_t)nid[c + 1] * 3 + a) - ldg_coherent<CG>(p + (size_t)nid[0] * 3 + a);
    const M3<float> f = mul(ds, dm_inv);
    const M3<float> r = polar_fixed4(f);
    const M3<float> s = mul(transpose(r), f);
    M3<float> strain;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) strain(i, j) = 0.5f * (s(i, j) + s(j, i));
#pragma unroll
    for (int i = 0; i < 3; ++i) strain(i, i) -= 1.0f;
    const float trace = strain(0, 0) + strain(1, 1) + strain(2, 2);
    M3<float> stress;
#pragma unroll
    for (int k = 0; k < 9; ++k) stress.m[k] = 2.0f * mu * strain.m[k];
#pragma unroll
    for (int i = 0; i < 3; ++i) stress(i, i) += lambda * trace;
    const M3<float> h = mul(mul(r, stress), transpose(dm_inv));
    const unsigned sid[4] = {sl.x, sl.y, sl.z, sl.w};
    float f0[3] = {0.0f, 0.0f, 0.0f};
    float4* slots = reinterpret_cast<float4*>(slot_array);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float v[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            v[a] = scale * h(a, c);
            f0[a] -= v[a];
        }
        slots[sid[c + 1]] = make_float4(v[0], v[1], v[2], 0.0f);
    }
    slots[sid[0]] = make_float4(f0[0], f0[1], f0[2], 0.0f);
}

// REF32: a free node of fem::stepCpu's loop (fem.cpp:196-214).
__device__ __forceinline__ void ref32_node(float m, const float (&force)[3], float dt, float damping, float* vel, float* pos) {
    const float inv_mass = 1.0f / m;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float v = vel[k] + force[k] * inv_mass * dt;
        v *= damping;
        vel[k] = v;
        pos[k] += v * dt;
    }
}

__global__ void __launch_bounds__(kBlock) ref32_forces(TetDevice<float> d, float lambda, float mu) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long tr = t < d.tets ? t : d.tets - 1;
    const uint4 idx = d.index[tr], sl = d.slot[tr];
    M3<float> dm_inv;
#pragma unroll
    for (int k = 0; k < 9; ++k) dm_inv.m[k] = d.rest_inv[(size_t)k * d.tets + tr];
    const float scale = -d.rest_vol[tr];
    pdl_wait();
    pdl_next();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const long long s = d.counter[0];
        d.counter[1] = s;
        d.counter[0] = s + 1;
    }
    if (t >= d.tets) return;
    ref32_element<false>(d.position, idx, sl, dm_inv, scale, lambda, mu, d.slots);
}

// REF32: fem::stepCpu's node loop (fem.cpp:196-214).
__global__ void __launch_bounds__(kTetNodeBlock) ref32_nodes(TetDevice<float> d, float dt, float gravity,
                                                      float damping) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nr = n < d.nodes ? n : d.nodes - 1;
    const SlotRun run = slot_run(d.run[nr]);
    const float m = d.mass[nr];
    const bool held = d.fixed[nr] != 0;
    pdl_wait();
    pdl_next();
    if (n >= d.nodes) return;
    float* vel = d.velocity + (size_t)n * 3;
    if (held) {
        vel[0] = 0.0f;
        vel[1] = 0.0f;
        vel[2] = 0.0f;
        return;
    }
    float force[3] = {0.0f, 0.0f, -gravity * m};
    const float4* slots = reinterpret_cast<const float4*>(d.slots);
    for_run<8>(
        run, [&](uint32_t k) { return slots[k]; },
        [&](const float4& f) {
            force[0] += f.x;
            force[1] += f.y;
            force[2] += f.z;
        });
    ref32_node(m, force, dt, damping, vel, d.position + (size_t)n * 3);
}

// `steps` steps of a small mesh in one cluster (common.cuh), with the two kernels' arithmetic.
__global__ void __launch_bounds__(512) ref32_cluster(TetDevice<float> d, float lambda, float mu, float dt, float gravity,
                                                     float damping, int steps) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, ni = cluster_node_group() * 128 + (threadIdx.x & 127);
    const bool tet = i < d.tets, node = ni < d.nodes;
    const long long t = tet ? i : 0;
    const uint4 idx = d.index[t], sl = d.slot[t];
    M3<float> dm_inv;
#pragma unroll
    for (int k = 0; k < 9; ++k) dm_inv.m[k] = d.rest_inv[(size_t)k * d.tets + t];
    const float scale = -d.rest_vol[t];
    const int n = node ? ni : 0;
    const SlotRun run = slot_run(d.run[n]);
    const float m = d.mass[n];
    const bool held = !node || d.fixed[n] != 0;
    const float4* slots = reinterpret_cast<const float4*>(d.slots);
    float vel[3], pos[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        vel[k] = held ? 0.0f : d.velocity[(size_t)n * 3 + k];
        pos[k] = d.position[(size_t)n * 3 + k];
    }
    const long long first = d.counter[0];
    for (int s = 0; s < steps; ++s) {
        if (tet) ref32_element<true>(d.position, idx, sl, dm_inv, scale, lambda, mu, d.slots);
        cluster_barrier();
        if (!held) {
            float force[3] = {0.0f, 0.0f, -gravity * m};
            for_run<12>(
                run, [&](uint32_t k) { return __ldcg(slots + k); },
                [&](const float4& f) {
                    force[0] += f.x;
                    force[1] += f.y;
                    force[2] += f.z;
                });
            ref32_node(m, force, dt, damping, vel, pos);
#pragma unroll
            for (int k = 0; k < 3; ++k) d.position[(size_t)n * 3 + k] = pos[k];
        }
        cluster_barrier();
    }
    if (node) {
#pragma unroll
        for (int k = 0; k < 3; ++k) d.velocity[(size_t)n * 3 + k] = vel[k];
    }
    if (i == 0) {
        d.counter[0] = first + steps;
        d.counter[1] = first + steps - 1;
    }
}

// ---------------------------------------------------------------------------------
// F64: the J2 tet.

// plasticity::update for linear isotropic hardening with no kinematic hardening and
// no failure (plasticity.cpp:333-456): elastic predictor, radial return with the
// bracketed Newton on the consistency condition, the committed plastic strain.  The
// arithmetic order is the CPU's, term for term.
struct J2Out {
    double dissipation;
    bool yielded;
};

__device__ __forceinline__ J2Out j2_return_f64(const double strain[6], double ps[7], double mu, double kappa,
                                               double yield, double hardening, double stress[6]) {
    J2Out out{0.0, false};
    const double root23 = sqrt(2.0 / 3.0);
    double elastic[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) elastic[i] = strain[i] - ps[i];
    const double volumetric = elastic[0] + elastic[1] + elastic[2];
    const double pressure = kappa * volumetric;
    double trial[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        trial[i] = 2.0 * mu * (elastic[i] - volumetric / 3.0);
        trial[3 + i] = mu * elastic[3 + i];
    }
    double relative[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) relative[i] = trial[i] - 0.0;
    const double norm2 = relative[0] * relative[0] + relative[1] * relative[1] + relative[2] * relative[2] +
                         2.0 * (relative[3] * relative[3] + relative[4] * relative[4] + relative[5] * relative[5]);
    const double relative_norm = sqrt(norm2);
    const double pp0 = ps[6] > 0.0 ? ps[6] : 0.0;
    const double yield_radius = root23 * (yield + hardening * pp0);
    const double excess = relative_norm - yield_radius;
    if (!(excess > 0.0)) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            stress[i] = pressure + trial[i];
            stress[3 + i] = trial[3 + i];
        }
        return out;
    }
    out.yielded = true;
    const double linear_part = 2.0 * mu + (2.0 / 3.0) * 0.0;
    double lo = 0.0, hi = excess / linear_part;
    double gamma = hi;
#pragma unroll 1
    for (int iterations = 0; iterations < 50; ++iterations) {
        const double accumulated = ps[6] + root23 * gamma;
        const double pa = accumulated > 0.0 ? accumulated : 0.0;
        const double residual = relative_norm - linear_part * gamma - root23 * (yield + hardening * pa);
        if (residual > 0.0)
            lo = gamma;
        else
            hi = gamma;
        if (fabs(residual) <= 1e-14 * yield_radius) break;
        const double slope = -linear_part - (2.0 / 3.0) * hardening;
        double next = gamma - residual / slope;
        if (!(next > lo && next < hi)) next = 0.5 * (lo + hi);
        if (fabs(next - gamma) <= 1e-15 * gamma) {
            gamma = next;
            break;
        }
        gamma = next;
    }
    double direction[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) direction[i] = relative[i] / relative_norm;
    double dp[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        dp[i] = gamma * direction[i];
        dp[3 + i] = 2.0 * gamma * direction[3 + i];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        stress[i] = pressure + trial[i] - 2.0 * mu * gamma * direction[i];
        stress[3 + i] = trial[3 + i] - 2.0 * mu * gamma * direction[3 + i];
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) s += (stress[i] - (0.0 + (2.0 / 3.0) * 0.0 * gamma * direction[i])) * dp[i];
    out.dissipation = s;
#pragma unroll
    for (int i = 0; i < 6; ++i) ps[i] += dp[i];
    ps[6] += root23 * gamma;
    return out;
}

// One tet of the FP64 step (every thread of its 128-thread group calls it, `live` or not):
// its Dm^-1 and volume in the park's rows (their copies under way), its plastic state
// copied there too; corner forces to their slots.  CG: in a cluster run, where other SMs
// wrote the positions in this launch and the rows stay in the park from step to step.
template <bool CG>
__device__ __forceinline__ void f64_element(const TetDevice<double>& d, const TetParams& p, PolarPark& park, long long t,
                                            bool live, const uint4& idx, double& diss, double& energy) {
    const int tid = threadIdx.x & 127;
    diss = energy = 0.0;
    M3<double> f;
    if (live) {
        const unsigned nid[4] = {idx.x, idx.y, idx.z, idx.w};
        const double* x = d.position;
        const auto load = [](const double* at) { return CG ? __ldcg(at) : *at; };
        M3<double> ds, dm_inv;
        if (!CG) {
#pragma unroll
            for (int i = 0; i < 7; ++i) cp_async8(&park.rows[10 + i][tid], d.plastic + (size_t)i * d.tets + t);
            cp_async_commit();
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int a = 0; a < 3; ++a) ds(a, c) = load(x + (size_t)nid[c + 1] * 3 + a) - load(x + (size_t)nid[0] * 3 + a);
        if (!CG) cp_async_wait_one();  // a thread reads back only what it copied: no barrier
#pragma unroll
        for (int k = 0; k < 9; ++k) dm_inv.m[k] = park.rows[k][tid];
        f = mul(ds, dm_inv);
#pragma unroll
        for (int k = 0; k < 9; ++k) park.f[k][tid] = f.m[k];
    }
    const M3<double> r = polar_block<CG>(f, live, park);
    if (live) {
        if (!CG) cp_async_wait_all();
#pragma unroll
        for (int k = 0; k < 9; ++k) f.m[k] = park.f[k][tid];
        const M3<double> sm = mul(transpose(r), f);
        double strain[6];
        strain[0] = 0.5 * (sm(0, 0) + sm(0, 0)) - 1.0;
        strain[1] = 0.5 * (sm(1, 1) + sm(1, 1)) - 1.0;
        strain[2] = 0.5 * (sm(2, 2) + sm(2, 2)) - 1.0;
        strain[3] = 2.0 * (0.5 * (sm(0, 1) + sm(1, 0)));
        strain[4] = 2.0 * (0.5 * (sm(1, 2) + sm(2, 1)));
        strain[5] = 2.0 * (0.5 * (sm(2, 0) + sm(0, 2)));
        double ps[7];
#pragma unroll
        for (int i = 0; i < 7; ++i) ps[i] = park.rows[10 + i][tid];
        double sv[6];
        const J2Out j = j2_return_f64(strain, ps, p.mu, p.bulk, p.yield, p.hardening, sv);
        if (j.yielded) {
#pragma unroll
            for (int i = 0; i < 7; ++i) {
                d.plastic[(size_t)i * d.tets + t] = ps[i];
                if (CG) park.rows[10 + i][tid] = ps[i];
            }
        }
        const double vol = park.rows[9][tid];
        diss = vol * j.dissipation;
        // 1/2 sigma : C^-1 : sigma from the deviator and the trace, by the reciprocals
        const double tr = sv[0] + sv[1] + sv[2], pressure = tr * (1.0 / 3.0);
        const double e0 = sv[0] - pressure, e1 = sv[1] - pressure, e2 = sv[2] - pressure;
        const double dev = e0 * e0 + e1 * e1 + e2 * e2 + 2.0 * (sv[3] * sv[3] + sv[4] * sv[4] + sv[5] * sv[5]);
        energy = 0.5 * vol * (dev * p.inv_2mu + pressure * tr * p.inv_3bulk);

        M3<double> dm_inv;
#pragma unroll
        for (int k = 0; k < 9; ++k) dm_inv.m[k] = park.rows[k][tid];

        M3<double> stress;
        stress(0, 0) = sv[0];
        stress(1, 1) = sv[1];
        stress(2, 2) = sv[2];
        stress(0, 1) = stress(1, 0) = sv[3];
        stress(1, 2) = stress(2, 1) = sv[4];
        stress(2, 0) = stress(0, 2) = sv[5];
        const M3<double> h = mul(mul(r, stress), transpose(dm_inv));
        const double scale = -vol;
        const uint4 sl = d.slot[t];
        const unsigned sid[4] = {sl.x, sl.y, sl.z, sl.w};
        double f0[3] = {0.0, 0.0, 0.0};
        double2* xy = reinterpret_cast<double2*>(d.slots);
        double* z = d.slots + 2 * d.slot_count;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                v[a] = scale * h(a, c);
                f0[a] -= v[a];
            }
            xy[sid[c + 1]] = make_double2(v[0], v[1]);
            z[sid[c + 1]] = v[2];
        }
        xy[sid[0]] = make_double2(f0[0], f0[1]);
        z[sid[0]] = f0[2];
    }
}

__global__ void __launch_bounds__(kTet64Block, 5) f64_forces(TetDevice<double> d, TetParams p) {
    __shared__ double scratch[64];
    __shared__ PolarPark park;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = t < d.tets;
    uint4 idx = make_uint4(0, 0, 0, 0);
    if (live) {
        idx = d.index[t];
#pragma unroll
        for (int k = 0; k < 9; ++k) cp_async8(&park.rows[k][threadIdx.x], d.rest_inv + (size_t)k * d.tets + t);
        cp_async_commit();
        cp_async8(&park.rows[9][threadIdx.x], d.rest_vol + t);
    }
    pdl_wait();
    pdl_next();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const long long s = d.counter[0];
        d.counter[1] = s;
        d.counter[0] = s + 1;
    }
    double diss, energy;
    f64_element<false>(d, p, park, t, live, idx, diss, energy);
    block_sum2(diss, energy, scratch);  // valid in thread 0
    if (threadIdx.x == 0) {
        account_add(&d.e_diss[blockIdx.x], diss);
        d.e_strain[blockIdx.x] = energy;
    }
}

// A free node's update from the force on it (its external part included), and the step's
// external work and kinetic energy.
__device__ __forceinline__ void f64_node(const TetParams& p, double m, double inv_mass, const double (&force)[3],
                                         const double (&ext)[3], double* vel, double* pos, double& work, double& kin) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = vel[k] + force[k] * inv_mass * p.dt;
        v *= p.damping;
        vel[k] = v;
        pos[k] += v * p.dt;
        work += ext[k] * v * p.dt;
        kin += 0.5 * m * v * v;
    }
}

__global__ void __launch_bounds__(kTetNodeBlock) f64_nodes(TetDevice<double> d, TetParams p) {
    __shared__ double scratch[64];
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double work = 0.0, kin = 0.0, gwork = 0.0;
    const SlotRun run = slot_run(d.run[n < d.nodes ? n : d.nodes - 1]);
    pdl_wait();
    pdl_next();
    if (n < d.nodes) {
        double* vel = d.velocity + (size_t)n * 3;
        if (d.fixed[n]) {
            vel[0] = 0.0;
            vel[1] = 0.0;
            vel[2] = 0.0;
        } else {
            const double lf = ramp_factor(d.counter[1], p.ramp);
            const double m = d.mass[n];
            double force[3] = {0.0, 0.0, -p.gravity * m};
            const double2* xy = reinterpret_cast<const double2*>(d.slots);
            const double* z = d.slots + 2 * d.slot_count;
            for_run<8>(
                run,
                [&](uint32_t k) {
                    const double2 f = xy[k];
                    return make_double3(f.x, f.y, z[k]);
                },
                [&](const double3& f) {
                    force[0] += f.x;
                    force[1] += f.y;
                    force[2] += f.z;
                });
            double ext[3] = {0.0, 0.0, 0.0};
            if (d.ext) {
#pragma unroll
                for (int k = 0; k < 3; ++k) ext[k] = lf * d.ext[(size_t)n * 3 + k];
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) force[k] += ext[k];
            f64_node(p, m, 1.0 / m, force, ext, vel, d.position + (size_t)n * 3, work, kin);
            gwork = -p.gravity * m * vel[2] * p.dt;
        }
    }
    block_sum2(work, kin, scratch);  // valid in thread 0
    if (threadIdx.x == 0) {
        account_add(&d.n_work[blockIdx.x], work);
        d.n_kin[blockIdx.x] = kin;
    }
    if (p.gravity != 0.0) {
        gwork = block_sum(gwork, scratch);
        if (threadIdx.x == 0) account_add(&d.n_grav[blockIdx.x], gwork);
    }
}

// `steps` steps of a small mesh in one cluster (common.cuh), with the two kernels'
// arithmetic and sums.  A group of 128 threads has its own park; Dm^-1, volumes and the
// plastic state stay there for the run.
__global__ void __launch_bounds__(kCluster64Most / kClusterBlocks) f64_cluster(TetDevice<double> d, TetParams p, int steps) {
    extern __shared__ __align__(16) unsigned char parks[];
    __shared__ GroupSums esum, nsum, gsum;
    PolarPark& park = reinterpret_cast<PolarPark*>(parks)[threadIdx.x >> 7];
    const int i = blockIdx.x * blockDim.x + threadIdx.x, group = i >> 7, tid = threadIdx.x & 127;
    const int node_group = cluster_node_group(), ni = node_group * 128 + tid;
    const bool leader = tid == 0, tet = i < d.tets, node = ni < d.nodes;
    const long long t = tet ? i : 0;
    const uint4 idx = d.index[t];
#pragma unroll
    for (int k = 0; k < 9; ++k) park.rows[k][tid] = d.rest_inv[(size_t)k * d.tets + t];
    park.rows[9][tid] = d.rest_vol[t];
#pragma unroll
    for (int k = 0; k < 7; ++k) park.rows[10 + k][tid] = d.plastic[(size_t)k * d.tets + t];
    const int n = node ? ni : 0;
    const SlotRun run = slot_run(d.run[n]);
    const bool held = !node || d.fixed[n] != 0;
    const double m = d.mass[n], inv_mass = 1.0 / m;
    double load[3] = {0.0, 0.0, 0.0}, vel[3], pos[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (d.ext) load[k] = d.ext[(size_t)n * 3 + k];
        vel[k] = held ? 0.0 : d.velocity[(size_t)n * 3 + k];
        pos[k] = d.position[(size_t)n * 3 + k];
    }
    const double2* xy = reinterpret_cast<const double2*>(d.slots);
    const double* z = d.slots + 2 * d.slot_count;
    const bool eg = leader && (long long)group * 128 < d.tets, ng = leader && (long long)node_group * 128 < d.nodes;
    double dissipated = eg ? d.e_diss[group] : 0.0, strain = 0.0;
    double worked = ng ? d.n_work[node_group] : 0.0, kinetic = 0.0, fallen = ng ? d.n_grav[node_group] : 0.0;
    const long long first = d.counter[0];
    for (int s = 0; s < steps; ++s) {
        double diss, energy;
        f64_element<true>(d, p, park, t, tet, idx, diss, energy);
        esum.put(diss, energy);
        cluster_barrier();
        if (leader) {
            const double2 e = esum.get();
            if (e.x != 0.0) dissipated += e.x;
            strain = e.y;
        }
        double work = 0.0, kin = 0.0, gwork = 0.0;
        if (!held) {
            const double lf = ramp_factor(first + s, p.ramp);
            double force[3] = {0.0, 0.0, -p.gravity * m};
            for_run<8>(
                run,
                [&](uint32_t k) {
                    const double2 f = __ldcg(xy + k);
                    return make_double3(f.x, f.y, __ldcg(z + k));
                },
                [&](const double3& f) {
                    force[0] += f.x;
                    force[1] += f.y;
                    force[2] += f.z;
                });
            double ext[3] = {0.0, 0.0, 0.0};
            if (d.ext) {
#pragma unroll
                for (int k = 0; k < 3; ++k) ext[k] = lf * load[k];
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) force[k] += ext[k];
            f64_node(p, m, inv_mass, force, ext, vel, pos, work, kin);
#pragma unroll
            for (int k = 0; k < 3; ++k) d.position[(size_t)n * 3 + k] = pos[k];
            gwork = -p.gravity * m * vel[2] * p.dt;
        }
        nsum.put(work, kin);
        if (p.gravity != 0.0) gsum.put(gwork, 0.0);
        cluster_barrier();
        if (leader) {
            const double2 w = nsum.get();
            worked += w.x;
            kinetic = w.y;
            if (p.gravity != 0.0) fallen += gsum.get().x;
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
        if (p.gravity != 0.0) d.n_grav[node_group] = fallen;
    }
    if (i == 0) {
        d.counter[0] = first + steps;
        d.counter[1] = first + steps - 1;
    }
}

// ---------------------------------------------------------------------------------
// FP64 critical time step: per tet, the largest omega^2 of the lumped-mass element
// (4/rho) lambda_max(B^T C B) by power iteration, as solid_shell.cpp:1088-1133 does
// for the hex (Rayleigh quotient, at most 400 iterations, relative 1e-10, the same
// start vector).  max over elements bounds the assembled problem.
// Dm^-1 may be the FP64 array (single-mesh J2 step) or a pool's FP32 array, read
// from `first` with SoA stride `stride` and promoted to double.
template <typename In>
__global__ void __launch_bounds__(kBlock) tet_omega2(long long tets, const In* rest_inv, long long stride,
                                                     double lambda, double mu, double rho, double* block_max) {
    __shared__ double smax[kBlock];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double w2 = 0.0;
    if (t < tets) {
        double g[4][3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int a = 0; a < 3; ++a) g[c + 1][a] = (double)rest_inv[(size_t)(a * 3 + c) * stride + t];
#pragma unroll
        for (int a = 0; a < 3; ++a) g[0][a] = -(g[1][a] + g[2][a] + g[3][a]);
        w2 = tet_omega2_one(g, lambda, mu, rho);
    }
    smax[threadIdx.x] = w2;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) block_max[blockIdx.x] = smax[0];
}

__global__ void __launch_bounds__(1024) reduce_sum(const double* in, long long n, double* out) {
    __shared__ double scratch[32];
    double s = 0.0;
    for (long long i = threadIdx.x; i < n; i += blockDim.x) s += in[i];
    const double total = block_sum(s, scratch);
    if (threadIdx.x == 0) out[0] = total;
}

__global__ void __launch_bounds__(1024) reduce_max(const double* in, long long n, double* out) {
    __shared__ double smax[1024];
    double s = 0.0;
    for (long long i = threadIdx.x; i < n; i += blockDim.x) s = fmax(s, in[i]);
    smax[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = smax[0];
}

// computeRestState (fem.cpp:119-158) in FP64 on the device, with the host's operations
// in the host's order (tet_rest_state64 in api_common.cu, compiled without contraction
// as this file is): per tet Dm^-1 (SoA rows of `tets`), |det| / 6 and its quarter of
// the lumped mass.
__global__ void tet_rest64_kernel(const float* position, const uint32_t* index, long long tets, double density,
                                  double* inv, double* vol, double* quarter) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tets) return;
    const uint32_t* idx = index + t * 4;
    double a[9];  // column-major
    for (int c = 0; c < 3; ++c)
        for (int r = 0; r < 3; ++r)
            a[c * 3 + r] = (double)position[(size_t)idx[c + 1] * 3 + r] - (double)position[(size_t)idx[0] * 3 + r];
#define A(r, c) a[(c) * 3 + (r)]
    const double det = A(0, 0) * (A(1, 1) * A(2, 2) - A(1, 2) * A(2, 1)) -
                       A(0, 1) * (A(1, 0) * A(2, 2) - A(1, 2) * A(2, 0)) +
                       A(0, 2) * (A(1, 0) * A(2, 1) - A(1, 1) * A(2, 0));
    const double volume = fabs(det / 6.0);
    const double id = fabs(det) > 1e-300 ? 1.0 / det : 0.0;
    double r[9];
#define R(rr, cc) r[(cc) * 3 + (rr)]
    R(0, 0) = (A(1, 1) * A(2, 2) - A(1, 2) * A(2, 1)) * id;
    R(0, 1) = (A(0, 2) * A(2, 1) - A(0, 1) * A(2, 2)) * id;
    R(0, 2) = (A(0, 1) * A(1, 2) - A(0, 2) * A(1, 1)) * id;
    R(1, 0) = (A(1, 2) * A(2, 0) - A(1, 0) * A(2, 2)) * id;
    R(1, 1) = (A(0, 0) * A(2, 2) - A(0, 2) * A(2, 0)) * id;
    R(1, 2) = (A(0, 2) * A(1, 0) - A(0, 0) * A(1, 2)) * id;
    R(2, 0) = (A(1, 0) * A(2, 1) - A(1, 1) * A(2, 0)) * id;
    R(2, 1) = (A(0, 1) * A(2, 0) - A(0, 0) * A(2, 1)) * id;
    R(2, 2) = (A(0, 0) * A(1, 1) - A(0, 1) * A(1, 0)) * id;
#undef R
#undef A
    for (int k = 0; k < 9; ++k) inv[(size_t)k * tets + t] = r[k];
    vol[t] = volume;
    quarter[t] = density * volume * 0.25;
}

// Each node's lumped mass: its tets' quarters summed over its CSR run, which lists its
// corners in ascending tet order -- the order the host's loop adds them in.
__global__ void tet_mass64_kernel(const uint32_t* offset, const uint32_t* entry, long long nodes, const double* quarter,
                                  double* mass) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nodes) return;
    double m = 0.0;
    for (uint32_t k = offset[n]; k < offset[n + 1]; ++k) m += quarter[entry[k] >> 2];
    mass[n] = m;
}

// The FP32 modes' copies of the FP64 rest state, rounded once.
__global__ void tet_rest_f32_kernel(const double* inv, const double* vol, long long tets, float* inv32, float* vol32) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tets) return;
    for (int k = 0; k < 9; ++k) inv32[(size_t)k * tets + t] = (float)inv[(size_t)k * tets + t];
    vol32[t] = (float)vol[t];
}

__global__ void tet_mass_f32_kernel(const double* mass, long long nodes, float* mass32, float* inv_mass32) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nodes) return;
    mass32[n] = (float)mass[n];
    inv_mass32[n] = mass[n] > 0.0 ? (float)(1.0 / mass[n]) : 0.0f;
}

__global__ void widen_kernel(const float* in, long long n, double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (double)in[i];
}

}  // namespace

void launch_tet_rest64(const float* position, const uint32_t* index, long long tets, double density, double* inv,
                       double* vol, double* quarter, cudaStream_t stream) {
    tet_rest64_kernel<<<blocks_for(tets, kBlock), kBlock, 0, stream>>>(position, index, tets, density, inv, vol,
                                                                       quarter);
}

void launch_tet_mass64(const uint32_t* offset, const uint32_t* entry, long long nodes, const double* quarter,
                       double* mass, cudaStream_t stream) {
    tet_mass64_kernel<<<blocks_for(nodes, kBlock), kBlock, 0, stream>>>(offset, entry, nodes, quarter, mass);
}

void launch_tet_rest_f32(const double* inv, const double* vol, long long tets, const double* mass, long long nodes,
                         float* inv32, float* vol32, float* mass32, float* inv_mass32, cudaStream_t stream) {
    tet_rest_f32_kernel<<<blocks_for(tets, kBlock), kBlock, 0, stream>>>(inv, vol, tets, inv32, vol32);
    tet_mass_f32_kernel<<<blocks_for(nodes, kBlock), kBlock, 0, stream>>>(mass, nodes, mass32, inv_mass32);
}

void launch_widen(const float* in, long long n, double* out, cudaStream_t stream) {
    widen_kernel<<<blocks_for(n, kBlock), kBlock, 0, stream>>>(in, n, out);
}

void launch_ref32_step(const TetDevice<float>& d, const TetParams& p, cudaStream_t stream, int parts) {
    const float lambda = (float)p.lambda, mu = (float)p.mu;
    if (parts & kElementPart) launch_pdl(ref32_forces, blocks_for(d.tets, kBlock), kBlock, 0, stream, d, lambda, mu);
    if (parts & kNodePart)
        launch_pdl(ref32_nodes, blocks_for(d.nodes, kTetNodeBlock), kTetNodeBlock, 0, stream, d, (float)p.dt,
                   (float)p.gravity, (float)p.damping);
}

bool launch_ref32_cluster(const TetDevice<float>& d, const TetParams& p, int steps, cudaStream_t stream) {
    int blocks, threads;
    cluster_shape(std::max(d.tets, d.nodes), blocks, threads);
    return launch_cluster(ref32_cluster, blocks, threads, 0, stream, d, (float)p.lambda, (float)p.mu, (float)p.dt,
                          (float)p.gravity, (float)p.damping, steps);
}

bool launch_f64_cluster(const TetDevice<double>& d, const TetParams& p, int steps, cudaStream_t stream) {
    int blocks, threads;
    cluster_shape(std::max(d.tets, d.nodes), blocks, threads);
    return launch_cluster(f64_cluster, blocks, threads, sizeof(PolarPark) * (threads / 128), stream, d, p, steps);
}

void launch_f64_step(const TetDevice<double>& d, const TetParams& p, cudaStream_t stream, int parts) {
    if (parts & kElementPart) launch_pdl(f64_forces, blocks_for(d.tets, kTet64Block), kTet64Block, 0, stream, d, p);
    if (parts & kNodePart) launch_pdl(f64_nodes, blocks_for(d.nodes, kTetNodeBlock), kTetNodeBlock, 0, stream, d, p);
}

void launch_tet_omega2(long long tets, const double* rest_inv, double E, double nu, double rho,
                       double* per_block_max, int blocks, cudaStream_t stream) {
    const double lambda = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
    const double mu = E / (2.0 * (1.0 + nu));
    tet_omega2<double><<<blocks, kBlock, 0, stream>>>(tets, rest_inv, tets, lambda, mu, rho, per_block_max);
}

void launch_tet_omega2_f32(long long tets, const float* rest_inv, long long stride, double E, double nu, double rho,
                           double* per_block_max, int blocks, cudaStream_t stream) {
    const double lambda = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
    const double mu = E / (2.0 * (1.0 + nu));
    tet_omega2<float><<<blocks, kBlock, 0, stream>>>(tets, rest_inv, stride, lambda, mu, rho, per_block_max);
}

void launch_reduce_sum(const double* in, long long n, double* out, cudaStream_t stream) {
    reduce_sum<<<1, 1024, 0, stream>>>(in, n, out);
}

void launch_reduce_max(const double* in, long long n, double* out, cudaStream_t stream) {
    reduce_max<<<1, 1024, 0, stream>>>(in, n, out);
}

}  // namespace fs
