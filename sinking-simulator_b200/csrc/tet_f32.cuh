// tet_f32.cuh -- the FP32 J2 tet element and node updates, shared by the single-mesh
// step (tet_fast.cu) and the batched / served pool (pool.cu).
//
// Same element and node update as the FP64 step (fem.cpp's co-rotational tet,
// plasticity::update's radial return, fem.cpp's node loop with a ramped external load),
// re-formulated so that FP32 keeps the digits that matter:
//
//   * nodes carry the displacement u = x - X (rest X fixed), not the position, so a
//     step's increment v dt ~ 1e-7 m is added to a number of size |u| ~ 1e-3 m rather
//     than |x| ~ 1 m.  The compensated variant adds it with Kahan summation and keeps
//     the pair (u, c), true value u - c, as a double-float: the element forms a
//     neighbour difference as (u_b - u_a) - (c_b - c_a), where the first difference is
//     exact (the two are within a factor of two, Sterbenz) and the second restores the
//     low bits u alone has lost.  A strain of 1e-4 on a displacement of 1e-2 m keeps
//     its digits instead of losing eleven bits to the subtraction;
//   * the element works on the displacement gradient H = Du Dm^-1 and the rotation's
//     deviation from identity Q = R - I, never on F = I + H and R themselves, so the
//     strain R^T F - I = H + Q^T + Q^T H is formed from small terms with no
//     cancellation.  The Higham iteration R <- (R + R^-T)/2 is carried in Q:
//     Q <- (Q - (M Q)^T)/2 with M = (I + Q)^-1 (fem.cpp:62-69), for as many steps as
//     FP32 needs at the tet's stretch (two for elastic steel, up to the reference's
//     four);
//   * the plastic strain is accumulated with Kahan compensation in the compensated
//     variant.
//
// Every file that includes this one is compiled without FMA contraction
// (-fmad=false); the fused multiply-adds below are written out (__fmaf_rn).  The
// arithmetic is then the same in every kernel that inlines these functions -- the
// single-mesh step, the pool's launches and its persistent kernel -- so a mesh gets
// the same bits whichever of them steps it.
#pragma once

#include "common.cuh"
#include "tet.hpp"

namespace fs {

__device__ __forceinline__ void kahan_add(float& sum, float& comp, float x) {
    const float y = x - comp;
    const float t = sum + y;
    comp = (t - sum) - y;
    sum = t;
}

// a * b with each entry an explicit FMA chain: (a_i0 b_0j + a_i1 b_1j) + a_i2 b_2j
__device__ __forceinline__ M3<float> mul_fma(const M3<float>& a, const M3<float>& b) {
    M3<float> r;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i) r(i, c) = __fmaf_rn(a(i, 2), b(2, c), __fmaf_rn(a(i, 1), b(1, c), a(i, 0) * b(0, c)));
    return r;
}

// (I + Q)^-1 by the adjugate with FMA cofactors, for the Higham step.  A singular
// matrix (|det| <= tiny) gives zero, as fem.cpp's inverse does.
__device__ __forceinline__ M3<float> inverse_fma(const M3<float>& a, float tiny) {
    const float c00 = __fmaf_rn(a(1, 1), a(2, 2), -(a(1, 2) * a(2, 1)));
    const float c01 = __fmaf_rn(a(1, 2), a(2, 0), -(a(1, 0) * a(2, 2)));
    const float c02 = __fmaf_rn(a(1, 0), a(2, 1), -(a(1, 1) * a(2, 0)));
    const float det = __fmaf_rn(a(0, 2), c02, __fmaf_rn(a(0, 1), c01, a(0, 0) * c00));
    const float id = fabsf(det) > tiny ? 1.0f / det : 0.0f;
    M3<float> r;
    r(0, 0) = c00 * id;
    r(1, 0) = c01 * id;
    r(2, 0) = c02 * id;
    r(0, 1) = __fmaf_rn(a(0, 2), a(2, 1), -(a(0, 1) * a(2, 2))) * id;
    r(1, 1) = __fmaf_rn(a(0, 0), a(2, 2), -(a(0, 2) * a(2, 0))) * id;
    r(2, 1) = __fmaf_rn(a(0, 1), a(2, 0), -(a(0, 0) * a(2, 1))) * id;
    r(0, 2) = __fmaf_rn(a(0, 1), a(1, 2), -(a(0, 2) * a(1, 1))) * id;
    r(1, 2) = __fmaf_rn(a(0, 2), a(1, 0), -(a(0, 0) * a(1, 2))) * id;
    r(2, 2) = __fmaf_rn(a(0, 0), a(1, 1), -(a(0, 1) * a(1, 0))) * id;
    return r;
}

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

struct TetElementRefs {
    const uint4* index;     // [stride] node ids
    const uint4* slot;      // [stride] node-major slot of each corner
    const float* rest_inv;  // [9][stride]
    const float* rest_vol;  // [stride]
    float* plastic;         // [7][stride]
    float* plastic_c;       // [7][stride] (compensated variant)
    const float4* disp;     // [N] (ux, uy, uz, 0)
    const float4* disp_c;   // [N] Kahan compensation (compensated variant)
    float4* slots;          // [4 * stride]: one (fx, fy, fz, 0) per corner
    long long stride;       // SoA stride (tets, or the pool's tet capacity)
};

struct J2f {
    float mu, kappa, yield, hardening;
    // for the strain-energy density: 1 / (2 mu), 1 / (3 kappa)
    float inv_2mu_f, inv_3kappa_f;
};

// The material record of the FP32 J2 tet from the FP64 constants.
__host__ __device__ inline J2f make_j2f(double mu, double kappa, double yield, double hardening) {
    return J2f{(float)mu, (float)kappa, (float)yield, (float)hardening, (float)(1.0 / (2.0 * mu)),
               (float)(1.0 / (3.0 * kappa))};
}

// L2 prefetch of the per-tet rows of tets [begin, end) -- one 128-byte line per thread
// of the block: index (16 B per tet), slot map (16 B), Dm^-1 (9 rows of 4 B), volume
// and the plastic state (7 rows).  A block issues it for the tile one wave ahead, so
// that block's first loads, the ones whose results the gathers wait for, hit L2.  Every
// address lies inside [begin, end) of its row.
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

__device__ __forceinline__ void prefetch_tet_rows(const TetElementRefs& d, long long begin, long long end) {
    if (end <= begin) return;
    const int x = threadIdx.x;
    const long long n = end - begin;
    const int wide = (int)((n * 16 + 127) >> 7);   // lines of a 16-byte row
    const int narrow = (int)((n * 4 + 127) >> 7);  // lines of a 4-byte row
    // each 4-byte row gets a power-of-two count of threads (no integer division);
    // threads past the row's last line issue nothing
    const int span = narrow <= 1 ? 1 : 1 << (32 - __clz(narrow - 1));
    const int shift = 31 - __clz(span);
    int k = x;
    if (k < wide) {
        prefetch_l2(reinterpret_cast<const char*>(d.index + begin) + ((long long)k << 7));
        return;
    }
    k -= wide;
    if (k < wide) {
        prefetch_l2(reinterpret_cast<const char*>(d.slot + begin) + ((long long)k << 7));
        return;
    }
    k -= wide;
    const int row = k >> shift, line = k & (span - 1);
    if (line >= narrow) return;
    const float* base;
    if (row < 9)
        base = d.rest_inv + (size_t)row * d.stride;
    else if (row == 9)
        base = d.rest_vol;
    else if (row < 17)
        base = d.plastic + (size_t)(row - 10) * d.stride;
    else
        return;
    prefetch_l2(reinterpret_cast<const char*>(base + begin) + ((long long)line << 7));
}

// Where a tet's own rows (node ids, slot map, Dm^-1, volume, plastic state) are read:
// straight from global memory, or from a block's copy of its tile in shared memory.
struct GlobalRows {
    const TetElementRefs& d;
    __device__ __forceinline__ uint4 index(long long t) const { return d.index[t]; }
    __device__ __forceinline__ uint4 slot(long long t) const { return d.slot[t]; }
    __device__ __forceinline__ float inv(int k, long long t) const { return d.rest_inv[(size_t)k * d.stride + t]; }
    __device__ __forceinline__ float vol(long long t) const { return d.rest_vol[t]; }
    __device__ __forceinline__ float plastic(int i, long long t) const { return d.plastic[(size_t)i * d.stride + t]; }
};

// The rows no step changes already in registers (loaded before the step's other data may
// be touched), the plastic state from global memory.
struct LoadedRows {
    uint4 idx, slt;
    float dm[9], v;
    const TetElementRefs& d;
    __device__ __forceinline__ LoadedRows(const TetElementRefs& refs, long long t) : d(refs) {
        idx = refs.index[t];
        slt = refs.slot[t];
#pragma unroll
        for (int k = 0; k < 9; ++k) dm[k] = refs.rest_inv[(size_t)k * refs.stride + t];
        v = refs.rest_vol[t];
    }
    __device__ __forceinline__ uint4 index(long long) const { return idx; }
    __device__ __forceinline__ uint4 slot(long long) const { return slt; }
    __device__ __forceinline__ float inv(int k, long long) const { return dm[k]; }
    __device__ __forceinline__ float vol(long long) const { return v; }
    __device__ __forceinline__ float plastic(int i, long long t) const { return d.plastic[(size_t)i * d.stride + t]; }
};

// A tile's rows in shared memory: index and slot map per tet from `first`, and 17
// float rows (Dm^-1 0..8, volume 9, plastic state 10..16) of `pitch` floats each from
// `base` (`first` rounded down to a multiple of 4, the 16-byte boundary of a row).
struct SharedRows {
    const uint4* idx;
    const uint4* slt;
    const float* rows;
    int pitch;
    long long first, base;
    __device__ __forceinline__ uint4 index(long long t) const { return idx[t - first]; }
    __device__ __forceinline__ uint4 slot(long long t) const { return slt[t - first]; }
    __device__ __forceinline__ float inv(int k, long long t) const { return rows[k * pitch + (int)(t - base)]; }
    __device__ __forceinline__ float vol(long long t) const { return rows[9 * pitch + (int)(t - base)]; }
    __device__ __forceinline__ float plastic(int i, long long t) const {
        return rows[(10 + i) * pitch + (int)(t - base)];
    }
};

// The rotation's deviation Q = R - I and the co-rotated strain U - I (engineering shears)
// of F = I + H = R U, from the displacement gradient H.
//
// At a small stretch, by series: with B = (H + H^T + H^T H) / 2 = (U^2 - I) / 2 exactly, its
// square root E = U - I by the fixed point E <- B - E^2 / 2 from E = B, and Q by
// Q <- X - Q E from Q = X = H - E (from R U = F).  Each round gains a factor |E|: after
// n rounds E is off by |E|^(n+2) / 2 and Q by |X| |E|^(n+1), so two rounds reach FP32's
// precision at elastic strains and three up to |E| of about 1e-2.  Beyond, by the Higham
// iteration Q <- (Q - (M Q)^T) / 2, M = (I + Q)^-1 (fem.cpp:62-69), which squares the
// stretch error and halves it: three steps up to 0.1, the reference's four beyond.
// The series has no divide and, in two rounds, 160 operations against 300 for two Higham
// steps and R^T F (a tiled element pass of 3.9 M tets: 127 M -> 109 M warp instructions).
// The squares are summed apart, so an entry of E takes one rounding at its own size:
// at rotations of 1e-3 to 0.5 rad the strain's relative error is 0.1 to 1 of what it was
// as R^T F - I (5.6e-7 for 4.8e-6 at 0.1 rad and a strain of 1e-3), and where nothing
// rotates 4.5e-8 for 3.7e-8; the solvers' errors against 64 bits are unchanged or smaller.
constexpr float kSeriesTwo = 1.25e-3f, kSeriesThree = 6e-3f;  // on the largest entry of B

// One round: E <- B - E^2 / 2.
__device__ __forceinline__ void series_round(const float (&b)[6], float (&e)[6]) {
    // entries xx yy zz xy yz zx
    const float xx = e[0], yy = e[1], zz = e[2], xy = e[3], yz = e[4], zx = e[5];
    e[0] = __fmaf_rn(-0.5f, __fmaf_rn(zx, zx, __fmaf_rn(xy, xy, xx * xx)), b[0]);
    e[1] = __fmaf_rn(-0.5f, __fmaf_rn(yz, yz, __fmaf_rn(xy, xy, yy * yy)), b[1]);
    e[2] = __fmaf_rn(-0.5f, __fmaf_rn(zx, zx, __fmaf_rn(yz, yz, zz * zz)), b[2]);
    e[3] = __fmaf_rn(-0.5f, __fmaf_rn(zx, yz, __fmaf_rn(xy, yy, xx * xy)), b[3]);
    e[4] = __fmaf_rn(-0.5f, __fmaf_rn(yz, zz, __fmaf_rn(yy, yz, xy * zx)), b[4]);
    e[5] = __fmaf_rn(-0.5f, __fmaf_rn(zz, zx, __fmaf_rn(yz, xy, zx * xx)), b[5]);
}

// Q <- X - Q E.
__device__ __forceinline__ void series_rotate(const M3<float>& x, const float (&e)[6], M3<float>& q) {
    const int at[3][3] = {{0, 3, 5}, {3, 1, 4}, {5, 4, 2}};
    M3<float> r;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            r(i, j) = __fmaf_rn(-q(i, 2), e[at[2][j]], __fmaf_rn(-q(i, 1), e[at[1][j]], __fmaf_rn(-q(i, 0), e[at[0][j]], x(i, j))));
    q = r;
}

__device__ __forceinline__ void tet_polar_f32(const M3<float>& h, M3<float>& q, float (&strain)[6]) {
    float b[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int j = (i + 1) % 3;
        b[i] = __fmaf_rn(0.5f, __fmaf_rn(h(2, i), h(2, i), __fmaf_rn(h(1, i), h(1, i), h(0, i) * h(0, i))), h(i, i));
        b[3 + i] = 0.5f * ((h(i, j) + h(j, i)) +
                           __fmaf_rn(h(2, i), h(2, j), __fmaf_rn(h(1, i), h(1, j), h(0, i) * h(0, j))));
    }
    const float big = fmaxf(fmaxf(fmaxf(fabsf(b[0]), fabsf(b[1])), fmaxf(fabsf(b[2]), fabsf(b[3]))),
                            fmaxf(fabsf(b[4]), fabsf(b[5])));
    if (big <= kSeriesThree) {
        float e[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) e[i] = b[i];
        series_round(b, e);
        series_round(b, e);
        const bool third = big > kSeriesTwo;
        if (third) series_round(b, e);
        const M3<float> x = [&] {
            M3<float> d = h;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int j = (i + 1) % 3;
                d(i, i) -= e[i];
                d(i, j) -= e[3 + i];
                d(j, i) -= e[3 + i];
            }
            return d;
        }();
        q = x;
        series_rotate(x, e, q);
        series_rotate(x, e, q);
        if (third) series_rotate(x, e, q);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            strain[i] = e[i];
            strain[3 + i] = 2.0f * e[3 + i];
        }
        return;
    }
    const int higham_steps = big <= 0.1f ? 3 : 4;
    q = h;
#pragma unroll 1
    for (int it = 0; it < higham_steps; ++it) {
        M3<float> ipq = q;
        ipq(0, 0) += 1.0f;
        ipq(1, 1) += 1.0f;
        ipq(2, 2) += 1.0f;
        const M3<float> mq = mul_fma(inverse_fma(ipq, 1e-30f), q);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) ipq(i, j) = 0.5f * (q(i, j) - mq(j, i));
        q = ipq;
    }
    const M3<float> qt = transpose(q);
    const M3<float> qth = mul_fma(qt, h);
    strain[0] = h(0, 0) + qt(0, 0) + qth(0, 0);
    strain[1] = h(1, 1) + qt(1, 1) + qth(1, 1);
    strain[2] = h(2, 2) + qt(2, 2) + qth(2, 2);
    strain[3] = (h(0, 1) + qt(0, 1) + qth(0, 1)) + (h(1, 0) + qt(1, 0) + qth(1, 0));
    strain[4] = (h(1, 2) + qt(1, 2) + qth(1, 2)) + (h(2, 1) + qt(2, 1) + qth(2, 1));
    strain[5] = (h(2, 0) + qt(2, 0) + qth(2, 0)) + (h(0, 2) + qt(0, 2) + qth(0, 2));
}

// One tet from its four corners' displacements un (and compensations cn), however
// they were fetched: its four corner forces into fc (x, y, z, 0), its plastic state
// advanced; the dissipation and strain energy of the element in diss / energy (FP64,
// for the energy account).  The arithmetic is the same whichever `Rows` supplies the
// tet's own rows.
template <bool KAHAN, class Rows>
__device__ __forceinline__ void tet_element_f32_eval(const TetElementRefs& d, const Rows& rows, long long t,
                                                     const J2f& m, const float4 (&un)[4], const float4 (&cn)[4],
                                                     double& diss, double& energy, float4 (&fc)[4]) {
    M3<float> du, dm_inv;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        du(0, c) = un[c + 1].x - un[0].x;
        du(1, c) = un[c + 1].y - un[0].y;
        du(2, c) = un[c + 1].z - un[0].z;
        if (KAHAN) {  // true value u - c
            du(0, c) -= cn[c + 1].x - cn[0].x;
            du(1, c) -= cn[c + 1].y - cn[0].y;
            du(2, c) -= cn[c + 1].z - cn[0].z;
        }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) dm_inv.m[k] = rows.inv(k, t);
    const M3<float> h = mul_fma(du, dm_inv);  // displacement gradient
    M3<float> q;
    float strain[6];
    tet_polar_f32(h, q, strain);

    // radial return, linear isotropic hardening (plasticity.cpp:333-456); for a linear
    // curve the consistency condition is affine in dgamma and its root is the closed
    // form below, which the CPU's Newton reaches in one step.
    float ps[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) ps[i] = rows.plastic(i, t);
    float el[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) el[i] = strain[i] - ps[i];
    const float vol_strain = el[0] + el[1] + el[2];
    const float pressure = m.kappa * vol_strain;
    const float two_mu = 2.0f * m.mu, third = vol_strain * (1.0f / 3.0f);
    float trial[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        trial[i] = two_mu * (el[i] - third);
        trial[3 + i] = m.mu * el[3 + i];
    }
    const float shear2 = __fmaf_rn(trial[5], trial[5], __fmaf_rn(trial[4], trial[4], trial[3] * trial[3]));
    const float norm2 = __fmaf_rn(
        2.0f, shear2, __fmaf_rn(trial[2], trial[2], __fmaf_rn(trial[1], trial[1], trial[0] * trial[0])));
    const float root23 = 0.81649658092772603f;
    const float radius = root23 * __fmaf_rn(m.hardening, fmaxf(ps[6], 0.0f), m.yield);
    // an elastic tet needs no square root: norm > radius is decided on the squares
    float norm = 0.0f, excess = 0.0f;
    if (norm2 > radius * fabsf(radius)) {
        norm = sqrtf(norm2);
        excess = norm - radius;
    }
    float dev = norm2;  // s : s of the final stress, for the energy
    float sv[6];
    diss = 0.0;
    if (excess > 0.0f) {
        const float gamma = excess / __fmaf_rn(2.0f / 3.0f, m.hardening, two_mu);
        const float inv_norm = 1.0f / norm;
        const float k = two_mu * gamma * inv_norm;
        const float left = __fmaf_rn(-two_mu, gamma, norm);
        dev = left * left;
        float dp[6];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            dp[i] = gamma * (trial[i] * inv_norm);
            sv[i] = pressure + __fmaf_rn(-k, trial[i], trial[i]);
        }
#pragma unroll
        for (int i = 3; i < 6; ++i) {
            dp[i] = 2.0f * gamma * (trial[i] * inv_norm);
            sv[i] = __fmaf_rn(-k, trial[i], trial[i]);
        }
        float dsum = 0.0f;
#pragma unroll
        for (int i = 0; i < 6; ++i) dsum += sv[i] * dp[i];
        diss = (double)dsum;
        const float deq = root23 * gamma;
        if (KAHAN) {
            // the compensation is read only where the state changes
            float pc[7];
#pragma unroll
            for (int i = 0; i < 7; ++i) pc[i] = d.plastic_c[(size_t)i * d.stride + t];
#pragma unroll
            for (int i = 0; i < 6; ++i) kahan_add(ps[i], pc[i], dp[i]);
            kahan_add(ps[6], pc[6], deq);
#pragma unroll
            for (int i = 0; i < 7; ++i) d.plastic_c[(size_t)i * d.stride + t] = pc[i];
        } else {
#pragma unroll
            for (int i = 0; i < 6; ++i) ps[i] += dp[i];
            ps[6] += deq;
        }
#pragma unroll
        for (int i = 0; i < 7; ++i) d.plastic[(size_t)i * d.stride + t] = ps[i];
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            sv[i] = pressure + trial[i];
            sv[3 + i] = trial[3 + i];
        }
    }
    const float volf = rows.vol(t);
    diss *= (double)volf;
    // 1/2 sigma : C^-1 : sigma = 1/2 [s : s / (2 mu) + p tr(sigma) / (3 kappa)], tr(sigma) =
    // 3 p, the engineering shears counted twice in s : s; the density in FP32 (a relative
    // error of a few ulps per tet), the account summed in FP64
    energy = (double)(volf * 0.5f * __fmaf_rn(dev, m.inv_2mu_f, 3.0f * pressure * pressure * m.inv_3kappa_f));
    // P = R sigma = sigma + Q sigma; nodal forces f_c = -V (P Dm^-T) column c, with -V
    // taken into sigma
    const float scale = -volf;
    M3<float> sig, pk;
    sig(0, 0) = scale * sv[0];
    sig(1, 1) = scale * sv[1];
    sig(2, 2) = scale * sv[2];
    sig(0, 1) = sig(1, 0) = scale * sv[3];
    sig(1, 2) = sig(2, 1) = scale * sv[4];
    sig(2, 0) = sig(0, 2) = scale * sv[5];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            pk(i, c) = __fmaf_rn(q(i, 2), sig(2, c), __fmaf_rn(q(i, 1), sig(1, c), __fmaf_rn(q(i, 0), sig(0, c), sig(i, c))));
    const M3<float> hf = mul_fma(pk, transpose(dm_inv));
#pragma unroll
    for (int c = 0; c < 3; ++c) fc[c + 1] = make_float4(hf(0, c), hf(1, c), hf(2, c), 0.0f);
    fc[0] = make_float4(-hf(0, 0) - hf(0, 1) - hf(0, 2), -hf(1, 0) - hf(1, 1) - hf(1, 2),
                        -hf(2, 0) - hf(2, 1) - hf(2, 2), 0.0f);
}

// The same with the corner forces written to the node-major slots (one 16-byte store
// each).
template <bool KAHAN, class Rows>
__device__ __forceinline__ void tet_element_f32_corners(const TetElementRefs& d, const Rows& rows, long long t,
                                                        const J2f& m, const float4 (&un)[4], const float4 (&cn)[4],
                                                        double& diss, double& energy) {
    float4 fc[4];
    tet_element_f32_eval<KAHAN, Rows>(d, rows, t, m, un, cn, diss, energy, fc);
    const uint4 sl = rows.slot(t);
    d.slots[sl.y] = fc[1];
    d.slots[sl.z] = fc[2];
    d.slots[sl.w] = fc[3];
    d.slots[sl.x] = fc[0];
}

template <bool KAHAN, bool CG = false, class Rows = GlobalRows>
__device__ __forceinline__ void tet_element_f32(const TetElementRefs& d, const Rows& rows, long long t, const J2f& m,
                                                double& diss, double& energy) {
    const uint4 idx = rows.index(t);
    const unsigned nid[4] = {idx.x, idx.y, idx.z, idx.w};
    float4 un[4], cn[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) un[c] = ldg_coherent4<CG>(d.disp + nid[c]);
    if (KAHAN) {
#pragma unroll
        for (int c = 0; c < 4; ++c) cn[c] = ldg_coherent4<CG>(d.disp_c + nid[c]);
    }
    tet_element_f32_corners<KAHAN, Rows>(d, rows, t, m, un, cn, diss, energy);
}

template <bool KAHAN, bool CG = false>
__device__ __forceinline__ void tet_element_f32(const TetElementRefs& d, long long t, const J2f& m, double& diss,
                                                double& energy) {
    tet_element_f32<KAHAN, CG, GlobalRows>(d, GlobalRows{d}, t, m, diss, energy);
}

struct TetNodeRefs {
    const float4* slots;
    const uint8_t* fixed;
    const float* mass;
    const float* inv_mass;
    const float* ext;        // may be null
    float* velocity;
    float4* disp;            // (ux, uy, uz, 0)
    float4* disp_c;          // compensated variant
};

// One node: its run of slots summed in order, external load, symplectic Euler on the
// displacement.  BATCH slots' loads go out together; 0: a contiguous run, in the few
// registers the pool's node pass has.
template <bool KAHAN, bool CG = false, int BATCH = 8>
__device__ __forceinline__ void tet_node_f32(const TetNodeRefs& d, const SlotRun& run, long long n, float lf, float dt, float gravity,
                                             float damping, double& work, double& kin, double& gwork) {
    work = kin = gwork = 0.0;
    float* vel = d.velocity + (size_t)n * 3;
    if (d.fixed[n]) {
        vel[0] = 0.0f;
        vel[1] = 0.0f;
        vel[2] = 0.0f;
        return;
    }
    const float m = d.mass[n];
    float force[3] = {0.0f, 0.0f, -gravity * m};
    const auto add = [&](const float4& f) {
        force[0] += f.x;
        force[1] += f.y;
        force[2] += f.z;
    };
    if constexpr (BATCH == 0) {
        const uint32_t end = run.start + run.count;
#pragma unroll 4
        for (uint32_t k = run.start; k < end; ++k) add(ldg_coherent4<CG>(d.slots + k));
    } else {
        for_run<BATCH>(
            run, [&](uint32_t k) { return ldg_coherent4<CG>(d.slots + k); }, add);
    }
    float ext[3] = {0.0f, 0.0f, 0.0f};
    if (d.ext) {
#pragma unroll
        for (int k = 0; k < 3; ++k) ext[k] = lf * d.ext[(size_t)n * 3 + k];
    }
    const float im = d.inv_mass[n];
    float4 u4 = d.disp[n], c4 = KAHAN ? d.disp_c[n] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float* u = &u4.x;
    float* cu = &c4.x;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float v = vel[k] + (force[k] + ext[k]) * im * dt;
        v *= damping;
        vel[k] = v;
        const float du = v * dt;
        if (KAHAN)
            kahan_add(u[k], cu[k], du);
        else
            u[k] += du;
        work += (double)ext[k] * (double)v * (double)dt;
        kin += 0.5 * (double)m * (double)v * (double)v;
    }
    d.disp[n] = u4;
    if (KAHAN) d.disp_c[n] = c4;
    gwork = -(double)gravity * (double)m * (double)vel[2] * (double)dt;
}

}  // namespace fs
