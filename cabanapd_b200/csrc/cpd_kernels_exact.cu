// Plain-FP64 particle kernels of the hot path.
//
// This translation unit is compiled with --fmad=false: every per-bond
// expression is evaluated with separately rounded IEEE double operations in
// the reference's operand order, so per-particle sums walked in the same
// neighbour order are bit-identical to a scalar CPU evaluation of the
// reference's code. sqrt and '/' on doubles are the IEEE-rounded CUDA
// operations.
//
// Work decomposition: one thread per particle row. A thread keeps particle
// i's position, displacement and running force in registers and walks its
// padded-ELL row; the k-th loads of a warp's 32 consecutive rows are
// contiguous in the column-major list, and neighbour gathers of a lattice in
// x-fastest order are contiguous as well. Broken-bond state is one bit per
// bond, read and written a 32-bond word at a time.
#include <cuda_runtime.h>

#include "cpd_internal.cuh"
#include "cpd_epilogue.cuh"

namespace cpd {
namespace {

constexpr int kBlock = 256;

inline int blocks_for(int64_t rows) { return (int)((rows + kBlock - 1) / kBlock); }

struct ModelDev {
    double c, theta_coeff, s_coeff, bond_break_coeff;
    double Rs, Es, coeff_h_n, coeff_h_d, radius;
};

ModelDev to_dev(const Model& m)
{
    return ModelDev{m.c,  m.theta_coeff, m.s_coeff,   m.bond_break_coeff, m.Rs,
                    m.Es, m.coeff_h_n,   m.coeff_h_d, m.radius};
}

// Correctly rounded square roots and quotients of a bond, from one reciprocal
// square root per length. The IEEE operations each carry their own iteration
// and special cases; a bond has two roots and four quotients by its two
// lengths, which share the iterations here:
//   sqrt  g = a y, s = RN(g + (a - g^2) y / 2) with the residual exact by
//         FMA; s is the rounded root unless the sum lies next to a midpoint
//         of two doubles (within 2^-21 of a unit, found from the part of the
//         sum that s leaves, against errors of 2^-50 of a unit);
//   1 / b two Newton steps on y, correctly rounded unless b's significand is
//         all ones; quotients by two corrections with exact remainders
//         (P. W. Markstein, IBM J. Res. Dev. 34, 1990).
// Next to a midpoint and for a divisor that ends in ones settle() decides, and
// outside the middle of the exponent range (where a residual could round) the
// IEEE operations are taken, so every result is the IEEE one, but for the sign of a
// zero: the quotient of -0 is +0 here. The callers add their quotients to sums
// that start at +0, where neither zero changes anything. (The root's test is by
// the unit above a power of two; below one only the double next under an even
// power has its root next to a midpoint, and every y within an ulp of its
// reciprocal root gives a sum on the upper side, where the test sees it.)
// Issue-bound (68%; FP64 pipe 56%). Plates of 1.0 M and 80 thousand rows: 924
// and 100 us per step, 1095 and 132 with IEEE operations throughout; LPS boxes
// of the same sizes 1947 and 160, 2520 and 197.
__device__ __forceinline__ bool mid_square(double v)  // v in [2^-900, 2^900)
{
    return (uint32_t)(__double2hiint(v) - 0x07b00000) < 0x70800000u;
}
__device__ __forceinline__ uint32_t value_range(double v)  // below 0x7d000000: see mid_value
{
    return ((uint32_t)__double2hiint(v) << 1) - 0x41600000u;
}
__device__ __forceinline__ bool mid_value(double v)  // |v| in [2^-500, 2^500), or zero
{
    return value_range(v) < 0x7d000000u || v == 0.0;
}
// A divisor: y = RN(1 / b) when fast.
struct Divisor {
    double b, y;
    bool fast;
};
__device__ __forceinline__ Divisor divisor(double b, double y, bool fast)
{
    y = fma(y, fma(-b, y, 1.0), y);
    y = fma(y, fma(-b, y, 1.0), y);
    return Divisor{b, y, fast && __double2loint(b) != -1};
}
__device__ __forceinline__ double quotient(double a, const Divisor& d)  // a a middle value
{
    double q = a * d.y;
    q = fma(fma(-q, d.b, a), d.y, q);
    return fma(fma(-q, d.b, a), d.y, q);
}
__device__ __forceinline__ double divide(double a, const Divisor& d)
{
    return d.fast && mid_value(a) ? quotient(a, d) : a / d.b;
}
// RN(sqrt(a)) from y within an ulp of 1 / sqrt(a) where ok stays set.
__device__ __forceinline__ double root(double a, double y, bool& ok)
{
    const double g = a * y;
    const double e = fma(-g, g, a), h = 0.5 * y;
    const double r = fma(e, h, g);
    const double left = fma(e, h, g - r);  // the sum less r: at most half a unit of r
    // High words: half a unit of r is 2^-53 of its power of two.
    const int32_t half = (__double2hiint(r) & 0x7ff00000) - (53 << 20);
    ok = ok && (__double2hiint(left) & 0x7fffffff) < half - 1;
    return r;
}
// Where root() or divisor() could not tell: r, next to RN(sqrt(a)), to the
// rounded root by the signs of a less the products with its neighbours (the
// Tuckerman test), and its reciprocal; all ones are 2^e (1 - 2^-53), whose
// reciprocal rounds to 2^-e (1 + 2^-52). Lengths just below a power of two are
// no rarity: on a lattice of 24, 48 or 96 cells to the unit three spacings are
// one, six bonds of every row (cubes of 24, 48 and 96 cells: 71, 137 and 855 us
// per step, 83, 153 and 939 with the IEEE root and quotients for both lengths).
__device__ __forceinline__ void settle(double a, double& r, Divisor& d)
{
    if (!mid_square(a)) {
        r = sqrt(a);
        d = Divisor{r, 0.0, false};
        return;
    }
    const double up = __longlong_as_double(__double_as_longlong(r) + 1);
    const double down = __longlong_as_double(__double_as_longlong(r) - 1);
    if (fma(-r, up, a) > 0.0)
        r = up;
    else if (fma(-r, down, a) <= 0.0)
        r = down;
    const int32_t high = __double2hiint(r);
    d = divisor(r, d.y, true);
    if (__double2loint(r) == -1 && (high & 0xfffff) == 0xfffff)
        d.y = __hiloint2double((2045 - (high >> 20)) << 20, 1);
    d.fast = true;
}

// CabanaPD_Force.hpp:74-93 getDistance for the pair (i, j); particle i's
// position and displacement are already in registers. R: r as a divisor; X:
// xi.
struct BondEnd {
    double x0, x1, x2, u0, u1, u2;
};
struct Geometry {
    double xi, r, s, rx, ry, rz, xx, xy, xz;
    Divisor R, X;
};
__device__ __forceinline__ BondEnd bond_end(const double* __restrict__ x,
                                            const double* __restrict__ u, int64_t np, int64_t j)
{
    return BondEnd{__ldg(x + j), __ldg(x + np + j), __ldg(x + 2 * np + j),
                   __ldg(u + j), __ldg(u + np + j), __ldg(u + 2 * np + j)};
}
__device__ __forceinline__ void bond_geometry(const BondEnd& a, const BondEnd& b, Geometry& g)
{
    g.xx = b.x0 - a.x0;
    const double eta_u = b.u0 - a.u0;
    g.xy = b.x1 - a.x1;
    const double eta_v = b.u1 - a.u1;
    g.xz = b.x2 - a.x2;
    const double eta_w = b.u2 - a.u2;
    g.rx = g.xx + eta_u;
    g.ry = g.xy + eta_v;
    g.rz = g.xz + eta_w;
    const double r2 = g.rx * g.rx + g.ry * g.ry + g.rz * g.rz;
    const double x2 = g.xx * g.xx + g.xy * g.xy + g.xz * g.xz;
    bool ok_r = mid_square(r2), ok_x = mid_square(x2);
    const double yr = rsqrt(r2), yx = rsqrt(x2);
    g.r = root(r2, yr, ok_r);
    g.xi = root(x2, yx, ok_x);
    g.X = divisor(g.xi, yx, ok_x);
    g.R = divisor(g.r, yr, ok_r);
    // (r - xi is exact or far above the range where a remainder could round.)
    g.s = quotient(g.r - g.xi, g.X);
    if (!(g.X.fast && g.R.fast)) {
        if (!g.R.fast) settle(r2, g.r, g.R);
        if (!g.X.fast) settle(x2, g.xi, g.X);
        g.s = divide(g.r - g.xi, g.X);
    }
}
// The form the passes without a force take.
__device__ __forceinline__ void bond_geometry(
    const double* __restrict__ x, const double* __restrict__ u, int64_t np,
    int64_t j, double xi0, double xi1, double xi2, double ui0, double ui1,
    double ui2, double& xi, double& r, double& s, double& rx, double& ry,
    double& rz, double& xx, double& xy, double& xz, Divisor* X = nullptr)
{
    Geometry g;
    bond_geometry(BondEnd{xi0, xi1, xi2, ui0, ui1, ui2}, bond_end(x, u, np, j), g);
    xi = g.xi;
    r = g.r;
    s = g.s;
    rx = g.rx;
    ry = g.ry;
    rz = g.rz;
    xx = g.xx;
    xy = g.xy;
    xz = g.xz;
    if (X) *X = g.X;
}

// CabanaPD_Force.hpp:114-129 getLinearizedDistance.
__device__ __forceinline__ void bond_linearized(
    const double* __restrict__ x, const double* __restrict__ u, int64_t np,
    int64_t j, double xi0, double xi1, double xi2, double ui0, double ui1,
    double ui2, double& xi, double& s, double& xx, double& xy, double& xz)
{
    xx = __ldg(x + j) - xi0;
    const double eta_u = __ldg(u + j) - ui0;
    xy = __ldg(x + np + j) - xi1;
    const double eta_v = __ldg(u + np + j) - ui1;
    xz = __ldg(x + 2 * np + j) - xi2;
    const double eta_w = __ldg(u + 2 * np + j) - ui2;
    xi = sqrt(xx * xx + xy * xy + xz * xz);
    s = (xx * eta_u + xy * eta_v + xz * eta_w) / (xi * xi);
}

// force_models/CabanaPD_LPS.hpp:85-98.
template <int INFL>
__device__ __forceinline__ double influence(const Divisor& xi)
{
    if (INFL == 1) return xi.fast ? xi.y : 1.0 / xi.b;
    return 1.0;
}

// ---------------------------------------------------------------------------
// LPS weighted volume: force/CabanaPD_LPS.hpp:89-112 (NoFracture) and
// :287-329 (Fracture). m_i = sum_k mu_k * omega(xi) xi^2 vol_j.
template <int INFL, bool FRACTURE>
__global__ void __launch_bounds__(kBlock, 4)
    k_lps_weighted_volume(ParticleView p, EllView nl)
{
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    const double xi0 = p.x[i], xi1 = p.x[np + i], xi2 = p.x[2 * np + i];
    const double ui0 = p.u[i], ui1 = p.u[np + i], ui2 = p.u[2 * np + i];
    const int cnt = nl.count[i];
    double mi = 0.0;
    uint32_t word = 0;
    int32_t jn = cnt > 0 ? __ldg(nl.idx + i) : 0;  // (read one bond ahead)
    for (int k = 0; k < cnt; ++k) {
        if (FRACTURE && (k & 31) == 0) word = nl.mu[(int64_t)(k >> 5) * np + i];
        const int64_t j = jn;
        if (k + 1 < cnt) jn = __ldg(nl.idx + (int64_t)(k + 1) * np + i);
        double xi, r, s, rx, ry, rz, xx, xy, xz;
        Divisor X;
        bond_geometry(p.x, p.u, np, j, xi0, xi1, xi2, ui0, ui1, ui2, xi, r, s, rx,
                      ry, rz, xx, xy, xz, &X);
        const double wv = influence<INFL>(X) * xi * xi * __ldg(p.vol + j);
        if (FRACTURE)
            mi += (double)((word >> (k & 31)) & 1u) * wv;
        else
            mi += wv;
    }
    p.m[i] = mi;
}

// LPS dilatation: force/CabanaPD_LPS.hpp:114-141 (NoFracture), :331-378
// (Fracture). Also stores the per-particle factors of the force coefficient
// (force_models/CabanaPD_LPS.hpp:118-134): a = theta_coeff*theta/m and
// b = s_coeff/m, the exact subexpressions the force loop would otherwise
// recompute for every bond.
template <int INFL, bool FRACTURE>
__global__ void __launch_bounds__(kBlock, 4)
    k_lps_dilatation(ParticleView p, EllView nl, ModelDev md)
{
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    const double xi0 = p.x[i], xi1 = p.x[np + i], xi2 = p.x[2 * np + i];
    const double ui0 = p.u[i], ui1 = p.u[np + i], ui2 = p.u[2 * np + i];
    const double m_i = p.m[i];
    const Divisor M = divisor(m_i, 1.0 / m_i, mid_value(m_i) && m_i != 0.0);
    const int cnt = nl.count[i];
    double th = 0.0;
    uint32_t word = 0;
    int32_t jn = cnt > 0 ? __ldg(nl.idx + i) : 0;  // (read one bond ahead)
    for (int k = 0; k < cnt; ++k) {
        if (FRACTURE && (k & 31) == 0) word = nl.mu[(int64_t)(k >> 5) * np + i];
        const int64_t j = jn;
        if (k + 1 < cnt) jn = __ldg(nl.idx + (int64_t)(k + 1) * np + i);
        double xi, r, s, rx, ry, rz, xx, xy, xz;
        Divisor X;
        bond_geometry(p.x, p.u, np, j, xi0, xi1, xi2, ui0, ui1, ui2, xi, r, s, rx,
                      ry, rz, xx, xy, xz, &X);
        const double theta_i = influence<INFL>(X) * s * xi * xi * __ldg(p.vol + j);
        const double term = divide(3.0 * theta_i, M);
        if (FRACTURE) {
            if (m_i > 0) th += (double)((word >> (k & 31)) & 1u) * term;
        } else {
            th += term;
        }
    }
    p.theta[i] = th;
    p.lps_a[i] = md.theta_coeff * th / m_i;
    p.lps_b[i] = md.s_coeff / m_i;
}

// ---------------------------------------------------------------------------
// PD force. PMB: force/CabanaPD_PMB.hpp:89-125 (NoFracture), :222-287
// (Fracture); LinearPMB :406-455; LPS: force/CabanaPD_LPS.hpp:143-181
// (NoFracture), :380-447 (Fracture). LinearLPS systems run as LPS.
// The force is written (not accumulated): CabanaPD_Force.hpp:187-189 zeroes
// f before the kernel, and 0.0 + t == t.
enum { M_PMB = 0, M_LPS = 1, M_LINEAR_PMB = 2 };

template <int MODEL, int INFL, bool FRACTURE>
__global__ void __launch_bounds__(kBlock, 3)
    k_pd_force(ParticleView p, EllView nl, ModelDev md)
{
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    const double xi0 = p.x[i], xi1 = p.x[np + i], xi2 = p.x[2 * np + i];
    const double ui0 = p.u[i], ui1 = p.u[np + i], ui2 = p.u[2 * np + i];
    constexpr bool lps = MODEL == M_LPS;
    constexpr bool linear = MODEL == M_LINEAR_PMB;
    double a_i = 0.0, b_i = 0.0;
    if (lps) {
        a_i = p.lps_a[i];
        b_i = p.lps_b[i];
    }
    const bool nofail_i = FRACTURE ? (p.nofail[i] != 0) : false;
    const int cnt = nl.count[i];
    double fx = 0.0, fy = 0.0, fz = 0.0;
    uint32_t word = 0;
    bool dirty = false;
    const int32_t* __restrict__ const row = nl.idx + i;
    if (linear) {
        int32_t jn = cnt > 0 ? __ldg(row) : 0;  // (read one bond ahead)
        for (int k = 0; k < cnt; ++k) {
            const int64_t j = jn;
            if (k + 1 < cnt) jn = __ldg(row + (int64_t)(k + 1) * np);
            const double vol_j = __ldg(p.vol + j);
            double xi, ls, xx, xy, xz;
            bond_linearized(p.x, p.u, np, j, xi0, xi1, xi2, ui0, ui1, ui2, xi, ls,
                            xx, xy, xz);
            const double coeff = md.c * ls * vol_j;
            fx += coeff * xx / xi;
            fy += coeff * xy / xi;
            fz += coeff * xz / xi;
        }
    } else {
        // PMB takes two bonds at a time: their geometry and quotients are
        // independent chains, which the FP64 latency would otherwise leave in
        // series; their breaking and sums stay in row order. Indices are read
        // a pair ahead. (An odd row's last pair holds its last bond twice; the
        // copy adds nothing.) LPS carries two more gathers per bond and is
        // faster with one bond at a time (box of 1.0 M rows: 2.26 against 2.4 ms
        // per step) and at three blocks of 256 per SM (2.16; four: 2.26, with
        // the spills of 64 registers). Whether a bond breaks is decided beside
        // its force, so that its lengths need not be kept.
        constexpr int NB = lps ? 1 : 2;
        const BondEnd me{xi0, xi1, xi2, ui0, ui1, ui2};
        int32_t jn[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b)
            jn[b] = cnt > 0 ? __ldg(row + (int64_t)min(b, cnt - 1) * np) : 0;
        for (int k = 0; k < cnt; k += NB) {
            if (FRACTURE && (k & 31) == 0) {
                if (dirty) nl.mu[(int64_t)((k >> 5) - 1) * np + i] = word;
                dirty = false;
                word = nl.mu[(int64_t)(k >> 5) * np + i];
            }
            double qx[NB], qy[NB], qz[NB];
            bool breaks[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const int64_t j = jn[b];
                if (k + NB < cnt) jn[b] = __ldg(row + (int64_t)min(k + NB + b, cnt - 1) * np);
                const double vol_j = __ldg(p.vol + j);
                // LPS tests nofail(i) twice (force/CabanaPD_LPS.hpp:417-418),
                // PMB nofail(i) and nofail(j).
                const bool safe = FRACTURE && (nofail_i || (!lps && __ldg(p.nofail + j) != 0));
                Geometry g;
                bond_geometry(me, bond_end(p.x, p.u, np, j), g);
                // CabanaPD_ForceModels.hpp:123-128.
                breaks[b] = FRACTURE && g.r * g.r >= md.bond_break_coeff * g.xi * g.xi && !safe;
                double coeff;
                if (lps) {
                    const double a_j = __ldg(p.lps_a + j), b_j = __ldg(p.lps_b + j);
                    coeff = (a_i + a_j + g.s * (b_i + b_j)) * influence<INFL>(g.X) *
                            g.xi * vol_j;
                } else {
                    coeff = md.c * g.s * vol_j;
                }
                const double px = coeff * g.rx, py = coeff * g.ry, pz = coeff * g.rz;
                qx[b] = quotient(px, g.R);
                qy[b] = quotient(py, g.R);
                qz[b] = quotient(pz, g.R);
                if (!(g.R.fast &&
                      max(max(value_range(px), value_range(py)), value_range(pz)) < 0x7d000000u) &&
                    !(g.R.fast && mid_value(px) && mid_value(py) && mid_value(pz))) {
                    qx[b] = px / g.r;
                    qy[b] = py / g.r;
                    qz[b] = pz / g.r;
                }
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                if (k + b >= cnt) continue;
                bool intact = true;
                if (FRACTURE) {
                    const uint32_t bit = 1u << ((k + b) & 31);
                    if (breaks[b]) {
                        if (word & bit) {
                            word &= ~bit;
                            dirty = true;
                        }
                        intact = false;
                    } else {
                        intact = (word & bit) != 0;
                    }
                }
                // mu == 1 here, and 1.0 * coeff == coeff.
                if (intact) {
                    fx += qx[b];
                    fy += qy[b];
                    fz += qz[b];
                }
            }
        }
    }
    if (FRACTURE && dirty && cnt > 0) nl.mu[(int64_t)((cnt - 1) >> 5) * np + i] = word;
    p.f[i] = fx;
    p.f[np + i] = fy;
    p.f[2 * np + i] = fz;
}

// ---------------------------------------------------------------------------
// Strain energy density and damage: force/CabanaPD_PMB.hpp:127-155
// (NoFracture), :289-339 (Fracture), :458-491 (LinearPMB);
// force/CabanaPD_LPS.hpp:183-219, :449-504.
// Per particle W_i and phi_i are exact; the block partial sums of
// (sum_k w_k vol_i or W_i vol_i, phi_i) are reduced in a fixed tree order.
template <int MODEL, int INFL, bool FRACTURE>
__global__ void __launch_bounds__(kBlock, 3)
    k_pd_energy(ParticleView p, EllView nl, ModelDev md, double* partials)
{
    __shared__ double s_phi[kBlock];
    __shared__ double s_dmg[kBlock];
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double Phi_i = 0.0, dmg_i = 0.0;
    if (i < p.n) {
        const int64_t np = p.npad;
        const double xi0 = p.x[i], xi1 = p.x[np + i], xi2 = p.x[2 * np + i];
        const double ui0 = p.u[i], ui1 = p.u[np + i], ui2 = p.u[2 * np + i];
        constexpr bool lps = MODEL == M_LPS;
        constexpr bool linear = MODEL == M_LINEAR_PMB;
        const int cnt = nl.count[i];
        const double vol_i = p.vol[i];
        double m_i = 0.0, th_i = 0.0;
        if (lps) {
            m_i = p.m[i];
            th_i = p.theta[i];
        }
        double num_bonds = (double)cnt;
        if (FRACTURE && lps) {
            num_bonds = 0.0;
            for (int k = 0; k < cnt; ++k) {
                const uint32_t word = nl.mu[(int64_t)(k >> 5) * np + i];
                num_bonds += (double)((word >> (k & 31)) & 1u);
            }
        }
        // The row's constants of the LPS energy, as the formula associates them.
        const double w_theta =
            lps ? 1.0 / num_bonds * 0.5 * md.theta_coeff / 3.0 * (th_i * th_i) : 0.0;
        const double half_b = lps ? 0.5 * (md.s_coeff / m_i) : 0.0;
        double Wi = 0.0, phi_sum = 0.0, vol_H = 0.0;
        uint32_t word = 0;
        int32_t jn = cnt > 0 ? __ldg(nl.idx + i) : 0;  // (read one bond ahead)
        for (int k = 0; k < cnt; ++k) {
            if (FRACTURE && (k & 31) == 0) word = nl.mu[(int64_t)(k >> 5) * np + i];
            const int64_t j = jn;
            if (k + 1 < cnt) jn = __ldg(nl.idx + (int64_t)(k + 1) * np + i);
            const double vol_j = __ldg(p.vol + j);
            double s, xi;
            Divisor X;
            if (linear) {
                double xx, xy, xz;
                bond_linearized(p.x, p.u, np, j, xi0, xi1, xi2, ui0, ui1, ui2, xi, s,
                                xx, xy, xz);
            } else {
                double r, rx, ry, rz, xx, xy, xz;
                bond_geometry(p.x, p.u, np, j, xi0, xi1, xi2, ui0, ui1, ui2, xi, r, s,
                              rx, ry, rz, xx, xy, xz, &X);
            }
            double w;
            if (lps) {
                // force_models/CabanaPD_LPS.hpp:136-148
                w = w_theta + half_b * influence<INFL>(X) * s * s * xi * xi * vol_j;
            } else {
                // force_models/CabanaPD_PMB.hpp:64-71
                w = 0.25 * md.c * s * s * xi * vol_j;
            }
            if (FRACTURE) {
                const double mu = (double)((word >> (k & 31)) & 1u);
                w = mu * w;
                Wi += w;
                phi_sum += mu * vol_j;
                vol_H += vol_j;
            } else {
                Wi += w;
                Phi_i += w * vol_i;
            }
        }
        p.W[i] = Wi;
        if (FRACTURE) {
            dmg_i = 1 - phi_sum / vol_H;
            p.phi[i] = dmg_i;
            Phi_i = Wi * vol_i;
        }
    }
    s_phi[threadIdx.x] = Phi_i;
    s_dmg[threadIdx.x] = dmg_i;
    __syncthreads();
    for (int w = kBlock / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            s_phi[threadIdx.x] += s_phi[threadIdx.x + w];
            s_dmg[threadIdx.x] += s_dmg[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x + 0] = s_phi[0];
        partials[2 * blockIdx.x + 1] = s_dmg[0];
    }
}

// Per-particle stress: force/CabanaPD_PMB.hpp:157-202 (NoFracture), :341-401
// (Fracture), :492-537 (LinearPMB); force/CabanaPD_LPS.hpp:221-267
// (NoFracture), :506-572 (Fracture: intact bonds only). Half the pair force
// times the reference bond vector, sigma(i, a, b) = sum_k f_a xi_b over the
// row in row order (the caller zeroes sigma first, CabanaPD_Force.hpp:
// 229-231). Component-major: sigma[(3 a + b) npad + i]. LPS uses the factors
// a = theta_coeff theta / m and b = s_coeff / m of the last force update,
// exact subexpressions of the reference's coefficient.
template <int MODEL, int INFL, bool FRACTURE>
__global__ void __launch_bounds__(kBlock)
    k_pd_stress(ParticleView p, EllView nl, ModelDev md, double* __restrict__ sigma)
{
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    const double xi0 = p.x[i], xi1 = p.x[np + i], xi2 = p.x[2 * np + i];
    const double ui0 = p.u[i], ui1 = p.u[np + i], ui2 = p.u[2 * np + i];
    constexpr bool lps = MODEL == M_LPS;
    constexpr bool linear = MODEL == M_LINEAR_PMB;
    double a_i = 0.0, b_i = 0.0;
    if (lps) {
        a_i = p.lps_a[i];
        b_i = p.lps_b[i];
    }
    const int cnt = nl.count[i];
    double S[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    uint32_t word = 0;
    int32_t jn = cnt > 0 ? __ldg(nl.idx + i) : 0;  // (read one bond ahead)
    for (int k = 0; k < cnt; ++k) {
        if (FRACTURE && (k & 31) == 0) word = nl.mu[(int64_t)(k >> 5) * np + i];
        const int64_t j = jn;
        if (k + 1 < cnt) jn = __ldg(nl.idx + (int64_t)(k + 1) * np + i);
        const double vol_j = __ldg(p.vol + j);
        double fx, fy, fz, xx, xy, xz;
        if (linear) {
            double xi, ls;
            bond_linearized(p.x, p.u, np, j, xi0, xi1, xi2, ui0, ui1, ui2, xi, ls, xx, xy,
                            xz);
            const double coeff = 0.5 * (md.c * ls * vol_j);
            fx = coeff * xx / xi;
            fy = coeff * xy / xi;
            fz = coeff * xz / xi;
        } else {
            const double mu = FRACTURE ? (double)((word >> (k & 31)) & 1u) : 1.0;
            if (FRACTURE && lps && !(mu > 0.0)) continue;
            double xi, r, s, rx, ry, rz;
            Divisor X;
            bond_geometry(p.x, p.u, np, j, xi0, xi1, xi2, ui0, ui1, ui2, xi, r, s, rx, ry,
                          rz, xx, xy, xz, &X);
            double coeff;
            if (lps) {
                const double a_j = __ldg(p.lps_a + j), b_j = __ldg(p.lps_b + j);
                coeff = (a_i + a_j + s * (b_i + b_j)) * influence<INFL>(X) * xi * vol_j;
                coeff *= 0.5;
            } else {
                coeff = 0.5 * (md.c * s * vol_j);
            }
            if (FRACTURE) {
                fx = mu * coeff * rx / r;
                fy = mu * coeff * ry / r;
                fz = mu * coeff * rz / r;
            } else {
                fx = coeff * rx / r;
                fy = coeff * ry / r;
                fz = coeff * rz / r;
            }
        }
        S[0] += fx * xx;
        S[4] += fy * xy;
        S[8] += fz * xz;
        S[1] += fx * xy;
        S[3] += fy * xx;
        S[2] += fx * xz;
        S[6] += fz * xx;
        S[5] += fy * xz;
        S[7] += fz * xy;
    }
    for (int c = 0; c < 9; ++c) sigma[(int64_t)c * np + i] = S[c];
}

// Fixed-order sums of two-column partials: block b adds rows [b seg, (b + 1)
// seg) of n, `step` rows apart, and leaves the sums in out, or in its
// segment's first row where out is null.
constexpr int kSumBlock = 1024;
__global__ void __launch_bounds__(kSumBlock)
    k_sum_partials(double2* partials, int64_t n, int64_t seg, int64_t step, double* out)
{
    __shared__ double s[2][kSumBlock / 32];
    const int64_t first = blockIdx.x * seg, last = min(n, first + seg);
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int64_t r = first + threadIdx.x; r < last; r += kSumBlock) {
        const double2 v = partials[r * step];
        acc.x += v.x;
        acc.y += v.y;
    }
    for (int half = 0; half < 2; ++half) {
        for (int o = 16; o > 0; o >>= 1) {
            acc.x += __shfl_down_sync(0xffffffffu, acc.x, o);
            acc.y += __shfl_down_sync(0xffffffffu, acc.y, o);
        }
        if (half) break;
        if ((threadIdx.x & 31) == 0) {
            s[0][threadIdx.x >> 5] = acc.x;
            s[1][threadIdx.x >> 5] = acc.y;
        }
        __syncthreads();
        if (threadIdx.x >= 32) return;
        acc = make_double2(s[0][threadIdx.x], s[1][threadIdx.x]);
    }
    if (threadIdx.x != 0) return;
    if (out) {  // (the caller's, aligned as doubles)
        out[0] = acc.x;
        out[1] = acc.y;
    } else {
        partials[first * step] = acc;
    }
}

__global__ void __launch_bounds__(kBlock)
    k_max_partials(const double* partials, int nblocks, double* out)
{
    __shared__ double s[kBlock];
    double acc = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += kBlock) acc = fmax(acc, partials[b]);
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = kBlock / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] = fmax(s[threadIdx.x], s[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = s[0];
}

// ---------------------------------------------------------------------------
// Hertzian contact: force/CabanaPD_Contact.hpp:119-168 with
// force_models/CabanaPD_Hertzian.hpp:58-87 (normalForce; tangentialForce is
// a no-op that adds 0.0). With per-particle radii the pair uses
// R* = R_i (R_j / (R_i + R_j)), overlap r - (R_i + R_j) and
// m* = m_i (m_j / (m_i + m_j)), which round to the single-radius values when
// R_i == R_j.
// EPI: a contact-only fused step; the epilogue finishes the row (force BC,
// half steps, next displacement and velocity into the second buffers).
//
// The overlap cancels (about 1e-4 of r), so the pair vector, r^2 and r round
// as the reference's; the force law behind it does not amplify rounding and
// is factored: with w = sqrt(R* d) and d the overlap,
//   (4/3) E* sqrt(R*) d^(3/2) = (4/3) E* d w,  S_n = 2 E* w,
// so a contact costs three square roots, three divisions and no pow (five,
// seven and one as the formulas stand). Bound by the FP64 pipe and the latency
// of its root and division sequences: four blocks per SM (two: 0.50, three:
// 0.37, four: 0.35 ms per launch over 4.0 M spheres with six contacts each;
// the formulas as they stand at three blocks: 0.66 ms).
template <bool PER_PARTICLE, bool EPI = false>
__global__ void __launch_bounds__(kBlock, 4)
    k_hertz_force(ParticleView p, EllView nl, ModelDev md, bool reset, StepEpilogue ep)
{
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    const double xi0 = p.x[i], xi1 = p.x[np + i], xi2 = p.x[2 * np + i];
    const double ui0 = p.u[i], ui1 = p.u[np + i], ui2 = p.u[2 * np + i];
    const double vi0 = p.v[i], vi1 = p.v[np + i], vi2 = p.v[2 * np + i];
    const double vol_i = p.vol[i], mi = p.rho[i] * vol_i;
    const double inv_vol = 1.0 / vol_i;
    const double R_i = PER_PARTICLE ? p.radius[i] : 0.0;
    double fx = reset ? 0.0 : p.f[i];
    double fy = reset ? 0.0 : p.f[np + i];
    double fz = reset ? 0.0 : p.f[2 * np + i];
    const int cnt = nl.count[i];
    int32_t jn = cnt > 0 ? __ldg(nl.idx + i) : 0;
    for (int k = 0; k < cnt; ++k) {
        const int64_t j = jn;
        if (k + 1 < cnt) jn = __ldg(nl.idx + (int64_t)(k + 1) * np + i);
        const double rx = (__ldg(p.x + j) - xi0) + (__ldg(p.u + j) - ui0);
        const double ry = (__ldg(p.x + np + j) - xi1) + (__ldg(p.u + np + j) - ui1);
        const double rz = (__ldg(p.x + 2 * np + j) - xi2) + (__ldg(p.u + 2 * np + j) - ui2);
        const double r2 = rx * rx + ry * ry + rz * rz;
        const double R_j = PER_PARTICLE ? __ldg(p.radius + j) : 0.0;
        const double sum_r = PER_PARTICLE ? R_i + R_j : 2.0 * md.radius;
        // Without overlap the pair adds a zero: skip it (the sum is unchanged;
        // at most a zero sum keeps the sign the reference's + 0.0 would
        // clear). The first test leaves out pairs clearly apart before their
        // square root (its margin is far above the rounding of both sides).
        if (r2 > sum_r * sum_r * (1.0 + 1e-14)) continue;
        const double r = sqrt(r2);
        const double delta_n = r - sum_r;
        if (!(delta_n < 0.0)) continue;
        const double rinv = 1.0 / r;
        const double vx = __ldg(p.v + j) - vi0;
        const double vy = __ldg(p.v + np + j) - vi1;
        const double vz = __ldg(p.v + 2 * np + j) - vi2;
        const double vn = fma(vz, rz, fma(vy, ry, vx * rx)) * rinv;
        double Rs, ms;
        if (PER_PARTICLE) {
            Rs = R_i * (R_j / sum_r);
            const double mj = __ldg(p.rho + j) * __ldg(p.vol + j);
            ms = mi * (mj / (mi + mj));
        } else {
            Rs = md.Rs;
            ms = mi / 2.0;
        }
        const double w = sqrt(Rs * -delta_n);
        const double h = 4.0 / 3.0 * md.Es * delta_n * w;  // minus the elastic force
        const double coeff = fma(-md.coeff_h_d * sqrt(2.0 * md.Es * w * ms), vn, h);
        const double kf = coeff * inv_vol * rinv;
        fx = fma(kf, rx, fx);
        fy = fma(kf, ry, fy);
        fz = fma(kf, rz, fz);
    }
    if (EPI) {
        step_epilogue<false>(p, ep, i, fx, fy, fz);
        return;
    }
    p.f[i] = fx;
    p.f[np + i] = fy;
    p.f[2 * np + i] = fz;
}

// ---------------------------------------------------------------------------
// Normal repulsion: force/CabanaPD_Contact.hpp:52-92 with
// NormalRepulsionModel::forceCoeff (force_models/CabanaPD_Contact.hpp:82-88).
// A pair whose current distance r is below the contact radius adds
// ((15 c) sc) vol_j r_d / r per component, sc = (r - radius) / delta_c; the
// coefficient is negative, so the pair pushes i away from j. Pairs farther
// apart add a zero and are skipped (only the sign of a zero sum can differ).
// The reference distance and stretch of getDistance are not used here.
__global__ void __launch_bounds__(kBlock)
    k_repulsion_force(ParticleView p, EllView nl, double radius, double c15,
                      double delta, bool reset)
{
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    const double xi0 = p.x[i], xi1 = p.x[np + i], xi2 = p.x[2 * np + i];
    const double ui0 = p.u[i], ui1 = p.u[np + i], ui2 = p.u[2 * np + i];
    double fx = reset ? 0.0 : p.f[i];
    double fy = reset ? 0.0 : p.f[np + i];
    double fz = reset ? 0.0 : p.f[2 * np + i];
    const int cnt = nl.count[i];
    for (int k = 0; k < cnt; ++k) {
        const int64_t j = __ldg(nl.idx + (int64_t)k * np + i);
        const double xx = __ldg(p.x + j) - xi0;
        const double eu = __ldg(p.u + j) - ui0;
        const double xy = __ldg(p.x + np + j) - xi1;
        const double ev = __ldg(p.u + np + j) - ui1;
        const double xz = __ldg(p.x + 2 * np + j) - xi2;
        const double ew = __ldg(p.u + 2 * np + j) - ui2;
        const double rx = xx + eu, ry = xy + ev, rz = xz + ew;
        const double r = sqrt(rx * rx + ry * ry + rz * rz);
        if (!(r < radius)) continue;
        const double sc = (r - radius) / delta;
        const double coeff = c15 * sc * p.vol[j];
        fx += coeff * rx / r;
        fy += coeff * ry / r;
        fz += coeff * rz / r;
    }
    p.f[i] = fx;
    p.f[np + i] = fy;
    p.f[2 * np + i] = fz;
}

// ---------------------------------------------------------------------------
// Velocity Verlet: CabanaPD_Integrate.hpp:89-116 (NoContact), :151-193
// (Contact: also the largest displacement since the last list build).
template <bool TRACK>
__global__ void __launch_bounds__(kBlock)
    k_vv_initial(ParticleView p, double dt, double half_dt, double* block_max, double* u_out)
{
    __shared__ double s_max[kBlock];
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double um = 0.0;
    if (i < p.n) {
        const int64_t np = p.npad;
        const double half_dt_m = half_dt / p.rho[i];
        double v0 = p.v[i] + half_dt_m * p.f[i];
        double v1 = p.v[np + i] + half_dt_m * p.f[np + i];
        double v2 = p.v[2 * np + i] + half_dt_m * p.f[2 * np + i];
        p.v[i] = v0;
        p.v[np + i] = v1;
        p.v[2 * np + i] = v2;
        const double u0 = p.u[i] + dt * v0;
        const double u1 = p.u[np + i] + dt * v1;
        const double u2 = p.u[2 * np + i] + dt * v2;
        u_out[i] = u0;
        u_out[np + i] = u1;
        u_out[2 * np + i] = u2;
        if (TRACK)
            um = norm3d(u0 - p.u_neigh[i], u1 - p.u_neigh[np + i],
                        u2 - p.u_neigh[2 * np + i]);
    }
    if (TRACK) {
        s_max[threadIdx.x] = um;
        __syncthreads();
        for (int w = kBlock / 2; w > 0; w >>= 1) {
            if ((int)threadIdx.x < w)
                s_max[threadIdx.x] = fmax(s_max[threadIdx.x], s_max[threadIdx.x + w]);
            __syncthreads();
        }
        if (threadIdx.x == 0) block_max[blockIdx.x] = s_max[0];
    }
}

__global__ void __launch_bounds__(kBlock) k_vv_final(ParticleView p, double half_dt)
{
    const int64_t i = p.frozen + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    const double half_dt_m = half_dt / p.rho[i];
    p.v[i] += half_dt_m * p.f[i];
    p.v[np + i] += half_dt_m * p.f[np + i];
    p.v[2 * np + i] += half_dt_m * p.f[2 * np + i];
}

// CabanaPD_Boundary.hpp:94-113, :138-157 and the custom-functor form.
__global__ void __launch_bounds__(kBlock)
    k_force_bc(ParticleView p, int kind, int comp, int64_t count, const int32_t* idx,
               const double* values, double value)
{
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    const int64_t q = idx[b];
    const int64_t np = p.npad;
    if (kind == CPD_BC_FORCE_VALUE) {
        for (int d = 0; d < 3; d++) p.f[d * np + q] = value;
    } else if (kind == CPD_BC_FORCE_UPDATE) {
        for (int d = 0; d < 3; d++) p.f[d * np + q] += value;
    } else {
        p.f[comp * np + q] += values[b];
    }
}

// ---------------------------------------------------------------------------
// Pre-notch: CabanaPD_Prenotch.hpp:24-172 geometry, :215-263 create.
struct V3 {
    double a[3];
};
__device__ __forceinline__ double dot3(V3 a, V3 b)
{
    double v = 0;
    for (int d = 0; d < 3; d++) v += (a.a[d]) * (b.a[d]);
    return v;
}
__device__ __forceinline__ double norm3(V3 a) { return sqrt(dot3(a, a)); }
__device__ __forceinline__ V3 cross3(V3 a, V3 b)
{
    V3 c;
    c.a[0] = a.a[1] * b.a[2] - a.a[2] * b.a[1];
    c.a[1] = -(a.a[0] * b.a[2] - a.a[2] * b.a[0]);
    c.a[2] = a.a[0] * b.a[1] - a.a[1] * b.a[0];
    return c;
}
__device__ __forceinline__ V3 scale3(V3 a, double n)
{
    for (int d = 0; d < 3; d++) a.a[d] *= n;
    return a;
}
__device__ __forceinline__ V3 diff3(V3 a, V3 b)
{
    V3 c;
    for (int d = 0; d < 3; d++) c.a[d] = a.a[d] - b.a[d];
    return c;
}
__device__ __forceinline__ V3 sum3(V3 a, V3 b)
{
    V3 c;
    for (int d = 0; d < 3; d++) c.a[d] = a.a[d] + b.a[d];
    return c;
}

__device__ int bond_prenotch_intersection(V3 v1, V3 v2, V3 p0, V3 x_i, V3 x_j)
{
    const double tol = 1e-10;
    V3 cv = cross3(v1, v2);
    double ncv = norm3(cv);
    V3 n = scale3(cv, 1.0 / ncv);
    V3 l0 = x_i;
    V3 l = diff3(x_j, x_i);
    int flag;
    if (fabs(dot3(l, n)) < tol)
        flag = (fabs(dot3(diff3(p0, l0), n)) < tol) ? 1 : 2;
    else
        flag = 3;
    int keep = 1;
    if (flag == 1) {
        double n2 = ncv * ncv;
        double li1 = dot3(cross3(diff3(x_i, p0), v2), cv) / n2;
        double li2 = -dot3(cross3(diff3(x_i, p0), v1), cv) / n2;
        double lj1 = dot3(cross3(diff3(x_j, p0), v2), cv) / n2;
        double lj2 = -dot3(cross3(diff3(x_j, p0), v1), cv) / n2;
        if (!(fmin(li1, lj1) > 1 + tol || fmax(li1, lj1) < -tol ||
              fmin(li2, lj2) > 1 + tol || fmax(li2, lj2) < -tol))
            keep = 0;
    } else if (flag == 3) {
        double dd = dot3(diff3(p0, l0), n) / dot3(l, n);
        if (-tol < dd && dd < 1 + tol) {
            V3 q = sum3(l0, scale3(l, dd));
            double n2 = ncv * ncv;
            double l1 = dot3(cross3(diff3(q, p0), v2), cv) / n2;
            double l2 = -dot3(cross3(diff3(q, p0), v1), cv) / n2;
            if (-tol < fmin(l1, l2) && fmax(l1, l2) < 1 + tol) keep = 0;
        }
    }
    return keep;
}

// One notch per launch (as the reference). Particles whose horizon ball
// cannot reach the notch's bounding box (grown by `margin`) are skipped;
// the test is conservative, so the cut bond set is unchanged.
__global__ void __launch_bounds__(kBlock)
    k_prenotch(ParticleView p, EllView nl, V3 v1, V3 v2, V3 p0, V3 box_lo,
               V3 box_hi)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int64_t np = p.npad;
    V3 xi{{p.x[i], p.x[np + i], p.x[2 * np + i]}};
    for (int d = 0; d < 3; d++)
        if (xi.a[d] < box_lo.a[d] || xi.a[d] > box_hi.a[d]) return;
    const int cnt = nl.count[i];
    for (int w = 0; w * 32 < cnt; ++w) {
        uint32_t word = nl.mu[(int64_t)w * np + i];
        const uint32_t old = word;
        for (int b = 0; b < 32 && w * 32 + b < cnt; ++b) {
            const int k = w * 32 + b;
            const int64_t j = nl.idx[(int64_t)k * np + i];
            V3 xj{{p.x[j], p.x[np + j], p.x[2 * np + j]}};
            if (!bond_prenotch_intersection(v1, v2, p0, xi, xj)) word &= ~(1u << b);
        }
        if (word != old) nl.mu[(int64_t)w * np + i] = word;
    }
}

}  // namespace

// ===========================================================================
// Launchers.
int energy_blocks(int64_t nrows) { return nrows > 0 ? blocks_for(nrows) : 1; }
int vv_blocks(int64_t nrows) { return nrows > 0 ? blocks_for(nrows) : 1; }

int launch_vv_initial(const ParticleView& p, double dt, bool track_max,
                      double* block_max, int, double* u_out, cudaStream_t st)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    const double half_dt = 0.5 * dt;
    if (track_max)
        k_vv_initial<true><<<blocks_for(rows), kBlock, 0, st>>>(p, dt, half_dt, block_max, u_out);
    else
        k_vv_initial<false><<<blocks_for(rows), kBlock, 0, st>>>(p, dt, half_dt, nullptr, u_out);
    return 1;
}

int launch_vv_final(const ParticleView& p, double dt, cudaStream_t st)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    k_vv_final<<<blocks_for(rows), kBlock, 0, st>>>(p, 0.5 * dt);
    return 1;
}

int launch_lps_weighted_volume(const ParticleView& p, const EllView& nl,
                               const Model& md, cudaStream_t st)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    const int g = blocks_for(rows);
    if (md.influence == 1) {
        if (md.fracture)
            k_lps_weighted_volume<1, true><<<g, kBlock, 0, st>>>(p, nl);
        else
            k_lps_weighted_volume<1, false><<<g, kBlock, 0, st>>>(p, nl);
    } else {
        if (md.fracture)
            k_lps_weighted_volume<0, true><<<g, kBlock, 0, st>>>(p, nl);
        else
            k_lps_weighted_volume<0, false><<<g, kBlock, 0, st>>>(p, nl);
    }
    return 1;
}

int launch_lps_dilatation(const ParticleView& p, const EllView& nl,
                          const Model& md, cudaStream_t st)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    const int g = blocks_for(rows);
    const ModelDev d = to_dev(md);
    if (md.influence == 1) {
        if (md.fracture)
            k_lps_dilatation<1, true><<<g, kBlock, 0, st>>>(p, nl, d);
        else
            k_lps_dilatation<1, false><<<g, kBlock, 0, st>>>(p, nl, d);
    } else {
        if (md.fracture)
            k_lps_dilatation<0, true><<<g, kBlock, 0, st>>>(p, nl, d);
        else
            k_lps_dilatation<0, false><<<g, kBlock, 0, st>>>(p, nl, d);
    }
    return 1;
}


#define CPD_PD_DISPATCH(KERNEL, GRID, BLOCK, ...)                                   \
    do {                                                                            \
        const int infl = md.influence == 1 ? 1 : 0;                                 \
        switch (md.pd) {                                                            \
        case CPD_PD_PMB:                                                            \
            if (md.fracture)                                                        \
                KERNEL<M_PMB, 1, true><<<GRID, BLOCK, 0, st>>>(__VA_ARGS__);       \
            else                                                                    \
                KERNEL<M_PMB, 1, false><<<GRID, BLOCK, 0, st>>>(__VA_ARGS__);      \
            break;                                                                  \
        case CPD_PD_LINEAR_PMB:                                                     \
            KERNEL<M_LINEAR_PMB, 1, false><<<GRID, BLOCK, 0, st>>>(__VA_ARGS__);   \
            break;                                                                  \
        case CPD_PD_LPS:                                                            \
            if (md.fracture) {                                                      \
                if (infl)                                                           \
                    KERNEL<M_LPS, 1, true><<<GRID, BLOCK, 0, st>>>(__VA_ARGS__);   \
                else                                                                \
                    KERNEL<M_LPS, 0, true><<<GRID, BLOCK, 0, st>>>(__VA_ARGS__);   \
            } else {                                                                \
                if (infl)                                                           \
                    KERNEL<M_LPS, 1, false><<<GRID, BLOCK, 0, st>>>(__VA_ARGS__);  \
                else                                                                \
                    KERNEL<M_LPS, 0, false><<<GRID, BLOCK, 0, st>>>(__VA_ARGS__);  \
            }                                                                       \
            break;                                                                  \
        default:                                                                    \
            return 0;                                                               \
        }                                                                           \
    } while (0)

int launch_pd_force(const ParticleView& p, const EllView& nl, const Model& md,
                    cudaStream_t st)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    // Blocks of half the size spread more evenly over the SMs (plates, per step
    // in blocks of 128 / 256: 20 thousand rows 62 / 65 us, 80: 102 / 107, 200:
    // 201 / 209, 440: 419 / 427, 800: 762 / 770; an LPS box of 2.0 M: 4.52 / 4.54
    // ms).
    constexpr int block = kBlock / 2;
    const int g = (int)((rows + block - 1) / block);
    const ModelDev d = to_dev(md);
    CPD_PD_DISPATCH(k_pd_force, g, block, p, nl, d);
    return 1;
}

int launch_pd_energy(const ParticleView& p, const EllView& nl, const Model& md,
                     double* partials, int nblocks, cudaStream_t st)
{
    const ModelDev d = to_dev(md);
    CPD_PD_DISPATCH(k_pd_energy, nblocks, kBlock, p, nl, d, partials);
    return 1;
}

int launch_pd_stress(const ParticleView& p, const EllView& nl, const Model& md, double* sigma,
                     cudaStream_t st)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    const int g = blocks_for(rows);
    const ModelDev d = to_dev(md);
    CPD_PD_DISPATCH(k_pd_stress, g, kBlock, p, nl, d, sigma);
    return 1;
}

// One block adds up to 4096 rows in a few microseconds; longer columns (the
// output step of a large body has one row per 32 particles) take one block
// per SM first, each leaving its sum in its own segment: 360 thousand rows in
// 12 us, 430 us by one block of 256.
int launch_sum_partials(double* partials, int n, double* out, cudaStream_t st)
{
    double2* const p = reinterpret_cast<double2*>(partials);
    if (n <= 4 * kSumBlock) {
        k_sum_partials<<<1, kSumBlock, 0, st>>>(p, n, n, 1, out);
        return 1;
    }
    const int64_t seg = (n + 147) / 148;
    const int g = (int)((n + seg - 1) / seg);
    k_sum_partials<<<g, kSumBlock, 0, st>>>(p, n, seg, 1, nullptr);
    k_sum_partials<<<1, kSumBlock, 0, st>>>(p, g, g, seg, out);
    return 2;
}

int launch_max_partials(const double* partials, int nblocks, double* out,
                        cudaStream_t st)
{
    k_max_partials<<<1, kBlock, 0, st>>>(partials, nblocks, out);
    return 1;
}

int launch_hertz_force(const ParticleView& p, const EllView& nl,
                       const Model& md, bool reset, cudaStream_t st, const StepEpilogue* ep)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    const ModelDev d = to_dev(md);
    const StepEpilogue e = ep ? *ep : StepEpilogue{};
    const int g = blocks_for(rows);
    if (ep) {
        if (md.per_particle_radius)
            k_hertz_force<true, true><<<g, kBlock, 0, st>>>(p, nl, d, true, e);
        else
            k_hertz_force<false, true><<<g, kBlock, 0, st>>>(p, nl, d, true, e);
    } else if (md.per_particle_radius) {
        k_hertz_force<true><<<g, kBlock, 0, st>>>(p, nl, d, reset, e);
    } else {
        k_hertz_force<false><<<g, kBlock, 0, st>>>(p, nl, d, reset, e);
    }
    return 1;
}

int launch_repulsion_force(const ParticleView& p, const EllView& nl, const Model& md,
                           bool reset, cudaStream_t st)
{
    const int64_t rows = p.n - p.frozen;
    if (rows <= 0) return 0;
    k_repulsion_force<<<blocks_for(rows), kBlock, 0, st>>>(
        p, nl, md.radius, 15.0 * md.c_contact, md.contact_horizon, reset);
    return 1;
}

int launch_force_bc(const ParticleView& p, const BoundaryCondition& bc,
                    cudaStream_t st)
{
    if (bc.count <= 0) return 0;
    k_force_bc<<<blocks_for(bc.count), kBlock, 0, st>>>(p, bc.kind, bc.component,
                                                       bc.count, bc.idx, bc.values,
                                                       bc.value);
    return 1;
}

int launch_prenotch(const ParticleView& p, const EllView& nl, const double* v1,
                    const double* v2, const double* p0, double margin,
                    cudaStream_t st)
{
    if (p.n <= 0) return 0;
    V3 a{{v1[0], v1[1], v1[2]}}, b{{v2[0], v2[1], v2[2]}}, o{{p0[0], p0[1], p0[2]}};
    V3 lo, hi;
    for (int d = 0; d < 3; d++) {
        double c[4] = {o.a[d], o.a[d] + a.a[d], o.a[d] + b.a[d], o.a[d] + a.a[d] + b.a[d]};
        double mn = c[0], mx = c[0];
        for (int q = 1; q < 4; q++) {
            mn = c[q] < mn ? c[q] : mn;
            mx = c[q] > mx ? c[q] : mx;
        }
        lo.a[d] = mn - margin;
        hi.a[d] = mx + margin;
    }
    k_prenotch<<<blocks_for(p.n), kBlock, 0, st>>>(p, nl, a, b, o, lo, hi);
    return 1;
}

}  // namespace cpd
