// Pair terms shared by more than one kernel.
#pragma once

#include "ctx.h"

namespace capac {

// exp(-x^2) and erfc(x) with x = alpha r, and 1/r, of one damped Coulomb pair,
// for alpha r < kDsfMaxX: no branch and no call, ~63 FP64 operations where
// sqrt, the division, exp and erfc take about 200.
//
// 1/r: the hardware's approximation y and one step of the series of r^2 y^2 = 1 - e,
// 1/r = y (1 - e)^(-1/2), to e^2: third order (remainder 5/16 e^3 of an e below
// 2^-19).  exp(-x^2): -alpha^2 r^2 with the product's rounding error (from r already
// rounded it would carry 2 x^2 of that rounding: 3.0e-16 for 5.1e-17 at the alpha
// and r below), 2^n split off, and 1 + f + f^2 q(f) on |f| <= ln2 / 2 with q a
// Chebyshev interpolant (1.6e-17 of the result).  erfc(x) = exp(-x^2) R(x), R the
// scaled complementary error function as a polynomial of degree 18 in
// u = (x - 3.5) / (x + 3.5), Chebyshev interpolant on [0, 5] (3.7e-17 of R with
// the rounded coefficients); both polynomials in two chains.  R changes by up to
// twice the relative change of u, so u is rounded once: without the sum's and the
// quotient's remainders erfc's error was 2.2e-16 where it is 1.05e-16.
//
// Rms relative error against 64 bits of alpha 2, r 0.12 .. 1.2 (CUDA's functions on
// the same r^2 in brackets): Gaussian 5.1e-17 (4.8e-17), erfc 1.05e-16 (1.8e-16);
// the damped Coulomb force and energy of unit charges, absolute, 1.48e-14 (1.55e-14)
// and 1.70e-16 (1.83e-16).
//
// CLOSE = false: without the remainders of u and of the last addition, for a caller
// that needs erfc to an absolute 1e-17 only, beyond x = 1.5 (metal blocks).
//
// W of them side by side (the three widths of a metal pair share the constants'
// moves).  Two pairs a lane in k_pair take ~160 registers, twelve warps per SM
// instead of sixteen: 398 us for 350 at 24,000 atoms.
constexpr double kDsfMaxX = 5.0;
struct Dsf {
    double rinv, r, eg, ec;
};
template <int W, bool CLOSE = true>
__device__ __forceinline__ void dsf_terms(const double (&alpha)[W], const double (&r2)[W], Dsf (&d)[W])
{
    double y[W], e[W], x2[W], kd[W], f[W], f2[W], a[W], b[W], u[W], u2[W];
    auto each = [](auto op) {
#pragma unroll
        for (int w = 0; w < W; ++w) op(w);
    };
    auto chain = [&](double (&p)[W], const double (&t)[W], double c) { each([&](int w) { p[w] = fma(p[w], t[w], c); }); };
    each([&](int w) {
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y[w]) : "d"(r2[w]));
        e[w] = fma(-r2[w] * y[w], y[w], 1.0);
        d[w].rinv = fma(y[w] * e[w], fma(0.375, e[w], 0.5), y[w]);
        d[w].r = r2[w] * d[w].rinv;
    });
    // exp(-x^2): n = round(-x^2 log2 e) from the low word of an addition to 1.5 2^52
    each([&](int w) {
        const double al2 = alpha[w] * alpha[w];
        x2[w] = al2 * r2[w];
        const double lo = fma(al2, r2[w], -x2[w]);
        kd[w] = fma(x2[w], -1.4426950408889634, 0x1.8p52);
        const double n = kd[w] - 0x1.8p52;
        f[w] = fma(n, -0x1.473de6af278edp-34, fma(n, -0x1.62e42fef00000p-1, -x2[w])) - lo;
        f2[w] = f[w] * f[w];
        a[w] = fma(2.51003759291859252e-08, f2[w], 2.75572684801069265e-06);
        b[w] = fma(2.76200760056313823e-07, f2[w], 2.48015213221045905e-05);
    });
    chain(a, f2, 1.98412698630406751e-04);
    chain(b, f2, 1.38888889171968899e-03);
    chain(a, f2, 8.33333333333006500e-03);
    chain(b, f2, 4.16666666666241636e-02);
    chain(a, f2, 1.66666666666666685e-01);
    chain(b, f2, 5.00000000000000111e-01);
    each([&](int w) {
        const double g = 1.0 + fma(f2[w], fma(a[w], f[w], b[w]), f[w]);
        d[w].eg = __hiloint2double(__double2hiint(g) + (__double2loint(kd[w]) << 20), __double2loint(g));
        // R(x): u = 1 - 7 / (x + 3.5), the sum as z and its rounding error, the
        // quotient as q and the rest of its division
        const double z = fma(alpha[w], d[w].r, 3.5), dz = fma(alpha[w], d[w].r, 3.5 - z);
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y[w]) : "d"(z));
        e[w] = fma(-z, y[w], 1.0);
        if (CLOSE) {
            y[w] = fma(y[w], e[w], y[w]);
            const double q = 7.0 * y[w];
            u[w] = fma(-y[w], fma(-dz, q, fma(-z, q, 7.0)), 1.0 - q);
        } else {
            u[w] = fma(-7.0, fma(y[w], fma(e[w], e[w], e[w]), y[w]), 1.0);
        }
        u2[w] = u[w] * u[w];
        a[w] = fma(1.44851080807840048e-07, u2[w], 9.39502676422655287e-07);
        b[w] = fma(1.21445591197839242e-08, u2[w], 6.32563657300747914e-07);
    });
    chain(a, u2, -1.35300964606639283e-06);
    chain(b, u2, -1.03347250494745519e-06);
    chain(a, u2, -4.65943681772681595e-06);
    chain(b, u2, 1.34428888195974961e-05);
    chain(a, u2, 2.88553311039605571e-04);
    chain(b, u2, -1.08088183803848795e-04);
    chain(a, u2, -4.24223856269931136e-03);
    chain(b, u2, 2.67384873232049400e-04);
    chain(a, u2, -4.54367611836835258e-02);
    chain(b, u2, 1.69767609425404628e-02);
    chain(a, u2, -1.61338524764510272e-01);
    chain(b, u2, 9.44278069090268707e-02);
    chain(a, u2, -2.89265044832767437e-01);
    chain(b, u2, 2.33130481600251627e-01);
    chain(b, u2, 1.55293655608894299e-01);
    each([&](int w) {  // CLOSE: with the last addition's rounding error
        const double R = fma(a[w], u[w], b[w]);
        d[w].ec = CLOSE ? fma(d[w].eg, R, d[w].eg * fma(a[w], u[w], b[w] - R)) : d[w].eg * R;
    });
}
__device__ __forceinline__ Dsf dsf_terms(double alpha, double r2)
{
    const double al[1] = {alpha}, in[1] = {r2};
    Dsf d[1];
    dsf_terms<1>(al, in, d);
    return d[0];
}

// The same for any x, by the library's functions.
__device__ __forceinline__ Dsf dsf_terms_any(double alpha, double r2)
{
    Dsf d;
    d.r = sqrt(r2);
    d.rinv = 1.0 / d.r;
    d.eg = exp(-alpha * alpha * r2);
    d.ec = erfc(alpha * d.r);
    return d;
}

// cpim_charge_pair with the damped form and alpha r < kDsfMaxX.
__device__ __forceinline__ Dsf cpim_charge_pair_dsf(const DevParams &P, const double r[3], double r2, double q_perm,
                                                    double q_ind, const double p[3], double f[3], double &a0)
{
    const Dsf d = dsf_terms(P.w_alpha, r2);
    const double r2inv = d.rinv * d.rinv, ir3 = r2inv * d.rinv, al3 = P.w_alpha * P.w_alpha * P.w_alpha;
    const double s = kFQQ * q_perm, sp = s / kNm2Bohr;
    a0 = (fma(d.ec, r2inv, P.w_a2_sqrtpi * d.eg * d.rinv) - P.w_const) * d.rinv;
    const double a1 = ir3 * r2inv * fma(P.w_a2_sqrtpi * d.r, d.eg, d.ec), b1 = 4.0 * kInvSqrtPi * al3 * r2inv * d.eg,
                 c1 = P.w_const * ir3;
    const double pr = p[0] * r[0] + p[1] * r[1] + p[2] * r[2];
    // sum_a T_ab p_a, T_ab = a1 (3 r_a r_b - d_ab r^2) + b1 r_a r_b - c1 (r_a r_b - d_ab r^2)
    const double along = fma(a0, s * q_ind, -(3.0 * a1 + b1 - c1) * pr * sp), off = (a1 - c1) * r2 * sp;
#pragma unroll
    for (int b = 0; b < 3; ++b) f[b] = fma(along, r[b], off * p[b]);
    return d;
}

// Force on the metal atom from the permanent charge q of a non-metal atom at
// metal - atom separation r (nm); the atom receives the opposite force.
// cpff.c:604-702.  Returns through f[3]; also gives const_a0 for energy [11].
__device__ __forceinline__ void cpim_charge_pair(const DevParams &P, const double r[3], double r2, double q_perm,
                                                 double q_ind, const double p_ind[3], double f[3], double &a0,
                                                 double &ec_out)
{
    const double rr = sqrt(r2);
    double ec = 0.0, eg = 0.0;
    if (P.use_coulomb == 1) {
        ec = erfc(P.w_alpha * rr);
        eg = exp(-P.w_alpha * P.w_alpha * r2);
        a0 = (ec / r2 + P.w_a2_sqrtpi * eg / rr - P.w_const) / rr;
    } else {
        a0 = 1.0 / (r2 * rr);
    }
    ec_out = ec;
#pragma unroll
    for (int a = 0; a < 3; ++a) f[a] = a0 * r[a] * kFQQ * q_perm * q_ind;
    if (P.use_coulomb == 1) {
        const double al3 = P.w_alpha * P.w_alpha * P.w_alpha;
        const double a1 = 1.0 / (rr * rr * rr * rr * rr) * (ec + P.w_a2_sqrtpi * rr * eg);
        const double b1 = 4.0 * kInvSqrtPi * al3 / r2 * eg;
        const double c1 = P.w_const / (rr * rr * rr);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const double dab = a == b ? 1.0 : 0.0;
                f[b] += -(a1 * (3.0 * r[a] * r[b] - dab * r2) + b1 * r[a] * r[b] - c1 * (r[a] * r[b] - dab * r2)) *
                        kFQQ * q_perm * p_ind[a] / kNm2Bohr;
            }
    } else {
        const double ir5 = 1.0 / (rr * rr * rr * rr * rr);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const double dab = a == b ? 1.0 : 0.0;
                f[b] += -((3.0 * r[a] * r[b] - dab * r2) * ir5) * kFQQ * q_perm * p_ind[a] / kNm2Bohr;
            }
    }
}

// The 4x4 CPIM block of the ordered metal pair (i, j) in FP64, entries
// e[4*row + col] over (p_x, p_y, p_z, q): mpi_cpff_mat_relay_COO,
// cpff.c:245-436.  r = r_j - r_i (pbc_12) in Bohr; diagonal block when same.
// Entries with |e| <= 1e-15 are dropped as in the reference (typedef.h:89-93).
__device__ __forceinline__ void cpim_block(const DevParams &P, const double4 &pi, const double4 &pj, bool same,
                                           double e[16])
{
#pragma unroll
    for (int k = 0; k < 16; ++k) e[k] = 0.0;
    if (same) {
        e[0] = e[5] = e[10] = keep_entry(P.inv_polar);
        e[15] = keep_entry(-P.inv_capac);
        return;
    }
    double r[3] = {pj.x - pi.x, pj.y - pi.y, pj.z - pi.z};
    image(r[0], r[1], r[2], P.box);
    r[0] *= kNm2Bohr;
    r[1] *= kNm2Bohr;
    r[2] *= kNm2Bohr;
    // the three widths' Gaussians and erf = 1 - erfc side by side.  Beyond the fitted
    // range R is a polynomial continued outside its interval: it grows no faster
    // than the Chebyshev polynomial of degree 18, and times 3.7e-17 of R and
    // erfc(x) that is below 1e-24 everywhere beyond x = 5.  x is held below 26, where
    // all is zero.  Below 1.5 the library's erf; beyond, erfc's error (2.2e-16 of at
    // most 0.034) is below the rounding of 1 - erfc.
    const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    const double ip[3] = {P.inv_r_pp, P.inv_r_pq, P.inv_r_qq};
    double al[3], er[3], g[3];
    const double rs[3] = {r2, r2, r2};
    Dsf d[3];
    const double top = 26.0 * rsqrt(r2);
#pragma unroll
    for (int k = 0; k < 3; ++k) al[k] = fmin(ip[k], top);
    dsf_terms<3, false>(al, rs, d);
    const double rr = d[0].r, rinv = d[0].rinv, r2inv = rinv * rinv, ir3 = r2inv * rinv;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        g[k] = d[k].eg;
        er[k] = rr * ip[k] < 1.5 ? erf(sqrt(r2) * ip[k]) : 1.0 - d[k].ec;
    }
    const double c1 = ir3 * r2inv * (er[0] - 2.0 * kInvSqrtPi * ip[0] * rr * g[0]);
    const double c2 = 4.0 * kInvSqrtPi * (ip[0] * ip[0] * ip[0]) * r2inv * g[0];
    const double c3 = ir3 * (er[1] - 2.0 * kInvSqrtPi * ip[1] * rr * g[1]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const double dab = a == b ? 1.0 : 0.0;
            e[4 * a + b] = keep_entry(-(c1 * (3.0 * r[a] * r[b] - dab * r2) - c2 * r[a] * r[b]));
        }
        e[4 * a + 3] = keep_entry(c3 * r[a]);
        e[12 + a] = keep_entry(-c3 * r[a]);
    }
    e[15] = keep_entry(-er[2] * rinv);
}

}  // namespace capac
