// Nonbonded pair forces over the full neighbour list (FP64 and mixed).
//
// Per pair this is compute_nonbonded / compute_erf_vdw / compute_morse /
// compute_buckingham (force.c:591-816) as dispatched by mpi_nonb_pair
// (force.c:1476-1528): LJ shifted force + damped shifted force Coulomb
// (funct 1), Buckingham (2), Morse (3), erf-damped vdW (4).
//
// One warp owns an atom i at a time (grid-stride over atoms) and walks its
// list; every pair is visited from both ends, so forces need no atomics and
// each end adds half of the pair energy and virial.  The cut-off test is done
// in FP64 with the reference's r^2 rounding, so both precisions keep exactly
// the reference's pair set.  Two passes: candidates (63% of the entries are
// inside rc at a skin of 0.2) are first tested in FP32, with a margin that keeps
// every pair the FP64 test accepts, and the entries that pass are compacted in
// shared memory, 4 bytes each; then full warps form the FP64 difference, test it
// and compute, their positions loaded one set ahead.  In FP64 the terms of an
// ordinary pair are dsf_terms' ~63 operations.  Bound by latency and issue together:
// at 24,000 atoms (FP64) 499 -> 336 us a launch, at 91,122 2.28 -> 1.45 ms with issue
// slots 52% busy, FP64 pipe 30%, sixteen warps per SM of 128 registers.
//
// The same traversal adds, on each charged non-metal atom, the force from the
// induced charges and dipoles of metal neighbours inside the cut-off: the
// water side of the metal-water loop of mpi_cpff_force (cpff.c:578-724).  The
// metal side, with energies [10],[11] and the virial, is k_cpim_metal.
//
// Mixed path: coordinate differences and the cut-off in FP64, the pair terms
// in FP32, force sums per lane with Kahan compensation, energies and virial
// gathered per atom in FP32 and summed across atoms in FP64.
#include <algorithm>

#include "terms.cuh"

namespace capac {

namespace {

constexpr int kPairWarps = 4;  // warps per block: a block ends with its longest row (24,000 atoms, eight: 2% more)

// FP32 constants of the run.
struct PairConstsF {
    float rc, inv_rc, inv_rc12, inv_rc6, alpha, a2_sqrtpi, w_const, w_erfc_arcut, fqq, rc2;
    float gauss2, gauss2_lo;  // -alpha^2 log2(e) as a sum of two
    int use_vdw, use_coulomb;
    double iL[3];  // 1 / box edge
};

// One type pair in FP32, with the shifted-force constants of funct 1
// precomputed: fc = 12 c12 / rc^12 - 6 c6 / rc^6, es = c12 / rc^12 - c6 / rc^6.
struct TypePairF {
    float c6, c12, a, b, fc, es;
    int fn, pad;
};

__device__ __forceinline__ TypePairF make_type_pair_f(const DevParams &P, const PairConstsF &K, int k)
{
    const double4 pd = P.nb_par[k];
    TypePairF t;
    t.c6 = (float)pd.x;
    t.c12 = (float)pd.y;
    t.a = (float)pd.z;
    t.b = (float)pd.w;
    t.fc = (float)(12.0 * pd.y * P.inv_rc12 - 6.0 * pd.x * P.inv_rc6);
    t.es = (float)(pd.y * P.inv_rc12 - pd.x * P.inv_rc6);
    t.fn = P.nb_funct[k];
    t.pad = 0;
    return t;
}

// 1/x by the hardware approximation (rcp.approx.ftz.f32, within about one
// ulp); 1 <= x <= 3.5 here.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// erfc(x) for 0 <= x in FP32 as exp(-x^2) R(x), with R(x) = erfc(x) exp(x^2)
// (the scaled complementary error function) fitted on [0, 5] by a degree-9
// polynomial in t = 1 / (1 + x / 2), least squares in relative error
// (relative error of R below 4e-8 in exact arithmetic, 3e-7 in FP32).  The
// caller has exp(-x^2) already, for the Gaussian term of the same pair.
__device__ __forceinline__ float erfc_from_gauss_f(float x, float gauss)
{
    const float t = rcp_approx(fmaf(0.5f, x, 1.0f));
    float r = -3.71903017e-02f;
    r = fmaf(r, t, 1.64898831e-01f);
    r = fmaf(r, t, -2.03180485e-01f);
    r = fmaf(r, t, -1.05265965e-01f);
    r = fmaf(r, t, 2.97262422e-01f);
    r = fmaf(r, t, 2.51787793e-02f);
    r = fmaf(r, t, 3.06175054e-01f);
    r = fmaf(r, t, 2.68365236e-01f);
    r = fmaf(r, t, 2.83852814e-01f);
    r = fmaf(r, t, -9.64172679e-05f);
    return gauss * r;
}
// The same for any x: the library's beyond the fitted range.
__device__ __forceinline__ float erfc_any_f(float x, float gauss)
{
    return x >= 5.0f ? erfcf(x) : erfc_from_gauss_f(x, gauss);
}

// FP64 pair term (force on j = f * rvec), reference formulas with the
// divisions by r, r^2, r^6, r^12 turned into products with 1/r.
__device__ __forceinline__ double pair_term(const DevParams &P, int k, double qi, double qj, double r2,
                                            double &e_qq, double &e_vdw)
{
    const int fn = P.nb_funct[k];
    const double4 pr = P.nb_par[k];  // (c6, c12, a, b)
    const double r = sqrt(r2), rinv = 1.0 / r, r2inv = rinv * rinv;
    if (fn == 4) {  // compute_erf_vdw, force.c:591-632 (width = a)
        if (pr.x != 0.0 || pr.y != 0.0) {
            const double r6inv = r2inv * r2inv * r2inv;
            const double a12 = pr.y * r6inv * r6inv, a6 = pr.x * r6inv, u = r / pr.z, eu = erf(u);
            e_vdw += (a12 - a6) * eu;
            return ((12.0 * a12 - 6.0 * a6) * rinv * eu - (a12 - a6) * 2.0 * kInvSqrtPi * exp(-u * u) / pr.z) * rinv;
        }
        return 0.0;
    }
    if (fn == 3) {  // compute_morse, force.c:639-667 (D = A, a = B, R = C6)
        const double e1 = exp(-pr.w * (r - pr.x)), e2 = e1 * e1;
        e_vdw += pr.z * (e2 - 2.0 * e1);
        return 2.0 * pr.z * pr.w * (e2 - e1) * rinv;
    }
    if (fn == 2) {  // compute_buckingham, force.c:674-703 (A, B, C6)
        const double r6inv = r2inv * r2inv * r2inv, eb = exp(-pr.w * r);
        e_vdw += pr.z * eb - pr.x * r6inv;
        return pr.z * eb * pr.w * rinv - 6.0 * pr.x * r6inv * r2inv;
    }
    // funct 1: compute_nonbonded, force.c:710-816 (not a 1-4 pair)
    double f = 0.0;
    if (pr.x != 0.0 || pr.y != 0.0) {
        const double r6inv = r2inv * r2inv * r2inv, r12inv = r6inv * r6inv;
        if (P.use_vdw == 1) {
            const double fr = 12.0 * pr.y * r12inv - 6.0 * pr.x * r6inv;
            const double fc = 12.0 * pr.y * P.inv_rc12 - 6.0 * pr.x * P.inv_rc6;
            f = (fr - fc) * r2inv;
            e_vdw += (pr.y * r12inv - pr.x * r6inv) + (r - P.rc) * fc / P.rc - (pr.y * P.inv_rc12 - pr.x * P.inv_rc6);
        } else {
            f = (pr.y * 2.0 * r12inv - pr.x * r6inv) * 6.0 * r2inv;
            e_vdw += pr.y * r12inv - pr.x * r6inv;
        }
    }
    if (qi != 0.0 && qj != 0.0) {
        const double qq = kFQQ * qi * qj;
        if (P.use_coulomb == 1) {
            const double a = P.w_alpha, ec = erfc(a * r);
            f += qq * ((ec * r2inv + P.w_a2_sqrtpi * exp(-a * a * r2) * rinv) - P.w_const) * rinv;
            e_qq += qq * (ec * rinv - P.w_erfc_arcut + P.w_const * (r - P.rc));
        } else {
            f += qq * r2inv * rinv;
            e_qq += qq * rinv;
        }
    }
    return f;
}

// The same terms in FP32, from the FP32 type pair.
__device__ __forceinline__ float pair_term_f(const PairConstsF &K, const TypePairF &tp, float qi, float qj, float r2,
                                             float &e_qq, float &e_vdw)
{
    const int fn = tp.fn;
    const float c6 = tp.c6, c12 = tp.c12, pa = tp.a, pb = tp.b;
    const float rinv = rsqrtf(r2), r = r2 * rinv, r2inv = rinv * rinv;
    if (fn == 4) {
        if (c6 != 0.f || c12 != 0.f) {
            const float r6inv = r2inv * r2inv * r2inv;
            const float a12 = c12 * r6inv * r6inv, a6 = c6 * r6inv, u = r / pa, eu = erff(u);
            e_vdw += (a12 - a6) * eu;
            return ((12.f * a12 - 6.f * a6) * rinv * eu - (a12 - a6) * 2.f * (float)kInvSqrtPi * expf(-u * u) / pa) *
                   rinv;
        }
        return 0.f;
    }
    if (fn == 3) {
        const float e1 = expf(-pb * (r - c6)), e2 = e1 * e1;
        e_vdw += pa * (e2 - 2.f * e1);
        return 2.f * pa * pb * (e2 - e1) * rinv;
    }
    if (fn == 2) {
        const float r6inv = r2inv * r2inv * r2inv, eb = expf(-pb * r);
        e_vdw += pa * eb - c6 * r6inv;
        return pa * eb * pb * rinv - 6.f * c6 * r6inv * r2inv;
    }
    float f = 0.f;
    if (c6 != 0.f || c12 != 0.f) {
        const float r6inv = r2inv * r2inv * r2inv, r12inv = r6inv * r6inv;
        if (K.use_vdw == 1) {
            const float fr = 12.f * c12 * r12inv - 6.f * c6 * r6inv;
            f = (fr - tp.fc) * r2inv;
            e_vdw += (c12 * r12inv - c6 * r6inv) + (r - K.rc) * tp.fc * K.inv_rc - tp.es;
        } else {
            f = (c12 * 2.f * r12inv - c6 * r6inv) * 6.f * r2inv;
            e_vdw += c12 * r12inv - c6 * r6inv;
        }
    }
    if (qi != 0.f && qj != 0.f) {
        const float qq = K.fqq * qi * qj;
        if (K.use_coulomb == 1) {
            const float ar = K.alpha * r, eg = expf(-ar * ar), ec = erfc_any_f(ar, eg);
            f += qq * ((ec * r2inv + K.a2_sqrtpi * eg * rinv) - K.w_const) * rinv;
            e_qq += qq * (ec * rinv - K.w_erfc_arcut + K.w_const * (r - K.rc));
        } else {
            f += qq * r2inv * rinv;
            e_qq += qq * rinv;
        }
    }
    return f;
}

// CPIM force on a metal atom from a permanent charge (the atom receives the
// opposite), FP32; r = metal - atom (cpim_charge_pair in FP32).
__device__ __forceinline__ void cpim_charge_pair_f(const PairConstsF &K, const float r[3], float r2, float q_perm,
                                                   float q_ind, const float p[3], float f[3])
{
    const float rinv = rsqrtf(r2), rr = r2 * rinv, r2inv = rinv * rinv;
    float a0, ec = 0.f, eg = 0.f;
    if (K.use_coulomb == 1) {
        const float ar = K.alpha * rr;
        eg = expf(-ar * ar);
        ec = erfc_any_f(ar, eg);
        a0 = (ec * r2inv + K.a2_sqrtpi * eg * rinv - K.w_const) * rinv;
    } else {
        a0 = r2inv * rinv;
    }
    const float s = K.fqq * q_perm;
#pragma unroll
    for (int a = 0; a < 3; ++a) f[a] = a0 * r[a] * s * q_ind;
    const float pr = p[0] * r[0] + p[1] * r[1] + p[2] * r[2];
    const float sp = s / (float)kNm2Bohr;
    const float ir3 = r2inv * rinv, ir5 = ir3 * r2inv;
    if (K.use_coulomb == 1) {
        const float al3 = K.alpha * K.alpha * K.alpha;
        const float a1 = ir5 * (ec + K.a2_sqrtpi * rr * eg);
        const float b1 = 4.f * (float)kInvSqrtPi * al3 * r2inv * eg;
        const float c1 = K.w_const * ir3;
        // sum_a T_ab p_a, T_ab = a1 (3 r_a r_b - d_ab r^2) + b1 r_a r_b - c1 (r_a r_b - d_ab r^2)
#pragma unroll
        for (int b = 0; b < 3; ++b)
            f[b] -= (a1 * (3.f * pr * r[b] - p[b] * r2) + b1 * pr * r[b] - c1 * (pr * r[b] - p[b] * r2)) * sp;
    } else {
#pragma unroll
        for (int b = 0; b < 3; ++b) f[b] -= (3.f * pr * r[b] - p[b] * r2) * ir5 * sp;
    }
}

// Per-lane force accumulator: plain FP64, or Kahan-compensated FP32.
template <typename Real>
struct Acc;
template <>
struct Acc<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double v) { s += v; }
    __device__ __forceinline__ double value() const { return s; }
};
template <>
struct Acc<float> {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float v)
    {
        const float y = v - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

// Type-pair tables staged in shared memory when the type count allows.
constexpr int kSmemTypes = 16;

// FP64 terms of a shifted-force Lennard-Jones and damped Coulomb pair (funct 1,
// use_vdw = use_coulomb = 1, alpha rc < kDsfMaxX); t: c6, c12 and the type pair's
// shifts of force and energy.
__device__ __forceinline__ double pair_term_short(const DevParams &P, double inv_rc, const double4 &t, bool vdw, double qq,
                                                  double r2, double &e_qq, double &e_vdw)
{
    const Dsf d = dsf_terms(P.w_alpha, r2);
    const double r2inv = d.rinv * d.rinv;
    double f = 0.0;
    if (qq != 0.0) {
        f = qq * (fma(d.ec, r2inv, P.w_a2_sqrtpi * d.eg * d.rinv) - P.w_const) * d.rinv;
        e_qq = fma(qq, fma(d.ec, d.rinv, -P.w_erfc_arcut) + P.w_const * (d.r - P.rc), e_qq);
    }
    if (vdw && (t.x != 0.0 || t.y != 0.0)) {
        const double r6inv = r2inv * r2inv * r2inv, a6 = t.x * r6inv, a12 = t.y * (r6inv * r6inv);
        f += (12.0 * a12 - 6.0 * a6 - t.z) * r2inv;
        e_vdw += (a12 - a6) + (d.r - P.rc) * (t.z * inv_rc) - t.w;
    }
    return f;
}

// The FP32 cut-off of the candidates of an atom at p (see k_pair): a pair whose
// FP64 difference is inside rc has an FP32 r^2 below it.  Its coordinates are at
// most A = max |p| + L + rc, so each FP32 coordinate is off by 2^-24 A, the
// difference by less than 2^-21 (A + L) with the shift and its roundings; where the
// shift itself is decided otherwise, the two images are equally far within that.
__device__ __forceinline__ float candidate_cut(const DevParams &P, const double4 &p)
{
    const double L = fmax(P.box.L[0], fmax(P.box.L[1], P.box.L[2]));
    const double A = fmax(fabs(p.x), fmax(fabs(p.y), fabs(p.z))) + 2.0 * L + P.rc;
    const double r = P.rc + 0x1p-19 * A;
    return __double2float_ru(r * r * 1.000001);
}
__device__ __forceinline__ float image1_f(float d, float L, float H) { return fabsf(d) > H ? d - copysignf(L, d) : d; }
// pbc_12's single conditional shift of one axis (image)
__device__ __forceinline__ double image1(double d, double L, double H) { return fabs(d) > H ? d - copysign(L, d) : d; }

// One warp per atom i (grid-stride); see the file comment.
template <typename Real, bool NONBONDED, bool CPIM>
__global__ void __launch_bounds__(kPairWarps * 32, sizeof(Real) == 4 ? 6 : 4) k_pair(
    DevParams P, PairConstsF K, const double4 *__restrict__ pos4, const float4 *__restrict__ pos4f,
    const uint32_t *__restrict__ nbr, const int *__restrict__ nnb, int cap, const double *__restrict__ vec_pq,
    double *__restrict__ fx, double *__restrict__ fy, double *__restrict__ fz, double *__restrict__ partials)
{
    // chunks of 32 candidates tested together; one where the FP64 CPIM terms need
    // the registers (9,309 atoms in 3,000 waters: two take 3.5% more of a step, without
    // those terms one takes 2% more)
    constexpr int NB = sizeof(Real) == 8 && CPIM ? 1 : 2;
    __shared__ uint32_t queue[kPairWarps][32 * (NB + 1)];  // < 32 left over and NB x 32 appended
    __shared__ double sh[32 * 11];
    __shared__ double wacc[kPairWarps][8];  // per warp: e_qq, e_vdw, virial xx xy xz yy yz zz
    // type-pair table: double4 parameters (FP64) or TypePairF records (mixed), 32 B each
    __shared__ __align__(16) unsigned char s_tab[kSmemTypes * kSmemTypes * 32];
    __shared__ double4 s_lj[sizeof(Real) == 8 ? kSmemTypes * kSmemTypes : 1];  // c6, c12 and pair_term's shift constants
    __shared__ int s_fn[kSmemTypes * kSmemTypes];
    __shared__ unsigned char s_metal[kSmemTypes];
    double4 *s_par = reinterpret_cast<double4 *>(s_tab);
    TypePairF *s_tpf = reinterpret_cast<TypePairF *>(s_tab);
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    uint32_t *Q = queue[wib];
    if (lane < 8) wacc[wib][lane] = 0.0;
    const bool smem_types = P.n_types <= kSmemTypes;
    if (smem_types) {
        const int nt2 = P.n_types * P.n_types;
        for (int k = threadIdx.x; k < nt2; k += blockDim.x) {
            if constexpr (sizeof(Real) == 8) {
                const double4 t = P.nb_par[k];
                s_par[k] = t;
                s_lj[k] = make_double4(t.x, t.y, 12.0 * t.y * P.inv_rc12 - 6.0 * t.x * P.inv_rc6,
                                       t.y * P.inv_rc12 - t.x * P.inv_rc6);
            } else {
                s_tpf[k] = make_type_pair_f(P, K, k);
            }
            s_fn[k] = P.nb_funct[k];
        }
        for (int k = threadIdx.x; k < P.n_types; k += blockDim.x) s_metal[k] = P.type_metal[k];
    }
    __syncthreads();
    // the type-pair table as the pair terms read it
    DevParams Pt = P;
    if (smem_types) {
        Pt.nb_par = s_par;
        Pt.nb_funct = s_fn;
    }
    const bool metal_by_type = smem_types && P.metal_by_type;
    const bool damped = P.use_coulomb == 1 && P.w_alpha * P.rc < kDsfMaxX;
    const bool shrt = smem_types && P.use_vdw == 1 && damped;
    const double inv_rc = 1.0 / P.rc;
    const float Lf[3] = {(float)P.box.L[0], (float)P.box.L[1], (float)P.box.L[2]};
    const float Hf[3] = {(float)P.box.H[0], (float)P.box.H[1], (float)P.box.H[2]};
    const int stride = gridDim.x * kPairWarps;
    for (int i = blockIdx.x * kPairWarps + wib; i < P.N; i += stride) {
        const double4 pi = pos4[i];
        const float xf = (float)pi.x, yf = (float)pi.y, zf = (float)pi.z, cut = candidate_cut(P, pi);
        const int trow = P.type[i] * P.n_types;
        const bool cpim_i = CPIM && P.is_metal[i] == 0 && pi.w != 0.0;
        bool vdw_i = false;  // a type pair of this atom has Lennard-Jones terms
        if (shrt)
            for (int t = 0; t < P.n_types; ++t) vdw_i = vdw_i || s_par[trow + t].x != 0.0 || s_par[trow + t].y != 0.0;
        const double qi = kFQQ * pi.w;
        const int n = nnb[i];
        const uint32_t *row = nbr + (size_t)i * cap;
        Acc<Real> f0, f1, f2;
        Real e_qq = 0, e_vdw = 0;
        Real v[6];  // the pair virial is symmetric: xx xy xz yy yz zz
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = 0;

        auto process = [&](uint32_t e, const double4 &pj, bool valid) {
            const double ddx = image1(pj.x - pi.x, P.box.L[0], P.box.H[0]);
            const double ddy = image1(pj.y - pi.y, P.box.L[1], P.box.H[1]);
            const double ddz = image1(pj.z - pi.z, P.box.L[2], P.box.H[2]);
            const Real dx = (Real)ddx, dy = (Real)ddy, dz = (Real)ddz;
            Real r2;
            bool ok;
            if constexpr (sizeof(Real) == 8) {
                // the reference's rounding of r^2: the FP64 pair set is the reference's
                r2 = norm2_exact(ddx, ddy, ddz);
                ok = valid && r2 < P.rc2;
            } else {
                // mixed: r^2 and the cut-off in FP32 from the FP64 minimum-image
                // difference; pairs within rounding of the cut-off contribute
                // nothing (shifted force and energy vanish there)
                r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                ok = valid && r2 < K.rc2;
            }
            if (!ok) return;
            const int tj = nb_type(e);
            if (NONBONDED) {
                Real f;
                if constexpr (sizeof(Real) == 8) {
                    if (shrt && s_fn[trow + tj] == 1)
                        f = pair_term_short(P, inv_rc, s_lj[trow + tj], vdw_i, qi * pj.w, r2, e_qq, e_vdw);
                    else
                        f = pair_term(Pt, trow + tj, pi.w, pj.w, r2, e_qq, e_vdw);
                } else {
                    f = pair_term_f(K, smem_types ? s_tpf[trow + tj] : make_type_pair_f(P, K, trow + tj), (float)pi.w,
                                    (float)pj.w, r2, e_qq, e_vdw);
                }
                const Real gx = f * dx, gy = f * dy, gz = f * dz;
                f0.add(-gx);
                f1.add(-gy);
                f2.add(-gz);
                v[0] -= dx * gx; v[1] -= dx * gy; v[2] -= dx * gz;
                v[3] -= dy * gy; v[4] -= dy * gz; v[5] -= dz * gz;
            }
            if (cpim_i) {
                const int j = nb_index(e);
                const bool mj = metal_by_type ? s_metal[tj] != 0 : P.is_metal[j] != 0;
                if (mj) {
                    const int jm = j - P.metal_min;
                    Real g[3];
                    const Real r[3] = {dx, dy, dz};  // metal - atom
                    const Real p[3] = {(Real)vec_pq[3 * jm], (Real)vec_pq[3 * jm + 1], (Real)vec_pq[3 * jm + 2]};
                    const Real q = (Real)vec_pq[3 * P.M + jm];
                    if constexpr (sizeof(Real) == 8) {
                        double a0, ec;
                        if (damped)
                            cpim_charge_pair_dsf(P, r, r2, pi.w, q, p, g, a0);
                        else
                            cpim_charge_pair(P, r, r2, pi.w, q, p, g, a0, ec);
                    } else {
                        cpim_charge_pair_f(K, r, r2, (float)pi.w, q, p, g);
                    }
                    f0.add(-g[0]);
                    f1.add(-g[1]);
                    f2.add(-g[2]);
                }
            }
        };

        // candidates: entries and FP32 positions of the next batch are loaded while
        // this one is tested (the list streams from HBM once per step, evict-first)
        uint32_t ev[NB], nxt[NB];
        float4 pf[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int k = u * 32 + lane, k2 = (NB + u) * 32 + lane;
            ev[u] = k < n ? __ldcs(row + k) : 0u;
            nxt[u] = k2 < n ? __ldcs(row + k2) : 0u;
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) pf[u] = pos4f[nb_index(ev[u])];
        // survivors: popped 32 at a time, their FP64 positions loaded one pop ahead
        int qn = 0, base = 0, cnt = -1;  // queue fill, next batch, size of the popped set (warp-uniform)
        uint32_t ec = 0;
        double4 pc = make_double4(0.0, 0.0, 0.0, 0.0);
        for (;;) {
            while (qn < 32 && base < n) {
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    const float dx = image1_f(pf[u].x - xf, Lf[0], Hf[0]), dy = image1_f(pf[u].y - yf, Lf[1], Hf[1]),
                                dz = image1_f(pf[u].z - zf, Lf[2], Hf[2]);
                    const bool ok = base + u * 32 + lane < n && fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < cut;
                    const unsigned ballot = __ballot_sync(0xffffffffu, ok);
                    if (ok) Q[qn + __popc(ballot & lt_mask)] = ev[u];
                    qn += __popc(ballot);
                }
                base += 32 * NB;
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    ev[u] = nxt[u];
                    pf[u] = pos4f[nb_index(ev[u])];
                    const int k = base + (NB + u) * 32 + lane;
                    nxt[u] = k < n ? __ldcs(row + k) : 0u;
                }
                __syncwarp();
            }
            const int take = min(qn, 32);
            uint32_t e2 = 0;
            double4 p2 = pc;
            if (lane < take) {
                e2 = Q[qn - take + lane];
                p2 = pos4[nb_index(e2)];
            }
            qn -= take;
            __syncwarp();
            if (cnt > 0) process(ec, pc, lane < cnt);
            if (take == 0) break;
            ec = e2;
            pc = p2;
            cnt = take;
        }

        const double s0 = warp_sum(f0.value()), s1 = warp_sum(f1.value()), s2 = warp_sum(f2.value());
        if (lane == 0) {
            fx[i] += s0;
            fy[i] += s1;
            fz[i] += s2;
        }
        if (NONBONDED) {
            double t[8] = {(double)e_qq, (double)e_vdw, (double)v[0], (double)v[1], (double)v[2], (double)v[3],
                           (double)v[4], (double)v[5]};
            const double w = warp_sum_halving<8>(t, lane);
            if ((lane & 3) == 0) wacc[wib][lane >> 2] += 0.5 * w;
        }
    }
    if (NONBONDED) {
        __syncthreads();
        // acc: e_qq, e_vdw, virial[9] (mirrored from the symmetric six)
        double acc[11] = {0.0};
        if (threadIdx.x < kPairWarps) {
            const double *w = wacc[threadIdx.x];
            acc[0] = w[0];
            acc[1] = w[1];
            acc[2] = w[2]; acc[3] = w[3]; acc[4] = w[4];
            acc[5] = w[3]; acc[6] = w[5]; acc[7] = w[6];
            acc[8] = w[4]; acc[9] = w[6]; acc[10] = w[7];
        }
        block_partials<11>(acc, sh, partials);
    }
}

// Mixed path on the cluster list (k_list.cu): one warp per cluster of up to
// four atoms.  Each entry (a j atom, its type, the mask of members it is a
// list neighbour of) is loaded once; j's minimum-image difference from the
// cluster centroid is formed in FP64 and rounded once, and the members' FP32
// offsets from the centroid give each member's difference and r^2 in FP32,
// cut as in k_pair.  The survivors go through the same per-warp queue and
// pair terms as k_pair, tagged with their member.  Each lane adds its pair's
// force in FP64 to its own slot of a shared-memory accumulator per member
// and axis; at the end of the cluster the 32 slots are summed in a fixed
// order, so the FP32 pair forces are summed without loss and run to run
// identically.  Pair energies are summed per lane in FP64 too.  Per chunk of
// 32 entries the four member tests run in straight-line code and append up to
// 128 pairs to the warp's queue (dynamic shared memory, kClQueue entries);
// full flushes of 32 follow at one site, which keeps the pair terms in the
// code once.
constexpr int kClQueue = 160;  // < 32 left over + 4 x 32 appended
constexpr int kClWarps = 8;      // warps per block of the cluster kernel
constexpr int kClMinBlocks = 2;  // resident blocks per SM the register budget allows
constexpr int kHalfWarps = 4, kHalfBlocks = 5;  // the same for k_pair_half
constexpr size_t kClQueueBytes = (size_t)kClWarps * kClQueue * (sizeof(float4) + sizeof(uint32_t));
// A warp's queue as two arrays: the neighbour's FP32 difference from the
// cluster centroid with its charge, and the list entry with the member
// index in its mask bits; the flush forms the member's difference from them
// by the same operations as the member test, so the pair's r^2 is the one
// the test accepted.  An append or a read is one 16-byte and one 4-byte
// shared-memory access.
struct ClQueue {
    float4 *a;
    uint32_t *b;
};
struct ClPair {
    float dx, dy, dz, r2, qj;
    uint32_t e;
};
template <bool NONBONDED, bool CPIM>
__global__ void __launch_bounds__(kClWarps * 32, kClMinBlocks) k_pair_cl(DevParams P, PairConstsF K, const double4 *__restrict__ pos4,
                                                              const int4 *__restrict__ cl_atoms,
                                                              const int *__restrict__ n_cl,
                                                              const uint32_t *__restrict__ nbr,
                                                              const int *__restrict__ nnb,
                                                              const unsigned char *__restrict__ cl_metal, int cap,
                                                              const double *__restrict__ vec_pq,
                                                              double *__restrict__ fx, double *__restrict__ fy,
                                                              double *__restrict__ fz, double *__restrict__ partials)
{
    constexpr int NB = 2;
    extern __shared__ __align__(16) unsigned char s_dyn[];  // the warps' queues
    __shared__ float4 s_mem[kClWarps][4];  // member offset from the centroid, charge
    __shared__ int s_trow[kClWarps][4];    // member type * n_types
    __shared__ unsigned char s_cpim[kClWarps][4];  // the member takes the CPIM force of metal neighbours
    __shared__ double s_acc[kClWarps][12][32];  // force on (member, axis) per lane slot
    __shared__ double sh[32 * 11];
    __shared__ double wacc[kClWarps][8];
    __shared__ __align__(16) TypePairF s_tpf[kSmemTypes * kSmemTypes];
    __shared__ unsigned char s_metal[kSmemTypes];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    ClQueue Q;
    Q.a = reinterpret_cast<float4 *>(s_dyn) + wib * kClQueue;
    Q.b = reinterpret_cast<uint32_t *>(s_dyn + (size_t)kClWarps * kClQueue * sizeof(float4)) + wib * kClQueue;
    if (lane < 8) wacc[wib][lane] = 0.0;
    const bool smem_types = P.n_types <= kSmemTypes;
    if (smem_types) {
        const int nt2 = P.n_types * P.n_types;
        for (int k = threadIdx.x; k < nt2; k += blockDim.x) s_tpf[k] = make_type_pair_f(P, K, k);
        for (int k = threadIdx.x; k < P.n_types; k += blockDim.x) s_metal[k] = P.type_metal[k];
    }
    __syncthreads();
    const bool metal_by_type = smem_types && P.metal_by_type;
    const double L[3] = {P.box.L[0], P.box.L[1], P.box.L[2]};
    const double iL[3] = {1.0 / L[0], 1.0 / L[1], 1.0 / L[2]};
    const int ncl = *n_cl;
    // fixed grid-stride order, which keeps the energy and virial sums in the
    // same order from run to run
    for (int cl = blockIdx.x * kClWarps + wib; cl < ncl; cl += gridDim.x * kClWarps) {
        const int4 A = cl_atoms[cl];
        const int nk = 1 + (A.y >= 0) + (A.z >= 0) + (A.w >= 0);
        const int mine = lane == 0 ? A.x : lane == 1 ? A.y : lane == 2 ? A.z : A.w;
        double4 pm = make_double4(0.0, 0.0, 0.0, 0.0);
        if (lane < nk) pm = pos4[mine];
        const double x0 = __shfl_sync(0xffffffffu, pm.x, 0), y0 = __shfl_sync(0xffffffffu, pm.y, 0),
                     z0 = __shfl_sync(0xffffffffu, pm.z, 0);
        double ox = 0.0, oy = 0.0, oz = 0.0;
        if (lane < nk) {
            ox = min_image(pm.x - x0, L[0], iL[0]);
            oy = min_image(pm.y - y0, L[1], iL[1]);
            oz = min_image(pm.z - z0, L[2], iL[2]);
        }
        // member mean offset: lanes 0..3 hold the offsets, the others zero
        double sx = ox, sy = oy, sz = oz;
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sy += __shfl_xor_sync(0xffffffffu, sy, o);
            sz += __shfl_xor_sync(0xffffffffu, sz, o);
        }
        const double inv_nk = 1.0 / nk;
        const double mx = __shfl_sync(0xffffffffu, sx, 0) * inv_nk, my = __shfl_sync(0xffffffffu, sy, 0) * inv_nk,
                     mz = __shfl_sync(0xffffffffu, sz, 0) * inv_nk;
        const double cx = x0 + mx, cy = y0 + my, cz = z0 + mz;
        if (lane < nk) {
            s_mem[wib][lane] = make_float4((float)(ox - mx), (float)(oy - my), (float)(oz - mz), (float)pm.w);
            s_trow[wib][lane] = P.type[mine] * P.n_types;
            s_cpim[wib][lane] = CPIM && P.is_metal[mine] == 0 && pm.w != 0.0;
        }
#pragma unroll
        for (int q = 0; q < 12; ++q) s_acc[wib][q][lane] = 0.0;
        __syncwarp();
        const bool cpim_cl = CPIM && cl_metal[cl] != 0;
        const int n = nnb[cl];
        const uint32_t *row = nbr + (size_t)cl * cap;
        double e_qq = 0.0, e_vdw = 0.0;  // per pair in FP64: a cluster's lane sums ~100 pairs
        float v[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = 0.f;

        // pair terms of the queue entries head .. head + cnt - 1 into the
        // lanes' slots
        auto flush = [&](int head, int cnt) {
            if (lane < cnt) {
                float g0 = 0.f, g1 = 0.f, g2 = 0.f;
                const float4 bq4 = Q.a[head + lane];
                ClPair c;
                c.e = Q.b[head + lane];
                const int k = (int)((c.e >> kClMaskShift) & 3u);
                const int tj = (int)(c.e >> kClTypeShift);
                const float4 mk = s_mem[wib][k];
                c.dx = bq4.x - mk.x;
                c.dy = bq4.y - mk.y;
                c.dz = bq4.z - mk.z;
                c.r2 = fmaf(c.dz, c.dz, fmaf(c.dy, c.dy, c.dx * c.dx));
                c.qj = bq4.w;
                if (NONBONDED) {
                    const int tp = s_trow[wib][k] + tj;
                    float eq = 0.f, ev = 0.f;
                    const float f = pair_term_f(K, smem_types ? s_tpf[tp] : make_type_pair_f(P, K, tp), mk.w, c.qj,
                                                c.r2, eq, ev);
                    e_qq += (double)eq;
                    e_vdw += (double)ev;
                    const float gx = f * c.dx, gy = f * c.dy, gz = f * c.dz;
                    g0 = -gx;
                    g1 = -gy;
                    g2 = -gz;
                    v[0] -= c.dx * gx; v[1] -= c.dx * gy; v[2] -= c.dx * gz;
                    v[3] -= c.dy * gy; v[4] -= c.dy * gz; v[5] -= c.dz * gz;
                }
                if (cpim_cl && s_cpim[wib][k]) {
                    const int j = (int)(c.e & kClIdxMask);
                    const bool mj = metal_by_type ? s_metal[tj] != 0 : P.is_metal[j] != 0;
                    if (mj) {
                        const int jm = j - P.metal_min;
                        const float r[3] = {c.dx, c.dy, c.dz};  // metal - atom
                        const float p[3] = {(float)vec_pq[3 * jm], (float)vec_pq[3 * jm + 1],
                                            (float)vec_pq[3 * jm + 2]};
                        float g[3];
                        cpim_charge_pair_f(K, r, c.r2, mk.w, (float)vec_pq[3 * P.M + jm], p, g);
                        g0 -= g[0];
                        g1 -= g[1];
                        g2 -= g[2];
                    }
                }
                s_acc[wib][3 * k][lane] += (double)g0;
                s_acc[wib][3 * k + 1][lane] += (double)g1;
                s_acc[wib][3 * k + 2][lane] += (double)g2;
            }
        };

        int qn = 0;  // queue fill, warp-uniform
        uint32_t nxt[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int k = u * 32 + lane;
            nxt[u] = k < n ? __ldcs(row + k) : 0u;
        }
        for (int base = 0; base < n; base += 32 * NB) {
            uint32_t ev[NB];
            bool valid[NB];
#pragma unroll
            for (int u = 0; u < NB; ++u) {
                valid[u] = base + u * 32 + lane < n;
                ev[u] = nxt[u];
                const int k = base + (NB + u) * 32 + lane;
                nxt[u] = k < n ? __ldcs(row + k) : 0u;
            }
            double4 pj[NB];
#pragma unroll
            for (int u = 0; u < NB; ++u)
                if (valid[u]) pj[u] = pos4[ev[u] & kClIdxMask];
            static_assert(NB == 2, "the member loop selects between two chunks");
            float dxc[NB], dyc[NB], dzc[NB], qj[NB];
            unsigned mask[NB];
            uint32_t keep[NB];
#pragma unroll
            for (int u = 0; u < NB; ++u) {
                dxc[u] = dyc[u] = dzc[u] = qj[u] = 0.f;
                mask[u] = 0;
                if (valid[u]) {
                    dxc[u] = (float)min_image(pj[u].x - cx, L[0], iL[0]);
                    dyc[u] = (float)min_image(pj[u].y - cy, L[1], iL[1]);
                    dzc[u] = (float)min_image(pj[u].z - cz, L[2], iL[2]);
                    qj[u] = (float)pj[u].w;
                    mask[u] = (ev[u] >> kClMaskShift) & 15u;
                }
                keep[u] = ev[u] & ~(15u << kClMaskShift);
            }
            // per chunk: the member tests in straight-line code (mask bits
            // exist only for members < nk), the survivors appended to the
            // queue, then the full flushes and the remainder moved to the front
#pragma unroll 1
            for (int u = 0; u < NB; ++u) {
                const bool hi = u == 1;
                const float bx = hi ? dxc[1] : dxc[0], by = hi ? dyc[1] : dyc[0], bz = hi ? dzc[1] : dzc[0];
                const float bq = hi ? qj[1] : qj[0];
                const unsigned bm = hi ? mask[1] : mask[0];
                const uint32_t bk = hi ? keep[1] : keep[0];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const float4 mk = s_mem[wib][kk];
                    const float dx = bx - mk.x, dy = by - mk.y, dz = bz - mk.z;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    const bool ok = ((bm >> kk) & 1u) && r2 < K.rc2;
                    const unsigned ballot = __ballot_sync(0xffffffffu, ok);
                    if (ok) {
                        const int at = qn + __popc(ballot & lt_mask);
                        Q.a[at] = make_float4(bx, by, bz, bq);
                        Q.b[at] = bk | ((uint32_t)kk << kClMaskShift);
                    }
                    qn += __popc(ballot);
                }
                __syncwarp();
                int head = 0;
                while (qn - head >= 32) {
                    flush(head, 32);
                    head += 32;
                }
                if (head > 0) {
                    const int rest = qn - head;
                    float4 ta;
                    uint32_t tb = 0;
                    if (lane < rest) {
                        ta = Q.a[head + lane];
                        tb = Q.b[head + lane];
                    }
                    __syncwarp();
                    if (lane < rest) {
                        Q.a[lane] = ta;
                        Q.b[lane] = tb;
                    }
                    __syncwarp();
                    qn = rest;
                }
            }
        }
        if (qn > 0) flush(0, qn);
        __syncwarp();

        // member forces: lane 3 k + a sums the 32 slots of (k, a), starting
        // at its own slot (no bank conflicts), in a fixed order
        if (lane < 3 * nk) {
            const int k = lane / 3, a = lane - 3 * k;
            double s = 0.0;
#pragma unroll 8
            for (int q = 0; q < 32; ++q) s += s_acc[wib][lane][(q + lane) & 31];
            const int atom = k == 0 ? A.x : k == 1 ? A.y : k == 2 ? A.z : A.w;
            double *f = a == 0 ? fx : (a == 1 ? fy : fz);
            f[atom] += s;
        }
        if (NONBONDED) {
            const double t[8] = {warp_sum(e_qq), warp_sum(e_vdw), warp_sum((double)v[0]),
                                 warp_sum((double)v[1]), warp_sum((double)v[2]), warp_sum((double)v[3]),
                                 warp_sum((double)v[4]), warp_sum((double)v[5])};
            if (lane == 0) {
#pragma unroll
                for (int q = 0; q < 8; ++q) wacc[wib][q] += 0.5 * t[q];
            }
        }
        __syncwarp();
    }
    if (NONBONDED) {
        __syncthreads();
        double acc[11] = {0.0};
        if (threadIdx.x < kClWarps) {
            const double *w = wacc[threadIdx.x];
            acc[0] = w[0];
            acc[1] = w[1];
            acc[2] = w[2]; acc[3] = w[3]; acc[4] = w[4];
            acc[5] = w[3]; acc[6] = w[5]; acc[7] = w[6];
            acc[8] = w[4]; acc[9] = w[6]; acc[10] = w[7];
        }
        block_partials<11>(acc, sh, partials);
    }
}

// A float times 2^-896 as a double, in three integer operations: the conversion
// instruction runs at an eighth of their rate, and the half-list kernel takes five
// a pair.  Moving the bits without correcting the exponent's bias gives the scale;
// it is exact, zero and subnormals included, so sums formed at this scale and
// multiplied by 2^896 at the end have the bits of plain FP64 sums.  Infinities and
// NaN are not preserved and take scaled_any.
constexpr float kScaledLimit = 1e30f;
__device__ __forceinline__ double scaled(float v)
{
    const int u = __float_as_int(v);
    return __hiloint2double((u >> 3) & 0x8fffffff, u << 29);
}
__device__ __forceinline__ double scaled_any(float v) { return (double)v * 0x1p-896; }

__device__ __forceinline__ float exp2_approx(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// min_image with the rounding by an addition of 1.5 2^52 instead of the rounding
// instruction, which runs at a fraction of the FP64 rate.
__device__ __forceinline__ double min_image_fma(double d, double L, double inv_L)
{
    return d - L * (fma(d, inv_L, 0x1.8p52) - 0x1.8p52);
}

__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Mixed path on the half cluster list (pair_list 0, the default, or 2; every
// pair listed once, k_list.cu): one warp per cluster of up to four atoms, a lane
// per entry.  A lane forms its neighbour's minimum-image difference from the
// centroid in FP64, rounds it once, and goes through the cluster's members: the
// pair's difference, r^2 and cut-off in FP32 as on the full list, and the pair
// terms in place for the lanes that pass.  The members' forces and the energies
// accumulate in the lane in FP64 (summed over the lanes at the end of the
// cluster); the neighbour's force over its at most four pairs in FP32, added to
// the atom by FP64 atomic adds.  The atomic adds make the order of the
// neighbour-side sums vary from run to run (FP64 rounding of FP32 terms).
//
// Bound by instruction issue (70% of the slots, 20 of 32 lanes active: about 45%
// of the lanes pass a member test, ~75 instructions a test with survivors).
// Queueing the survivors so that the pair terms run on full warps, as the full
// list does, costs more than the idle lanes: scans, 20 bytes written and read per
// pair in shared memory, the forces read and added in shared slots, shuffles for
// the neighbour's sum; 2.31 ms a call at 452,057 atoms and 0.51 at 91,122.
// Pairs in place 2.99 and 0.69 with the general terms in the four unrolled
// members (instruction cache misses); 1.51 and 0.44 with the short route below;
// 1.39 and 0.34 with the positions loaded a chunk ahead, the general terms in a
// rolled loop and five blocks of four warps (96 registers, no spills).
//
// Routes, chosen per cluster: `plain` where every type pair that can occur (all
// of them for a cluster next to metal, else those of non-metal types) has funct 1
// and the options are the shifted-force van der Waals and the damped Coulomb
// form with alpha rc < 5, the range of the fitted erfc; `general` otherwise
// (pair_term_f, all forms; also with more types than the shared tables hold).
// The short route takes the Gaussian as 2^(-alpha^2 log2(e) r^2) from r^2 itself,
// the constant as a sum of two (rounded to one, the Gaussian is off by up to 6e-8
// (alpha r)^2 of one sign in all pairs alike), and sharpens 1/r by a Newton step.
// Against 64 bits, alpha 2, r 0.12..1.2 nm: the Gaussian within 4e-7 and its mean
// within 2e-10 (expf of the rounded (alpha r)^2: 1.5e-6, 9e-10).  Net forces, rms
// relative error with expf and rsqrtf -> one rounded constant -> now: 7.58e-7 ->
// 7.91e-7 -> 7.45e-7 (8,000 waters around Au561), 6.86e-7 -> 6.97e-7 -> 6.94e-7
// (30,000 waters, two Au561).  The virial from the entry's
// summed force instead of per pair is 1% faster and 15% less accurate.
//
// The water-side CPIM term walks the entries a second time, only for clusters next
// to metal; taken from whichever end holds the metal.
template <bool NONBONDED, bool CPIM>
__global__ void __launch_bounds__(kHalfWarps * 32, kHalfBlocks) k_pair_half(
    DevParams P, PairConstsF K, const double4 *__restrict__ pos4, const int4 *__restrict__ cl_atoms,
    const int *__restrict__ n_cl, const uint32_t *__restrict__ nbr, const int *__restrict__ nnb,
    const unsigned char *__restrict__ cl_metal, int cap, const double *__restrict__ vec_pq, double *__restrict__ fx,
    double *__restrict__ fy, double *__restrict__ fz, double *__restrict__ partials, int *__restrict__ next,
    const int *__restrict__ sel)
{
    __shared__ float4 s_mem[kHalfWarps][4];  // member offset from the centroid, charge
    __shared__ int s_type[kHalfWarps][4];    // member type * n_types
    __shared__ int s_mmetal[kHalfWarps][4];  // the member's metal index, -1 not metal
    __shared__ double sh[32 * 11];
    __shared__ double wacc[kHalfWarps][8];
    __shared__ __align__(16) TypePairF s_tpf[kSmemTypes * kSmemTypes];
    __shared__ unsigned char s_metal[kSmemTypes], s_vdw[kSmemTypes];  // s_vdw: 1 with a non-metal type, 2 with a metal
    __shared__ __align__(16) float4 s_lj[kSmemTypes * kSmemTypes];     // c6, c12, fc, es
    bool plain_near = false, plain_far = false;  // all type pairs, or all of non-metal types, have funct 1
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane < 8) wacc[wib][lane] = 0.0;
    const bool smem_types = P.n_types <= kSmemTypes;
    const bool metal_by_type = smem_types && P.metal_by_type;
    if (smem_types) {
        const int nt = P.n_types;
        for (int k = threadIdx.x; k < nt * nt; k += blockDim.x) s_tpf[k] = make_type_pair_f(P, K, k);
        for (int k = threadIdx.x; k < nt; k += blockDim.x) s_metal[k] = P.type_metal[k];
        __syncthreads();
        for (int k = threadIdx.x; k < nt; k += blockDim.x) {
            int f = metal_by_type ? 0 : 3;
            for (int j = 0; j < nt; ++j) {
                const TypePairF &t = s_tpf[k * nt + j];
                if (t.fn != 1 || t.c6 != 0.f || t.c12 != 0.f) f |= s_metal[j] ? 2 : 1;
            }
            s_vdw[k] = (unsigned char)f;
        }
        bool near = true, far = true;
        for (int k = threadIdx.x; k < nt * nt; k += blockDim.x) {
            const TypePairF &t = s_tpf[k];
            s_lj[k] = make_float4(t.c6, t.c12, t.fc, t.es);
            near = near && t.fn == 1;
            far = far && (t.fn == 1 || (metal_by_type && (s_metal[k / nt] || s_metal[k % nt])));
        }
        const bool dsf = K.use_vdw == 1 && K.use_coulomb == 1 && K.alpha * K.rc < 5.0f;
        plain_near = __syncthreads_and(near) && dsf;
        plain_far = __syncthreads_and(far) && dsf;
    }
    __syncthreads();
    const double L[3] = {P.box.L[0], P.box.L[1], P.box.L[2]};
    const double iL[3] = {K.iL[0], K.iL[1], K.iL[2]};
    const int ncl = *n_cl;
    const float rc2 = K.rc2;
    // a resident grid whose warps take the next cluster from the counter
    // (zeroed before the launch), so list lengths that differ from cluster to
    // cluster leave no warp idle at the end; sel: only the listed clusters
    for (;;) {
        int ci = 0;
        if (lane == 0) ci = atomicAdd(next, 1);
        ci = __shfl_sync(0xffffffffu, ci, 0);
        if (ci >= ncl) break;
        const int cl = sel ? __ldg(sel + ci) : ci;
        const int n = nnb[cl];
        const uint32_t *row = nbr + (size_t)cl * cap;
        const uint32_t first = lane < n ? __ldcs(row + lane) : 0u;
        const int4 A = cl_atoms[cl];
        const int nk = 1 + (A.y >= 0) + (A.z >= 0) + (A.w >= 0);
        const int mine = lane == 0 ? A.x : lane == 1 ? A.y : lane == 2 ? A.z : A.w;
        double4 pm = make_double4(0.0, 0.0, 0.0, 0.0);
        if (lane < nk) pm = pos4[mine];
        const double x0 = __shfl_sync(0xffffffffu, pm.x, 0), y0 = __shfl_sync(0xffffffffu, pm.y, 0),
                     z0 = __shfl_sync(0xffffffffu, pm.z, 0);
        double ox = 0.0, oy = 0.0, oz = 0.0;
        if (lane < nk) {
            ox = min_image(pm.x - x0, L[0], iL[0]);
            oy = min_image(pm.y - y0, L[1], iL[1]);
            oz = min_image(pm.z - z0, L[2], iL[2]);
        }
        // member mean offset: lanes 0..3 hold the offsets, the others zero
        double sx = ox, sy = oy, sz = oz;
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sy += __shfl_xor_sync(0xffffffffu, sy, o);
            sz += __shfl_xor_sync(0xffffffffu, sz, o);
        }
        const double inv_nk = 1.0 / nk;
        const double mx = __shfl_sync(0xffffffffu, sx, 0) * inv_nk, my = __shfl_sync(0xffffffffu, sy, 0) * inv_nk,
                     mz = __shfl_sync(0xffffffffu, sz, 0) * inv_nk;
        const double cx = x0 + mx, cy = y0 + my, cz = z0 + mz;
        const bool near_metal = cl_metal[cl] != 0, cpim_cl = CPIM && near_metal;
        bool vdw = false;
        __syncwarp();
        if (lane < nk) {
            const int ty = P.type[mine];
            s_mem[wib][lane] = make_float4((float)(ox - mx), (float)(oy - my), (float)(oz - mz), (float)pm.w);
            s_type[wib][lane] = ty * P.n_types;
            vdw = smem_types && (s_vdw[ty] & (near_metal ? 3 : 1)) != 0;
            s_mmetal[wib][lane] = P.is_metal[mine] != 0 ? mine - P.metal_min : -1;
        }
        const unsigned vmask = __ballot_sync(0xffffffffu, vdw);
        const bool plain = NONBONDED && (near_metal ? plain_near : plain_far);
        __syncwarp();
        double f[16];  // force on member k, axis a at 3 k + a
#pragma unroll
        for (int q = 0; q < 16; ++q) f[q] = 0.0;
        double e_qq = 0.0, e_vdw = 0.0;
        float v[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = 0.f;

        // the entries of the row, `pairs` with each one's difference from the centroid
        auto walk = [&](auto pairs) {
            // the next chunk's positions are loaded while this one is computed, the
            // entries one further ahead
            uint32_t e = first, nxt = 32 + lane < n ? __ldcs(row + 32 + lane) : 0u;
            double4 pj = pos4[e & kClIdxMask];
            for (int base = 0; base < n; base += 32) {
                const float bx = (float)min_image_fma(pj.x - cx, L[0], iL[0]);
                const float by = (float)min_image_fma(pj.y - cy, L[1], iL[1]);
                const float bz = (float)min_image_fma(pj.z - cz, L[2], iL[2]);
                const float bq = (float)pj.w;
                pj = pos4[nxt & kClIdxMask];
                const uint32_t cur = e;
                e = nxt;
                const int k = base + 64 + lane;
                nxt = k < n ? __ldcs(row + k) : 0u;
                const int j = (int)(cur & kClIdxMask);
                float h[3] = {0.f, 0.f, 0.f};  // force on the neighbour
                // lanes past the end hold a zero entry: no mask bits
                pairs(j, (int)(cur >> kClTypeShift), (cur >> kClMaskShift) & 15u, bx, by, bz, bq, h);
                if (h[0] != 0.f || h[1] != 0.f || h[2] != 0.f) {
                    atomicAdd(fx + j, (double)h[0]);
                    atomicAdd(fy + j, (double)h[1]);
                    atomicAdd(fz + j, (double)h[2]);
                }
            }
        };
        // pairs of any form with the members in `mask`; h null: only the sums that `scaled` takes
        auto general = [&](int tj, unsigned mask, float bx, float by, float bz, float bq, float *h) {
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const float4 mk = s_mem[wib][k];
                const float dx = bx - mk.x, dy = by - mk.y, dz = bz - mk.z;
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                if (!(((mask >> k) & 1u) && r2 < rc2)) continue;
                const int tp = s_type[wib][k] + tj;
                float eq = 0.f, ev = 0.f;
                const float fp = pair_term_f(K, smem_types ? s_tpf[tp] : make_type_pair_f(P, K, tp), mk.w, bq, r2, eq,
                                             ev);
                const float gx = fp * dx, gy = fp * dy, gz = fp * dz;
                const double sx = scaled_any(gx), sy = scaled_any(gy), sz = scaled_any(gz);
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (m == k) {
                        f[3 * m] -= sx;
                        f[3 * m + 1] -= sy;
                        f[3 * m + 2] -= sz;
                    }
                e_qq += scaled_any(eq);
                e_vdw += scaled_any(ev);
                if (h) {
                    h[0] += gx;
                    h[1] += gy;
                    h[2] += gz;
                    v[0] -= dx * gx; v[1] -= dx * gy; v[2] -= dx * gz;
                    v[3] -= dy * gy; v[4] -= dy * gz; v[5] -= dz * gz;
                }
            }
        };
        if (plain) {
            walk([&](int, int tj, unsigned mask, float bx, float by, float bz, float bq, float *h) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 mk = s_mem[wib][k];
                    const float dx = bx - mk.x, dy = by - mk.y, dz = bz - mk.z;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    if (!(((mask >> k) & 1u) && r2 < rc2)) continue;
                    const float y = rsqrt_approx(r2), rinv = fmaf(0.5f * y, fmaf(-(r2 * y), y, 1.0f), y), r = r2 * rinv,
                                r2inv = rinv * rinv;
                    float fp = 0.f, eq = 0.f, ev = 0.f;
                    if ((vmask >> k) & 1u) {
                        const float4 t = s_lj[s_type[wib][k] + tj];
                        if (t.x != 0.f || t.y != 0.f) {
                            const float r6inv = r2inv * r2inv * r2inv, a6 = t.x * r6inv, a12 = t.y * (r6inv * r6inv);
                            fp = (12.f * a12 - 6.f * a6 - t.z) * r2inv;
                            ev = (a12 - a6) + (r - K.rc) * t.z * K.inv_rc - t.w;
                        }
                    }
                    if (mk.w != 0.f && bq != 0.f) {
                        const float qq = K.fqq * mk.w * bq, eg = exp2_approx(fmaf(K.gauss2, r2, K.gauss2_lo * r2)),
                                    ec = erfc_from_gauss_f(K.alpha * r, eg);
                        fp += qq * ((ec * r2inv + K.a2_sqrtpi * eg * rinv) - K.w_const) * rinv;
                        eq = qq * (ec * rinv - K.w_erfc_arcut + K.w_const * (r - K.rc));
                    }
                    const float gx = fp * dx, gy = fp * dy, gz = fp * dz;
                    if (fabsf(fp) < kScaledLimit) {
                        f[3 * k] -= scaled(gx);
                        f[3 * k + 1] -= scaled(gy);
                        f[3 * k + 2] -= scaled(gz);
                        e_qq += scaled(eq);
                        e_vdw += scaled(ev);
                    } else {
                        f[3 * k] -= scaled_any(gx);
                        f[3 * k + 1] -= scaled_any(gy);
                        f[3 * k + 2] -= scaled_any(gz);
                        e_qq += scaled_any(eq);
                        e_vdw += scaled_any(ev);
                    }
                    h[0] += gx;
                    h[1] += gy;
                    h[2] += gz;
                    v[0] -= dx * gx; v[1] -= dx * gy; v[2] -= dx * gz;
                    v[3] -= dy * gy; v[4] -= dy * gz; v[5] -= dz * gz;
                }
            });
        } else if (NONBONDED) {
            walk([&](int, int tj, unsigned mask, float bx, float by, float bz, float bq, float *h) {
                general(tj, mask, bx, by, bz, bq, h);
            });
        }
        if (NONBONDED) {
            double t[8] = {0x1p896 * e_qq, 0x1p896 * e_vdw, (double)v[0], (double)v[1], (double)v[2], (double)v[3],
                           (double)v[4], (double)v[5]};
            const double w = warp_sum_halving<8>(t, lane);
            if ((lane & 3) == 0) wacc[wib][lane >> 2] += w;
        }
        if (cpim_cl) {
            walk([&](int j, int tj, unsigned mask, float bx, float by, float bz, float bq, float *h) {
                const bool mj = metal_by_type ? s_metal[tj] != 0 : mask != 0 && P.is_metal[j] != 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 mk = s_mem[wib][k];
                    const float dx = bx - mk.x, dy = by - mk.y, dz = bz - mk.z;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    const int mm = s_mmetal[wib][k];
                    if (!(((mask >> k) & 1u) && r2 < rc2) || mj == (mm >= 0)) continue;
                    // one of the two is metal
                    const int m = mj ? j - P.metal_min : mm;
                    const float q = mj ? mk.w : bq, sgn = mj ? 1.f : -1.f;
                    if (q == 0.f) continue;
                    const float r[3] = {sgn * dx, sgn * dy, sgn * dz};  // metal - atom
                    const float p[3] = {(float)vec_pq[3 * m], (float)vec_pq[3 * m + 1], (float)vec_pq[3 * m + 2]};
                    float g[3];
                    cpim_charge_pair_f(K, r, r2, q, (float)vec_pq[3 * P.M + m], p, g);
                    if (mj) {
                        f[3 * k] -= scaled_any(g[0]);
                        f[3 * k + 1] -= scaled_any(g[1]);
                        f[3 * k + 2] -= scaled_any(g[2]);
                    } else {
                        h[0] -= g[0];
                        h[1] -= g[1];
                        h[2] -= g[2];
                    }
                }
            });
        }

        // member forces: summed over the lanes, value q = 3 k + a in lane 2 q
        const double sum = 0x1p896 * warp_sum_halving<16>(f, lane);
        const int q = lane >> 1, k = q / 3, a = q - 3 * k;
        if ((lane & 1) == 0 && k < nk) {
            const int atom = k == 0 ? A.x : k == 1 ? A.y : k == 2 ? A.z : A.w;
            double *out = a == 0 ? fx : (a == 1 ? fy : fz);
            atomicAdd(out + atom, sum);  // other clusters add to this atom as a neighbour
        }
    }
    if (NONBONDED) {
        __syncthreads();
        double acc[11] = {0.0};
        if (threadIdx.x < kHalfWarps) {
            const double *w = wacc[threadIdx.x];
            acc[0] = w[0];
            acc[1] = w[1];
            acc[2] = w[2]; acc[3] = w[3]; acc[4] = w[4];
            acc[5] = w[3]; acc[6] = w[5]; acc[7] = w[6];
            acc[8] = w[4]; acc[9] = w[6]; acc[10] = w[7];
        }
        block_partials<11>(acc, sh, partials);
    }
}

// Mixed path on the cluster-pair list (pair_list 4, k_list.cu): one warp per
// cluster I at a time (taken from a counter, as on the half cluster list),
// two entries (clusters J) per step.  Lane l works on member k = l & 3 of I
// with member m = (l >> 2) & 3 of entry h = l >> 4: the 32 lanes cover the
// 2 x 16 member pairs with no compaction, and a pair that is masked at the
// build or outside the cut-off now contributes nothing.  I's member stays in
// the lane's registers for the whole list; each step a lane loads J's
// centroid, its member's offset and charge, and its atom and type (the four
// lanes of one J member read the same addresses).  The pair difference is
// the FP64 minimum image of the centroid difference, rounded once, plus the
// FP32 offsets; the FP32 cut-off decides the pair as in k_pair.  Each pair
// counts once: the force on I's member accumulates in FP64 in the lane (the
// eight lanes of a member summed at the end, then added with FP64 atomic
// adds, since other clusters add to the same atom), the force on J's member
// is summed over its four lanes by shuffles and added with FP64 atomic adds;
// pair energies are summed per lane in FP64, the virial per lane in FP32 per
// cluster.  CPIM: on entries where either cluster has a metal member, the
// CPIM force on a charged non-metal atom from a metal atom of the pair,
// whichever end holds the metal.
constexpr int kCpWarps = 8;
constexpr int kCpMinBlocks = 2;
template <bool NONBONDED, bool CPIM>
__global__ void __launch_bounds__(kCpWarps * 32, kCpMinBlocks)
    k_pair_cp(DevParams P, PairConstsF K, const double4 *__restrict__ cent, const float4 *__restrict__ off,
              const int *__restrict__ ti, const uint2 *__restrict__ list, const int *__restrict__ cnt, int cap,
              int ncl, const double *__restrict__ vec_pq, double *__restrict__ fx, double *__restrict__ fy,
              double *__restrict__ fz, double *__restrict__ partials, int *__restrict__ next)
{
    __shared__ double sh[32 * 11];
    __shared__ double wacc[kCpWarps][8];
    __shared__ __align__(16) TypePairF s_tpf[kSmemTypes * kSmemTypes];
    __shared__ unsigned char s_metal[kSmemTypes];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ki = lane & 3, mj = (lane >> 2) & 3, h = lane >> 4;
    if (lane < 8) wacc[wib][lane] = 0.0;
    const bool smem_types = P.n_types <= kSmemTypes;
    if (smem_types) {
        const int nt2 = P.n_types * P.n_types;
        for (int k = threadIdx.x; k < nt2; k += blockDim.x) s_tpf[k] = make_type_pair_f(P, K, k);
        for (int k = threadIdx.x; k < P.n_types; k += blockDim.x) s_metal[k] = P.type_metal[k];
    }
    __syncthreads();
    const bool metal_by_type = smem_types && P.metal_by_type;
    const double L[3] = {P.box.L[0], P.box.L[1], P.box.L[2]};
    const double iL[3] = {1.0 / L[0], 1.0 / L[1], 1.0 / L[2]};
    for (;;) {
        int ic = 0;
        if (lane == 0) ic = atomicAdd(next, 1);
        ic = __shfl_sync(0xffffffffu, ic, 0);
        if (ic >= ncl) break;
        const double4 ci = cent[ic];
        const float4 oi = off[4 * ic + ki];
        const int tii = ti[4 * ic + ki];
        const bool vi = tii >= 0;
        const int ai = tii & kCpIdxMask;
        const int tyi = vi ? (tii >> kCpTypeShift) : 0;
        const int trow = tyi * P.n_types;
        const bool metal_i = vi && (metal_by_type ? s_metal[tyi] != 0 : P.is_metal[ai] != 0);
        const int mi = metal_i ? ai - P.metal_min : 0;
        const bool water_i = CPIM && vi && !metal_i && oi.w != 0.f;  // takes the CPIM force of metal atoms
        double fix = 0.0, fiy = 0.0, fiz = 0.0, e_qq = 0.0, e_vdw = 0.0;
        float v[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = 0.f;
        const int n = cnt[ic];
        const uint2 *row = list + (size_t)ic * cap;
        for (int q0 = 0; q0 < n; q0 += 2) {
            const int q = q0 + h;
            const bool ve = q < n;
            const uint2 e = ve ? row[q] : make_uint2((uint32_t)ic, 0u);
            const int jc = (int)e.x;
            const double4 cj = cent[jc];
            const float4 oj = off[4 * jc + mj];
            const int tij = ti[4 * jc + mj];
            const float dcx = (float)min_image(cj.x - ci.x, L[0], iL[0]);
            const float dcy = (float)min_image(cj.y - ci.y, L[1], iL[1]);
            const float dcz = (float)min_image(cj.z - ci.z, L[2], iL[2]);
            const float dx = dcx + (oj.x - oi.x), dy = dcy + (oj.y - oi.y), dz = dcz + (oj.z - oi.z);
            const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            const bool act = ((e.y >> (4 * ki + mj)) & 1u) && r2 < K.rc2;
            float gx = 0.f, gy = 0.f, gz = 0.f;  // force on I's member
            float hx = 0.f, hy = 0.f, hz = 0.f;  // force on J's member
            if (act) {
                const int aj = tij & kCpIdxMask, tyj = tij >> kCpTypeShift;
                if (NONBONDED) {
                    const int tp = trow + tyj;
                    float eq = 0.f, ev = 0.f;
                    const float f = pair_term_f(K, smem_types ? s_tpf[tp] : make_type_pair_f(P, K, tp), oi.w, oj.w,
                                                r2, eq, ev);
                    e_qq += (double)eq;
                    e_vdw += (double)ev;
                    hx = f * dx;
                    hy = f * dy;
                    hz = f * dz;
                    gx = -hx;
                    gy = -hy;
                    gz = -hz;
                    v[0] -= dx * hx; v[1] -= dx * hy; v[2] -= dx * hz;
                    v[3] -= dy * hy; v[4] -= dy * hz; v[5] -= dz * hz;
                }
                if (CPIM && (e.y & kCpMetalBit)) {
                    const bool metal_j = metal_by_type ? s_metal[tyj] != 0 : P.is_metal[aj] != 0;
                    if (water_i && metal_j) {
                        const int jm = aj - P.metal_min;
                        const float r[3] = {dx, dy, dz};  // metal - atom
                        const float p[3] = {(float)vec_pq[3 * jm], (float)vec_pq[3 * jm + 1], (float)vec_pq[3 * jm + 2]};
                        float g[3];
                        cpim_charge_pair_f(K, r, r2, oi.w, (float)vec_pq[3 * P.M + jm], p, g);
                        gx -= g[0];
                        gy -= g[1];
                        gz -= g[2];
                    } else if (metal_i && !metal_j && oj.w != 0.f) {
                        const float r[3] = {-dx, -dy, -dz};  // metal - atom
                        const float p[3] = {(float)vec_pq[3 * mi], (float)vec_pq[3 * mi + 1], (float)vec_pq[3 * mi + 2]};
                        float g[3];
                        cpim_charge_pair_f(K, r, r2, oj.w, (float)vec_pq[3 * P.M + mi], p, g);
                        hx -= g[0];
                        hy -= g[1];
                        hz -= g[2];
                    }
                }
            }
            fix += (double)gx;
            fiy += (double)gy;
            fiz += (double)gz;
            // J's member: the four lanes of (h, m) summed, added by the first
#pragma unroll
            for (int o = 1; o <= 2; o <<= 1) {
                hx += __shfl_xor_sync(0xffffffffu, hx, o);
                hy += __shfl_xor_sync(0xffffffffu, hy, o);
                hz += __shfl_xor_sync(0xffffffffu, hz, o);
            }
            if (ki == 0 && (hx != 0.f || hy != 0.f || hz != 0.f)) {
                const int aj = tij & kCpIdxMask;
                atomicAdd(fx + aj, (double)hx);
                atomicAdd(fy + aj, (double)hy);
                atomicAdd(fz + aj, (double)hz);
            }
        }
        // I's member: its eight lanes summed in a fixed order
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            fix += __shfl_xor_sync(0xffffffffu, fix, o);
            fiy += __shfl_xor_sync(0xffffffffu, fiy, o);
            fiz += __shfl_xor_sync(0xffffffffu, fiz, o);
        }
        if (lane < 4 && vi && (fix != 0.0 || fiy != 0.0 || fiz != 0.0)) {
            atomicAdd(fx + ai, fix);
            atomicAdd(fy + ai, fiy);
            atomicAdd(fz + ai, fiz);
        }
        if (NONBONDED) {
            const double t[8] = {warp_sum(e_qq), warp_sum(e_vdw), warp_sum((double)v[0]),
                                 warp_sum((double)v[1]), warp_sum((double)v[2]), warp_sum((double)v[3]),
                                 warp_sum((double)v[4]), warp_sum((double)v[5])};
            if (lane == 0) {
#pragma unroll
                for (int q = 0; q < 8; ++q) wacc[wib][q] += t[q];
            }
        }
        __syncwarp();
    }
    if (NONBONDED) {
        __syncthreads();
        double acc[11] = {0.0};
        if (threadIdx.x < kCpWarps) {
            const double *w = wacc[threadIdx.x];
            acc[0] = w[0];
            acc[1] = w[1];
            acc[2] = w[2]; acc[3] = w[3]; acc[4] = w[4];
            acc[5] = w[3]; acc[6] = w[5]; acc[7] = w[6];
            acc[8] = w[4]; acc[9] = w[6]; acc[10] = w[7];
        }
        block_partials<11>(acc, sh, partials);
    }
}

PairConstsF pair_consts_f(const capac_ctx *c)
{
    PairConstsF K;
    K.rc = (float)c->P.rc;
    K.inv_rc = (float)(1.0 / c->P.rc);
    K.inv_rc12 = (float)c->P.inv_rc12;
    K.inv_rc6 = (float)c->P.inv_rc6;
    K.alpha = (float)c->P.w_alpha;
    K.a2_sqrtpi = (float)c->P.w_a2_sqrtpi;
    K.w_const = (float)c->P.w_const;
    K.w_erfc_arcut = (float)c->P.w_erfc_arcut;
    K.fqq = (float)kFQQ;
    K.rc2 = (float)c->P.rc2;
    const double g2 = -c->P.w_alpha * c->P.w_alpha * 1.4426950408889634074;
    K.gauss2 = (float)g2;
    K.gauss2_lo = (float)(g2 - (double)K.gauss2);
    K.use_vdw = c->P.use_vdw;
    K.use_coulomb = c->P.use_coulomb;
    for (int a = 0; a < 3; ++a) K.iL[a] = 1.0 / c->P.box.L[a];
    return K;
}

template <typename Real>
void launch_pair_t(capac_ctx *c, int mode, unsigned grid)
{
    const PairConstsF K = pair_consts_f(c);
    const bool cpim = c->M > 0 && c->use_cpff;
    double *part = force_partials(c, FP_PAIR);
    ProfScope ps(c, K_PAIR);
    if (mode == 0 && cpim)
        k_pair<Real, true, true><<<grid, kPairWarps * 32, 0, c->stream>>>(c->P, K, c->pos4, c->pos4f, c->nbr, c->nnb, c->cap,
                                                                          c->vec_pq, c->fx, c->fy, c->fz, part);
    else if (mode == 0)
        k_pair<Real, true, false><<<grid, kPairWarps * 32, 0, c->stream>>>(c->P, K, c->pos4, c->pos4f, c->nbr, c->nnb, c->cap,
                                                                           c->vec_pq, c->fx, c->fy, c->fz, part);
    else
        k_pair<Real, false, true><<<grid, kPairWarps * 32, 0, c->stream>>>(c->P, K, c->pos4, c->pos4f, c->nbr, c->nnb, c->cap,
                                                                           c->vec_pq, c->fx, c->fy, c->fz, part);
    ++c->launches;
}

// The full-list cluster kernel.
template <bool NONBONDED, bool CPIM>
void launch_pair_cl_t(capac_ctx *c, unsigned grid, double *partials)
{
    // the queues and the static arrays together exceed the default 48 KB
    CAPAC_CUDA(cudaFuncSetAttribute(k_pair_cl<NONBONDED, CPIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kClQueueBytes));
    k_pair_cl<NONBONDED, CPIM><<<grid, kClWarps * 32, kClQueueBytes, c->stream>>>(
        c->P, pair_consts_f(c), c->pos4, c->cl_atoms, c->cl_cell_start + c->n_cells, c->cl_nbr, c->cl_nnb, c->cl_metal,
        c->cl_cap, c->vec_pq, c->fx, c->fy, c->fz, partials);
}

// The half-list cluster kernel on stream st, its block partials to `partials`;
// sel: only the clusters with a metal member or neighbour.
template <bool NONBONDED, bool CPIM>
void launch_pair_half_t(capac_ctx *c, unsigned grid, cudaStream_t st, double *partials, bool sel)
{
    CAPAC_CUDA(cudaMemsetAsync(c->cl_next, 0, sizeof(int), st));
    k_pair_half<NONBONDED, CPIM><<<grid, kHalfWarps * 32, 0, st>>>(
        c->P, pair_consts_f(c), c->pos4, c->cl_atoms, sel ? c->n_cl_sel : c->cl_cell_start + c->n_cells, c->cl_nbr,
        c->cl_nnb, c->cl_metal, c->cl_cap, c->vec_pq, c->fx, c->fy, c->fz, partials, c->cl_next,
        sel ? c->cl_sel : nullptr);
}

template <bool NONBONDED, bool CPIM>
void launch_pair_cp_t(capac_ctx *c, unsigned grid)
{
    CAPAC_CUDA(cudaMemsetAsync(c->cl_next, 0, sizeof(int), c->stream));
    k_pair_cp<NONBONDED, CPIM><<<grid, kCpWarps * 32, 0, c->stream>>>(
        c->P, pair_consts_f(c), c->cp_cent, c->cp_off, c->cp_ti, c->cp_list, c->cp_n, c->cp_cap, c->n_clusters,
        c->vec_pq, c->fx, c->fy, c->fz, force_partials(c, FP_PAIR), c->cl_next);
}

// The cluster frames of the current positions, then the cluster-pair kernel.
void launch_pair_cpairs(capac_ctx *c, int mode, unsigned grid)
{
    const bool cpim = c->M > 0 && c->use_cpff;
    ProfScope ps(c, K_PAIR);
    launch_cluster_frames(c, false);
    if (mode == 0 && cpim)
        launch_pair_cp_t<true, true>(c, grid);
    else if (mode == 0)
        launch_pair_cp_t<true, false>(c, grid);
    else
        launch_pair_cp_t<false, true>(c, grid);
    ++c->launches;
}

void launch_pair_clusters(capac_ctx *c, int mode, unsigned grid)
{
    const bool cpim = c->M > 0 && c->use_cpff;
    double *part = force_partials(c, FP_PAIR);
    ProfScope ps(c, K_PAIR);
    if (c->cl_half) {
        if (mode == 0 && cpim && c->pair_split) {
            // the pair terms without the CPIM branches, then the water-side
            // CPIM term over the clusters with a metal member or neighbour
            launch_pair_half_t<true, false>(c, grid, c->stream, part, false);
            launch_pair_half_t<false, true>(c, grid, c->stream, part, true);
            ++c->launches;
        } else if (mode == 0 && cpim)
            launch_pair_half_t<true, true>(c, grid, c->stream, part, false);
        else if (mode == 0)
            launch_pair_half_t<true, false>(c, grid, c->stream, part, false);
        else
            launch_pair_half_t<false, true>(c, grid, c->stream, part, false);
    } else if (mode == 0 && cpim)
        launch_pair_cl_t<true, true>(c, grid, part);
    else if (mode == 0)
        launch_pair_cl_t<true, false>(c, grid, part);
    else
        launch_pair_cl_t<false, true>(c, grid, part);
    ++c->launches;
}

}  // namespace

// Blocks of the pair launch: one warp per atom (or per cluster), at most 16
// blocks per SM (grid-stride beyond); on the half cluster list the resident
// blocks only (its warps take clusters from a counter).
unsigned pair_grid(const capac_ctx *c)
{
    if (c->cpairs) return (unsigned)c->num_sms * kCpMinBlocks;
    const long units = c->clusters ? c->n_clusters : c->N;
    const int warps = c->clusters ? (c->cl_half ? kHalfWarps : kClWarps) : kPairWarps;
    const long need = (units + warps - 1) / warps;
    const long cap = (long)c->num_sms * (c->clusters && c->cl_half ? kHalfBlocks : 16);
    return (unsigned)std::max(1L, std::min(need, cap));
}

// Overlap, first half (on stream2, once `stream` has reached this point):
// the nonbonded terms of the half cluster list, two blocks per SM so that the
// CPIM solve's blocks find room beside it; energies and virial into
// partials2.  The forces go to fx, fy, fz by atomic adds only, so the
// kernels that run meanwhile on `stream` must leave them alone (the CPIM
// right-hand side, matrix and solve do).
void launch_pair_nonbonded_async(capac_ctx *c)
{
    CAPAC_CUDA(cudaEventRecord(c->ev_fork, c->stream));
    CAPAC_CUDA(cudaStreamWaitEvent(c->stream2, c->ev_fork, 0));
    c->work_stream = c->stream2;
    {
        ProfScope ps(c, K_PAIR);
        // two blocks (eight warps) per SM, and no more blocks than warps have clusters to take
        c->async_grid = std::min(2u * (unsigned)c->num_sms, pair_grid(c));
        launch_pair_half_t<true, false>(c, c->async_grid, c->stream2, c->partials2, false);
    }
    c->work_stream = nullptr;
    ++c->launches;
    CAPAC_CUDA(cudaEventRecord(c->ev_join, c->stream2));
}

// Overlap, second half (on `stream`, after the solve): wait for the first,
// sum its energies and virial, then the CPIM forces on water atoms from the
// solved induced vector over the clusters with a metal member or neighbour.
void launch_pair_join(capac_ctx *c)
{
    CAPAC_CUDA(cudaStreamWaitEvent(c->stream, c->ev_join, 0));
    static const int pot_slots[11] = {7, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1};
    static const int vir_slots[11] = {-1, -1, 0, 1, 2, 3, 4, 5, 6, 7, 8};
    launch_finalize(c, (int)c->async_grid, 11, pot_slots, vir_slots, c->partials2);
    {
        ProfScope ps(c, K_PAIR);
        launch_pair_half_t<false, true>(c, pair_grid(c), c->stream, c->partials, true);
    }
    ++c->launches;
}

void launch_pair_forces(capac_ctx *c, int mode)
{
    const unsigned grid = pair_grid(c);
    if (c->cpairs)
        launch_pair_cpairs(c, mode, grid);
    else if (c->clusters)
        launch_pair_clusters(c, mode, grid);
    else if (c->opt.precision == CAPAC_PREC_MIXED)
        launch_pair_t<float>(c, mode, grid);
    else
        launch_pair_t<double>(c, mode, grid);
    if (mode == 0 && c->defer) {
        c->fs.pair = force_partials(c, FP_PAIR);
        c->fs.n_pair = (int)grid;
    } else if (mode == 0) {
        static const int pot_slots[11] = {7, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1};
        static const int vir_slots[11] = {-1, -1, 0, 1, 2, 3, 4, 5, 6, 7, 8};
        launch_finalize(c, (int)grid, 11, pot_slots, vir_slots);
    }
}

}  // namespace capac
