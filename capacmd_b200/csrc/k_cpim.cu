// Sutton-Chen and CPIM kernels, FP64, plus the deterministic reductions.
//
// Metal atoms are contiguous (MM_METAL min..max).  The CPIM system of size
// n_mat = 4M + n_NPs is the reference's (cpff.c:205-519): per ordered metal
// pair (i, j) a 4x4 block over (p_x, p_y, p_z, q) of each atom,
//
//     [ A_ij (3x3)   m_ij ]     A_ij = -(c1 (3 r r^T - r^2 I) - c2 r r^T)
//     [ -m_ij^T      C_ij ]     m_ij = c3 r,  C_ij = -erf(r/R_qq)/r
//
// with diagonal blocks diag(1/polar x3, -1/capac), and the charge-neutrality
// rows/columns (+1 between an NP's Lagrange multiplier and its charges).
// Blocks are stored densely (the reference has no cut-off here either) as 16
// planes per block row: mat[(i*16 + e)*Mp + j], e = 4*row + col, so a warp
// reading consecutive j of one plane is fully coalesced.
#include "terms.cuh"

namespace capac {

// ---------------------------------------------------------- reductions

struct Slots {
    int pot[24];
    int vir[24];
};

// One block per value k (the slots of one launch are distinct, checked on
// the host), each summing its column of the per-block partials in a fixed
// order.
__global__ void __launch_bounds__(256) k_finalize(const double *__restrict__ partials, int nblocks, int K,
                                                  Slots s, double *pot, double *vir)
{
    __shared__ double sh[32];
    const int k = blockIdx.x;
    double v = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) v += partials[(size_t)b * K + k];
    double t[1] = {v};
    block_sum<1>(t, sh);
    if (threadIdx.x == 0) {
        if (s.pot[k] >= 0) pot[s.pot[k]] += t[0];
        if (s.vir[k] >= 0) vir[s.vir[k]] += t[0];
    }
}

void launch_finalize(capac_ctx *c, int nblocks, int K, const int *slots_pot, const int *slots_vir, const double *src)
{
    Slots s;
    for (int k = 0; k < 24; ++k) {
        s.pot[k] = k < K ? slots_pot[k] : -1;
        s.vir[k] = k < K ? slots_vir[k] : -1;
    }
    // the values are summed by separate blocks: no two may share a slot
    for (int a = 0; a < K; ++a)
        for (int b = a + 1; b < K; ++b)
            if ((s.pot[a] >= 0 && s.pot[a] == s.pot[b]) || (s.vir[a] >= 0 && s.vir[a] == s.vir[b]))
                throw Error(CAPAC_ERR_INVALID, "finalize: two values share an energy or virial slot");
    k_finalize<<<K, 256, 0, c->stream>>>(src ? src : c->partials, nblocks, K, s, c->pot, c->vir);
    ++c->launches;
}

// All of a force call's block partials at once: block k sums one energy or
// virial slot over its sources in a fixed order (a launch per source took
// 2-3 us each).
__global__ void __launch_bounds__(256) k_force_sums(ForceSums f, double *pot, double *vir)
{
    __shared__ double sh[32];
    static const int kPot[9] = {1, 7, 8, 9, 10, 11, 12, 13, 14};
    const int k = blockIdx.x;
    double t[1] = {0.0};
    auto add = [&](const double *p, int n, int K, int col) {
        for (int b = threadIdx.x; b < n; b += blockDim.x) t[0] += p[(size_t)b * K + col];
    };
    if (k < 9) {
        if (k == 0) add(f.qsc, f.n_qsc, 10, 0);
        if (k == 1 || k == 2) add(f.pair, f.n_pair, 11, k - 1);
        if (k >= 3) add(f.metal, f.n_metal, 15, k - 3);
        if (k == 3) add(f.field, f.n_field, 1, 0);
    } else {
        add(f.qsc, f.n_qsc, 10, k - 8);
        add(f.pair, f.n_pair, 11, k - 7);
        add(f.metal, f.n_metal, 15, k - 3);
    }
    block_sum<1>(t, sh);
    if (threadIdx.x == 0) (k < 9 ? pot[kPot[k]] : vir[k - 9]) += t[0];
}

void launch_force_sums(capac_ctx *c)
{
    k_force_sums<<<18, 256, 0, c->stream>>>(c->fs, c->pot, c->vir);
    ++c->launches;
}

// --------------------------------------------------------- Sutton-Chen

// (a/r)^e of an exponent e from t = (a/r)^2.  The reference's
// exponents are integers: products of t (a square root more where odd) then
// take 4-5 operations where log and exp take ~60.  Real exponents (parameter
// gradients) go through exp(e log(a/r)), within ~1e-15 of pow.
struct QscPower {
    double e;
    int half;  // floor(e / 2), -1: not an integer of 0..64
    bool odd;
    __device__ __forceinline__ explicit QscPower(double x) : e(x)
    {
        const bool whole = x >= 0.0 && x <= 64.0 && x == floor(x);
        half = whole ? (int)x >> 1 : -1;
        odd = whole && ((int)x & 1);
    }
    // log_t: log(t), read where the exponent is no such integer
    __device__ __forceinline__ double operator()(double t, double log_t) const
    {
        if (half < 0) return exp(0.5 * e * log_t);
        double y = odd ? sqrt(t) : 1.0, b = t;
        for (int k = half; k; k >>= 1, b *= b)
            if (k & 1) y *= b;
        return y;
    }
};

// mpi_qsc_dens, force.c:385-461: rho_i = sum_{j != i, r < rc} (a/r)^m.
// A block per atom here and below: with a warp per atom (as many warps on the chip
// as the metal has atoms) a warp waited for one load of its row after another.
constexpr int kQscBlock = 128;
__global__ void __launch_bounds__(kQscBlock) k_qsc_density(DevParams P, const double4 *__restrict__ pos4, double *isd)
{
    __shared__ double sh[32];
    const int i = blockIdx.x;
    const double4 pi = pos4[P.metal_min + i];
    double rho[1] = {0.0};
    const QscPower pm(P.qsc_m);
    const double a2 = P.qsc_a * P.qsc_a;
#pragma unroll 2
    for (int j = threadIdx.x; j < P.M; j += kQscBlock) {
        const double4 pj = pos4[P.metal_min + j];
        double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
        image(dx, dy, dz, P.box);
        const double r2 = norm2_exact(dx, dy, dz);
        if (j != i && r2 < P.rc2) {
            const double t = a2 / r2;
            rho[0] += pm(t, pm.half < 0 ? log(t) : 0.0);
        }
    }
    block_sum<1>(rho, sh);
    if (threadIdx.x == 0) isd[i] = 1.0 / sqrt(rho[0]);
}

// mpi_qsc_force, force.c:468-542: forces on i only, virial halved.
__global__ void __launch_bounds__(kQscBlock) k_qsc_force(DevParams P, const double4 *__restrict__ pos4,
                                                         const double *__restrict__ isd, double *fx, double *fy,
                                                         double *fz, double *partials)
{
    __shared__ double sh[32 * 10];
    const int i = blockIdx.x;
    const double4 pi = pos4[P.metal_min + i];
    const double isd_i = isd[i], cm2 = P.qsc_c * P.qsc_m / 2.0;
    const QscPower pn(P.qsc_n), pm(P.qsc_m);
    const double a2 = P.qsc_a * P.qsc_a;
    double acc[10] = {0.0};  // (a/r)^n, virial xx xy xz yy yz zz, force
#pragma unroll 2
    for (int j = threadIdx.x; j < P.M; j += kQscBlock) {
        const double4 pj = pos4[P.metal_min + j];
        const double isd_j = isd[j];
        double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
        image(dx, dy, dz, P.box);
        const double r2 = norm2_exact(dx, dy, dz);
        if (j == i || r2 >= P.rc2) continue;
        const double r2inv = 1.0 / r2, t = a2 * r2inv, lt = pn.half < 0 || pm.half < 0 ? log(t) : 0.0;
        const double an = pn(t, lt), am = pm(t, lt);
        const double f = P.qsc_eps * (P.qsc_n * an - cm2 * (isd_i + isd_j) * am) * r2inv;
        const double gx = f * dx, gy = f * dy, gz = f * dz;
        acc[0] += an;
        acc[1] -= dx * gx; acc[2] -= dx * gy; acc[3] -= dx * gz;
        acc[4] -= dy * gy; acc[5] -= dy * gz; acc[6] -= dz * gz;
        acc[7] -= gx; acc[8] -= gy; acc[9] -= gz;
    }
    block_sum<10>(acc, sh);
    if (threadIdx.x == 0) {
        const int a = P.metal_min + i;
        fx[a] += acc[7];
        fy[a] += acc[8];
        fz[a] += acc[9];
        double *out = partials + (size_t)i * 10;  // energy, virial[9]
        out[0] = 0.5 * P.qsc_eps * acc[0] - P.qsc_eps * P.qsc_c / isd_i;
        out[1] = 0.5 * acc[1];
        out[2] = out[4] = 0.5 * acc[2];
        out[3] = out[7] = 0.5 * acc[3];
        out[5] = 0.5 * acc[4];
        out[6] = out[8] = 0.5 * acc[5];
        out[9] = 0.5 * acc[6];
    }
}

void launch_qsc(capac_ctx *c)
{
    const unsigned grid = (unsigned)c->M;
    {
        ProfScope ps(c, K_QSC);
        k_qsc_density<<<grid, kQscBlock, 0, c->stream>>>(c->P, c->pos4, c->isd);
        k_qsc_force<<<grid, kQscBlock, 0, c->stream>>>(c->P, c->pos4, c->isd, c->fx, c->fy, c->fz,
                                                       force_partials(c, FP_QSC));
    }
    c->launches += 2;
    if (c->defer) {
        c->fs.qsc = force_partials(c, FP_QSC);
        c->fs.n_qsc = (int)grid;
        return;
    }
    static const int pot_slots[10] = {1, -1, -1, -1, -1, -1, -1, -1, -1, -1};
    static const int vir_slots[10] = {-1, 0, 1, 2, 3, 4, 5, 6, 7, 8};
    launch_finalize(c, (int)grid, 10, pot_slots, vir_slots);
}

// ------------------------------------------------------------ CPIM RHS

// mpi_cpff_vec_ext, cpff.c:43-198: field and potential of the permanent
// charges inside the cut-off at each metal atom, converted to atomic units,
// plus the uniform external field; NP total charges in the last rows.  A block
// per metal atom: a warp each left the chip idle up to a few hundred atoms.
constexpr int kRhsBlock = 128;
__global__ void __launch_bounds__(kRhsBlock) k_cpim_rhs(DevParams P, const double4 *__restrict__ pos4,
                                                  const uint32_t *__restrict__ nbr, const int *__restrict__ nnb,
                                                  int cap, double *vec_ext)
{
    __shared__ double sh[32 * 4];
    const int i = blockIdx.x;
    if (i == 0)
        for (int k = threadIdx.x; k < P.n_nps; k += kRhsBlock) vec_ext[4 * P.M + k] = P.np_charge[k];
    const int im = P.metal_min + i, n = nnb[im];
    const double4 pi = pos4[im];
    const bool shrt = P.w_alpha * P.rc < kDsfMaxX;
    double t[4] = {0.0, 0.0, 0.0, 0.0};  // field, potential
    const uint32_t *row = nbr + (size_t)im * cap;
    for (int k = threadIdx.x; k < n; k += kRhsBlock) {
        const int j = nb_index(row[k]);
        const double4 pj = pos4[j];
        if (pj.w == 0.0 || P.is_metal[j]) continue;
        double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        image(dx, dy, dz, P.box);
        const double r2 = norm2_exact(dx, dy, dz);
        if (r2 >= P.rc2) continue;
        double ef, vf;
        if (P.use_coulomb == 1) {
            const Dsf d = shrt ? dsf_terms(P.w_alpha, r2) : dsf_terms_any(P.w_alpha, r2);
            ef = kFQQ * pj.w * (fma(d.ec, d.rinv * d.rinv, P.w_a2_sqrtpi * d.eg * d.rinv) - P.w_const) * d.rinv;
            vf = kFQQ * pj.w * (fma(d.ec, d.rinv, -P.w_erfc_arcut) + P.w_const * (d.r - P.rc));
        } else {
            const double r = sqrt(r2);
            ef = kFQQ * pj.w / (r2 * r);
            vf = kFQQ * pj.w / r;
        }
        const double s = ef * kConvE;
        t[0] = fma(s, dx, t[0]);
        t[1] = fma(s, dy, t[1]);
        t[2] = fma(s, dz, t[2]);
        t[3] = fma(vf, kConvV, t[3]);
    }
    block_sum<4>(t, sh);
    if (threadIdx.x == 0) {
        vec_ext[3 * i + 0] = t[0] + P.efield[0] * kConvE;
        vec_ext[3 * i + 1] = t[1] + P.efield[1] * kConvE;
        vec_ext[3 * i + 2] = t[2] + P.efield[2] * kConvE;
        const double vext = P.efield[0] * pi.x + P.efield[1] * pi.y + P.efield[2] * pi.z;
        vec_ext[3 * P.M + i] = t[3] - vext * kConvV;
    }
}

void launch_cpim_rhs(capac_ctx *c)
{
    ProfScope ps(c, K_CPIM_RHS);
    k_cpim_rhs<<<c->M, kRhsBlock, 0, c->stream>>>(c->P, c->pos4, c->nbr, c->nnb, c->cap, c->vec_ext);
    ++c->launches;
}

// ------------------------------------------------------- CPIM matrix

// One thread per ordered pair (i, j); 16 coalesced plane writes.  The entries
// are computed in FP64 and stored as T (double on the FP64 path, float on the
// mixed path).
template <typename T>
__global__ void __launch_bounds__(128) k_cpim_matrix(DevParams P, const double4 *__restrict__ pos4, int Mp,
                                                     T *__restrict__ mat)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= Mp) return;
    double e[16];
    if (j < P.M) {
        cpim_block(P, pos4[P.metal_min + i], pos4[P.metal_min + j], i == j, e);
    } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) e[k] = 0.0;
    }
    T *base = mat + (size_t)i * 16 * Mp + j;
#pragma unroll
    for (int k = 0; k < 16; ++k) base[(size_t)k * Mp] = (T)e[k];
}

constexpr long kPrecondEvery = 10;
// the coarse correction (A Z, E^-1, W) is refreshed at every kCoarseEvery-th
// refresh of the inverse blocks: its group sums change more slowly than the
// blocks, and its inversion costs ~10 ms for 261 coarse columns
constexpr long kCoarseEvery = 5;

// Dense FP64 4x4 blocks of metal rows i0 .. i0 + rows - 1 against every metal
// column j: out[((i - i0) M + j) 16 + 4 r + c], the entries of cpim_block
// (the reference's |e| <= 1e-15 drop applied), diagonal blocks diag(1/polar
// x3, -1/capac).
__global__ void __launch_bounds__(128) k_cpim_block_rows(DevParams P, const double4 *__restrict__ pos4, int i0,
                                                         int rows, double *__restrict__ out)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= P.M || (int)blockIdx.y >= rows) return;
    const int i = i0 + (int)blockIdx.y;
    double e[16];
    cpim_block(P, pos4[P.metal_min + i], pos4[P.metal_min + j], i == j, e);
    double *o = out + ((size_t)blockIdx.y * P.M + j) * 16;
#pragma unroll
    for (int k = 0; k < 16; ++k) o[k] = e[k];
}

void launch_cpim_block_rows(capac_ctx *c, int i0, int rows, double *out)
{
    dim3 grid(grid_for(c->M, 128), rows);
    k_cpim_block_rows<<<grid, 128, 0, c->stream>>>(c->P, c->pos4, i0, rows, out);
    ++c->launches;
}

void launch_cpim_matrix(capac_ctx *c)
{
    if (c->msym) {
        // (the dense solver forms the mixed path's matrix from the positions
        // itself: the tiles then serve the coarse refreshes only, whose result it
        // does not use)
        const bool due = c->dinv && c->precond_age % kPrecondEvery == 0;
        const bool coarse = due && c->twolevel && (c->precond_age == 0 || c->coarse_age % kCoarseEvery == 0);
        if (!c->dense_ex || c->opt.precision != CAPAC_PREC_MIXED || coarse) launch_sym_assemble(c);
        // the preconditioner only steers the inner solves (the FP64 residual
        // defines the answer), so its inverse blocks are refreshed every
        // kPrecondEvery matrix builds, not every step
        if (c->dinv && c->precond_age++ % kPrecondEvery == 0) {
            launch_block_inverse(c);
            if (c->twolevel && c->precond_age <= 1) c->coarse_age = 0;  // fresh positions: fresh coarse part
            if (c->twolevel && c->coarse_age++ % kCoarseEvery == 0) launch_coarse_refresh(c);
            if (c->twolevel && !c->dense_ex) launch_coarse_kw(c);
        }
        return;
    }
    dim3 grid(grid_for(c->Mp, 128), c->M);
    ProfScope ps(c, K_MATRIX);
    if (c->matf)
        k_cpim_matrix<float><<<grid, 128, 0, c->stream>>>(c->P, c->pos4, c->Mp, c->matf);
    else
        k_cpim_matrix<double><<<grid, 128, 0, c->stream>>>(c->P, c->pos4, c->Mp, c->mat);
    ++c->launches;
}

// ------------------------------------------------------------ SpMV

// y = A x for the CPIM system, one block per row block (metal atom) plus one
// block per Lagrange row.  Epilogue: per-block dot partials
//   DOT_R0:  (r0, y)            -> partials[b*2]
//   DOT_KT:  Kt = K y; (Kt, z), (Kt, Kt) -> partials[b*2], partials[b*2+1]
enum { DOT_NONE = 0, DOT_R0 = 1, DOT_KT = 2 };

// T: stored entry type (double, or float on the mixed path; accumulation is
// FP64 either way).  FREE: no stored matrix, every block is recomputed in FP64
// from the positions (the FP64 residual of the mixed path's refinement).
template <int DOT, typename T, bool FREE>
__global__ void __launch_bounds__(256) k_spmv(DevParams P, int Mp, const T *__restrict__ mat,
                                              const double4 *__restrict__ pos4,
                                              const double *__restrict__ x, double *__restrict__ y,
                                              const double *__restrict__ d1, const double *__restrict__ d2,
                                              double *__restrict__ partials, const SolverScalars *ss)
{
    __shared__ double sh[32 * 4];
    if (ss && ss->done) return;
    const int M = P.M;
    const int b = blockIdx.x;
    if (b < M) {
        const T *row = FREE ? nullptr : mat + (size_t)b * 16 * Mp;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        double4 pb = FREE ? pos4[P.metal_min + b] : make_double4(0, 0, 0, 0);
        for (int j = threadIdx.x; j < M; j += blockDim.x) {
            const double xv[4] = {x[3 * j], x[3 * j + 1], x[3 * j + 2], x[3 * M + j]};
            if (FREE) {
                double e[16];
                cpim_block(P, pb, pos4[P.metal_min + j], j == b, e);
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) acc[r] += e[4 * r + cc] * xv[cc];
            } else {
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) acc[r] += (double)row[(size_t)(4 * r + cc) * Mp + j] * xv[cc];
            }
        }
        block_sum<4>(acc, sh);
        if (threadIdx.x == 0) {
            const int im = P.metal_min + b;
            for (int k = 0; k < P.n_nps; ++k)
                if (im >= P.np_start[k] && im <= P.np_end[k]) acc[3] += x[4 * M + k];
            const int rows[4] = {3 * b, 3 * b + 1, 3 * b + 2, 3 * M + b};
            double p0 = 0.0, p1 = 0.0;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                y[rows[r]] = acc[r];
                if (DOT == DOT_R0) p0 += d1[rows[r]] * acc[r];
                if (DOT == DOT_KT) {
                    const double kt = d2[rows[r]] * acc[r];
                    p0 += kt * d1[rows[r]];
                    p1 += kt * kt;
                }
            }
            if (DOT != DOT_NONE) {
                partials[2 * b] = p0;
                partials[2 * b + 1] = p1;
            }
        }
    } else {
        const int k = b - M;
        double acc[1] = {0.0};
        for (int a = P.np_start[k] + threadIdx.x; a <= P.np_end[k]; a += blockDim.x)
            acc[0] += x[3 * M + (a - P.metal_min)];
        block_sum<1>(acc, sh);
        if (threadIdx.x == 0) {
            const int rowi = 4 * M + k;
            y[rowi] = acc[0];
            if (DOT == DOT_R0) partials[2 * b] = d1[rowi] * acc[0], partials[2 * b + 1] = 0.0;
            if (DOT == DOT_KT) {
                const double kt = acc[0];  // K = 1 on Lagrange rows
                partials[2 * b] = kt * d1[rowi];
                partials[2 * b + 1] = kt * kt;
            }
        }
    }
}

// ------------------------------------------------------------ BiCGSTAB

// Work vector slots inside bw (bicg_stab.c:280-290).
enum { W_AX = 0, W_R0, W_R, W_P, W_V, W_S, W_T, W_Y, W_Z, W_KT, W_K };

// Fixed-order sum of `nb` two-wide partials into out[0..1] (single block).
__device__ __forceinline__ void sum_partials2(const double *partials, int nb, double *sh, double &s0, double &s1)
{
    double v[2] = {0.0, 0.0};
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        v[0] += partials[2 * b];
        v[1] += partials[2 * b + 1];
    }
    block_sum<2>(v, sh);
    s0 = v[0];
    s1 = v[1];
}

__global__ void __launch_bounds__(256) k_vec_dot(int n, const double *__restrict__ a, const double *__restrict__ b,
                                                 double *partials)
{
    __shared__ double sh[64];
    double v[2] = {0.0, 0.0};
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) v[0] = a[k] * b[k];
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = v[0];
        partials[2 * blockIdx.x + 1] = 0.0;
    }
}

// bTb, early exit and criterion (bicg_stab.c:296-303).  `skip` is the
// absolute threshold of the reference's two early exits (bTb < 1e-10 and, on
// the first iteration, rho < 1e-10); refinement sweeps, whose right-hand
// sides are small residuals, pass a threshold that only catches exact zero.
__global__ void k_bcg_start(const double *partials, int nb, double tol, double skip, int max_iter,
                            SolverScalars *ss)
{
    __shared__ double sh[64];
    double s0, s1;
    sum_partials2(partials, nb, sh, s0, s1);
    if (threadIdx.x == 0) {
        ss->bTb = s0;
        ss->crit = s0 * tol;
        ss->rho_old = ss->alpha = ss->omega = 1.0;
        ss->iter = 0;
        ss->status = 0;
        ss->skip = skip;
        ss->max_iter = max_iter;
        ss->done = s0 < skip ? 1 : 0;
        ss->rTr = 0.0;
    }
}

// r0 = r = b - Ax, p = v = 0, K = 1/diag (1 on Lagrange rows); (r0, r) partials.
__global__ void __launch_bounds__(256) k_bcg_init(int n, int n4, const double *__restrict__ b,
                                                  const double *__restrict__ diag, double *bw, double *partials,
                                                  const SolverScalars *ss)
{
    __shared__ double sh[64];
    if (ss->done) return;
    double v[2] = {0.0, 0.0};
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) {
        const double r = b[k] - bw[W_AX * n + k];
        bw[W_R0 * n + k] = r;
        bw[W_R * n + k] = r;
        bw[W_V * n + k] = 0.0;
        bw[W_P * n + k] = 0.0;
        bw[W_K * n + k] = k < n4 ? 1.0 / diag[k] : 1.0;
        v[0] = r * r;
    }
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = v[0];
        partials[2 * blockIdx.x + 1] = 0.0;
    }
}

__global__ void k_bcg_rho0(const double *partials, int nb, SolverScalars *ss)
{
    __shared__ double sh[64];
    if (ss->done) return;
    double s0, s1;
    sum_partials2(partials, nb, sh, s0, s1);
    if (threadIdx.x == 0) {
        ss->rho = s0;  // (r0, r) with r = r0
        ss->rTr = s0;
        ss->rr0 = s0;
    }
}

// p = r + beta (p - omega v), y = K p (bicg_stab.c:371-404); the iteration-0
// early exit on rho < 1e-10 (bicg_stab.c:368).
__global__ void __launch_bounds__(256) k_bcg_p(int n, double *bw, SolverScalars *ss)
{
    if (ss->done) return;
    if (ss->iter == 0 && ss->rho < ss->skip) {
        if (blockIdx.x == 0 && threadIdx.x == 0) ss->done = 1;
        return;
    }
    const double beta = (ss->rho / ss->rho_old) * (ss->alpha / ss->omega), om = ss->omega;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double p = bw[W_R * n + k] + beta * (bw[W_P * n + k] - om * bw[W_V * n + k]);
    bw[W_P * n + k] = p;
    bw[W_Y * n + k] = p * bw[W_K * n + k];
}

// Status when BiCGSTAB breaks down (a zero or non-finite alpha or omega, which
// the reference does not guard against and which it would carry into NaN):
// the iterate stays at the last finite x.  Accepted like the reference's
// MAX_ITER fallback when rTr < 100 crit (status 1), otherwise an error (-1).
// rTr of iteration 0 is the initial residual, stored by k_bcg_rho0.
__device__ __forceinline__ int breakdown_status(const SolverScalars *ss)
{
    return ss->rTr < ss->crit * 100.0 ? 1 : -2;  // -2: restartable breakdown
}

__global__ void k_bcg_alpha(const double *partials, int nb, SolverScalars *ss)
{
    __shared__ double sh[64];
    if (ss->done) return;
    double s0, s1;
    sum_partials2(partials, nb, sh, s0, s1);
    if (threadIdx.x == 0) {
        const double a = ss->rho / s0;
        if (isfinite(a)) {
            ss->alpha = a;
        } else {  // breakdown: keep x as it is and judge the last residual
            ss->done = 1;
            ss->status = breakdown_status(ss);
        }
    }
}

// s = r - alpha v, z = K s (bicg_stab.c:418-449).
__global__ void __launch_bounds__(256) k_bcg_s(int n, double *bw, const SolverScalars *ss)
{
    if (ss->done) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double s = bw[W_R * n + k] - ss->alpha * bw[W_V * n + k];
    bw[W_S * n + k] = s;
    bw[W_Z * n + k] = s * bw[W_K * n + k];
}

__global__ void k_bcg_omega(const double *partials, int nb, SolverScalars *ss)
{
    __shared__ double sh[64];
    if (ss->done) return;
    double s0, s1;
    sum_partials2(partials, nb, sh, s0, s1);
    if (threadIdx.x == 0) {
        const double w = s0 / s1;
        if (isfinite(w) && w != 0.0) {
            ss->omega = w;
        } else {  // breakdown before x is touched
            ss->done = 1;
            ss->status = breakdown_status(ss);
        }
    }
}

// x += alpha y + omega z, r = s - omega t; (r, r) and (r0, r) partials
// (bicg_stab.c:490-529).
__global__ void __launch_bounds__(256) k_bcg_x(int n, double *bw, double *x, double *partials,
                                               const SolverScalars *ss)
{
    __shared__ double sh[64];
    if (ss->done) return;
    double v[2] = {0.0, 0.0};
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) {
        x[k] += ss->alpha * bw[W_Y * n + k] + ss->omega * bw[W_Z * n + k];
        const double r = bw[W_S * n + k] - ss->omega * bw[W_T * n + k];
        bw[W_R * n + k] = r;
        v[0] = r * r;
        v[1] = bw[W_R0 * n + k] * r;
    }
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = v[0];
        partials[2 * blockIdx.x + 1] = v[1];
    }
}

// Convergence test and MAX_ITER handling (bicg_stab.c:523-571).
__global__ void k_bcg_check(const double *partials, int nb, SolverScalars *ss)
{
    __shared__ double sh[64];
    if (ss->done) return;
    double rTr, r0r;
    sum_partials2(partials, nb, sh, rTr, r0r);
    if (threadIdx.x == 0) {
        ss->rho_old = ss->rho;
        ss->rho = r0r;
        ss->rTr = rTr;
        ss->iter += 1;
        if (rTr < ss->crit) {
            ss->done = 1;
        } else if (ss->iter > ss->max_iter) {
            ss->done = 1;
            ss->status = rTr < ss->crit * 100.0 ? 1 : -1;  // 1: loosened criterion accepted
        }
    }
}

namespace {

void spmv(capac_ctx *c, int dot, const double *x, double *y, const double *d1, const double *d2,
          const SolverScalars *ss)
{
    if (c->msym) {
        launch_sym_spmv(c, dot, x, y, d1, d2, ss);
        return;
    }
    const int nb = c->M + c->n_nps;
    ProfScope ps(c, K_SPMV);
    cudaStream_t s = c->stream;
    if (c->matf) {
        if (dot == DOT_R0)
            k_spmv<DOT_R0, float, false><<<nb, 256, 0, s>>>(c->P, c->Mp, c->matf, c->pos4, x, y, d1, d2, c->partials, ss);
        else if (dot == DOT_KT)
            k_spmv<DOT_KT, float, false><<<nb, 256, 0, s>>>(c->P, c->Mp, c->matf, c->pos4, x, y, d1, d2, c->partials, ss);
        else
            k_spmv<DOT_NONE, float, false><<<nb, 256, 0, s>>>(c->P, c->Mp, c->matf, c->pos4, x, y, d1, d2, c->partials,
                                                              ss);
    } else {
        if (dot == DOT_R0)
            k_spmv<DOT_R0, double, false><<<nb, 256, 0, s>>>(c->P, c->Mp, c->mat, c->pos4, x, y, d1, d2, c->partials, ss);
        else if (dot == DOT_KT)
            k_spmv<DOT_KT, double, false><<<nb, 256, 0, s>>>(c->P, c->Mp, c->mat, c->pos4, x, y, d1, d2, c->partials, ss);
        else
            k_spmv<DOT_NONE, double, false><<<nb, 256, 0, s>>>(c->P, c->Mp, c->mat, c->pos4, x, y, d1, d2,
                                                               c->partials, ss);
    }
    ++c->launches;
}

}  // namespace

void launch_cpim_spmv(capac_ctx *c, const double *x, double *y)
{
    // the grouped solver's tiles are in its own atom order: the product in
    // the reference layout comes from the blocks rebuilt in FP64
    if (c->grouped) {
        spmv_free(c, x, y);
        return;
    }
    spmv(c, DOT_NONE, x, y, nullptr, nullptr, nullptr);
}

// y = A x with every block recomputed in FP64 from the positions.
void spmv_free(capac_ctx *c, const double *x, double *y)
{
    if (c->sympart) {  // symmetric tiles: every unordered pair once
        launch_sym_spmv_free(c, x, y);
        return;
    }
    const int nb = c->M + c->n_nps;
    ProfScope ps(c, K_RESID);
    k_spmv<DOT_NONE, double, true><<<nb, 256, 0, c->stream>>>(c->P, c->Mp, nullptr, c->pos4, x, y, nullptr, nullptr,
                                                              c->partials, nullptr);
    ++c->launches;
}

// r = b - Ax; partials of (r, r).
__global__ void __launch_bounds__(256) k_residual(int n, const double *__restrict__ b, const double *__restrict__ Ax,
                                                  double *__restrict__ r, double *partials)
{
    __shared__ double sh[64];
    double v[2] = {0.0, 0.0};
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) {
        const double rk = b[k] - Ax[k];
        r[k] = rk;
        v[0] = rk * rk;
    }
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = v[0];
        partials[2 * blockIdx.x + 1] = 0.0;
    }
}

__global__ void k_residual_final(const double *partials, int nb, SolverScalars *ss)
{
    __shared__ double sh[64];
    double s0, s1;
    sum_partials2(partials, nb, sh, s0, s1);
    if (threadIdx.x == 0) ss->res0 = s0;
}

__global__ void __launch_bounds__(256) k_axpy1(int n, const double *__restrict__ d, double *__restrict__ x)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) x[k] += d[k];
}

// Warm-start predictor: polynomial extrapolation of the last solutions.
// x is the last solution x_n, hist holds x_{n-1}, x_{n-2}, x_{n-3} (n each);
// order 1: 2 x_n - x_{n-1}; 2: 3 x_n - 3 x_{n-1} + x_{n-2};
// 3: 4 x_n - 6 x_{n-1} + 4 x_{n-2} - x_{n-3}; 0 or less only records x_n.
__global__ void __launch_bounds__(256) k_predict(int n, int order, double *__restrict__ x, double *__restrict__ hist)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double t = x[k], h1 = hist[k], h2 = hist[n + k], h3 = hist[2 * (size_t)n + k];
    if (order == 1) x[k] = 2.0 * t - h1;
    else if (order == 2) x[k] = 3.0 * (t - h1) + h2;
    else if (order == 3) x[k] = 4.0 * (t + h2) - 6.0 * h1 - h3;
    hist[2 * (size_t)n + k] = h2;
    hist[n + k] = h1;
    hist[k] = t;
}

// Jacobi-preconditioned BiCGSTAB (bicg_stab.c:253-573) on A x = b with the
// stored matrix (FP64, or FP32 on the mixed path), x warm-started.  The host
// polls the done flag every few iterations.  Returns the status; the solver
// scalars are left in c->h_ss.
int bicgstab_core(capac_ctx *c, const double *b, double *x, double tol, double skip)
{
    if (c->coop_grid > 0) return bicgstab_coop(c, b, x, tol, skip);
    const int n = c->n_mat, n4 = 4 * c->M;
    const int nbv = (int)grid_for(n, 256);
    const int nbm = c->msym ? sym_reduce_blocks(c) : c->M + c->n_nps;  // blocks writing SpMV dot partials
    cudaStream_t s = c->stream;
    double *bw = c->bw;
    auto W = [&](int k) { return bw + (size_t)k * n; };

    k_vec_dot<<<nbv, 256, 0, s>>>(n, b, b, c->partials);
    k_bcg_start<<<1, 256, 0, s>>>(c->partials, nbv, tol, skip, solver_max_iter(c), c->ss);
    spmv(c, DOT_NONE, x, W(W_AX), nullptr, nullptr, c->ss);
    k_bcg_init<<<nbv, 256, 0, s>>>(n, n4, b, c->diag, bw, c->partials, c->ss);
    k_bcg_rho0<<<1, 256, 0, s>>>(c->partials, nbv, c->ss);
    c->launches += 4;

    const int chunk = 4;
    // One chunk of iterations; every kernel returns at once after convergence.
    auto issue_chunk = [&]() {
        for (int q = 0; q < chunk; ++q) {
            {
                ProfScope ps(c, K_SOLVER_VEC);
                k_bcg_p<<<nbv, 256, 0, s>>>(n, bw, c->ss);
            }
            spmv(c, DOT_R0, W(W_Y), W(W_V), W(W_R0), nullptr, c->ss);
            {
                ProfScope ps(c, K_SOLVER_VEC);
                k_bcg_alpha<<<1, 256, 0, s>>>(c->partials, nbm, c->ss);
                k_bcg_s<<<nbv, 256, 0, s>>>(n, bw, c->ss);
            }
            spmv(c, DOT_KT, W(W_Z), W(W_T), W(W_Z), W(W_K), c->ss);
            {
                ProfScope ps(c, K_SOLVER_VEC);
                k_bcg_omega<<<1, 256, 0, s>>>(c->partials, nbm, c->ss);
                k_bcg_x<<<nbv, 256, 0, s>>>(n, bw, x, c->partials, c->ss);
                k_bcg_check<<<1, 256, 0, s>>>(c->partials, nbv, c->ss);
            }
            c->launches += 6;
        }
    };
    // The chunk only touches buffers fixed for the context's lifetime, so it
    // is captured once per (b, x, profiling) and replayed as a CUDA graph.
    SolveGraph *g = nullptr;
    if (c->use_graphs) {
        for (auto &sg : c->graphs)
            if (sg.b == b && sg.x == x && sg.prof == c->prof.on) g = &sg;
        if (!g) {
            c->graphs.emplace_back();
            g = &c->graphs.back();
            g->b = b;
            g->x = x;
            g->prof = c->prof.on;
            const long l0 = c->launches;
            cudaGraph_t graph;
            CAPAC_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            c->capturing = g;
            issue_chunk();
            c->capturing = nullptr;
            CAPAC_CUDA(cudaStreamEndCapture(s, &graph));
            CAPAC_CUDA(cudaGraphInstantiate(&g->exec, graph, 0));
            CAPAC_CUDA(cudaGraphDestroy(graph));
            g->kernels = c->launches - l0;
            c->launches = l0;
        }
    }
    for (int it = 0; it <= solver_max_iter(c) + chunk; it += chunk) {
        if (g) {
            CAPAC_CUDA(cudaGraphLaunch(g->exec, s));
            c->launches += g->kernels;
        } else {
            issue_chunk();
        }
        CAPAC_CUDA(cudaMemcpyAsync(c->h_ss, c->ss, sizeof(SolverScalars), cudaMemcpyDeviceToHost, s));
        CAPAC_CUDA(cudaStreamSynchronize(s));
        if (g) prof_graph_replayed(c, *g);
        if (c->h_ss->done) break;
    }
    if (c->prof.on && c->h_ss->bTb >= skip) c->prof.spmv_effective += 1 + 2L * c->h_ss->iter;
    if (!c->h_ss->done || c->h_ss->status < 0) return CAPAC_ERR_NOT_CONVERGED;
    return c->h_ss->status == 1 ? 1 : CAPAC_OK;
}

// The reference's solve: rTr < tol * bTb with its early exits.
int run_bicgstab(capac_ctx *c, bool defer)
{
    const double tol = c->opt.solver_tol > 0.0 ? c->opt.solver_tol : 1.0e-8;
    if (c->dense_ex) {  // one launch, with the restarts after a breakdown
        bicgstab_dense(c, c->vec_ext, c->vec_pq, tol, 1.0e-10, nullptr, 0, true);
        c->pending_solve = true;
        if (defer) return CAPAC_OK;
        CAPAC_CUDA(cudaStreamSynchronize(c->stream));
        return settle_solve(c);
    }
    int st = bicgstab_core(c, c->vec_ext, c->vec_pq, tol, 1.0e-10);
    int iters = c->h_ss->iter, starts = 1;
    // A breakdown (zero or non-finite alpha/omega) leaves x at its last finite
    // value; restart from there with a fresh shadow residual, as is standard
    // for BiCGSTAB (the reference would carry the NaN to MAX_ITER and exit).
    while (c->h_ss->status == -2 && starts < 8) {
        // not the reference's first iteration: only an exact zero ends it early
        st = bicgstab_core(c, c->vec_ext, c->vec_pq, tol, 1.0e-300);
        iters += c->h_ss->iter;
        ++starts;
    }
    c->last_iters = iters;
    c->last_outer = starts;
    c->last_rel_res = c->h_ss->bTb > 0 ? sqrt(c->h_ss->rTr / c->h_ss->bTb) : 0.0;
    c->last_init_res = c->h_ss->bTb > 0 ? sqrt(c->h_ss->rr0 / c->h_ss->bTb) : 0.0;
    if (st == 1) fprintf(stderr, "Note: Loosen bicg_stab convergence criteria to 1e-6 for this step.\n");
    return st < 0 ? st : CAPAC_OK;
}

// Mixed path: FP64 iterative refinement.  Each sweep recomputes the residual
// r = b - A x in FP64 (matrix-free: every block rebuilt from the positions in
// FP64, so no FP64 matrix is stored), solves A d = r with BiCGSTAB on the FP32
// matrix (FP64 vectors, inner products and accumulation) to a relative
// residual of 1e-5 (on the last sweep only as far as the target needs), and
// updates x += d, until |r| <= refine_tol |b|.  The reference's zero-field
// early exit (bTb < 1e-10) is kept.
constexpr double kInnerReduction = 1.0e-5;
// an inner solve whose (r, r) has not halved for this many iterations stops
// and returns its iterate to the refinement
constexpr int kInnerStall = 60;
// The status of a refinement that ended at (r, r) = rr, short of its target or not.
static int refined_status(bool missed, double rr, double bTb)
{
    if (!missed) return CAPAC_OK;
    if (rr < 1.0e-8 * bTb) {  // the reference's own criterion still holds
        fprintf(stderr, "Note: refinement stopped at relative residual %.3e\n", sqrt(rr / bTb));
        return CAPAC_OK;
    }
    return CAPAC_ERR_NOT_CONVERGED;
}

// The status and statistics of a dense solve whose scalars have landed in h_ss.
int settle_solve(capac_ctx *c)
{
    if (!c->pending_solve) return CAPAC_OK;
    c->pending_solve = false;
    const bool mixed = c->opt.precision == CAPAC_PREC_MIXED;
    const int st = dense_status(c, 1.0e-10);
    const SolverScalars &S = *c->h_ss;
    if (!mixed) {
        c->last_iters = S.iter;
        c->last_outer = std::max(1, S.outer);
        c->last_rel_res = S.bTb > 0 ? sqrt(S.rTr / S.bTb) : 0.0;
        c->last_init_res = S.bTb > 0 ? sqrt(S.rr0 / S.bTb) : 0.0;
        if (st == 1) fprintf(stderr, "Note: Loosen bicg_stab convergence criteria to 1e-6 for this step.\n");
        return st < 0 ? st : CAPAC_OK;
    }
    c->last_iters = c->last_outer = 0;
    c->last_rel_res = 0.0;
    if (S.bTb < 1.0e-10) return CAPAC_OK;  // zero right-hand side: keep x
    ++c->n_solves;
    c->last_iters = S.iter;
    c->last_outer = S.outer;
    c->last_init_res = sqrt(S.rr0 / S.bTb);
    c->last_rel_res = sqrt(S.rTr / S.bTb);
    return refined_status(st < 0 || !(S.rTr <= c->pending_tol * S.bTb), S.rTr, S.bTb);
}

int run_refined_solve(capac_ctx *c, bool defer)
{
    const int n = c->n_mat;
    const int nbv = (int)grid_for(n, 256);
    cudaStream_t s = c->stream;
    const double rtol = c->opt.refine_tol > 0.0 ? c->opt.refine_tol : 1.0e-10;
    const int max_sweeps = 12;

    if (c->dense_ex) {  // small systems: predictor, solve and residual in one launch
        const bool hist = c->opt.predictor > 0 && c->xprev;
        bicgstab_dense(c, c->vec_ext, c->vec_pq, rtol * rtol, 1.0e-10, hist ? c->xprev : nullptr,
                       std::min(c->opt.predictor, c->n_solves - 1), true);
        c->pending_solve = true;
        c->pending_tol = rtol * rtol;
        if (defer) return CAPAC_OK;
        CAPAC_CUDA(cudaStreamSynchronize(s));
        return settle_solve(c);
    }
    k_vec_dot<<<nbv, 256, 0, s>>>(n, c->vec_ext, c->vec_ext, c->partials);
    k_bcg_start<<<1, 256, 0, s>>>(c->partials, nbv, 1.0, 1.0e-10, solver_max_iter(c), c->ss);
    c->launches += 2;
    CAPAC_CUDA(cudaMemcpyAsync(c->h_ss, c->ss, sizeof(SolverScalars), cudaMemcpyDeviceToHost, s));
    CAPAC_CUDA(cudaStreamSynchronize(s));
    c->last_iters = 0;
    c->last_outer = 0;
    c->last_rel_res = 0.0;
    if (c->h_ss->done) return CAPAC_OK;  // zero right-hand side: keep x
    const double bTb = c->h_ss->bTb;
    if (c->opt.predictor > 0 && c->xprev) {
        // the warm start of the first solve is not a solution: history
        // entries count from the second solve on
        k_predict<<<nbv, 256, 0, s>>>(n, std::min(c->opt.predictor, c->n_solves - 1), c->vec_pq, c->xprev);
        ++c->launches;
    }
    ++c->n_solves;
    double rr = 0.0;
    int total = 0, sweep = 0;
    for (;; ++sweep) {
        spmv_free(c, c->vec_pq, c->bw + (size_t)W_AX * n);
        k_residual<<<nbv, 256, 0, s>>>(n, c->vec_ext, c->bw + (size_t)W_AX * n, c->rres, c->partials);
        k_residual_final<<<1, 256, 0, s>>>(c->partials, nbv, c->ss);
        c->launches += 2;
        CAPAC_CUDA(cudaMemcpyAsync(c->h_ss, c->ss, sizeof(SolverScalars), cudaMemcpyDeviceToHost, s));
        CAPAC_CUDA(cudaStreamSynchronize(s));
        rr = c->h_ss->res0;
        if (sweep == 0) c->last_init_res = sqrt(rr / bTb);
        if (rr <= rtol * rtol * bTb || sweep == max_sweeps) break;
        CAPAC_CUDA(cudaMemsetAsync(c->dcorr, 0, sizeof(double) * n, s));
        // reduce the residual by 1e-5, or, on the last sweep, by what is
        // left to the target with a margin of 3
        const double need = 0.3 * rtol * sqrt(bTb / rr);
        const double tau = std::min(std::max(need, kInnerReduction), 0.1);
        struct StallGuard {  // the guard applies to this inner solve only
            capac_ctx *c;
            ~StallGuard() { c->inner_stall = 0; }
        } guard{c};
        c->inner_stall = kInnerStall;
        const int st = bicgstab_core(c, c->rres, c->dcorr, tau * tau, 1.0e-300);
        c->inner_stall = 0;
        total += c->h_ss->iter;
        if (st == 1 && c->h_ss->rTr >= c->h_ss->crit) ++c->inner_stalls;
        if (st < 0 && c->h_ss->iter == 0) break;  // no progress possible
        k_axpy1<<<nbv, 256, 0, s>>>(n, c->dcorr, c->vec_pq);
        ++c->launches;
    }
    c->last_iters = total;
    c->last_outer = sweep;
    c->last_rel_res = sqrt(rr / bTb);
    return refined_status(!(rr <= rtol * rtol * bTb), rr, bTb);
}

// ------------------------------------------------- CPIM metal-side forces

// One metal-metal pair of mpi_cpff_force (cpff.c:752-926) in the arithmetic
// type R, atomic units, r = r_j - r_i in Bohr: f is the pair force the
// reference subtracts from atom i, e the halves of the charge-charge,
// charge-dipole and dipole-dipole energies (each pair is visited from both
// atoms).
template <typename R>
__device__ __forceinline__ void metal_pair(const R r[3], R qi, const R pi[3], R qj, const R pj[3], R iqq, R ipq,
                                           R ipp, R f[3], R e[3])
{
    const R isp = (R)kInvSqrtPi, fq2 = (R)kFqqAu2, fq1 = (R)kFqqAu1, half = (R)0.5;
    const R ipq3 = ipq * ipq * ipq, ipp3 = ipp * ipp * ipp, ipp5 = ipp3 * ipp * ipp;
    const R r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2], rr = sqrt(r2);
    const R ir3 = (R)1 / (r2 * rr), ir5 = ir3 / r2, ir7 = ir5 / r2;
    f[0] = f[1] = f[2] = (R)0;
    e[0] = e[1] = e[2] = (R)0;
    // the tensors T1_ab, T2_abc contracted with the dipoles by hand: p . r and
    // pi . pj stand for the sums over their indices
    const R dpi = pi[0] * r[0] + pi[1] * r[1] + pi[2] * r[2], dpj = pj[0] * r[0] + pj[1] * r[1] + pj[2] * r[2];
    const R dpp = pi[0] * pj[0] + pi[1] * pj[1] + pi[2] * pj[2];
    // charge - charge
    const R gqq = exp(-(r2 * iqq * iqq)), erq = erf(rr * iqq);
    const R A0 = ir3 * (erq - (R)2 * isp * iqq * rr * gqq);
    R along = A0 * fq2 * qi * qj;
    e[0] += fq1 * qi * qj * erq / rr * half;
    // charge - dipole: T_ab = A1 (3 r_a r_b - d_ab r^2) - B1 r_a r_b
    const R gpq = exp(-(r2 * ipq * ipq));
    const R tpq = erf(rr * ipq) - (R)2 * isp * ipq * rr * gpq;
    const R Apq0 = ir3 * tpq, A1 = ir5 * tpq, B1 = (R)4 * isp * ipq3 / r2 * gpq;
    const R mix = qj * dpi - qi * dpj;
    along += fq2 * ((R)3 * A1 - B1) * mix;
    R ci = -fq2 * A1 * r2 * qj, cj = fq2 * A1 * r2 * qi;  // coefficients of pi and pj
    e[1] += fq1 * mix * Apq0 * half;
    // dipole - dipole: T_abc = A2 (5 r_a r_b r_c - r^2 (r_a d_bc + r_b d_ca + r_c d_ab)) - B2 r_a r_b r_c
    const R gpp = exp(-(r2 * ipp * ipp)), erp = erf(rr * ipp);
    const R App1 = ir5 * (erp - (R)2 * isp * ipp * rr * gpp);
    const R Bpp1 = (R)4 * isp * ipp3 / r2 * gpp;
    const R A2 = ir7 * ((R)3 * erp - (R)6 * isp * ipp * rr * gpp - (R)4 * (r2 * rr) * isp * ipp3 * gpp);
    const R B2 = (R)8 * isp * ipp5 / r2 * gpp;
    along -= fq2 * (((R)5 * A2 - B2) * dpi * dpj - A2 * r2 * dpp);
    ci += fq2 * A2 * r2 * dpj;
    cj += fq2 * A2 * r2 * dpi;
#pragma unroll
    for (int a = 0; a < 3; ++a) f[a] = along * r[a] + ci * pi[a] + cj * pj[a];
    e[2] -= fq1 * half * (((R)3 * dpi * dpj - r2 * dpp) * App1 - dpi * dpj * Bpp1);
}

// mpi_cpff_force (cpff.c:526-950) for one metal atom per block: metal -
// permanent-charge terms over its list, self terms, dense metal - metal
// damped T0/T1/T2 terms (forces on i only, virial halved), external field on
// the induced charge and dipole.  Energies [9..14] and the virial go to
// per-block partials.  The metal-metal pair terms are evaluated in R (FP32
// on the mixed path, FP64 otherwise); every sum is FP64.
template <typename R>
__global__ void __launch_bounds__(256) k_cpim_metal(DevParams P, const double4 *__restrict__ pos4,
                                                    const uint32_t *__restrict__ nbr, const int *__restrict__ nnb,
                                                    int cap, const double *__restrict__ pq, double *fx, double *fy,
                                                    double *fz, double *partials)
{
    __shared__ double sh[32 * 18];
    const int i = blockIdx.x;
    const int M = P.M;
    const int im = P.metal_min + i;
    const double4 pi4 = pos4[im];
    const double qi = pq[3 * M + i];
    const double pi[3] = {pq[3 * i], pq[3 * i + 1], pq[3 * i + 2]};
    // acc: f[3], e9..e14 (6), vir[9]
    double acc[18];
#pragma unroll
    for (int k = 0; k < 18; ++k) acc[k] = 0.0;

    // metal - permanent charge, MD units (cpff.c:578-724)
    const uint32_t *row = nbr + (size_t)im * cap;
    const bool shrt = P.use_coulomb == 1 && P.w_alpha * P.rc < kDsfMaxX;
    for (int k = threadIdx.x, n = nnb[im]; k < n; k += blockDim.x) {
        const int j = nb_index(row[k]);
        const double4 pj = pos4[j];
        if (pj.w == 0.0 || P.is_metal[j]) continue;
        double r[3] = {pi4.x - pj.x, pi4.y - pj.y, pi4.z - pj.z};
        image(r[0], r[1], r[2], P.box);
        const double r2 = norm2_exact(r[0], r[1], r[2]);
        if (r2 >= P.rc2) continue;
        double f[3], a0, v;
        if (shrt) {
            const Dsf d = cpim_charge_pair_dsf(P, r, r2, pj.w, qi, pi, f, a0);
            v = fma(d.ec, d.rinv, -P.w_erfc_arcut) + P.w_const * (d.r - P.rc);
        } else {
            double ec;
            cpim_charge_pair(P, r, r2, pj.w, qi, pi, f, a0, ec);
            const double rr = sqrt(r2);
            v = P.use_coulomb == 1 ? ec / rr - P.w_erfc_arcut + P.w_const * (rr - P.rc) : 1.0 / rr;
        }
        acc[4] += kFQQ * pj.w * qi * v;
        acc[5] -= kFQQ / kNm2Bohr * pj.w * a0 * (pi[0] * r[0] + pi[1] * r[1] + pi[2] * r[2]);
        acc[0] += f[0];
        acc[1] += f[1];
        acc[2] += f[2];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) acc[9 + 3 * a + b] += -r[a] * f[b];
    }

    // metal - metal, atomic units (cpff.c:752-926); the pair terms in R,
    // their sums in FP64
    const R iqq = (R)P.inv_r_qq, ipq = (R)P.inv_r_pq, ipp = (R)P.inv_r_pp;
    const R qiR = (R)qi, piR[3] = {(R)pi[0], (R)pi[1], (R)pi[2]};
    for (int j = threadIdx.x; j < M; j += blockDim.x) {
        if (j == i) continue;
        const double4 pj4 = pos4[P.metal_min + j];
        double rd[3] = {pj4.x - pi4.x, pj4.y - pi4.y, pj4.z - pi4.z};
        image(rd[0], rd[1], rd[2], P.box);
        const R r[3] = {(R)(rd[0] * kNm2Bohr), (R)(rd[1] * kNm2Bohr), (R)(rd[2] * kNm2Bohr)};
        const R qj = (R)pq[3 * M + j];
        const R pj[3] = {(R)pq[3 * j], (R)pq[3 * j + 1], (R)pq[3 * j + 2]};
        R f[3], e[3];
        metal_pair<R>(r, qiR, piR, qj, pj, iqq, ipq, ipp, f, e);
        acc[6] += (double)e[0];
        acc[7] += (double)e[1];
        acc[8] += (double)e[2];
        acc[0] -= (double)f[0];
        acc[1] -= (double)f[1];
        acc[2] -= (double)f[2];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) acc[9 + 3 * a + b] += -(double)r[a] * (double)f[b] * 0.5;
    }
    block_sum<18>(acc, sh);
    if (threadIdx.x == 0) {
        // self terms (cpff.c:729-742)
        acc[6] += 0.5 * kFQQ * qi * qi * (P.inv_capac * kNm2Bohr);
        for (int a = 0; a < 3; ++a) acc[8] += 0.5 * kFQQ * pi[a] * pi[a] * (P.inv_polar * kNm2Bohr);
        // external field on the induced charge and dipole (cpff.c:930-948)
        acc[0] += P.efield[0] * qi;
        acc[1] += P.efield[1] * qi;
        acc[2] += P.efield[2] * qi;
        acc[3] -= P.efield[0] * qi * pi4.x + P.efield[1] * qi * pi4.y + P.efield[2] * qi * pi4.z;
        acc[3] -= P.efield[0] * pi[0] + P.efield[1] * pi[1] + P.efield[2] * pi[2];
        fx[im] += acc[0];
        fy[im] += acc[1];
        fz[im] += acc[2];
        for (int k = 0; k < 15; ++k) partials[(size_t)blockIdx.x * 15 + k] = acc[3 + k];
    }
}

void launch_cpim_metal_forces(capac_ctx *c)
{
    {
        ProfScope ps(c, K_CPIM_METAL);
        if (c->opt.precision == CAPAC_PREC_MIXED)
            k_cpim_metal<float><<<c->M, 256, 0, c->stream>>>(c->P, c->pos4, c->nbr, c->nnb, c->cap, c->vec_pq, c->fx,
                                                             c->fy, c->fz, force_partials(c, FP_METAL));
        else
            k_cpim_metal<double><<<c->M, 256, 0, c->stream>>>(c->P, c->pos4, c->nbr, c->nnb, c->cap, c->vec_pq, c->fx,
                                                              c->fy, c->fz, force_partials(c, FP_METAL));
    }
    ++c->launches;
    if (c->defer) {
        c->fs.metal = force_partials(c, FP_METAL);
        c->fs.n_metal = c->M;
        return;
    }
    static const int pot_slots[15] = {9, 10, 11, 12, 13, 14, -1, -1, -1, -1, -1, -1, -1, -1, -1};
    static const int vir_slots[15] = {-1, -1, -1, -1, -1, -1, 0, 1, 2, 3, 4, 5, 6, 7, 8};
    launch_finalize(c, c->M, 15, pot_slots, vir_slots);
}

// ------------------------------------- external field on fixed charges

// force.c:2251-2260
__global__ void __launch_bounds__(256) k_external_field(DevParams P, const double4 *__restrict__ pos4, double *fx,
                                                        double *fy, double *fz, double *partials)
{
    __shared__ double sh[32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double e[1] = {0.0};
    if (i < P.N) {
        const double4 p = pos4[i];
        const double q = p.w;
        fx[i] += P.efield[0] * q;
        fy[i] += P.efield[1] * q;
        fz[i] += P.efield[2] * q;
        e[0] = -(P.efield[0] * q * p.x + P.efield[1] * q * p.y + P.efield[2] * q * p.z);
    }
    block_partials<1>(e, sh, partials);
}

void launch_external_field(capac_ctx *c)
{
    if (c->P.efield[0] == 0.0 && c->P.efield[1] == 0.0 && c->P.efield[2] == 0.0) return;
    const unsigned grid = grid_for(c->N, 256);
    k_external_field<<<grid, 256, 0, c->stream>>>(c->P, c->pos4, c->fx, c->fy, c->fz, force_partials(c, FP_FIELD));
    ++c->launches;
    if (c->defer) {
        c->fs.field = force_partials(c, FP_FIELD);
        c->fs.n_field = (int)grid;
        return;
    }
    static const int pot_slots[1] = {9};
    static const int vir_slots[1] = {-1};
    launch_finalize(c, (int)grid, 1, pot_slots, vir_slots);
}

// The areas of a force call's partials; returns their doubles.
size_t force_partial_areas(const capac_ctx *c, size_t off[4])
{
    const size_t pair = std::max((size_t)grid_for(c->N, 4), (size_t)c->num_sms * 5) * 11;  // or a resident grid
    const size_t n[4] = {(size_t)c->M * 10, pair, (size_t)c->M * 15,
                         (size_t)grid_for(c->N, 256)};
    size_t at = 0;
    for (int k = 0; k < 4; ++k) {
        off[k] = at;
        at += n[k];
    }
    return at;
}

size_t partials_needed(const capac_ctx *c)
{
    const size_t pair_blocks = grid_for(c->N, 4);  // k_pair: four warps of one atom each
    size_t need = pair_blocks * 11;
    need = std::max(need, (size_t)c->num_sms * 5 * 11);  // resident pair grids (at most five blocks per SM)
    need = std::max(need, (size_t)grid_for((long)c->N, 256) * 16);
    need = std::max(need, (size_t)(c->M + c->n_nps + 8) * 16);
    need = std::max(need, (size_t)grid_for((long)c->n_mols, 128) * 16);  // RATTLE blocks
    need = std::max(need, (size_t)grid_for((long)c->n_mat, 256) * 4);
    need = std::max(need, (size_t)c->M * 20);  // gradient sums (k_grad.cu)
    return need + 64;
}

}  // namespace capac
