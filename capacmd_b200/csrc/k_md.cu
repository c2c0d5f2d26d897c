// Velocity-Verlet MD step pieces on the device (mpi-main.c:874-1013):
// Nose-Hoover chain, half kicks, drift, RATTLE, kinetic energy, COM-velocity
// removal, apply_pbc and the force diagnostics.  Scalars (thermostat chain,
// kinetic energy, temperature) stay in device memory.
#include <algorithm>

#include "ctx.h"

namespace capac {

namespace {

struct MdParams {
    int N, n_mols, fix_metal, ndf;
    double dt, dt_2, q_mass;
    Box box;
};

MdParams md_params(const capac_ctx *c)
{
    MdParams m;
    m.N = c->N;
    m.n_mols = c->n_mols;
    m.fix_metal = c->fix_metal;
    m.ndf = c->c.ndf;
    m.dt = c->dt;
    m.dt_2 = c->c.dt_2;
    m.q_mass = c->c.q_mass;
    m.box = c->P.box;
    return m;
}

// Heating ramp of the reference temperature (mpi-main.c:879-891).
struct Heating {
    long step;
    int n;
};
__device__ __forceinline__ void heat(ThermoState *th, Heating h)
{
    if (h.step < h.n)
        th->ref_temp = th->first_temp + (th->ext_temp - th->first_temp) * h.step / h.n;
    else
        th->ref_temp = th->ext_temp;
    th->kT = kBoltz * th->ref_temp;
}

// exp(x) for |x| < 1/64: the Taylor sum to x^7, whose remainder there is 9e-20
// of the result, in pairs so that four dependent operations form it.
__device__ __forceinline__ double exp_small(double x)
{
    const double x2 = x * x;
    const double a = fma(x, 1.0 / 6.0, 0.5), b = fma(x, 1.0 / 120.0, 1.0 / 24.0), c = fma(x, 1.0 / 5040.0, 1.0 / 720.0);
    return 1.0 + fma(x2, fma(x2, fma(x2, c, b), a), x);
}

// The Nose-Hoover chain of k_nhc from the given velocities; returns the
// velocity scale.  SMALL: with exp_small; `most` is then the largest argument
// met, and the result holds only below 1/64.
template <bool SMALL>
__device__ __forceinline__ double nhc_chain(double (&vQ)[kNhc], double (&aQ)[kNhc], double ek, double NkT, double c0,
                                            double inv_q, double dt, double &most)
{
    const int Nc = 5, L = kNhc;
    const double w1 = 0.41449077179437571194, w3 = -0.65796308717750284778;
    const double w[5] = {w1, w1, w3, w1, w1};
    double scale = 1.0;
    most = 0.0;
    auto ex = [&](double x) {
        if (!SMALL) return exp(x);
        most = fmax(most, fabs(x));
        return exp_small(x);
    };
    aQ[0] = (ek - NkT) * inv_q;
#pragma unroll
    for (int k = 0; k < L - 1; ++k) aQ[k + 1] = fma(vQ[k], vQ[k], -c0);
    for (int c = 0; c < Nc; ++c) {
#pragma unroll
        for (int y = 0; y < 5; ++y) {
            const double h4 = w[y] * dt / (4 * Nc), h8 = w[y] * dt / (8 * Nc), h2 = w[y] * dt / (2 * Nc);
            vQ[L - 1] += aQ[L - 1] * h4;
#pragma unroll
            for (int k = L - 2; k >= 0; --k) {
                const double e = ex(-h8 * vQ[k + 1]);
                vQ[k] = e * fma(vQ[k], e, h4 * aQ[k]);
            }
            scale *= ex(-h2 * vQ[0]);
            aQ[0] = fma(ek * scale, scale, -NkT) * inv_q;
            double e[kNhc];
#pragma unroll
            for (int k = 0; k < L - 1; ++k) e[k] = ex(-h8 * vQ[k + 1]);
#pragma unroll
            for (int k = 0; k < L - 1; ++k) {
                vQ[k] = fma(h4 * e[k], aQ[k], vQ[k] * e[k] * e[k]);
                aQ[k + 1] = fma(vQ[k], vQ[k], -c0);
            }
            vQ[L - 1] += aQ[L - 1] * h4;
        }
    }
    return scale;
}

// nose_hoover_chain, thermostat.c:117-191: 10 links, Nc = 5, 5th-order
// Suzuki-Yoshida weights; the velocity scale is left in th->scale.  One
// thread: 25 sweeps down and up the chain, each link waiting for the last, so
// the length of one link's chain of operations is the time.  The exponentials'
// arguments are a time step over 40 times a thermostat velocity, far below the
// 1/64 up to which exp_small serves (else the chain runs again with the
// library's); on the way up they are those of velocities the way down left
// final, so only a multiply-add pair waits; the divisions by Q are folded into
// kT / Q.  41 us a launch with the library's exp and the divisions, 14.6 so.
__device__ void nhc(ThermoState *th, const MdParams &m)
{
    const double Q = m.q_mass, kT = th->kT, NkT = kT * m.ndf, ek = th->eksum, inv_q = 1.0 / Q;
    // the chain in registers (every index is fixed once the loops unroll),
    // written back at the end
    double vQ[kNhc], aQ[kNhc], most;
#pragma unroll
    for (int k = 0; k < kNhc; ++k) vQ[k] = th->vQ[k];
    double scale = nhc_chain<true>(vQ, aQ, ek, NkT, kT * inv_q, inv_q, m.dt, most);
    if (!(most < 0.015625)) {
#pragma unroll
        for (int k = 0; k < kNhc; ++k) vQ[k] = th->vQ[k];
        scale = nhc_chain<false>(vQ, aQ, ek, NkT, kT * inv_q, inv_q, m.dt, most);
    }
#pragma unroll
    for (int k = 0; k < kNhc; ++k) {
        th->vQ[k] = vQ[k];
        th->aQ[k] = aQ[k];
    }
    th->scale = scale;
    th->eksum = ek * (scale * scale);
    th->inst_temp *= scale * scale;
}

// The first chain of a step, after the heating ramp.
__global__ void k_nhc(ThermoState *th, MdParams m, Heating h)
{
    heat(th, h);
    nhc(th, m);
}

// Berendsen weak coupling (no counterpart in the reference, whose only
// thermostat is the Nose-Hoover chain): lambda = sqrt(1 + dt/tau (T0/T - 1))
// from the temperature after the second RATTLE (Berendsen et al., J. Chem.
// Phys. 81, 3684 (1984)), lambda^2 held to [0.64, 1.5625] and lambda = 1 at
// T = 0; the scale is left in th->scale.
__device__ void berendsen(ThermoState *th, double dt_over_tau)
{
    const double T = th->inst_temp;
    double s2 = 1.0;
    if (T > 0.0) s2 = fmin(fmax(1.0 + dt_over_tau * (th->ref_temp / T - 1.0), 0.64), 1.5625);
    const double s = sqrt(s2);
    th->scale = s;
    th->eksum *= s * s;
    th->inst_temp *= s * s;
}

// First half of a step: the thermostat's scale (nvt; else the heating ramp is
// done here), v += dt/2 F/m, old_r = r, r += dt v, the last three for atoms
// that move (mpi-main.c:900-932).
__global__ void k_kick_drift(MdParams m, const unsigned char *is_metal, const double *inv_mass, const double *fx,
                             const double *fy, const double *fz, double *vx, double *vy, double *vz, double *rx,
                             double *ry, double *rz, double *ox, double *oy, double *oz, ThermoState *th, int nvt,
                             Heating h)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (!nvt && i == 0) heat(th, h);
    if (i >= m.N) return;
    double a = vx[i], b = vy[i], c = vz[i];
    if (nvt) {
        const double s = th->scale;
        a *= s; b *= s; c *= s;
    }
    if (!(m.fix_metal == 1 && is_metal[i])) {
        const double im = inv_mass[i], x = rx[i], y = ry[i], z = rz[i];
        a += m.dt_2 * fx[i] * im;
        b += m.dt_2 * fy[i] * im;
        c += m.dt_2 * fz[i] * im;
        ox[i] = x; oy[i] = y; oz[i] = z;
        rx[i] = x + m.dt * a;
        ry[i] = y + m.dt * b;
        rz[i] = z + m.dt * c;
    }
    vx[i] = a; vy[i] = b; vz[i] = c;
}

// A step's second half after a solve that failed (md_step): nothing may change.
__device__ __forceinline__ bool halted(const SolverScalars *ss) { return ss && (ss->error | ss->failed) != 0; }

// v += dt/2 F/m for atoms that move.
__global__ void k_half_kick(MdParams m, const unsigned char *is_metal, const double *inv_mass, const double *fx,
                            const double *fy, const double *fz, double *vx, double *vy, double *vz,
                            const SolverScalars *ss)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.N || (m.fix_metal == 1 && is_metal[i]) || halted(ss)) return;
    const double im = inv_mass[i];
    vx[i] += m.dt_2 * fx[i] * im;
    vy[i] += m.dt_2 * fy[i] * im;
    vz[i] += m.dt_2 * fz[i] * im;
}

struct CstrView {
    const int *mol_first, *mol_type, *off, *cnt, *ci, *cj;
    const double *len;
    const double *inv_mass;
    const int *mol_atoms;  // atoms per molecule type
};

// Three-atom molecules with at most three constraints (the 3-site waters) are
// iterated in the constraints' own variables, in registers.  A correction g of
// constraint k moves atom t by sgn(t, k) m_t g times a vector d_k that does not
// change during the iteration (the old bond in the first stage, the bond in the
// second), so a bond's difference vector or projected velocity changes by
// weight(l, k) g d_k: the loop updates those and sums the g of each constraint,
// and the atoms are moved once at the end by the sums.  The same corrections
// and tests in the same order as on the atoms, to rounding; an iteration of a
// constraint waits for a few operations where the selects of its atoms'
// coordinates, the image shifts and the updates of positions and velocities
// made ~1,500 cycles of it (first and second stage, us a launch: 31 and 48 -> 14
// and 9 for 3,000 waters, 74 and 117 -> 45 and 25 for 150,000).
struct Bonds3 {
    int ca[3], cb[3];
    double im[3], d[3][3];  // inverse masses; d_k
    __device__ __forceinline__ void load(const CstrView &cv, int first, int c0, int nc)
    {
#pragma unroll
        for (int t = 0; t < 3; ++t) im[t] = cv.inv_mass[first + t];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            ca[k] = k < nc ? cv.ci[c0 + k] : 0;
            cb[k] = k < nc ? cv.cj[c0 + k] : 0;
        }
    }
    __device__ __forceinline__ double mass(int t) const { return t == 0 ? im[0] : (t == 1 ? im[1] : im[2]); }
    // the move of atom t per g of constraint k, along d_k
    __device__ __forceinline__ double move(int t, int k) const
    {
        return (t == ca[k] ? mass(t) : 0.0) - (t == cb[k] ? mass(t) : 0.0);
    }
    // the change of bond l's difference per g of constraint k, along d_k
    __device__ __forceinline__ double weight(int l, int k) const { return move(ca[l], k) - move(cb[l], k); }
    // bond k's difference of the atoms' values r
    __device__ __forceinline__ double diff(const double (&r)[3], int k) const
    {
        const double a = ca[k] == 0 ? r[0] : (ca[k] == 1 ? r[1] : r[2]);
        const double b = cb[k] == 0 ? r[0] : (cb[k] == 1 ? r[1] : r[2]);
        return a - b;
    }
};

// Threads of a block of the RATTLE kernels: one warp per scheduler, so that a
// few thousand molecules spread over as many SMs as they can.
constexpr int kRattleBlock = 128;

// rattle_1st, force.c:1907-1997: one thread per molecule.
__global__ void __launch_bounds__(kRattleBlock) k_rattle1(MdParams m, CstrView cv, double *rx, double *ry, double *rz, const double *ox,
                          const double *oy, const double *oz, double *vx, double *vy, double *vz, volatile int *failed)
{
    const int im = blockIdx.x * blockDim.x + threadIdx.x;
    if (im >= m.n_mols) return;
    const int first = cv.mol_first[im], mt = cv.mol_type[first];
    const int nc = cv.cnt[mt], c0 = cv.off[mt];
    if (nc == 0) return;
    const double tol2 = 2.0e-05, inv_dt = 1.0 / m.dt;  // the velocity update multiplies by 1/dt
    int iter = 0, done = 0;
    if (cv.mol_atoms[mt] == 3 && nc <= 3) {
        Bonds3 B;
        B.load(cv, first, c0, nc);
        double *const r[3] = {rx, ry, rz}, *const v[3] = {vx, vy, vz};
        const double *const o[3] = {ox, oy, oz};
        double x[3][3], p[3][3], len2[3], scale[3], w[3][3], G[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            double old[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                x[a][t] = r[a][first + t];
                old[t] = o[a][first + t];
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                p[k][a] = wrap1(B.diff(x[a], k), m.box.L[a]);
                B.d[k][a] = wrap1(B.diff(old, k), m.box.L[a]);
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double len = k < nc ? cv.len[c0 + k] : 0.0;
            len2[k] = len * len;
            scale[k] = 2.0 * (B.mass(B.ca[k]) + B.mass(B.cb[k]));
#pragma unroll
            for (int l = 0; l < 3; ++l) w[l][k] = B.weight(l, k);
        }
        while (!done) {
            done = 1;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (k >= nc) continue;
                const double diff = len2[k] - (p[k][0] * p[k][0] + p[k][1] * p[k][1] + p[k][2] * p[k][2]);
                if (fabs(diff) > len2[k] * tol2) {
                    const double g = diff / (scale[k] * (B.d[k][0] * p[k][0] + B.d[k][1] * p[k][1] + B.d[k][2] * p[k][2]));
                    G[k] += g;
#pragma unroll
                    for (int l = 0; l < 3; ++l) {
                        const double wg = w[l][k] * g;
#pragma unroll
                        for (int a = 0; a < 3; ++a) p[l][a] = fma(wg, B.d[k][a], p[l][a]);
                    }
                    done = 0;
                }
            }
            if (++iter > kMaxIter) break;
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            const double g0 = B.move(t, 0) * G[0], g1 = B.move(t, 1) * G[1], g2 = B.move(t, 2) * G[2];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const double dx = fma(g0, B.d[0][a], fma(g1, B.d[1][a], g2 * B.d[2][a]));
                r[a][first + t] = x[a][t] + dx;
                v[a][first + t] += dx * inv_dt;
            }
        }
        if (!done) *failed = 1;
        return;
    }
    while (!done) {
        done = 1;
        for (int k = 0; k < nc; ++k) {
            const int a = first + cv.ci[c0 + k], b = first + cv.cj[c0 + k];
            const double len2 = cv.len[c0 + k] * cv.len[c0 + k];
            const double px = wrap1(rx[a] - rx[b], m.box.L[0]);
            const double py = wrap1(ry[a] - ry[b], m.box.L[1]);
            const double pz = wrap1(rz[a] - rz[b], m.box.L[2]);
            const double diff = len2 - (px * px + py * py + pz * pz);
            if (fabs(diff) > len2 * tol2) {
                const double qx = wrap1(ox[a] - ox[b], m.box.L[0]);
                const double qy = wrap1(oy[a] - oy[b], m.box.L[1]);
                const double qz = wrap1(oz[a] - oz[b], m.box.L[2]);
                const double ma = cv.inv_mass[a], mb = cv.inv_mass[b];
                const double g = diff / (2.0 * (ma + mb) * (qx * px + qy * py + qz * pz));
                double dx = qx * g, dy = qy * g, dz = qz * g;
                rx[a] += ma * dx; ry[a] += ma * dy; rz[a] += ma * dz;
                rx[b] -= mb * dx; ry[b] -= mb * dy; rz[b] -= mb * dz;
                dx *= inv_dt; dy *= inv_dt; dz *= inv_dt;
                vx[a] += ma * dx; vy[a] += ma * dy; vz[a] += ma * dz;
                vx[b] -= mb * dx; vy[b] -= mb * dy; vz[b] -= mb * dz;
                done = 0;
            }
        }
        if (++iter > kMaxIter) break;
    }
    if (!done) *failed = 1;
}

// rattle_2nd, force.c:2004-2090: one thread per molecule; the constraint
// virial goes to per-block partials.
__global__ void __launch_bounds__(kRattleBlock) k_rattle2(MdParams m, CstrView cv, const double *rx, const double *ry,
                                                 const double *rz, double *vx, double *vy, double *vz,
                                                 volatile int *failed, double *partials,
                                                 const SolverScalars *ss)
{
    __shared__ double sh[32 * 9];
    if (halted(ss)) return;
    double vir[9] = {0.0};
    const int im = blockIdx.x * blockDim.x + threadIdx.x;
    if (im < m.n_mols) {
        const int first = cv.mol_first[im], mt = cv.mol_type[first];
        const int nc = cv.cnt[mt], c0 = cv.off[mt];
        // 1/(dt/2) and, per constraint of a three-atom molecule, the
        // reciprocal of its fixed denominator (m_a + m_b) len^2 taken once:
        // the iterations multiply where the reference divides (equal to
        // within a rounding of each product)
        const double tol = 1.0e-05, inv_hdt = 2.0 / m.dt;
        int iter = 0, done = nc == 0;
        const bool fast = !done && cv.mol_atoms[mt] == 3 && nc <= 3;
        if (fast) {
            Bonds3 B;
            B.load(cv, first, c0, nc);
            const double *const r[3] = {rx, ry, rz};
            double *const v[3] = {vx, vy, vz};
            double u[3][3], c[3] = {0.0, 0.0, 0.0}, inv_den[3], C[3][3], G[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                double x[3];
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    x[t] = r[a][first + t];
                    u[a][t] = v[a][first + t];
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    B.d[k][a] = wrap1(B.diff(x, k), m.box.L[a]);
                    c[k] = fma(B.d[k][a], B.diff(u[a], k), c[k]);  // projected relative velocity
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double len = k < nc ? cv.len[c0 + k] : 1.0;
                inv_den[k] = 1.0 / ((B.mass(B.ca[k]) + B.mass(B.cb[k])) * (len * len));
#pragma unroll
                for (int l = 0; l < 3; ++l)
                    C[l][k] = B.weight(l, k) * (B.d[l][0] * B.d[k][0] + B.d[l][1] * B.d[k][1] + B.d[l][2] * B.d[k][2]);
            }
            while (!done) {
                done = 1;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if (k >= nc) continue;
                    const double g = -c[k] * inv_den[k];
                    if (fabs(g) > tol) {
                        G[k] += g;
#pragma unroll
                        for (int l = 0; l < 3; ++l) c[l] = fma(C[l][k], g, c[l]);
                        done = 0;
                    }
                }
                if (++iter > kMaxIter) break;
            }
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const double g0 = B.move(t, 0) * G[0], g1 = B.move(t, 1) * G[1], g2 = B.move(t, 2) * G[2];
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    v[a][first + t] = u[a][t] + fma(g0, B.d[0][a], fma(g1, B.d[1][a], g2 * B.d[2][a]));
            }
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) vir[3 * a + b] -= B.d[k][a] * (B.d[k][b] * G[k] * inv_hdt);
        }
        while (!fast && !done) {
            done = 1;
            for (int k = 0; k < nc; ++k) {
                const int a = first + cv.ci[c0 + k], b = first + cv.cj[c0 + k];
                const double len2 = cv.len[c0 + k] * cv.len[c0 + k];
                const double ux = vx[a] - vx[b], uy = vy[a] - vy[b], uz = vz[a] - vz[b];
                const double px = wrap1(rx[a] - rx[b], m.box.L[0]);
                const double py = wrap1(ry[a] - ry[b], m.box.L[1]);
                const double pz = wrap1(rz[a] - rz[b], m.box.L[2]);
                const double ma = cv.inv_mass[a], mb = cv.inv_mass[b];
                const double g = -(px * ux + py * uy + pz * uz) / ((ma + mb) * len2);
                if (fabs(g) > tol) {
                    double dx = px * g, dy = py * g, dz = pz * g;
                    vx[a] += ma * dx; vy[a] += ma * dy; vz[a] += ma * dz;
                    vx[b] -= mb * dx; vy[b] -= mb * dy; vz[b] -= mb * dz;
                    dx *= inv_hdt; dy *= inv_hdt; dz *= inv_hdt;
                    vir[0] -= px * dx; vir[1] -= px * dy; vir[2] -= px * dz;
                    vir[3] -= py * dx; vir[4] -= py * dy; vir[5] -= py * dz;
                    vir[6] -= pz * dx; vir[7] -= pz * dy; vir[8] -= pz * dz;
                    done = 0;
                }
            }
            if (++iter > kMaxIter) break;
        }
        if (!done) *failed = 1;
    }
    block_partials<9>(vir, sh, partials);
}

// A block's K partial sums stored; true in the block that finds all others'
// stored (the last to arrive), which then sums them in block order.  The
// counter is left at zero for the next launch.
template <int K>
__device__ bool last_block_sum(double (&v)[K], double *sh, double *partials, int *count)
{
    __shared__ int last;
    block_partials<K>(v, sh, partials);
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(count, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] += __ldcg(partials + (size_t)K * b + k);
    block_sum<K>(v, sh);
    if (threadIdx.x == 0) *count = 0;
    return true;
}

// The velocity sums after the second half kick, kinetic_energy
// (thermostat.c:34-63) and remove_comm's momentum (:69-108), in one pass; the
// last block finishes them, runs the thermostat and leaves in th the scale and
// the scaled momentum's velocity for k_step_apply, and adds RATTLE's block
// partials of the virial.
__global__ void __launch_bounds__(256) k_step_sums(MdParams m, const double *__restrict__ mass,
                                                   const double *__restrict__ vx, const double *__restrict__ vy,
                                                   const double *__restrict__ vz, int thermostat, double dt_over_tau,
                                                   ThermoState *th, double *partials, int *count,
                                                   const double *__restrict__ rattle, int n_rattle, double *vir,
                                                   const SolverScalars *ss)
{
    __shared__ double sh[32 * 9];
    if (halted(ss)) return;
    double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m.N; i += gridDim.x * blockDim.x) {
        const double mm = mass[i];
        if (!(mm > 0.0)) continue;
        const double a = vx[i], b = vy[i], c = vz[i];
        v[0] += mm * a * a;
        v[1] += mm * b * b;
        v[2] += mm * c * c;
        v[3] += a * mm;
        v[4] += b * mm;
        v[5] += c * mm;
        v[6] += mm;
    }
    if (!last_block_sum<7>(v, sh, partials, count)) return;
    if (threadIdx.x == 0) {
        th->eksum = v[0] + v[1] + v[2];
        th->inst_temp = th->eksum / (kBoltz * m.ndf);
        if (thermostat == CAPAC_NVT) nhc(th, m);
        else if (thermostat == CAPAC_BERENDSEN) berendsen(th, dt_over_tau);
        else th->scale = 1.0;
        for (int a = 0; a < 3; ++a) th->vcom[a] = th->scale * v[3 + a] / v[6];
        th->vcom[3] = v[6];
    }
    if (n_rattle > 0) {
        double w[9] = {0.0};
        for (int b = threadIdx.x; b < n_rattle; b += blockDim.x)
#pragma unroll
            for (int k = 0; k < 9; ++k) w[k] += rattle[(size_t)9 * b + k];
        __syncthreads();
        block_sum<9>(w, sh);
        if (threadIdx.x == 0)
            for (int k = 0; k < 9; ++k) vir[k] += w[k];
    }
}

// v = scale v - v_com and the kinetic energy of the result (the last block
// finishes it), with sum_potential (force.c:322-331).
__global__ void __launch_bounds__(256) k_step_apply(MdParams m, const double *__restrict__ mass, double *vx, double *vy,
                                                    double *vz, ThermoState *th, double *partials, int *count,
                                                    double *pot, const SolverScalars *ss)
{
    __shared__ double sh[32 * 3];
    if (halted(ss)) return;
    const double s = th->scale, c0 = th->vcom[0], c1 = th->vcom[1], c2 = th->vcom[2];
    double v[3] = {0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m.N; i += gridDim.x * blockDim.x) {
        const double mm = mass[i];
        const bool real = mm > 0.0;
        const double a = s * vx[i] - (real ? c0 : 0.0), b = s * vy[i] - (real ? c1 : 0.0),
                     c = s * vz[i] - (real ? c2 : 0.0);
        vx[i] = a; vy[i] = b; vz[i] = c;
        if (real) {
            v[0] += mm * a * a;
            v[1] += mm * b * b;
            v[2] += mm * c * c;
        }
    }
    if (!last_block_sum<3>(v, sh, partials, count)) return;
    if (threadIdx.x == 0) {
        th->eksum = v[0] + v[1] + v[2];
        th->inst_temp = th->eksum / (kBoltz * m.ndf);
        double e = 0.0;
        for (int k = 1; k < 15; ++k) e += pot[k];
        pot[0] = e;
    }
}

// apply_pbc, force.c:127-165: one thread per molecule.
__global__ void k_apply_pbc(MdParams m, const int *mol_first, const int *mol_last, double *rx, double *ry,
                            double *rz)
{
    const int im = blockIdx.x * blockDim.x + threadIdx.x;
    if (im >= m.n_mols) return;
    const int lo = mol_first[im], hi = mol_last[im], mid = (lo + hi) / 2;
    double *r[3] = {rx, ry, rz};
    const double h[3] = {0.5 * m.box.L[0], 0.5 * m.box.L[1], 0.5 * m.box.L[2]};
    for (int a = 0; a < 3; ++a) {
        if (r[a][mid] > m.box.L[a]) r[a][mid] -= m.box.L[a];
        else if (r[a][mid] < 0.0) r[a][mid] += m.box.L[a];
    }
    for (int i = lo; i <= hi; ++i) {
        if (i == mid) continue;
        for (int a = 0; a < 3; ++a) {
            if (r[a][i] - r[a][mid] > h[a]) r[a][i] -= m.box.L[a];
            else if (r[a][i] - r[a][mid] < -h[a]) r[a][i] += m.box.L[a];
        }
    }
}

// get_fmax_rms, force.c:361-378
__global__ void __launch_bounds__(256) k_fmax(int N, const double *fx, const double *fy, const double *fz,
                                              double *partials)
{
    __shared__ double sh[32 * 2];
    __shared__ double shm[8];
    double v[2] = {0.0, 0.0};
    double mx = 0.0;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) {
        const double f2 = fx[i] * fx[i] + fy[i] * fy[i] + fz[i] * fz[i];
        v[0] = f2;
        mx = f2;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = mx;
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx = fmax(mx, shm[w]);
        partials[2 * blockIdx.x] = v[0];
        partials[2 * blockIdx.x + 1] = mx;
    }
}

__global__ void k_fmax_final(const double *partials, int nb, int N, ThermoState *th)
{
    __shared__ double sh[32 * 2];
    __shared__ double shm[32];
    double v[2] = {0.0, 0.0};
    double mx = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        v[0] += partials[2 * b];
        mx = fmax(mx, partials[2 * b + 1]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = mx;
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx = fmax(mx, shm[w]);
        th->fmax = sqrt(mx);
        th->frms = sqrt(v[0] / N);
    }
}

// (x, y, z) of each atom side by side.
__global__ void k_interleave(int N, const double *__restrict__ x, const double *__restrict__ y,
                             const double *__restrict__ z, double *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    out[3 * (size_t)i] = x[i];
    out[3 * (size_t)i + 1] = y[i];
    out[3 * (size_t)i + 2] = z[i];
}

// Energy minimisation step (mpi-main.c:730-756): old_r = r for every atom;
// r += s / f_max * em_length except for fixed metal atoms.
__global__ void k_em_move(MdParams m, const unsigned char *is_metal, const ThermoState *th, double em_length,
                          const double *__restrict__ sx, const double *__restrict__ sy,
                          const double *__restrict__ sz, double *rx, double *ry, double *rz, double *ox, double *oy,
                          double *oz)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.N) return;
    ox[i] = rx[i];
    oy[i] = ry[i];
    oz[i] = rz[i];
    if (m.fix_metal == 1 && is_metal[i]) return;
    const double fmax = th->fmax;
    rx[i] += sx[i] / fmax * em_length;
    ry[i] += sy[i] / fmax * em_length;
    rz[i] += sz[i] / fmax * em_length;
}

// s = F + gamma s, old F = F (mpi-main.c:843-852).
__global__ void k_em_direction(int N, double gamma, const double *__restrict__ fx, const double *__restrict__ fy,
                               const double *__restrict__ fz, double *sx, double *sy, double *sz, double *gx,
                               double *gy, double *gz)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    sx[i] = fx[i] + gamma * sx[i];
    sy[i] = fy[i] + gamma * sy[i];
    sz[i] = fz[i] + gamma * sz[i];
    gx[i] = fx[i];
    gy[i] = fy[i];
    gz[i] = fz[i];
}

// Partials of g22 = (F, F), g12 = (F_old, F), g11 = (F_old, F_old) for the
// conjugate-gradient gamma (mpi-main.c:823-840).
__global__ void __launch_bounds__(256) k_em_dots(int N, const double *__restrict__ fx, const double *__restrict__ fy,
                                                 const double *__restrict__ fz, const double *__restrict__ gx,
                                                 const double *__restrict__ gy, const double *__restrict__ gz,
                                                 double *partials)
{
    __shared__ double sh[32 * 3];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[3] = {0.0, 0.0, 0.0};
    if (i < N) {
        acc[0] = fx[i] * fx[i] + fy[i] * fy[i] + fz[i] * fz[i];
        acc[1] = gx[i] * fx[i] + gy[i] * fy[i] + gz[i] * fz[i];
        acc[2] = gx[i] * gx[i] + gy[i] * gy[i] + gz[i] * gz[i];
    }
    block_partials<3>(acc, sh, partials);
}

__global__ void k_sum_potential(double *pot)
{
    double s = 0.0;
    for (int k = 1; k < 15; ++k) s += pot[k];
    pot[0] = s;
}

CstrView cstr_view(const capac_ctx *c)
{
    CstrView v;
    v.mol_first = c->mol_first;
    v.mol_type = c->mol_type;
    v.off = c->cstr_off;
    v.cnt = c->cstr_cnt;
    v.ci = c->cstr_i;
    v.cj = c->cstr_j;
    v.len = c->cstr_r;
    v.inv_mass = c->inv_mass;
    v.mol_atoms = c->mol_atoms;
    return v;
}

}  // namespace

void launch_nhc(capac_ctx *c, long step)
{
    k_nhc<<<1, 1, 0, c->stream>>>(c->th, md_params(c), Heating{step, c->n_heating});
    ++c->launches;
}

void launch_md_kick_drift(capac_ctx *c, bool nvt, long step)
{
    k_kick_drift<<<grid_for(c->N, 256), 256, 0, c->stream>>>(
        md_params(c), c->is_metal, c->inv_mass, c->fx, c->fy, c->fz, c->vx, c->vy, c->vz, c->rx, c->ry, c->rz, c->ox,
        c->oy, c->oz, c->th, nvt ? 1 : 0, Heating{step, c->n_heating});
    ++c->launches;
}

void launch_md_half_kick(capac_ctx *c)
{
    k_half_kick<<<grid_for(c->N, 256), 256, 0, c->stream>>>(md_params(c), c->is_metal, c->inv_mass, c->fx, c->fy,
                                                           c->fz, c->vx, c->vy, c->vz, halting(c));
    ++c->launches;
}

void launch_step_sums(capac_ctx *c, int thermostat, bool rattle_virial)
{
    const unsigned grid = std::min(grid_for(c->N, 256), (unsigned)kSumBlocks);
    const int nr = rattle_virial ? (int)grid_for(c->n_mols, kRattleBlock) : 0;
    k_step_sums<<<grid, 256, 0, c->stream>>>(md_params(c), c->mass, c->vx, c->vy, c->vz, thermostat, c->dt_over_tau,
                                             c->th, c->spart, c->scount, c->partials, nr, c->vir, halting(c));
    k_step_apply<<<grid, 256, 0, c->stream>>>(md_params(c), c->mass, c->vx, c->vy, c->vz, c->th, c->spart,
                                              c->scount + 1, c->pot, halting(c));
    c->launches += 2;
}

void launch_rattle(capac_ctx *c, int second, bool in_step)
{
    if (!c->has_cstr) return;
    const unsigned grid = grid_for(c->n_mols, kRattleBlock);
    if (!second) {
        k_rattle1<<<grid, kRattleBlock, 0, c->stream>>>(md_params(c), cstr_view(c), c->rx, c->ry, c->rz, c->ox, c->oy, c->oz,
                                               c->vx, c->vy, c->vz, c->sig + 1);
        ++c->launches;
    } else {
        k_rattle2<<<grid, kRattleBlock, 0, c->stream>>>(md_params(c), cstr_view(c), c->rx, c->ry, c->rz, c->vx, c->vy, c->vz,
                                               c->sig + 2, c->partials, halting(c));
        ++c->launches;
        if (in_step) return;
        static const int pot_slots[9] = {-1, -1, -1, -1, -1, -1, -1, -1, -1};
        static const int vir_slots[9] = {0, 1, 2, 3, 4, 5, 6, 7, 8};
        launch_finalize(c, (int)grid, 9, pot_slots, vir_slots);
    }
}

void launch_apply_pbc(capac_ctx *c)
{
    k_apply_pbc<<<grid_for(c->n_mols, 256), 256, 0, c->stream>>>(md_params(c), c->mol_first, c->mol_last, c->rx,
                                                                c->ry, c->rz);
    ++c->launches;
}

void launch_interleave(capac_ctx *c, const double *x, const double *y, const double *z, double *out)
{
    k_interleave<<<grid_for(c->N, 256), 256, 0, c->stream>>>(c->N, x, y, z, out);
    ++c->launches;
}

void launch_fmax_rms(capac_ctx *c)
{
    const unsigned grid = grid_for(c->N, 256);
    k_fmax<<<grid, 256, 0, c->stream>>>(c->N, c->fx, c->fy, c->fz, c->partials);
    k_fmax_final<<<1, 256, 0, c->stream>>>(c->partials, (int)grid, c->N, c->th);
    c->launches += 2;
}

void launch_sum_potential(capac_ctx *c)
{
    k_sum_potential<<<1, 1, 0, c->stream>>>(c->pot);
    ++c->launches;
}

// em_buf layout: sx sy sz | old fx fy fz, N each
void launch_em_move(capac_ctx *c)
{
    const size_t N = c->N;
    k_em_move<<<grid_for(c->N, 256), 256, 0, c->stream>>>(md_params(c), c->is_metal, c->th, c->em_length, c->em_buf,
                                                         c->em_buf + N, c->em_buf + 2 * N, c->rx, c->ry, c->rz,
                                                         c->ox, c->oy, c->oz);
    ++c->launches;
}

void launch_em_direction(capac_ctx *c, double gamma)
{
    const size_t N = c->N;
    double *b = c->em_buf;
    k_em_direction<<<grid_for(c->N, 256), 256, 0, c->stream>>>(c->N, gamma, c->fx, c->fy, c->fz, b, b + N,
                                                              b + 2 * N, b + 3 * N, b + 4 * N, b + 5 * N);
    ++c->launches;
}

void launch_em_dots(capac_ctx *c)
{
    const size_t N = c->N;
    const double *b = c->em_buf;
    k_em_dots<<<grid_for(c->N, 256), 256, 0, c->stream>>>(c->N, c->fx, c->fy, c->fz, b + 3 * N, b + 4 * N,
                                                         b + 5 * N, c->partials);
    ++c->launches;
}

}  // namespace capac
