// Block-Jacobi preconditioner for the mixed path's inner BiCGSTAB.
//
// The reference preconditions BiCGSTAB with the matrix diagonal (Jacobi,
// bicg_stab.c:328-347); the FP64 path keeps that.  On the mixed path the
// inner solves only have to reduce the residual of an FP64 refinement
// sweep, so they may use a stronger preconditioner without changing the
// answer, which the FP64 residual defines.  The metal atoms are cut into
// groups of 32 along a Morton (Z-order) curve of their initial positions, so
// a group is a compact piece of the cluster; each group's 128 x 128 diagonal
// block of the CPIM matrix (its dipole-dipole, dipole-charge and
// charge-charge couplings plus the diagonal 1/polar, -1/capac) is inverted in
// FP64 and stored in FP32.  Applying the inverse couples the unknowns of
// neighbouring atoms that the diagonal alone leaves apart; on the 9.3k-atom
// system it cuts the iterations to a relative residual of 1e-10 from 117 to
// about 50.  The neutrality rows keep a unit preconditioner.  The inverse
// blocks are refreshed every 10 matrix builds (and after positions are set
// from outside): in MD the atoms move little between refreshes, and a
// slightly stale preconditioner changes only the inner iteration count.
//
// Layout: g_atoms[G * 32 + a] = metal index (0-based, -1 for padding) of slot
// a of group G; local row o = 4 a + c (c = 0..2 dipole, 3 charge);
// dinv[G][c][o] = (D_G^-1)[o][c] (column-major, so the threads of a warp
// reading one column for their rows are coalesced).
#include <algorithm>
#include <cstdint>
#include <vector>

#include "terms.cuh"

namespace capac {

namespace {

constexpr int kG = 32;             // atoms per group
constexpr int kN = 4 * kG;         // rows per block
constexpr int kInvThreads = 512;
constexpr int kInvRows = kN * kN / kInvThreads / 4;  // rows of a warp

// In-place Gauss-Jordan inversion with partial pivoting of the group's block
// in FP64, one block per group.  The matrix lives in registers, warp w holding
// rows 8 w .., lane l columns 4 l .. 4 l + 3: a pivot step then takes 4 reads of
// column factors and 2 of the pivot row from shared memory for 32 multiply-adds
// of a thread.  (Shared reads set the pace, a 16-byte one costing four cycles
// even when all lanes read the same: 32 rows of one column per thread, 16 such
// reads for the same 32, took 1.9 us a step; the whole matrix read and
// rewritten in shared memory 4.4.  128 steps: 568 -> 247 -> 152 us a launch,
// whatever the number of groups.)  Rows are not interchanged: row p_k serves as
// pivot of column k and is marked used, and the result is stored permuted,
// inverse[k][p_l] = B[p_k][l].  The pivot is the largest entry to 13 bits of
// mantissa (the rest of a 32-bit key holds the row), which is as good a pivot.
// A pivot below 1e-13 of the block's largest entry falls back to the Jacobi
// inverse for this group (never observed; it keeps a degenerate block harmless).
__global__ void __launch_bounds__(kInvThreads) k_block_inverse(DevParams P, const double4 *__restrict__ pos4,
                                                               const int *__restrict__ g_atoms, float *__restrict__ dinv)
{
    extern __shared__ __align__(16) double Dm[];  // kN * kN, row-major; then the inverse in FP32, rows of kN + 1
    // the pivot column, twice: as it is, for the pivot search, and as the
    // update's factors, where the pivot row's is replaced
    __shared__ __align__(16) double colk[2][kN], fac[2][kN], prow[kN];
    __shared__ double wv[kInvThreads / 32];
    __shared__ short piv[kN], row_of[kN];  // piv[k] = p_k, row_of[p_k] = k
    const int G = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int w = __shfl_sync(0xffffffffu, tid >> 5, 0), row0 = w * kInvRows;
    const int *atoms = g_atoms + (size_t)G * kG;

    // the block: diagonal terms and cpim_block for every ordered pair of the group
    for (int q = tid; q < kG * kG; q += blockDim.x) {
        const int a = q / kG, b = q % kG;
        const int ia = atoms[a], ib = atoms[b];
        double e[16];
        if (ia < 0 || ib < 0) {
#pragma unroll
            for (int k = 0; k < 16; ++k) e[k] = 0.0;
            if (a == b)
#pragma unroll
                for (int k = 0; k < 4; ++k) e[5 * k] = 1.0;  // padding slot: identity
        } else {
            cpim_block(P, pos4[P.metal_min + ia], pos4[P.metal_min + ib], a == b, e);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) Dm[(4 * a + r) * kN + 4 * b + cc] = e[4 * r + cc];
    }
    __syncthreads();
    double a[kInvRows][4], amax = 0.0;
#pragma unroll
    for (int r = 0; r < kInvRows; ++r)
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            const double2 v = *reinterpret_cast<const double2 *>(Dm + (row0 + r) * kN + 4 * lane + c);
            a[r][c] = v.x;
            a[r][c + 1] = v.y;
            amax = fmax(amax, fmax(fabs(v.x), fabs(v.y)));
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) {
        wv[w] = amax;
        double2 *u = reinterpret_cast<double2 *>(colk[0] + row0), *v = reinterpret_cast<double2 *>(fac[0] + row0);
#pragma unroll
        for (int r = 0; r < kInvRows; r += 2) u[r / 2] = v[r / 2] = make_double2(a[r][0], a[r + 1][0]);
    }
    __syncthreads();
    for (int q = 0; q < kInvThreads / 32; ++q) amax = fmax(amax, wv[q]);
    const double tiny = 1e-13 * amax;

    bool bad = false;
    unsigned used = 0;  // of rows lane, lane + 32, ..: every warp keeps its own copy
    for (int k4 = 0; k4 < kN && !bad; k4 += 4) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {  // column kk of lane k4 / 4
            const int k = k4 + kk;
            const double *col = colk[kk & 1];
            double *f = fac[kk & 1];
            unsigned key = 0;
#pragma unroll
            for (int q = 0; q < kN / 32; ++q) {
                const int i = lane + 32 * q;
                const unsigned h = (unsigned)__double2hiint(fabs(col[i]));
                if (!((used >> q) & 1u)) key = max(key, (h & ~(unsigned)(kN - 1)) | (unsigned)(kN - 1 - i));
            }
            const int p = kN - 1 - (int)(__reduce_max_sync(0xffffffffu, key) & (unsigned)(kN - 1));
            const double d = col[p];
            bad = !(fabs(d) > tiny);  // the same in every thread
            if (bad) break;
            if ((p & 31) == lane) used |= 1u << (p >> 5);
            const int pl = p - row0;  // the pivot row among this warp's
            // the pivot column becomes the unit vector of the pivot row
            if (lane == k4 / 4)
#pragma unroll
                for (int r = 0; r < kInvRows; ++r) a[r][kk] = r == pl ? 1.0 : 0.0;
            if ((unsigned)pl < (unsigned)kInvRows) {
                // the pivot row, before its division, from the warp that holds it
                double v[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    v[c] = a[0][c];
#pragma unroll
                    for (int r = 1; r < kInvRows; ++r) v[c] = r == pl ? a[r][c] : v[c];
                }
                double2 *u = reinterpret_cast<double2 *>(prow + 4 * lane);
                u[0] = make_double2(v[0], v[1]);
                u[1] = make_double2(v[2], v[3]);
                if (lane == 0) {
                    piv[k] = (short)p;
                    row_of[p] = (short)k;
                    f[p] = d - 1.0;  // v - (d - 1) v / d = v / d
                }
            }
            const double inv = 1.0 / d;
            __syncthreads();
            const double2 p0 = *reinterpret_cast<const double2 *>(prow + 4 * lane);
            const double2 p1 = *reinterpret_cast<const double2 *>(prow + 4 * lane + 2);
            const double rj[4] = {p0.x * inv, p0.y * inv, p1.x * inv, p1.y * inv};
#pragma unroll
            for (int r = 0; r < kInvRows; r += 2) {
                const double2 g = *reinterpret_cast<const double2 *>(f + row0 + r);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    a[r][c] = fma(-g.x, rj[c], a[r][c]);
                    a[r + 1][c] = fma(-g.y, rj[c], a[r + 1][c]);
                }
            }
            if (k + 1 < kN && lane == (k + 1) / 4) {
                double2 *u = reinterpret_cast<double2 *>(colk[(kk + 1) & 1] + row0);
                double2 *v = reinterpret_cast<double2 *>(fac[(kk + 1) & 1] + row0);
#pragma unroll
                for (int r = 0; r < kInvRows; r += 2)
                    u[r / 2] = v[r / 2] = make_double2(a[r][(kk + 1) & 3], a[r + 1][(kk + 1) & 3]);
            }
            __syncthreads();
        }
    }
    float *S = reinterpret_cast<float *>(Dm);
    __syncthreads();
    if (!bad) {
#pragma unroll
        for (int r = 0; r < kInvRows; ++r)  // out[c][o] = inverse[o][c], o = row_of[i], c = piv[j]
#pragma unroll
            for (int c = 0; c < 4; ++c) S[piv[4 * lane + c] * (kN + 1) + row_of[row0 + r]] = (float)a[r][c];
    } else {  // Jacobi for this group
        for (int q = tid; q < kN * kN; q += blockDim.x) {
            const int c = q / kN, o = q % kN, at = o >> 2, comp = o & 3;
            const double d = atoms[at] < 0 ? 1.0 : (comp < 3 ? P.inv_polar : -P.inv_capac);
            S[c * (kN + 1) + o] = c == o ? (float)(1.0 / d) : 0.0f;
        }
    }
    __syncthreads();
    float *out = dinv + (size_t)G * kN * kN;
    for (int q = tid; q < kN * kN; q += blockDim.x) out[q] = S[q / kN * (kN + 1) + q % kN];
}

// Interleave the low 21 bits of v with two zero bits after each (Morton key).
uint64_t spread3(uint64_t v)
{
    uint64_t out = 0;
    for (int b = 0; b < 21; ++b) out |= ((v >> b) & 1ull) << (3 * b);
    return out;
}

}  // namespace

int precond_groups(int M) { return (M + kG - 1) / kG; }
size_t precond_inverse_floats(int M) { return (size_t)precond_groups(M) * kN * kN; }

// Groups of 32 metal atoms along the Morton curve of the positions given
// (metal_min .. metal_min + M - 1), as g_atoms above.
std::vector<int> precond_group_atoms(int M, int metal_min, const double *rx, const double *ry, const double *rz)
{
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    const double *r[3] = {rx, ry, rz};
    for (int i = 0; i < M; ++i)
        for (int a = 0; a < 3; ++a) {
            lo[a] = std::min(lo[a], r[a][metal_min + i]);
            hi[a] = std::max(hi[a], r[a][metal_min + i]);
        }
    double span = 0.0;
    for (int a = 0; a < 3; ++a) span = std::max(span, hi[a] - lo[a]);
    if (span <= 0.0) span = 1.0;
    std::vector<std::pair<uint64_t, int>> key(M);
    for (int i = 0; i < M; ++i) {
        uint64_t k = 0;
        for (int a = 0; a < 3; ++a) {
            const uint64_t q = (uint64_t)std::min(1048575.0, (r[a][metal_min + i] - lo[a]) / span * 1048575.0);
            k |= spread3(q) << a;
        }
        key[i] = {k, i};
    }
    std::stable_sort(key.begin(), key.end(), [](const auto &x, const auto &y) { return x.first < y.first; });
    const int nG = precond_groups(M);
    std::vector<int> g((size_t)nG * kG, -1);
    for (int i = 0; i < M; ++i) g[i] = key[i].second;
    return g;
}

void launch_block_inverse(capac_ctx *c)
{
    const int nG = precond_groups(c->M);
    const size_t smem = sizeof(double) * kN * kN;
    CAPAC_CUDA(cudaFuncSetAttribute(k_block_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ProfScope ps(c, K_MATRIX);
    k_block_inverse<<<nG, kInvThreads, smem, c->stream>>>(c->P, c->pos4, c->g_atoms, c->dinv);
    ++c->launches;
}

}  // namespace capac
