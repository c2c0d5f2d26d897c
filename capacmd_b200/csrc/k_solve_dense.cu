// BiCGSTAB for small CPIM systems with the whole FP64 matrix on chip.
//
// A solve of a few hundred metal atoms is bound by the latency of its
// grid-wide exchanges, not by bytes or operations: the tiled solvers
// (k_solve_coop.cu) need four to six per iteration (tile partials, their
// reduction and the preconditioner, twice), each a grid barrier with dependent
// round trips to L2 on both sides, 19 us (FP64) and 29 us (mixed path) per
// iteration whatever the size.  Here block b holds 12 whole rows of the dense
// matrix, column e = tid + 256 m with thread tid, and every block carries all the
// vectors (the same elements in the same threads).  Up to three columns a thread
// all of it is in registers.  With five and seven (769 unknowns and more) 255
// registers do not hold the rows' 480 and 672 bytes beside the vectors: the
// compiler keeps 248 and 664 bytes a thread on the stack (mixed path 192 and 640),
// and the products read what of the rows is among them back through L1.  A
// product is 12 C fused multiply-adds per thread and a block reduction; what
// the blocks exchange is only their 12 new values, and all that follows (dots,
// scalars, vector updates) every block does on the same numbers in the same
// order, so all take the same branches.  Two exchanges per iteration.
//
// The exchange has no barrier: a value travels as two 64-bit words, each half
// of the double beside a 32-bit sequence number, which a reader polls until
// both carry the number of this exchange (64-bit accesses are single-copy
// atomic, so value and number cannot part).  One trip to L2 and back replaces
// write, fence, barrier arrival, barrier poll and read.  Two buffers by the
// parity of the number suffice: a block writes number q + 2 only after it has
// read all of q + 1, and each block wrote its part of q + 1 after it had read
// all of q.  Numbers grow from launch to launch.  A block's 12 values take two
// 128-byte lines of their own: lines written by several SMs while others poll
// them cost ~70 ns per writer (17 us per iteration with one flag word per
// block packed together).  The first read waits 600 cycles: earlier it misses
// and the polls slow the stores (n = 1,237: 7.0 us per iteration without the
// wait, 5.3 with it, 5.9 with 300; measured at that size only).  12 rows
// because fewer blocks read less from the same lines (n = 589: 4 rows on 148
// blocks 5.8 us, 12 on 50 4.6).
// Every poll is bounded (wait_polls); a block that gives up sets the error
// word, which ends the other blocks' polls, and all return.
//
// Two modes:
//   FP64 path: the reference's Jacobi-BiCGSTAB and stopping rules
//     (bicg_stab.c:253-573) on the assembled tiles.
//   Mixed path: right-preconditioned BiCGSTAB on B = A K (K the block-Jacobi
//     inverses of the 32-atom groups, k_precond.cu): A from the positions in
//     FP64 into shared memory, the block's rows of B formed once per solve into
//     the registers, so an iteration still is two products and two exchanges;
//     x += K u at the end of a sweep, and the residual b - A x then decides, as
//     in the refinement around the tiled solver.  The FP64 matrix is at hand,
//     so one sweep usually reaches refine_tol.
//
// Which systems: 12 rows per block, one block per SM, 256 x 7 columns: up to
// 443 metal atoms with one nanoparticle on 148 SMs, whose blocks have no rows for
// more.
// Cold solves of Au55/147/309 in water against the tiled solvers (one B200):
// FP64 to rTr < 1e-24 bTb 954 -> 349, 1,532 -> 346, 2,081 -> 621 us (6.2, 3.8
// and 5.3 us per iteration); mixed to 1e-10, with the sweeps and residuals
// that were launches of their own, 557 -> 136, 835 -> 235, 946 -> 362 us.
// (221 unknowns on 19 blocks take longer per iteration than 589 on 50: the
// trace shows blocks in two camps, on the two dies, seeing each other's
// stores ~1 us later than their own.)
#include <algorithm>
#include <cstdint>

#include "terms.cuh"

namespace capac {

namespace {

constexpr int kT = 32;
constexpr int kPlanes = 10;
constexpr int kGroup = 4 * kT;  // unknowns of a preconditioner group
constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
constexpr int kR = 12;          // matrix rows per block
constexpr int kSeg = 16;        // exchange slots per block (two 128-byte lines of eight)
constexpr int kMaxCols = 7;     // columns per thread
constexpr long kPollLimit = 1L << 24;
constexpr int kFirstRead = 600; // cycles from a block's store to its first read
constexpr int kStall = 60;      // iterations without a halving of (r, r) that end a sweep
constexpr int kSweeps = 12;
constexpr int kStarts = 8;      // FP64 path: starts after breakdowns
constexpr int kStageRows = 8;   // ring of inverse-block rows: stages(C) x 2 groups x 8 rows
constexpr int kStepsPerPair = kGroup / kStageRows;
constexpr long kWaitPolls = 1L << 20;
// 32 KB of them, 16 KB where the matrix rows leave no more
__host__ __device__ constexpr int stages(int cols) { return cols <= 5 ? 4 : 2; }

struct DenseArgs {
    int M, n, n_nps, metal_min, max_iter, nT;
    long spin_limit;
    double inv_polar, inv_capac, tol, skip;
    const int *np_start, *np_end;
    const double *tiles;  // FP64 path: symmetric packed tiles in the metal atoms' order
    const double *b;
    double *x;
    ulonglong2 *ex;       // two exchange buffers of kSeg slots per block
    unsigned seq;         // number of the first exchange of this launch
    SolverScalars *ss;    // the error word that ends all polls
    SolverScalars *out;   // pinned host memory: the result's scalars
    // mixed path
    DevParams P;
    const double4 *pos4;
    const int *g_atoms, *slot_np;
    const float *dinv;
    int nG;
    double *hist;         // warm-start history (null: x is the start)
    int order;            // extrapolation order, 0 or less: only record
};

__device__ __forceinline__ ulonglong2 ld_pair(const ulonglong2 *p)
{
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_value(ulonglong2 *p, double v, unsigned seq)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(v), f = (unsigned long long)seq << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"((u & 0xffffffffull) | f),
                 "l"((u >> 32) | f)
                 : "memory");
}
__device__ __forceinline__ bool arrived(const ulonglong2 &q, unsigned seq)
{
    return (unsigned)(q.x >> 32) == seq && (unsigned)(q.y >> 32) == seq;
}
__device__ __forceinline__ double value_of(const ulonglong2 &q)
{
    return __longlong_as_double((long long)((q.x & 0xffffffffull) | (q.y << 32)));
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// Bounded wait for a phase of the barrier (each try suspends up to 1 us).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity)
{
    for (long i = 0; i < kWaitPolls; ++i) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity), "r"(1000u)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Entry (row, col) of the dense matrix in the FP64 path's order (atom e / 4,
// component e % 4 = p_x, p_y, p_z, q; the constraint rows at 4 M), from the tiles.
__device__ double tile_entry(const DenseArgs &A, int row, int col)
{
    const int n4 = 4 * A.M;
    if (row >= n4 || col >= n4) {
        const int k = (row >= n4 ? row : col) - n4, o = row >= n4 ? col : row, im = A.metal_min + (o >> 2);
        return o < n4 && (o & 3) == 3 && im >= A.np_start[k] && im <= A.np_end[k] ? 1.0 : 0.0;
    }
    const int i = row >> 2, c = row & 3, j = col >> 2, d = col & 3;
    if (i == j) return c != d ? 0.0 : keep_entry(c < 3 ? A.inv_polar : -A.inv_capac);
    // the tile holds the block of the ordered pair (lo, hi), [A m; -m^T C];
    // that of (hi, lo) is [A -m; m^T C]
    const int lo = min(i, j), hi = max(i, j), I = lo / kT, J = hi / kT, a = lo % kT, bb = hi % kT;
    int plane;
    double sign = 1.0;
    if (c < 3 && d < 3) {
        const int l = min(c, d), h = max(c, d);
        plane = l == 0 ? h : (l == 1 ? 2 + h : 5);
    } else if (c == 3 && d == 3) {
        plane = 9;
    } else {
        plane = 6 + (c < 3 ? c : d);
        sign = (c == 3) == (i < j) ? -1.0 : 1.0;
    }
    const size_t t = (size_t)I * A.nT - (size_t)I * (I - 1) / 2 + (size_t)(J - I);
    return sign * __ldg(A.tiles + t * (kPlanes * kT * kT) + ((size_t)(plane * (kT / 4) + (bb >> 2))) * (kT * 4) +
                        a * 4 + (bb & 3));
}

// K sums over the block, the same in every thread (fixed order); false when
// a thread of the block calls with bad set.
template <int K>
__device__ __forceinline__ bool sum_all(double (&v)[K], double (*sh)[8], bool bad)
{
    static_assert(K <= 8, "the shared rows hold eight sums");
    constexpr int V = K == 1 ? 1 : (K == 2 ? 2 : 8);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double u[V];
#pragma unroll
    for (int k = 0; k < V; ++k) u[k] = k < K ? v[k] : 0.0;
    const double s = warp_sum_halving<V>(u, lane);
    constexpr int kStep = 32 / V;
    if (lane % kStep == 0) sh[w][lane / kStep] = s;
    if (__syncthreads_or(bad)) return false;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double t[kWarps];
#pragma unroll
        for (int q = 0; q < kWarps; ++q) t[q] = sh[q][k];
        v[k] = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    }
    return true;
}

// A bounded wait has run out: the other blocks' polls end, the host is told.
__device__ __forceinline__ void give_up(const DenseArgs &A)
{
    atomicExch(&A.ss->error, 1);
    *(volatile int *)&A.out->error = 1;
}

// Store the block's kR values (thread q < kR holds row q) for exchange seq.
__device__ __forceinline__ void publish(const DenseArgs &A, double v, unsigned seq)
{
    if (threadIdx.x < kR)
        st_value(A.ex + ((size_t)(seq & 1) * gridDim.x + blockIdx.x) * kSeg + threadIdx.x, v, seq);
}

// This block's rows of a product, from each thread's partial sums, stored for
// exchange seq.
__device__ __forceinline__ void publish_sums(const DenseArgs &A, const double (&part)[kR], double (*sh)[16],
                                             unsigned seq)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double acc[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) acc[r] = r < kR ? part[r] : 0.0;
    const double s = warp_sum_halving<16>(acc, lane);
    if ((lane & 1) == 0) sh[w][lane >> 1] = s;
    __syncthreads();
    if (threadIdx.x < kR) {
        double t[kWarps];
#pragma unroll
        for (int q = 0; q < kWarps; ++q) t[q] = sh[q][threadIdx.x];
        publish(A, ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7])), seq);
    }
}

// This thread's elements of exchange seq, `since` the clock at the block's own
// store; true when a poll gave up.
template <int C>
__device__ __forceinline__ bool receive(const DenseArgs &A, double (&out)[C], unsigned seq, long long since)
{
    const ulonglong2 *src = A.ex + (size_t)(seq & 1) * gridDim.x * kSeg;
    ulonglong2 q[C];
    while (clock64() - since < kFirstRead) {}
#pragma unroll
    for (int m = 0; m < C; ++m) {
        const int e = threadIdx.x + kBlock * m;
        if (e < A.n) q[m] = ld_pair(src + (e / kR) * kSeg + e % kR);
    }
    bool all = false, bad = false;
    long spins = 1;
    while (!all && !bad) {
        all = true;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const int e = threadIdx.x + kBlock * m;
            if (e < A.n && !arrived(q[m], seq)) {
                all = false;
                q[m] = ld_pair(src + (e / kR) * kSeg + e % kR);
            }
        }
        if (!all) {
            if (++spins > A.spin_limit) {
                give_up(A);
                bad = true;
            } else if ((spins & 63) == 0 && *(volatile int *)&A.ss->error != 0) {
                bad = true;
            }
        }
    }
#pragma unroll
    for (int m = 0; m < C; ++m) out[m] = threadIdx.x + kBlock * m < A.n ? value_of(q[m]) : 0.0;
    return bad;
}

// BJ: the mixed path's mode (see the head of the file).
template <int C, bool BJ>
__global__ void __launch_bounds__(kBlock, 1) k_bicgstab_dense(const __grid_constant__ DenseArgs A)
{
    // BJ: the block's rows of A (ld = n rounded up to even), then the ring of
    // inverse-block rows
    extern __shared__ __align__(128) double Asm[];
    constexpr int kStages = stages(C);
    __shared__ __align__(8) uint64_t bars[kStages];
    __shared__ double psh[kWarps][16];             // products
    __shared__ double vsh[kWarps][8];              // dots after the first product of an iteration
    __shared__ double tsh[kWarps][8];              // dots after the second
    __shared__ double r0s[C][kBlock], xs[C][kBlock];  // each thread's own elements
    __shared__ double us[BJ ? C : 1][kBlock];
    const int tid = threadIdx.x, n = A.n, row0 = blockIdx.x * kR;
    const int n4 = 4 * A.M, ld = (n + 1) & ~1;
    unsigned seq = A.seq;
    bool ok = true, broke = false;

    // row of the reference layout of internal unknown e, -1 for padding
    auto ref_row = [&](int e) {
        if (e >= n4) return 4 * A.M + (e - n4);
        const int at = BJ ? A.g_atoms[e >> 2] : e >> 2;
        return at < 0 ? -1 : ((e & 3) < 3 ? 3 * at + (e & 3) : 3 * A.M + at);
    };
    double a[kR][C], r[C], p[C], v[C], y[C];
    double d2[2] = {0.0, 0.0};
#pragma unroll
    for (int m = 0; m < C; ++m) {
        const int e = tid + kBlock * m;
        const int rr = e < n ? ref_row(e) : -1;
        const double bk = rr >= 0 ? A.b[rr] : 0.0;
        double xk = rr >= 0 ? A.x[rr] : 0.0;
        if (BJ && A.hist && rr >= 0) {  // polynomial extrapolation of the last solutions (k_predict)
            const size_t nm = 4 * (size_t)A.M + A.n_nps;
            const double h1 = A.hist[rr], h2 = A.hist[nm + rr], h3 = A.hist[2 * nm + rr];
            if (A.order == 1) xk = 2.0 * xk - h1;
            else if (A.order == 2) xk = 3.0 * (xk - h1) + h2;
            else if (A.order == 3) xk = 4.0 * (xk + h2) - 6.0 * h1 - h3;
        }
        xs[m][tid] = xk;
        r[m] = bk;
        y[m] = xk;
        p[m] = v[m] = 0.0;
        d2[0] += bk * bk;
        d2[1] += xk != 0.0 ? 1.0 : 0.0;
    }
    sum_all<2>(d2, vsh, false);
    const double bTb = d2[0], crit = bTb * A.tol;
    double rTr = 0.0, rr0 = 0.0;
    int iter = 0, status = 0, sweep = 0;
    bool done = bTb < A.skip;  // zero right-hand side: x stays (bicg_stab.c:303-307)
#pragma unroll
    for (int m = 0; m < C; ++m) {
        const int e = tid + kBlock * m;
#pragma unroll
        for (int q = 0; q < kR; ++q)
            a[q][m] = !BJ && !done && e < n && row0 + q < n ? tile_entry(A, row0 + q, e) : 0.0;
    }

    if (BJ && !done) {
        // K's blocks stream through a ring of kStages slots of kStageRows rows
        // of two groups (the two halves of the threads work on one each);
        // step t holds the rows kStageRows (t % kStepsPerPair) .. of groups
        // 2 (t / kStepsPerPair) and the next
        float *ring = reinterpret_cast<float *>(Asm + (size_t)kR * ld);
        const int steps = (A.nG + 1) / 2 * kStepsPerPair;
        auto issue = [&](int t) {
            const int g = 2 * (t / kStepsPerPair), c0 = t % kStepsPerPair * kStageRows, st = t % kStages;
            const int two = g + 1 < A.nG ? 2 : 1;
            constexpr unsigned bytes = kStageRows * kGroup * sizeof(float);
            mbar_expect(bars + st, two * bytes);
            for (int h = 0; h < two; ++h)
                bulk_copy(ring + (size_t)(2 * st + h) * kStageRows * kGroup,
                          A.dinv + ((size_t)(g + h) * kGroup + c0) * kGroup, bytes, bars + st);
        };
        if (tid == 0) {
            for (int st = 0; st < kStages; ++st) mbar_init(bars + st);
            mbar_init_fence();
            for (int t = 0; t < min(kStages, steps); ++t) issue(t);
        }
        // the block's rows of A: its atoms against every atom, the constraint
        // rows and columns
        const int slots = A.M;
        for (int q = tid; q < kR / 4 * slots; q += kBlock) {
            const int s = q / slots, j = q % slots, is = row0 / 4 + s;
            const int ia = is < slots ? A.g_atoms[is] : -1, ja = A.g_atoms[j];
            double e[16];
            if (ia >= 0 && ja >= 0) {
                cpim_block(A.P, A.pos4[A.metal_min + ia], A.pos4[A.metal_min + ja], ia == ja, e);
            } else {
#pragma unroll
                for (int k = 0; k < 16; ++k) e[k] = 0.0;
            }
            if (is < slots)
#pragma unroll
                for (int k = 0; k < 16; ++k) Asm[(4 * s + k / 4) * ld + 4 * j + k % 4] = e[k];
        }
        for (int q = 0; q < kR; ++q) {
            const int row = row0 + q;
            if (row < n4) {
                for (int k = tid; k < ld - n4; k += kBlock)
                    Asm[q * ld + n4 + k] = k < A.n_nps && (row & 3) == 3 && A.slot_np[row >> 2] == k ? 1.0 : 0.0;
            } else {
                for (int e = tid; e < ld; e += kBlock)
                    Asm[q * ld + e] = row < n && e < n4 && (e & 3) == 3 && A.slot_np[e >> 2] == row - n4 ? 1.0 : 0.0;
            }
        }
        __syncthreads();
        // rows of B = A K into the registers: thread (half h, o) of the block
        // forms column o of group 2 m + h, which is its element of index m;
        // dinv[g][c][o] is the entry (c, o) of K's block g.  The last group may
        // be short; the constraint columns (K = 1) follow it.
        const int o = tid & (kGroup - 1), h = tid / kGroup;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const int g = 2 * m + h, e = tid + kBlock * m;
            const double *col = Asm + g * kGroup;
            for (int t = m * kStepsPerPair; t < min((m + 1) * kStepsPerPair, steps); ++t) {
                const int st = t % kStages, c0 = t % kStepsPerPair * kStageRows, left = n4 - (g * kGroup + c0);
                const bool late = !mbar_wait(bars + st, (t / kStages) & 1);
                const float *K = ring + (size_t)(2 * st + h) * kStageRows * kGroup + o;
#pragma unroll
                for (int c = 0; c < kStageRows; c += 2) {
                    if (c >= left) continue;  // n4 is a multiple of 4; the same for the whole warp
                    const double k0 = (double)K[c * kGroup], k1 = (double)K[(c + 1) * kGroup];
#pragma unroll
                    for (int q = 0; q < kR; ++q) {
                        const double2 w = *reinterpret_cast<const double2 *>(col + q * ld + c0 + c);
                        a[q][m] = fma(w.x, k0, fma(w.y, k1, a[q][m]));
                    }
                }
                if (__syncthreads_or(late)) {
                    // the copies in flight land in this block's shared memory:
                    // wait for them (bounded) before leaving
                    if (tid == 0) {
                        give_up(A);
                        for (int u = t; u < min(t + kStages, steps); ++u) mbar_wait(bars + u % kStages, (u / kStages) & 1);
                    }
                    return;
                }
                if (tid == 0 && t + kStages < steps) issue(t + kStages);
            }
            if (e >= n4)
#pragma unroll
                for (int q = 0; q < kR; ++q) a[q][m] = e < n ? Asm[q * ld + e] : 0.0;
        }
    }

    // K of the FP64 path: the inverse diagonal, 1 on the constraint rows
    const double kp = 1.0 / A.inv_polar, kq = -1.0 / A.inv_capac;
    auto K = [&](int m) {
        if (BJ) return 1.0;
        const int e = tid + kBlock * m;
        return e >= n4 ? 1.0 : ((e & 3) < 3 ? kp : kq);
    };
    // out = A in (BJ: the matrix itself, from shared memory) or the matrix in registers
    auto product = [&](const double(&in)[C], bool matrix, long long &since) {
        double acc[kR];
#pragma unroll
        for (int q = 0; q < kR; ++q) acc[q] = 0.0;
        if (BJ && matrix) {
#pragma unroll
            for (int m = 0; m < C; ++m) {
                const int e = tid + kBlock * m;
                if (e < n)
#pragma unroll
                    for (int q = 0; q < kR; ++q) acc[q] = fma(Asm[q * ld + e], in[m], acc[q]);
            }
        } else {
#pragma unroll
            for (int m = 0; m < C; ++m)
#pragma unroll
                for (int q = 0; q < kR; ++q) acc[q] = fma(a[q][m], in[m], acc[q]);
        }
        publish_sums(A, acc, psh, seq);
        since = clock64();
    };
    long long since = 0;

    double rho = 0.0;
    if (!done) {
        if (d2[1] == 0.0) {
            rho = bTb;  // r = b - A 0
        } else {
            product(y, true, since);
            double ax[C], s[1] = {0.0};
            const bool bad = receive<C>(A, ax, seq, since);
            ++seq;
#pragma unroll
            for (int m = 0; m < C; ++m) {
                r[m] -= ax[m];
                s[0] = fma(r[m], r[m], s[0]);
            }
            ok = sum_all<1>(s, tsh, bad);
            rho = s[0];
        }
        rTr = rr0 = rho;
        if (BJ ? rTr <= crit : rho < A.skip) done = true;  // warm start already converged (bicg_stab.c:368)
    }
    while (ok && !done) {  // sweeps; on the FP64 path starts, a second one only after a breakdown
        const double goal = BJ ? 0.25 * crit : crit;
        double rho_old = 1.0, alpha = 1.0, omega = 1.0, mark = rTr;
        int it = 0, gain = 0;
        bool end = false;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            r0s[m][tid] = r[m];
            if (BJ) us[BJ ? m : 0][tid] = 0.0;
        }
        while (!end) {
            const double beta = (rho / rho_old) * (alpha / omega);
#pragma unroll
            for (int m = 0; m < C; ++m) {
                p[m] = it == 0 ? r[m] : fma(beta, fma(-omega, v[m], p[m]), r[m]);
                y[m] = K(m) * p[m];
            }
            product(y, false, since);
            bool bad = receive<C>(A, v, seq, since);
            ++seq;
            double r0v[1] = {0.0};
#pragma unroll
            for (int m = 0; m < C; ++m) r0v[0] = fma(r0s[m][tid], v[m], r0v[0]);
            if (!sum_all<1>(r0v, vsh, bad)) {
                ok = false;
                break;
            }
            const double al = rho / r0v[0];
            if (!isfinite(al)) {  // breakdown: x is the start of this iteration
                status = rTr < crit * 100.0 ? 1 : -2;
                broke = true;
                break;
            }
            alpha = al;
#pragma unroll
            for (int m = 0; m < C; ++m) {
                r[m] = fma(-alpha, v[m], r[m]);  // s
                y[m] = K(m) * r[m];              // z
            }
            product(y, false, since);
            double t[C];
            bad = receive<C>(A, t, seq, since);
            ++seq;
            double d[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int m = 0; m < C; ++m) {
                const double kt = K(m) * t[m], r0 = r0s[m][tid];
                d[0] = fma(kt, y[m], d[0]);
                d[1] = fma(kt, kt, d[1]);
                d[2] = fma(r0, r[m], d[2]);
                d[3] = fma(r0, t[m], d[3]);
                d[4] = fma(r[m], r[m], d[4]);
                d[5] = fma(r[m], t[m], d[5]);
                d[6] = fma(t[m], t[m], d[6]);
            }
            if (!sum_all<7>(d, tsh, bad)) {
                ok = false;
                break;
            }
            const double om = d[0] / d[1];
            if (!isfinite(om) || om == 0.0) {
                status = rTr < crit * 100.0 ? 1 : -2;
                broke = true;
                break;
            }
            omega = om;
            rho_old = rho;
            rho = fma(-omega, d[3], d[2]);
            rTr = fma(omega * omega, d[6], fma(-2.0 * omega, d[5], d[4]));
#pragma unroll
            for (int m = 0; m < C; ++m) {
                double &acc = BJ ? us[BJ ? m : 0][tid] : xs[m][tid];
                acc += alpha * (K(m) * p[m]) + omega * y[m];
                r[m] = fma(-omega, t[m], r[m]);
            }
            ++it;
            ++iter;
            if (rTr < goal) {
                end = true;
            } else if (it > A.max_iter) {
                status = rTr < crit * 100.0 ? 1 : -1;
                end = true;
            } else if (BJ) {
                if (rTr < 0.5 * mark) {
                    mark = rTr;
                    gain = it;
                } else if (it - gain >= kStall) {
                    end = true;
                }
            }
        }
        if (!ok) break;
        if (!BJ) {
            // a breakdown leaves x at its last finite value: start again from
            // there with a fresh shadow residual (the reference would carry the
            // NaN to MAX_ITER); only an exact zero now ends it early
            ++sweep;
            if (!broke || status != -2 || sweep == kStarts) break;
            broke = false;
            status = 0;
#pragma unroll
            for (int m = 0; m < C; ++m) y[m] = xs[m][tid];
            product(y, true, since);
            const bool bad = receive<C>(A, y, seq, since);
            ++seq;
            double s[1] = {0.0};
#pragma unroll
            for (int m = 0; m < C; ++m) {
                const int e = tid + kBlock * m, rr = e < n ? ref_row(e) : -1;
                r[m] = rr >= 0 ? A.b[rr] - y[m] : 0.0;
                s[0] = fma(r[m], r[m], s[0]);
            }
            ok = sum_all<1>(s, tsh, bad);
            rTr = rho = s[0];
            done = rho < 1.0e-300;
            continue;
        }
        // x += K u: the block's rows of K u, one warp per row, then the new x
        // to every block and its residual from the matrix itself
        if (it == 0) break;  // no progress possible
        ++sweep;
        status = 0;
        __syncthreads();
        double *uf = &us[0][0];  // us[m][tid] is element tid + 256 m
        for (int q = tid >> 5; q < kR; q += kWarps) {
            const int row = row0 + q, lane = tid & 31;
            double s = 0.0;
            if (row < n4) {
                const int g = row / kGroup, c = row % kGroup;
                const float *Kr = A.dinv + ((size_t)g * kGroup + c) * kGroup;
                for (int k = lane; k < min(kGroup, n4 - g * kGroup); k += 32)
                    s = fma((double)__ldg(Kr + k), uf[g * kGroup + k], s);
            } else if (row < n && lane == 0) {
                s = uf[row];
            }
            s = warp_sum(s);
            if (lane == 0) psh[0][q] = s;
        }
        __syncthreads();
        if (tid < kR) publish(A, psh[0][tid], seq);
        since = clock64();
        bool bad = receive<C>(A, y, seq, since);
        ++seq;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            xs[m][tid] += y[m];
            y[m] = xs[m][tid];
        }
        if (__syncthreads_or(bad)) {
            ok = false;
            break;
        }
        product(y, true, since);
        bad = receive<C>(A, y, seq, since);
        ++seq;
        double s[1] = {0.0};
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const int e = tid + kBlock * m, rr = e < n ? ref_row(e) : -1;
            r[m] = rr >= 0 ? A.b[rr] - y[m] : 0.0;
            s[0] = fma(r[m], r[m], s[0]);
        }
        ok = sum_all<1>(s, vsh, bad);
        rTr = rho = s[0];
        done = rTr <= crit || sweep == kSweeps || !isfinite(rTr);
        if (done && !(rTr <= crit)) status = rTr < crit * 100.0 ? 1 : -1;
    }
    if (!ok) return;
    if (!BJ && iter > 0 && !broke) {  // (r, r) of the final residual, summed directly
        double s[1] = {0.0};
#pragma unroll
        for (int m = 0; m < C; ++m) s[0] = fma(r[m], r[m], s[0]);
        sum_all<1>(s, vsh, false);
        rTr = s[0];
    }
    if (blockIdx.x == 0) {
        // every block has read x and the history before its first exchange
        const bool moved = iter > 0, predicted = BJ && A.hist && bTb >= A.skip;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const int e = tid + kBlock * m, rr = e < n ? ref_row(e) : -1;
            if (rr < 0) continue;
            if (predicted) {
                const size_t nm = 4 * (size_t)A.M + A.n_nps;
                A.hist[2 * nm + rr] = A.hist[nm + rr];
                A.hist[nm + rr] = A.hist[rr];
                A.hist[rr] = A.x[rr];
            }
            if (moved || predicted) A.x[rr] = xs[m][tid];
        }
        if (tid == 0) {
            // as settle_solve decides it
            if (BJ) A.ss->failed = bTb >= A.skip && (status < 0 || !(rTr <= crit)) && !(rTr < 1.0e-8 * bTb);
            else A.ss->failed = status < 0;
            volatile SolverScalars *ss = A.out;
            ss->bTb = bTb;
            ss->crit = crit;
            ss->rTr = rTr;
            ss->rr0 = rr0;
            ss->iter = iter;
            ss->done = 1;
            ss->status = status;
            ss->outer = sweep;
        }
    }
}

// The kernel for n unknowns on `sms` SMs, null when the matrix does not fit.
const void *dense_kernel(int n, int sms, bool bj)
{
    if ((n + kR - 1) / kR > sms) return nullptr;
    switch ((n + kBlock - 1) / kBlock) {
    case 1: return bj ? (const void *)k_bicgstab_dense<1, true> : (const void *)k_bicgstab_dense<1, false>;
    case 2: return bj ? (const void *)k_bicgstab_dense<2, true> : (const void *)k_bicgstab_dense<2, false>;
    case 3: return bj ? (const void *)k_bicgstab_dense<3, true> : (const void *)k_bicgstab_dense<3, false>;
    case 4:
    case 5: return bj ? (const void *)k_bicgstab_dense<5, true> : (const void *)k_bicgstab_dense<5, false>;
    case 6:
    case kMaxCols: return bj ? (const void *)k_bicgstab_dense<7, true> : (const void *)k_bicgstab_dense<7, false>;
    default: return nullptr;
    }
}

size_t dense_smem(int n, bool bj)
{
    const int c = (n + kBlock - 1) / kBlock;
    return bj ? sizeof(double) * kR * ((n + 1) & ~1) + sizeof(float) * 2 * stages(c) * kStageRows * kGroup : 0;
}

}  // namespace

// Whether the system's FP64 matrix fits the chip.
bool dense_fits(int device, int n, bool mixed)
{
    int coop = 0, sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop) return false;
    CAPAC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const void *k = dense_kernel(n, sms, mixed);
    if (!k) return false;
    // The limit on a launch's dynamic shared memory belongs to the kernel, which
    // contexts of other sizes launch too: all that a block can have, not this
    // system's need, so that creating one context takes nothing from another.
    const size_t smem = dense_smem(n, mixed);
    int most = 0;
    cudaFuncAttributes fa{};
    CAPAC_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    if (cudaFuncGetAttributes(&fa, k) != cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kBlock, smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return per_sm >= 1;
}

size_t dense_exchange_bytes(int n) { return (size_t)2 * ((n + kR - 1) / kR) * kSeg * sizeof(ulonglong2); }

// One launch: a solve on the FP64 path's tiles; on the mixed path the whole
// refined solve (hist set: with the warm-start predictor) to (r, r) <= tol
// (b, b), the residual from the positions.  The status as bicgstab_core
// returns it.
// `defer`: without waiting for it (dense_status reads it later).
int bicgstab_dense(capac_ctx *c, const double *b, double *x, double tol, double skip, double *hist, int order,
                   bool defer)
{
    const bool mixed = c->opt.precision == CAPAC_PREC_MIXED;
    DenseArgs A;
    A.M = c->M;
    A.n = c->n_mat;
    A.n_nps = c->n_nps;
    A.metal_min = c->P.metal_min;
    A.max_iter = solver_max_iter(c);
    A.nT = sym_tiles(c->M);
    A.spin_limit = c->opt.wait_polls > 0 ? c->opt.wait_polls : kPollLimit;
    A.inv_polar = c->P.inv_polar;
    A.inv_capac = c->P.inv_capac;
    A.tol = tol;
    A.skip = skip;
    A.np_start = c->np_start;
    A.np_end = c->np_end;
    A.tiles = mixed ? nullptr : static_cast<const double *>(c->msym);
    A.b = b;
    A.x = x;
    A.ex = static_cast<ulonglong2 *>(c->dense_ex);
    A.ss = c->ss;
    A.out = c->h_ss;
    A.P = c->P;
    A.pos4 = c->pos4;
    A.g_atoms = c->g_atoms;
    A.slot_np = c->slot_np;
    A.dinv = c->dinv;
    A.nG = mixed ? precond_groups(c->M) : 0;
    A.hist = hist;
    A.order = order;
    // two exchanges per iteration, two per sweep or start; the
    // numbers of a launch are not used again until they wrap, when the buffers
    // are cleared
    const unsigned long long need = 2ull * ((unsigned long long)A.max_iter + 4) * (mixed ? kSweeps : kStarts) + 2;
    if (c->dense_seq + need > 0xffffffffull) {
        CAPAC_CUDA(cudaMemsetAsync(c->dense_ex, 0, dense_exchange_bytes(A.n), c->stream));
        c->dense_seq = 1;
    }
    A.seq = (unsigned)c->dense_seq;
    c->dense_seq += need;
    void *args[] = {&A};
    {
        ProfScope ps(c, K_SOLVE);
        CAPAC_CUDA(cudaLaunchCooperativeKernel(dense_kernel(A.n, c->num_sms, mixed), dim3((A.n + kR - 1) / kR),
                                               dim3(kBlock), args, dense_smem(A.n, mixed), c->stream));
    }
    ++c->launches;
    if (defer) {
        CAPAC_CUDA(cudaEventRecord(c->ev_solve, c->stream));
        return CAPAC_OK;
    }
    CAPAC_CUDA(cudaStreamSynchronize(c->stream));
    return dense_status(c, skip);
}

int dense_status(capac_ctx *c, double skip)
{
    if (c->h_ss->error) {
        c->h_ss->error = 0;
        CAPAC_CUDA(cudaMemsetAsync(&c->ss->error, 0, sizeof(int), c->stream));
        throw Error(CAPAC_ERR_CUDA, "persistent solver: a bounded wait timed out");
    }
    if (c->prof.on && c->h_ss->bTb >= skip) c->prof.spmv_effective += 1 + 2L * c->h_ss->iter;
    if (c->h_ss->status < 0) return CAPAC_ERR_NOT_CONVERGED;
    return c->h_ss->status == 1 ? 1 : CAPAC_OK;
}

}  // namespace capac
