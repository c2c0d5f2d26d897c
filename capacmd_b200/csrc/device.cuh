// Device-side helpers shared by the kernels of the force-and-solve path.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace capac {

// Physical constants of the reference (typedef.h:44-93, cpff.c:72-75, 758-759).
constexpr double kFQQ = 138.935457696552;
constexpr double kNm2Bohr = 18.8972612456506;
constexpr double kBoltz = 0.00831446214546895;
constexpr double kInvSqrtPi = 0.564189583547756;
constexpr double kThreshold = 1.0e-15;
constexpr double kConvE = 2.01552955019358e-05;
constexpr double kConvV = 3.80879884583368e-04;
constexpr double kFqqAu2 = 49614.7526045429;
constexpr double kFqqAu1 = 2625.49964037578;
constexpr int kMaxIter = 1000;
constexpr int kNhc = 10;

// Rectangular box: edge lengths and half lengths (System.box[6], mpi-main.c:536-538).
struct Box {
    double L[3];
    double H[3];
};

// pbc_12 (force.c:111-121): a single conditional shift per axis.
__device__ __forceinline__ void image(double &x, double &y, double &z, const Box &b)
{
    if (x < -b.H[0]) x += b.L[0]; else if (x > b.H[0]) x -= b.L[0];
    if (y < -b.H[1]) y += b.L[1]; else if (y > b.H[1]) y -= b.L[1];
    if (z < -b.H[2]) z += b.L[2]; else if (z > b.H[2]) z -= b.L[2];
}

// dist_2 (force.c:41-44) with the reference's rounding: (x*x + y*y) + z*z,
// no fused multiply-add, so cut-off decisions match the CPU bit for bit.
__device__ __forceinline__ double norm2_exact(double x, double y, double z)
{
    return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// pbc (force.c:104-109): one conditional shift by the full box length.
__device__ __forceinline__ double wrap1(double dx, double L)
{
    if (dx < -0.5 * L) dx += L; else if (dx > 0.5 * L) dx -= L;
    return dx;
}

__device__ __forceinline__ double keep_entry(double e) { return fabs(e) > kThreshold ? e : 0.0; }

// Deterministic warp sum (fixed butterfly order).
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sumf(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of V values over the 32 lanes of a warp by recursive halving: at
// each step a lane keeps half of its values and adds the partner's copy of
// that half (V/2 + V/4 + ... + 1 exchanges), then plain exchanges for the
// remaining lane bits; V - 1 + 5 - log2 V shuffles instead of 5 V.  Lane l
// returns the sum of value l >> (5 - log2 V).  The order of additions is
// fixed.
template <int V, typename R>
__device__ __forceinline__ R warp_sum_halving(R (&v)[V], int lane)
{
    int m = 16;
#pragma unroll
    for (int half = V / 2; half >= 1; half >>= 1, m >>= 1) {
        const bool upper = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const R send = upper ? v[i] : v[i + half];
            const R keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    R s = v[0];
#pragma unroll
    for (; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    return s;
}

// Warp sums of v[k], k = A .. A + K - 1, into out[k], in groups of a power of two
// (10 values: 8 + 2, 16 shuffles for 50).
template <int A, int K, int N>
__device__ __forceinline__ void warp_sums_to(const double (&v)[N], double *out, int lane)
{
    constexpr int V = K >= 16 ? 16 : (K >= 8 ? 8 : (K >= 4 ? 4 : (K >= 2 ? 2 : 1)));
    double u[V];
#pragma unroll
    for (int k = 0; k < V; ++k) u[k] = v[A + k];
    const double s = warp_sum_halving<V>(u, lane);
    constexpr int kStep = 32 / V;
    if (lane % kStep == 0) out[A + lane / kStep] = s;
    if constexpr (K > V) warp_sums_to<A + V, K - V>(v, out, lane);
}

// Sum K <= 32 values over the block (blockDim.x a multiple of 32, at most 1024)
// in a fixed order; thread 0 receives the totals in v[].  `sh` needs 32*K
// doubles.
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double *sh)
{
    static_assert(K <= 32, "one warp adds the warps' sums");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    warp_sums_to<0, K>(v, sh + wid * K, lane);
    __syncthreads();
    if (wid == 0) {
        if (lane < K) {
            double s = sh[lane];
#pragma unroll 8
            for (int w = 1; w < nw; ++w) s += sh[w * K + lane];
            sh[lane] = s;
        }
        __syncwarp();
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) v[k] = sh[k];
        }
    }
    __syncthreads();
}

// Write a block's K partial sums to partials[blockIdx.x*K + k].
template <int K>
__device__ __forceinline__ void block_partials(double (&v)[K], double *sh, double *partials)
{
    block_sum<K>(v, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) partials[(size_t)blockIdx.x * K + k] = v[k];
    }
}

// Tiles (I <= J) of a symmetric nT x nT tile grid, row-major upper triangle
// including the diagonal.
__host__ __device__ __forceinline__ size_t tile_index(int I, int J, int nT)
{
    return (size_t)I * nT - (size_t)I * (I - 1) / 2 + (size_t)(J - I);
}
// The row I of tile t, J = I + t - tile_index(I, I): from the root of t =
// I (2 nT + 1 - I) / 2 in FP32 (the discriminant is exact before its rounding, so
// the root is within a row or so), then set right.  A search from row 0 took up to
// nT dependent steps, 0.3 us a call at nT = 36.
__device__ __forceinline__ int tile_row(size_t t, int nT)
{
    const long b = 2L * nT + 1;
    int I = (int)(0.5f * ((float)b - sqrtf((float)(b * b - 8 * (long)t))));
    I = I < 0 ? 0 : (I >= nT ? nT - 1 : I);
    while (I > 0 && tile_index(I, I, nT) > t) --I;
    while (I + 1 < nT && tile_index(I + 1, I + 1, nT) <= t) ++I;
    return I;
}

// splitmix64 finaliser, used for order-independent pair-set hashes.
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t x)
{
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}

// Neighbour-list entries carry the atom index in the low 24 bits and the
// atom type in the high 8 bits, so the pair kernel needs no type gather.
constexpr int kIdxBits = 24;
constexpr uint32_t kIdxMask = (1u << kIdxBits) - 1u;
__host__ __device__ __forceinline__ uint32_t pack_nb(int j, int t) { return (uint32_t)j | ((uint32_t)t << kIdxBits); }
__host__ __device__ __forceinline__ int nb_index(uint32_t e) { return (int)(e & kIdxMask); }
__host__ __device__ __forceinline__ int nb_type(uint32_t e) { return (int)(e >> kIdxBits); }

// Cluster-list entries: the j atom in the low 22 bits, in bits 22-25 the mask
// of the cluster members j is a list neighbour of, the j type in bits 26-31.
// In the pair kernel's queue bits 22-23 carry the member instead of the mask.
constexpr int kClIdxBits = 22, kClMaskShift = 22, kClTypeShift = 26;
constexpr uint32_t kClIdxMask = (1u << kClIdxBits) - 1u;
constexpr int kClMaxTypes = 64;
// cluster-pair list: a member slot holds atom | type << kCpTypeShift; an
// entry's second word the 16-bit member-pair mask and kCpMetalBit
constexpr int kCpTypeShift = 24;
constexpr int kCpIdxMask = (1 << kCpTypeShift) - 1;
constexpr uint32_t kCpMetalBit = 1u << 16;
__host__ __device__ __forceinline__ uint32_t pack_cl(int j, unsigned mask, int t)
{
    return (uint32_t)j | (mask << kClMaskShift) | ((uint32_t)t << kClTypeShift);
}

// Minimum image by rounding (any number of box lengths apart).
__device__ __forceinline__ double min_image(double d, double L, double inv_L) { return d - L * rint(d * inv_L); }

}  // namespace capac
