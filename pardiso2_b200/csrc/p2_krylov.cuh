// Vector kernels of the FP64 outer loop (flexible GMRES on the level-0
// system): dot products of the new vector with the stored basis, the
// orthogonalisation and the solution update.
//
// Vectors are the four level-0 fields in one allocation, read as 2 n pairs of
// doubles.  The basis is orthogonal but not normalised: ww[j] = (W_j, W_j).
// Per outer iteration with k + 1 stored vectors k_basis_dots reads k + 2
// vectors and k_basis_update reads k + 2 and writes one (and its copy for the
// V-cycle), all bound by HBM; the preconditioned vectors are read only once
// per restart, by k_basis_axpy.  16-byte loads, all loads of a pair
// independent of each other; the grid is fixed by the vector length, each
// block's partial sums are added in block order by the last block, so the
// sums do not depend on scheduling.  At 257^3 (543 MB a vector) with 4 / 8 /
// 12 / 16 stored vectors the dots take 0.40 / 0.87 / 0.97 / 1.28 ms (6.8 /
// 5.6 / 7.3 / 7.2 TB/s) and the update 0.53 / 1.09 / 1.18 / 2.03 ms (6.7 /
// 5.2 / 6.7 / 5.0 TB/s).
#pragma once

#include "p2_internal.cuh"

namespace p2 {

constexpr int kMaxBasis = 19;  // restart length (at most 18) + 1
constexpr int kBasisThreads = 256;

struct Basis {
    const double2 *v[kMaxBasis];
};

// hcol: h_0 .. h_{k}, then these (HC_ERROR: set by a smoother whose barrier ran out of time)
enum { HC_SIGMA = kMaxBasis, HC_QQ, HC_WW, HC_ERROR, HC_LEN };

inline unsigned basis_blocks(long n2, int u)
{
    const long b = (n2 + u * kBasisThreads - 1) / (u * kBasisThreads);
    return (unsigned)(b < kRedBlocks ? b : kRedBlocks);
}
// Pairs per thread and tile of k_basis_update: four (each block then reads
// 16 KB of a vector before the next one's turn; one pair at a time the same
// update took 2.69 against 1.18 ms with 12 vectors at 257^3) on vectors of at
// least four tiles per SM, one below, where the blocks would not fill the
// device.  The dots gain nothing from it (1.21 against 1.57 ms with 14).
inline int basis_unroll(long n2) { return n2 >= 4L * 148 * 4 * kBasisThreads ? 4 : 1; }

// Sum NS values over the block; the totals of block 0..gridDim-1 are added in
// that order by the last block to finish, which gets true and the sums in tot.
template <int NS>
__device__ __forceinline__ bool basis_reduce(double (&acc)[NS], double *partial, unsigned *ticket, double *tot)
{
    constexpr int kW = kBasisThreads / 32;
    __shared__ double sh[kW][NS];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < NS; j++) {
        double v = acc[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[w][j] = v;
    }
    __syncthreads();
    if (threadIdx.x < NS) {
        double v = 0;
#pragma unroll
        for (int q = 0; q < kW; q++) v += sh[q][threadIdx.x];
        partial[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = v;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    for (int j = w; j < NS; j += kW) {
        double v = 0;
        for (int q = lane; q < (int)gridDim.x; q += 32) v += __ldcg(partial + (size_t)j * gridDim.x + q);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) tot[j] = v;
    }
    if (threadIdx.x == 0) *ticket = 0;
    __syncthreads();
    return true;
}

// (q, W_j) for j < ND and (q, q), without the pinned pressure cell (flat
// index skip, -1 none).  ND = 0: hcol[HC_QQ] = ww[0] = (q, q).  ND > 0: also the
// coefficients h_j = (q, W_j) / (W_j, W_j) and the scale sigma that gives the
// orthogonalised vector about the norm of W_0, from the Pythagorean estimate
// of its norm (any sigma is exact, the true norm is summed in k_basis_update;
// it keeps the V-cycle's right-hand sides at one magnitude, as FP32 wants).
template <int ND>
__global__ void __launch_bounds__(kBasisThreads) k_basis_dots(long n2, const double2 *__restrict__ q, Basis W,
                                                              long skip, double *partial, unsigned *ticket,
                                                              double *ww, double *hcol)
{
    constexpr int U = ND <= 1 ? 4 : (ND <= 5 ? 2 : 1);
    __shared__ double tot[ND + 1];
    double acc[ND + 1];
#pragma unroll
    for (int j = 0; j <= ND; j++) acc[j] = 0;
    const long stride = (long)gridDim.x * kBasisThreads, skip2 = skip >= 0 ? skip >> 1 : -1;
#pragma unroll U
    for (long i = (long)blockIdx.x * kBasisThreads + threadIdx.x; i < n2; i += stride) {
        double2 a = __ldg(q + i);
        double2 b[ND > 0 ? ND : 1];
#pragma unroll
        for (int j = 0; j < ND; j++) b[j] = __ldg(W.v[j] + i);
        if (i == skip2) {
            if (skip & 1) a.y = 0;
            else a.x = 0;
        }
#pragma unroll
        for (int j = 0; j < ND; j++) acc[j] += a.x * b[j].x + a.y * b[j].y;
        acc[ND] += a.x * a.x + a.y * a.y;
    }
    if (!basis_reduce<ND + 1>(acc, partial, ticket, tot)) return;
    if (threadIdx.x == 0) {
        const double qq = tot[ND];
        hcol[HC_QQ] = qq;
        if (ND == 0) {
            ww[0] = qq;
            return;
        }
        double rest = qq;
        for (int j = 0; j < ND; j++) {
            const double h = tot[j] / ww[j];
            hcol[j] = h;
            rest -= h * tot[j];
        }
        rest = fmax(rest, 1e-12 * qq);
        hcol[HC_SIGMA] = qq > 0 ? sqrt(ww[0] / rest) : 0.0;
    }
}

// w = sigma (q - sum_j h_j W_j) in place of q, its copy for the V-cycle
// (rhs, the cycle's type) and ww[ND] = hcol[HC_WW] = (w, w).
template <int ND, int U, typename S2>
__global__ void __launch_bounds__(kBasisThreads) k_basis_update(long n2, double2 *__restrict__ q, Basis W,
                                                                S2 *__restrict__ rhs, long skip, double *partial,
                                                                unsigned *ticket, double *ww, double *hcol)
{
    __shared__ double tot[1];
    double h[ND];
#pragma unroll
    for (int j = 0; j < ND; j++) h[j] = hcol[j];
    const double sigma = hcol[HC_SIGMA];
    double acc[1] = {0};
    const long skip2 = skip >= 0 ? skip >> 1 : -1;
    constexpr int kTileN = U * kBasisThreads;
    for (long t = (long)blockIdx.x * kTileN; t < n2; t += (long)gridDim.x * kTileN) {
        double2 a[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = t + u * kBasisThreads + threadIdx.x;
            a[u] = i < n2 ? q[i] : make_double2(0, 0);
        }
#pragma unroll
        for (int j = 0; j < ND; j++) {
            double2 b[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const long i = t + u * kBasisThreads + threadIdx.x;
                b[u] = i < n2 ? __ldg(W.v[j] + i) : make_double2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                a[u].x -= h[j] * b[u].x;
                a[u].y -= h[j] * b[u].y;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = t + u * kBasisThreads + threadIdx.x;
            if (i >= n2) continue;
            a[u].x *= sigma;
            a[u].y *= sigma;
            q[i] = a[u];
            S2 c;
            c.x = a[u].x;
            c.y = a[u].y;
            rhs[i] = c;
            if (i == skip2) {
                if (skip & 1) a[u].y = 0;
                else a[u].x = 0;
            }
            acc[0] += a[u].x * a[u].x + a[u].y * a[u].y;
        }
    }
    if (!basis_reduce<1>(acc, partial, ticket, tot)) return;
    if (threadIdx.x == 0) ww[ND] = hcol[HC_WW] = tot[0];
}

// x += sum_j y_j Z_j over nv preconditioned vectors stored as pairs S2
template <typename S2>
struct Corrections {
    const S2 *v[kMaxBasis];
    double y[kMaxBasis];
};
template <typename S2>
__global__ void __launch_bounds__(kBasisThreads) k_basis_axpy(long n2, double2 *x, Corrections<S2> Z, int nv)
{
    const long i = (long)blockIdx.x * kBasisThreads + threadIdx.x;
    if (i >= n2) return;
    double2 a = x[i];
#pragma unroll 6
    for (int j = 0; j < nv; j++) {
        const S2 z = __ldg(Z.v[j] + i);
        a.x += Z.y[j] * (double)z.x;
        a.y += Z.y[j] * (double)z.y;
    }
    x[i] = a;
}

#define P2_BASIS_SIZES(X)                                                                                      \
    X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18)

inline cudaError_t launch_basis_dots(cudaStream_t st, int nd, long n2, const double *q, const Basis &W, long skip,
                                     double *partial, unsigned *ticket, double *ww, double *hcol)
{
    switch (nd) {
#define P2_CASE(N)                                                                                         \
    case N:                                                                                                \
        k_basis_dots<N><<<basis_blocks(n2, 1), kBasisThreads, 0, st>>>(n2, (const double2 *)q, W, skip, partial, \
                                                                       ticket, ww, hcol);                  \
        break;
        P2_CASE(0) P2_BASIS_SIZES(P2_CASE)
#undef P2_CASE
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename S2>
inline cudaError_t launch_basis_update(cudaStream_t st, int nd, long n2, double *q, const Basis &W, void *rhs, long skip,
                                       double *partial, unsigned *ticket, double *ww, double *hcol)
{
    switch (nd) {
#define P2_CASE(N)                                                                                             \
    case N:                                                                                                    \
        if (basis_unroll(n2) == 4)                                                                             \
            k_basis_update<N, 4, S2><<<basis_blocks(n2, 4), kBasisThreads, 0, st>>>(n2, (double2 *)q, W, (S2 *)rhs, \
                                                                                    skip, partial, ticket, ww, hcol); \
        else                                                                                                   \
            k_basis_update<N, 1, S2><<<basis_blocks(n2, 1), kBasisThreads, 0, st>>>(n2, (double2 *)q, W, (S2 *)rhs, \
                                                                                    skip, partial, ticket, ww, hcol); \
        break;
        P2_BASIS_SIZES(P2_CASE)
#undef P2_CASE
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace p2
