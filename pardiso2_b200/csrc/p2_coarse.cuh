// The coarsest level's direct solve as two kernels: the stored inverse (from
// p2_lu.cu) times the free unknowns' right-hand side, with the columns split
// over the grid's y, and the sum of the partial products written back over the
// whole level (the reference calls MKL PARDISO here,
// gaus3mg_SerieMG.c:170-216).
#pragma once

#include "p2_kernels.cuh"

namespace p2 {

template <typename T>
struct GemvVec;
template <>
struct GemvVec<float> {
    using V = float4;
    static constexpr int kN = 4;
};
template <>
struct GemvVec<double> {
    using V = double2;
    static constexpr int kN = 2;
};
constexpr int kGemvWarps = 8;
template <typename T>
constexpr int gemv_rows() { return 32 * GemvVec<T>::kN; }

// Splits of the columns so that about four blocks per SM share the matrix: one
// block per 32 rows left its columns to 8 warps and read a 53 MB inverse at
// 0.7 TB/s (73 us); split 21 ways it takes 14 us (3.7 TB/s), cold caches both.
template <typename T>
inline int gemv_splits(int n)
{
    const int groups = (n + gemv_rows<T>() - 1) / gemv_rows<T>();
    int s = (4 * 148 + groups - 1) / groups;
    s = s < 1 ? 1 : (s > 32 ? 32 : s);
    const int room = (int)((sizeof(T) * (size_t)n + 32767) / 32768);  // a split's right-hand side in 32 KB
    return s > room ? s : room;
}

// part[s][r] = sum of Ainv[r][c] b_c over the columns of split s (Ainv
// column-major n x n, n a multiple of the vector width); b_c is the
// right-hand side of the unknown of slot c (-1: 0).  Each lane holds one
// vector of adjacent rows.
template <typename T>
__global__ void __launch_bounds__(32 * kGemvWarps) k_gemv_split(int n, const T *__restrict__ A, const int *slots, Vec4<T> b,
                                                                T *part, int chunk)
{
    pdl_enter();
    using V = typename GemvVec<T>::V;
    constexpr int kN = GemvVec<T>::kN;
    extern __shared__ unsigned char smem_gemv[];
    T *bs = (T *)smem_gemv;
    __shared__ T red[kGemvWarps][gemv_rows<T>()];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c0 = blockIdx.y * chunk, c1 = min(n, c0 + chunk);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        const int uc = slots[c];
        bs[c - c0] = uc >= 0 ? b.c[uc & 3][uc >> 2] : (T)0;
    }
    __syncthreads();
    const int r = blockIdx.x * gemv_rows<T>() + lane * kN;
    T s[kN] = {};
    if (r < n) {
        const T *a = A + r;
#pragma unroll 8
        for (int c = c0 + w; c < c1; c += kGemvWarps) {
            const V v = __ldg((const V *)(a + (size_t)c * n));
            const T x = bs[c - c0];
            const T *e = (const T *)&v;
#pragma unroll
            for (int q = 0; q < kN; q++) s[q] += e[q] * x;
        }
    }
#pragma unroll
    for (int q = 0; q < kN; q++) red[w][lane * kN + q] = s[q];
    __syncthreads();
    for (int q = threadIdx.x; q < gemv_rows<T>(); q += blockDim.x) {
        const int row = blockIdx.x * gemv_rows<T>() + q;
        if (row >= n) continue;
        T t = 0;
#pragma unroll
        for (int v = 0; v < kGemvWarps; v++) t += red[v][q];
        part[(size_t)blockIdx.y * n + row] = t;
    }
}

// x over the whole level (4 nn unknowns): the sum of the partial products of
// its slot, or 0 where it has none.
template <typename T>
__global__ void k_coarse_write(int nn, int n, int splits, const int *slot_of, const T *part, Vec4<T> x)
{
    pdl_enter();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * nn) return;
    const int c = t / nn, u = t - c * nn;
    const int q = slot_of[u * 4 + c];
    T s = 0;
    if (q >= 0) {
#pragma unroll 8
        for (int p = 0; p < splits; p++) s += part[(size_t)p * n + q];
    }
    (c == 0 ? x.c[0] : (c == 1 ? x.c[1] : (c == 2 ? x.c[2] : x.c[3])))[u] = s;
}

}  // namespace p2
