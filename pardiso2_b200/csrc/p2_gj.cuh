// Explicit inverse of the coarsest operator by blocked Gauss-Jordan
// elimination without pivoting (Golub & Van Loan, Matrix Computations), FP64.
//
// The free unknowns are ordered velocities first, then pressures, each by
// z-plane.  The velocity block is definite in the inner product of the control
// volumes and so is the pressures' Schur complement, so no interchanges are
// needed (as the same block of one cell in k_vanka_factor); the caller checks
// the inverse and falls back to the pivoted band LU.  Both parts are padded
// to multiples of kGT with identity rows, so every tile is whole.  Per panel
// of kGT unknowns two launches: k_gj_panel forms D^-1 R and -C D^-1 of the
// panel's rows R and columns C, k_gj_update subtracts C (D^-1 R) from the rest,
// and its first block goes on to invert the next panel's diagonal block D, so
// that serial chain runs beside the other tiles.  A panel touches only the
// unknowns up to two planes ahead (the operator couples within two nodes), so
// the update runs on those rows and columns only.
//
// Bound by FP64 arithmetic: about 2 n^2 (nv / 3 + np) operations for nv
// velocities and np pressures.  n = 3648 (12^3 nodes): the full update 74 us,
// 23 TFLOP/s, the panel 8.5 us, the whole inverse 4.3 ms; the pivoted band LU
// and its triangular solves, a serial chain of 114 panels in one block, took
// 13 ms.  The LU's work grows with the band instead of n, so large and long
// levels take it from the start (gj_prefers_lu).
#pragma once

#include "p2_internal.cuh"

namespace p2 {

constexpr int kGThreads = 128;   // per tile: 4 warps of 32 x 32 values
constexpr int kGLd = kGT + 4;    // row stride of a tile in shared memory: fragment loads without bank conflicts
constexpr int kGjSmem = 2 * kGT * kGLd * (int)sizeof(double);

// active tiles of a panel: the first tv velocity tiles and the first tq
// pressure tiles (which start at tile np0)
struct GjTiles {
    int tv, tq, np0;
    __host__ __device__ int count() const { return tv + tq; }
    __host__ __device__ int at(int t) const { return t < tv ? t : np0 + t - tv; }
};

__device__ __forceinline__ void gj_copy16(double *s, const double *g)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(g) : "memory");
}
__device__ __forceinline__ void gj_copy_wait()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

// dst[k * kGLd + 0..63] = src[k * ld + 0..63], k < 64
__device__ __forceinline__ void gj_load(double *dst, const double *src, long ld)
{
#pragma unroll
    for (int t = 0; t < kGT * kGT / 2 / kGThreads; t++) {
        const int e = t * kGThreads + threadIdx.x, k = e / (kGT / 2), c = e % (kGT / 2) * 2;
        gj_copy16(dst + k * kGLd + c, src + k * ld + c);
    }
}

// acc(r, c) += sum_k As[k][r] Bs[k][c] on the FP64 tensor cores (m16n8k8, the
// columns c along m, so that a thread's values lie in pairs of adjacent rows of
// a column-major matrix).  With 8 x 4 register tiles and DFMA the update was
// bound by shared memory (83 % of its bandwidth, 20 TFLOP/s).
struct GjFrag {
    double v[2][4][4];  // [16 columns][8 rows][fragment]
    int row0, col0;     // of v[.][.][0]; [1] the next row, [2], [3] eight columns on
    __device__ GjFrag()
    {
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        row0 = (w & 1) * 32 + (l & 3) * 2;
        col0 = (w >> 1) * 32 + (l >> 2);
    }
    __device__ __forceinline__ int row(int n) const { return row0 + 8 * n; }
    __device__ __forceinline__ int col(int m, int h) const { return col0 + 16 * m + 8 * h; }
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int e = 0; e < 4; e++) v[m][n][e] = 0;
    }
    __device__ __forceinline__ void product(const double *As, const double *Bs)
    {
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31, g = l >> 2, t = l & 3;
        const double *pa = Bs + t * kGLd + (w >> 1) * 32 + g, *pb = As + t * kGLd + (w & 1) * 32 + g;
#pragma unroll 4
        for (int k = 0; k < kGT; k += 8) {
            double a[2][4], b[4][2];
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int e = 0; e < 4; e++) a[m][e] = pa[(k + 4 * (e >> 1)) * kGLd + 16 * m + 8 * (e & 1)];
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int e = 0; e < 2; e++) b[n][e] = pb[(k + 4 * e) * kGLd + 8 * n];
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int n = 0; n < 4; n++)
                    asm volatile(
                        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                        "{%0,%1,%2,%3};"
                        : "+d"(v[m][n][0]), "+d"(v[m][n][1]), "+d"(v[m][n][2]), "+d"(v[m][n][3])
                        : "d"(a[m][0]), "d"(a[m][1]), "d"(a[m][2]), "d"(a[m][3]), "d"(b[n][0]), "d"(b[n][1]));
        }
    }
};

// Inverse of the 64 x 64 block in sh ([column][row], stride kGLd) by Gauss-Jordan.  Threads
// 0..63 hold the even columns of their row in registers, 64..127 the odd ones,
// rotated so that the pivot column is register 0 of its half: the step is then
// the same code for every pair of pivots (unrolled over all 64 pivots the
// kernel was bound by fetching instructions: 50 us against 32 us).  Per step
// the pivot row and column are published in one of two buffers (w, 4 x 64
// doubles), one barrier.  D gets the inverse as [column][row], DT as
// [row][column].  A pivot that is not positive in magnitude sets *flag.
__device__ __forceinline__ void gj_invert(const double *sh, double *w, double *D, double *DT, int *flag)
{
    const int row = threadIdx.x & (kGT - 1), half = threadIdx.x / kGT;
    constexpr int kH = kGT / 2;
    double v[kH];
#pragma unroll
    for (int c = 0; c < kH; c++) v[c] = sh[(2 * c + half) * kGLd + row];
    bool bad = false;
    for (int j2 = 0; j2 < kH; j2++) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int j = 2 * j2 + q;
            double *prow = w + q * 2 * kGT, *pcol = prow + kGT;  // pivot row [half][c], pivot column
            if (half == q) pcol[row] = v[0];
            if (row == j) {
#pragma unroll
                for (int c = 0; c < kH; c++) prow[half * kH + c] = v[c];
            }
            __syncthreads();
            const double d = pcol[j];
            if (!(fabs(d) > 0)) bad = true;
            const double inv = 1.0 / d;
            const double f = row == j ? -inv : pcol[row] * inv;
            // pivot row: prow * inv; others: v - f prow.  The pivot column's half moves down one register and its
            // new entry (inv, or -f) goes last.
            const double keep = row == j ? 0.0 : 1.0;
            if (half == q) {
#pragma unroll
                for (int c = 0; c + 1 < kH; c++) v[c] = keep * v[c + 1] - f * prow[half * kH + c + 1];
                v[kH - 1] = -f;
            } else {
#pragma unroll
                for (int c = 0; c < kH; c++) v[c] = keep * v[c] - f * prow[half * kH + c];
            }
        }
    }
    if (bad) *flag = 1;
#pragma unroll
    for (int c = 0; c < kH; c++) {
        D[(2 * c + half) * kGT + row] = v[c];
        DT[row * kGT + 2 * c + half] = v[c];
    }
}

// +-1 by the bits of a hash of r
__device__ __forceinline__ double gj_sign(int r)
{
    unsigned h = (unsigned)r * 2654435761u;
    h ^= h >> 15;
    return (h & 0x400u) ? 1.0 : -1.0;
}

// X = A in the permuted order with identity padding, column-major n x n; the
// columns along the grid's x, whose y ends at 65535.  v: the check's vector.
__global__ void k_gj_gather(int n, int nF, const int *perm, const double *A, const double *scale, double *X, double *v)
{
    const int r = blockIdx.y * blockDim.x + threadIdx.x, c = blockIdx.x;
    if (r >= n) return;
    const int pr = perm[r], pc = perm[c];
    if (r == 0) {
        double s = pc >= 0 ? scale[pc] : 0.0;
        if (pc >= 0 && s == 0) s = fabs(A[(size_t)pc * nF + pc]);
        v[c] = gj_sign(c) * s;
    }
    X[(size_t)c * n + r] = pr >= 0 && pc >= 0 ? A[(size_t)pc * nF + pr] : (r == c ? 1.0 : 0.0);
}

__global__ void __launch_bounds__(kGThreads) k_gj_first(const double *X, int n, double *D, int *flag)
{
    __shared__ double sh[kGT * kGLd], w[4 * kGT];
    gj_load(sh, X, n);
    gj_copy_wait();
    __syncthreads();
    gj_invert(sh, w, D, D + kGT * kGT, flag);
}

// Block t < tiles: X[p, j] = U_j = D^-1 X[p, j] (U also to Ub[row][column]);
// block tiles + t: Lb[column][row] = -X[i, p], X[i, p] = -X[i, p] D^-1.
__global__ void __launch_bounds__(kGThreads) k_gj_panel(double *X, int n, int p, GjTiles T, const double *D,
                                                        double *Lb, double *Ub)
{
    extern __shared__ double sm[];
    double *As = sm, *Bs = sm + kGT * kGLd;
    const int nt = T.count();
    const bool rowside = (int)blockIdx.x < nt;
    const int t = T.at(rowside ? blockIdx.x : blockIdx.x - nt);
    double *P = X + (size_t)p * kGT * n + (size_t)p * kGT;
    if (t == p) {
        if (rowside)
            for (int e = threadIdx.x; e < kGT * kGT; e += kGThreads) P[(size_t)(e / kGT) * n + e % kGT] = D[e];
        return;
    }
    GjFrag acc;
    acc.zero();
    if (rowside) {
        double *R = X + (size_t)t * kGT * n + (size_t)p * kGT;
        gj_load(As, D, kGT);  // D as [k][row]
        // R as [k][column]: a warp takes 4 rows of 8 columns, so that neither side is strided throughout
        double v[kGT * kGT / kGThreads];
#pragma unroll
        for (int e = 0; e < kGT * kGT / kGThreads; e++) {
            const int g = e * (kGThreads / 32) + (threadIdx.x >> 5), l = threadIdx.x & 31;
            v[e] = R[(size_t)((g >> 4) * 8 + (l >> 2)) * n + (g & 15) * 4 + (l & 3)];
        }
#pragma unroll
        for (int e = 0; e < kGT * kGT / kGThreads; e++) {
            const int g = e * (kGThreads / 32) + (threadIdx.x >> 5), l = threadIdx.x & 31;
            Bs[((g & 15) * 4 + (l & 3)) * kGLd + (g >> 4) * 8 + (l >> 2)] = v[e];
        }
        gj_copy_wait();
        __syncthreads();
        acc.product(As, Bs);
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int r = acc.row(q), c = acc.col(m, h);
                    const double2 u = make_double2(acc.v[m][q][2 * h], acc.v[m][q][2 * h + 1]);
                    *(double2 *)(R + (size_t)c * n + r) = u;
                    Ub[(size_t)r * n + (size_t)t * kGT + c] = u.x;
                    Ub[(size_t)(r + 1) * n + (size_t)t * kGT + c] = u.y;
                }
    } else {
        double *C = X + (size_t)p * kGT * n + (size_t)t * kGT;
        gj_load(As, C, n);
        gj_load(Bs, D + kGT * kGT, kGT);  // D as [k][column]
        gj_copy_wait();
        __syncthreads();
        acc.product(As, Bs);
        for (int e = threadIdx.x; e < kGT * kGT; e += kGThreads)
            Lb[(size_t)(e / kGT) * n + (size_t)t * kGT + e % kGT] = -As[e / kGT * kGLd + e % kGT];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    *(double2 *)(C + (size_t)acc.col(m, h) * n + acc.row(q)) =
                        make_double2(-acc.v[m][q][2 * h], -acc.v[m][q][2 * h + 1]);
    }
}

// X[i, j] -= L_i U_j on the active tiles outside row and column p; the block
// of tile (next, next) comes first and inverts it for the next panel.
__global__ void __launch_bounds__(kGThreads, 3) k_gj_update(double *X, int n, int p, int next, GjTiles T,
                                                            const double *Lb, const double *Ub, double *Dn, int *flag)
{
    extern __shared__ double sm[];
    double *As = sm, *Bs = sm + kGT * kGLd;
    // tile 0 and the next panel's tile change places in both directions
    auto tile = [&](int b) {
        const int t = T.at(b);
        return b == 0 && next >= 0 ? next : (t == next ? T.at(0) : t);
    };
    const int i = tile(blockIdx.x), j = tile(blockIdx.y);
    if (i == p || j == p) return;
    gj_load(As, Lb + (size_t)i * kGT, n);
    gj_load(Bs, Ub + (size_t)j * kGT, n);
    double *Cp = X + (size_t)j * kGT * n + (size_t)i * kGT;
    GjFrag acc;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const double2 v = *(const double2 *)(Cp + (size_t)acc.col(m, h) * n + acc.row(q));
                acc.v[m][q][2 * h] = v.x;
                acc.v[m][q][2 * h + 1] = v.y;
            }
    gj_copy_wait();
    __syncthreads();
    acc.product(As, Bs);
    const bool first = i == next && j == next;
    if (first) __syncthreads();
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const double2 v = make_double2(acc.v[m][q][2 * h], acc.v[m][q][2 * h + 1]);
                *(double2 *)(Cp + (size_t)acc.col(m, h) * n + acc.row(q)) = v;
                if (first) *(double2 *)(As + acc.col(m, h) * kGLd + acc.row(q)) = v;
            }
    if (first) {
        __syncthreads();
        gj_invert(As, Bs, Dn, Dn + kGT * kGT, flag);
    }
}

// Check of the inverse: y = X v for v_r = +-s_r with the rows' scales s_r (their
// largest velocity entry: the diagonal of a momentum row, 1 / h of a continuity
// row), then flag when |A y - v| in a row is above kGjCheck
// s_r (or not a number).  That is the test of the inverse of A with its rows
// scaled to 1, so it does not depend on the units: rounding alone leaves about
// 1e-14 at equal viscosities and 1e-7 at a contrast of 1e4, in a unit box as in
// metres and Pa s, where an absolute bound on v = +-1 fails any inverse
// (momentum rows hold eta / h^2, continuity rows 1 / h; it failed the layered model
// at 257^3 too, 13 ms a solve).  An inverse that passes serves the FP64 cycle as the
// pivoted one does: the same iterations on 48 models at 33^3 to 65^3 with contrasts of
// 1e2 to 1e8.
constexpr double kGjCheck = 1e-4;
// row r of A b, the 32 warps of the block splitting the columns
constexpr int kCheckWarps = 32;
__device__ __forceinline__ double gj_rows(int n, const double *A, int r, const double *b, double (*part)[33])
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double s = 0;
    if (r < n) {
#pragma unroll 4
        for (int c = w; c < n; c += kCheckWarps) s += A[(size_t)c * n + r] * b[c];
    }
    part[w][lane] = s;
    __syncthreads();
    double t = 0;
    for (int q = 0; q < kCheckWarps; q++) t += part[q][lane];
    return t;
}
__global__ void __launch_bounds__(32 * kCheckWarps) k_gj_check_x(int n, const int *perm, const double *X, const double *v,
                                                                 double *y)
{
    __shared__ double part[kCheckWarps][33];
    const int r = blockIdx.x * 32 + (threadIdx.x & 31);
    const double t = gj_rows(n, X, r, v, part);
    if (threadIdx.x < 32 && r < n && perm[r] >= 0) y[perm[r]] = t;  // y in the order of A
}
__global__ void __launch_bounds__(32 * kCheckWarps) k_gj_check_a(int nF, const int *iperm, const double *A,
                                                                 const double *y, const double *v, int *flag)
{
    __shared__ double part[kCheckWarps][33];
    const int r = blockIdx.x * 32 + (threadIdx.x & 31);
    const double t = gj_rows(nF, A, r, y, part);
    if (threadIdx.x < 32 && r < nF) {
        const double want = v[iperm[r]];
        if (!(fabs(t - want) < kGjCheck * fabs(want))) *flag = 2;
    }
}

}  // namespace p2
