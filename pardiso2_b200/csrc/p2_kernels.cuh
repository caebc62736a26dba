// Stencil, transfer and reduction kernels of the p2cuda Stokes multigrid.
#pragma once

#include "p2_internal.cuh"

namespace p2 {

// Storage type of the stored cell factors of a V-cycle computing in T (the
// cycle's own type: bfloat16 factors for the FP32 cycle were measured to cost
// 26 -> 31 outer iterations at 257^3 for a 1 % faster pass, which is latency-
// rather than bandwidth-bound).
template <typename T>
using factor_t = T;

__device__ __forceinline__ float ld_factor(const float *p) { return __ldg(p); }
__device__ __forceinline__ double ld_factor(const double *p) { return __ldg(p); }
template <typename S>
__device__ __forceinline__ S to_factor(double v) { return (S)v; }

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------
// The three momentum rows at node (i, j, k), 1 <= i <= nx-2 and so on, from
// shared stresses: the upper cell's three normal stresses, the one along the
// row's axis of its lower x, y and z neighbours, three edges of each
// orientation; every velocity, viscosity and pressure loaded once.  The same
// terms as row_vx / row_vy / row_vz up to rounding (the deviatoric third is a
// multiplication by 1/3).
template <typename T, typename S>
__device__ __forceinline__ void node_rows(const LevelView<T> &L, const Fields<T, S> &x, int i, int j, int k, T r[3])
{
    const int sy = L.ny, sz = L.nx * L.ny, u = P2IDX(L, i, j, k);
    const S *vx = x.vx + u, *vy = x.vy + u, *vz = x.vz + u, *pp = x.p + u + sz + sy + 1;
    auto V = [](const S *q) { return (T)__ldg(q); };
    const T vx0 = V(vx), vxX = V(vx + sy), vxm = V(vx - sy), vxY = V(vx + 1), vxy_ = V(vx - 1), vxZ = V(vx + sz),
            vxz_ = V(vx - sz), vxXy = V(vx + sy - 1), vxXz = V(vx + sy - sz);
    const T vy0 = V(vy), vyY = V(vy + 1), vym = V(vy - 1), vyX = V(vy + sy), vyx_ = V(vy - sy), vyZ = V(vy + sz),
            vyz_ = V(vy - sz), vyYx = V(vy + 1 - sy), vyYz = V(vy + 1 - sz);
    const T vz0 = V(vz), vzZ = V(vz + sz), vzm = V(vz - sz), vzX = V(vz + sy), vzx_ = V(vz - sy), vzY = V(vz + 1),
            vzy_ = V(vz - 1), vzZx = V(vz + sz - sy), vzZy = V(vz + sz - 1);
    const T pA = V(pp), pL = V(pp - sy), pF = V(pp - 1), pD = V(pp - sz);
    const T third = (T)(1.0 / 3.0), two = (T)2.0;
    const T hx0 = L.ax.ih[i], hx1 = L.ax.ih[i + 1], hy0 = L.ay.ih[j], hy1 = L.ay.ih[j + 1], hz0 = L.az.ih[k],
            hz1 = L.az.ih[k + 1];
    const int c = u + sz + sy + 1;
    T sAx, sAy, sAz, sL, sF, sD;
    {
        const T a = (vxX - vx0) * hx1, b = (vyY - vy0) * hy1, d = (vzZ - vz0) * hz1, m = (a + b + d) * third;
        const T E = two * eta_at(L, L.ec, c);
        sAx = E * (a - m);
        sAy = E * (b - m);
        sAz = E * (d - m);
    }
    {
        const T a = (vx0 - vxm) * hx0, b = (vyYx - vyx_) * hy1, d = (vzZx - vzx_) * hz1;
        sL = two * eta_at(L, L.ec, c - sy) * (a - (a + b + d) * third);
    }
    {
        const T a = (vxXy - vxy_) * hx1, b = (vy0 - vym) * hy0, d = (vzZy - vzy_) * hz1;
        sF = two * eta_at(L, L.ec, c - 1) * (b - (a + b + d) * third);
    }
    {
        const T a = (vxXz - vxz_) * hx1, b = (vyYz - vyz_) * hy1, d = (vz0 - vzm) * hz0;
        sD = two * eta_at(L, L.ec, c - sz) * (d - (a + b + d) * third);
    }
    const T ex0 = L.ax.ihe[i], ex1 = L.ax.ihe[i + 1], ey0 = L.ay.ihe[j], ey1 = L.ay.ihe[j + 1], ez0 = L.az.ihe[k],
            ez1 = L.az.ihe[k + 1];
    const T xy0 = two * eta_at(L, L.exy, u) * ((vx0 - vxy_) * ey0 + (vy0 - vyx_) * ex0);
    const T xyY = two * eta_at(L, L.exy, u + 1) * ((vxY - vx0) * ey1 + (vyY - vyYx) * ex0);
    const T xyX = two * eta_at(L, L.exy, u + sy) * ((vxX - vxXy) * ey0 + (vyX - vy0) * ex1);
    const T xz0 = two * eta_at(L, L.exz, u) * ((vx0 - vxz_) * ez0 + (vz0 - vzx_) * ex0);
    const T xzZ = two * eta_at(L, L.exz, u + sz) * ((vxZ - vx0) * ez1 + (vzZ - vzZx) * ex0);
    const T xzX = two * eta_at(L, L.exz, u + sy) * ((vxX - vxXz) * ez0 + (vzX - vz0) * ex1);
    const T yz0 = two * eta_at(L, L.eyz, u) * ((vy0 - vyz_) * ez0 + (vz0 - vzy_) * ey0);
    const T yzZ = two * eta_at(L, L.eyz, u + sz) * ((vyZ - vy0) * ez1 + (vzZ - vzZy) * ey0);
    const T yzY = two * eta_at(L, L.eyz, u + 1) * ((vyY - vyYz) * ez0 + (vzY - vz0) * ey1);
    const T cx = L.ax.ihc[i], cy = L.ay.ihc[j], cz = L.az.ihc[k], wx = L.ax.ihv[i], wy = L.ay.ihv[j], wz = L.az.ihv[k];
    r[0] = (sAx - sL) * cx + (xyY - xy0) * wy + (xzZ - xz0) * wz - (pA - pL) * cx;
    r[1] = (sAy - sF) * cy + (xyX - xy0) * wx + (yzZ - yz0) * wz - (pA - pF) * cy;
    r[2] = (sAz - sD) * cz + (xzX - xz0) * wx + (yzY - yz0) * wy - (pA - pD) * cz;
}

// Rows: out = b - A x (mode 0) or out = A x (mode 1) on every non-boundary
// row; boundary rows and non-unknown positions get 0 here (boundary rows are
// written by k_bc_rows).  Optionally also writes a float copy (the FP32
// right-hand side of the mixed-precision V-cycle) or a copy of x (the outer
// loop's stored correction).  All four rows of a node in one thread from one
// set of loads: evaluated one after the other, with a store between them, each
// row loaded and derived its stresses anew.  Waits for loads: 8 (FP32) or 4
// (FP64) blocks of 128 threads an SM measured best of 5 .. 10 and 3 .. 6.  257^3:
// q = A c from FP32 with its copy 0.99 ms (and 0.17 ms for the copy) -> 0.72 ms,
// FP32 residual 0.66 -> 0.60 ms, 67^3 26 -> 20 us; the FP64 residual, once per
// restart, 1.08 -> 1.29 ms.
constexpr int kRowsThreads = 128;
template <typename T, typename S>
__global__ void __launch_bounds__(kRowsThreads, sizeof(T) == 4 ? 8 : 4) k_rows(LevelView<T> L, Fields<T, S> x,
                                                                             Vec4<T> b, Vec4<T> out,
                                                                             Vec4<float> out32, Vec4<S> copy, int mode)
{
    pdl_enter();
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= L.n) return;
    const int j = u % L.ny, i = (u / L.ny) % L.nx, k = u / (L.nx * L.ny);
    const uint8_t m = L.bcm[u];
    T v[4] = {0, 0, 0, 0}, r[3];
    if (i > 0 && j > 0 && k > 0) {
        if (!(m & BC_P)) v[0] = row_p(L, x, i, j, k);
        if (i < L.nx - 1 && j < L.ny - 1 && k < L.nz - 1 && (m & (BC_VX | BC_VY | BC_VZ)) != (BC_VX | BC_VY | BC_VZ)) {
            node_rows(L, x, i, j, k, r);
#pragma unroll
            for (int c = 1; c < 4; c++) v[c] = r[c - 1];
        }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const bool row = valid_pos(c, i, j, k, L.nx, L.ny, L.nz) && !(m & (1 << c));
        const T w = !row ? (T)0 : (mode == 0 ? b.c[c][u] - v[c] : v[c]);
        out.c[c][u] = w;
        if (out32.c[0]) out32.c[c][u] = (float)w;
        if (copy.c[0]) copy.c[c][u] = (c == 0 ? x.p : c == 1 ? x.vx : c == 2 ? x.vy : x.vz)[u];
    }
}

// Boundary rows x_u = b_u + koef * x_t: residual (mode 0) b_u + koef x_t - x_u,
// or operator (mode 1) x_u - koef x_t.
template <typename T, typename S>
__device__ __forceinline__ void bc_rows_item(int nbc, const int *bu, const int *bt, const float *bk,
                                             const Fields<T, S> &x, const Vec4<T> &b, const Vec4<T> &out,
                                             const Vec4<float> &out32, int mode, int q)
{
    if (q >= nbc) return;
    int uc = bu[q], c = uc & 3, u = uc >> 2, t = bt[q];
    const S *xs[4] = {x.p, x.vx, x.vy, x.vz};
    T xt = t >= 0 ? (T)bk[q] * (T)xs[t & 3][t >> 2] : (T)0;
    T v = mode == 0 ? b.c[c][u] + xt - (T)xs[c][u] : (T)xs[c][u] - xt;
    out.c[c][u] = v;
    if (out32.c[0]) out32.c[c][u] = (float)v;
}
template <typename T, typename S>
__global__ void k_bc_rows(int nbc, const int *bu, const int *bt, const float *bk, Fields<T, S> x, Vec4<T> b,
                          Vec4<T> out, Vec4<float> out32, int mode)
{
    pdl_enter();
    bc_rows_item(nbc, bu, bt, bk, x, b, out, out32, mode, blockIdx.x * blockDim.x + threadIdx.x);
}

// All boundary rows in one launch: each row walks its copy chain (the rows
// owning its successive targets, bnext) and evaluates it from the innermost
// row outwards, x = b + koef * x_target, the same arithmetic as applying the
// chain-depth groups one after another.  Only the final target (a regular
// unknown) is read from x, and each row writes only its own unknown.
constexpr int kMaxBcChain = 8;

template <typename T>
__device__ __forceinline__ void bc_set_chain_item(int nbc, const int *bu, const int *bt, const float *bk,
                                                  const int *bnext, const Vec4<T> &x, const Vec4<T> &b, int q)
{
    if (q >= nbc) return;
    int chain[kMaxBcChain];
    int m = 0, r = q;
    chain[m++] = r;
    while (bnext[r] >= 0 && m < kMaxBcChain) {
        r = bnext[r];
        chain[m++] = r;
    }
    const int t = bt[r];                      // innermost row's target (regular unknown or none)
    T v = t >= 0 ? (T)bk[r] * x.c[t & 3][t >> 2] : (T)0;
    int uc = bu[r];
    v = b.c[uc & 3][uc >> 2] + v;
    for (int s = m - 2; s >= 0; s--) {
        const int rr = chain[s];
        uc = bu[rr];
        v = b.c[uc & 3][uc >> 2] + (T)bk[rr] * v;
    }
    uc = bu[q];
    x.c[uc & 3][uc >> 2] = v;
}
template <typename T>
__global__ void k_bc_set_chain(int nbc, const int *bu, const int *bt, const float *bk, const int *bnext, Vec4<T> x,
                               Vec4<T> b)
{
    pdl_enter();
    bc_set_chain_item(nbc, bu, bt, bk, bnext, x, b, blockIdx.x * blockDim.x + threadIdx.x);
}

// Boundary rows between the colour passes of a smoothing call: the rows with a
// regular target, by their resolved target and the constant part that
// k_bc_begin left for them, x = c + k x_target.  Two dependent loads instead of
// the walk along the chain: V-cycle of 65^3 0.491 -> 0.444 ms, of 257^3 10.64 -> 10.21 ms.
template <typename T, bool kDouble>
__global__ void k_bc_follow(BcFollow R, const T *c, Vec4<T> x)
{
    pdl_enter();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= R.n) return;
    const int uc = __ldg(R.uc + q), t = __ldg(R.target + q);
    const T k = kDouble ? (T)__ldg(R.kd + q) : (T)__ldg(R.k + q);
    const T *s = (t & 3) == 0 ? x.c[0] : ((t & 3) == 1 ? x.c[1] : ((t & 3) == 2 ? x.c[2] : x.c[3]));
    T *d = (uc & 3) == 0 ? x.c[0] : ((uc & 3) == 1 ? x.c[1] : ((uc & 3) == 2 ? x.c[2] : x.c[3]));
    d[uc >> 2] = __ldg(c + q) + k * s[t >> 2];
}
// Start of a smoothing call: every boundary row of x (as k_bc_set_chain) and,
// in the second velocity buffer y, the same values, which the rows without a
// target keep; slot[r] is the row's place among the following ones or -1.
template <typename T>
__global__ void k_bc_begin(int nbc, const int *bu, const int *bt, const float *bk, const int *bnext, const int *slot,
                           Vec4<T> x, Vec4<T> y, Vec4<T> b, T *c)
{
    pdl_enter();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nbc) return;
    int chain[kMaxBcChain];
    int m = 0, r = q;
    chain[m++] = r;
    while (bnext[r] >= 0 && m < kMaxBcChain) {
        r = bnext[r];
        chain[m++] = r;
    }
    const int t = bt[r];
    int uc = bu[r];
    T c0 = b.c[uc & 3][uc >> 2], v = c0;
    if (t >= 0) v += (T)bk[r] * x.c[t & 3][t >> 2];
    for (int s = m - 2; s >= 0; s--) {
        const int rr = chain[s];
        uc = bu[rr];
        const T bb = b.c[uc & 3][uc >> 2], kk = (T)bk[rr];
        c0 = bb + kk * c0;
        v = bb + kk * v;
    }
    uc = bu[q];
    x.c[uc & 3][uc >> 2] = v;
    if (uc & 3) y.c[uc & 3][uc >> 2] = v;
    const int f = slot[q];
    if (f >= 0) c[f] = c0;
}

// ---------------------------------------------------------------------------
// Full cell-block variant: the cell's 6 face velocities and its pressure are
// solved together with the exact 7x7 cell system
//   [M g; cc^T 0] [dv; dp] = [r; rp],
// M the face-face block of the momentum rows.  Its off-diagonal entries come
// from the cell's normal stresses (every face enters e_xx, e_yy, e_zz and the
// divergence) and from the shear stresses on the edges two faces share; they
// are the coefficients of the row functions above (checked entry by entry
// against the assembled operator).  Faces under a boundary row are held; the
// pressure is held where the cell pressure is a boundary unknown.  M is
// eliminated without pivoting (-M is diagonally dominant).  Read/write
// pattern and buffering as k_vanka.
template <typename T>
__device__ __forceinline__ void face_block(const LevelView<T> &L, int i, int j, int k, T M[6][6])
{
    const T Ec = eta_at(L, L.ec, P2IDX(L, i, j, k));
    const T hx = L.ax.ih[i], hy = L.ay.ih[j], hz = L.az.ih[k];
    const T t43 = (T)(4.0 / 3.0), t23 = (T)(2.0 / 3.0);
    // d snn_d(cell) / d face, times Ec
    const T dn[3][6] = {{-t43 * hx, t43 * hx, t23 * hy, -t23 * hy, t23 * hz, -t23 * hz},
                        {t23 * hx, -t23 * hx, -t43 * hy, t43 * hy, t23 * hz, -t23 * hz},
                        {t23 * hx, -t23 * hx, t23 * hy, -t23 * hy, -t43 * hz, t43 * hz}};
    const T s0 = Ec * L.ax.ihc[i - 1], s1 = -Ec * L.ax.ihc[i], s2 = Ec * L.ay.ihc[j - 1], s3 = -Ec * L.ay.ihc[j],
            s4 = Ec * L.az.ihc[k - 1], s5 = -Ec * L.az.ihc[k];
#pragma unroll
    for (int b = 0; b < 6; b++) {
        M[0][b] = s0 * dn[0][b];
        M[1][b] = s1 * dn[0][b];
        M[2][b] = s2 * dn[1][b];
        M[3][b] = s3 * dn[1][b];
        M[4][b] = s4 * dn[2][b];
        M[5][b] = s5 * dn[2][b];
    }
    const T two = (T)2.0;
    const T exy00 = eta_at(L, L.exy, P2IDX(L, i - 1, j - 1, k - 1)), exy01 = eta_at(L, L.exy, P2IDX(L, i - 1, j, k - 1));
    const T exy10 = eta_at(L, L.exy, P2IDX(L, i, j - 1, k - 1)), exy11 = eta_at(L, L.exy, P2IDX(L, i, j, k - 1));
    const T exz00 = eta_at(L, L.exz, P2IDX(L, i - 1, j - 1, k - 1)), exz01 = eta_at(L, L.exz, P2IDX(L, i - 1, j - 1, k));
    const T exz10 = eta_at(L, L.exz, P2IDX(L, i, j - 1, k - 1)), exz11 = eta_at(L, L.exz, P2IDX(L, i, j - 1, k));
    const T eyz00 = eta_at(L, L.eyz, P2IDX(L, i - 1, j - 1, k - 1)), eyz01 = eta_at(L, L.eyz, P2IDX(L, i - 1, j - 1, k));
    const T eyz10 = eta_at(L, L.eyz, P2IDX(L, i - 1, j, k - 1)), eyz11 = eta_at(L, L.eyz, P2IDX(L, i - 1, j, k));
    const T hex0 = L.ax.ihe[i - 1], hex1 = L.ax.ihe[i], hey0 = L.ay.ihe[j - 1], hey1 = L.ay.ihe[j];
    const T hez0 = L.az.ihe[k - 1], hez1 = L.az.ihe[k];
    const T hvx = L.ax.ihv[i - 1], hvy = L.ay.ihv[j - 1], hvz = L.az.ihv[k - 1];
    // vx faces: shear with the vy (front/back) and vz (bottom/top) faces
    M[0][3] += two * exy01 * hex0 * hvy;  M[0][2] -= two * exy00 * hex0 * hvy;
    M[0][5] += two * exz01 * hex0 * hvz;  M[0][4] -= two * exz00 * hex0 * hvz;
    M[1][3] -= two * exy11 * hex1 * hvy;  M[1][2] += two * exy10 * hex1 * hvy;
    M[1][5] -= two * exz11 * hex1 * hvz;  M[1][4] += two * exz10 * hex1 * hvz;
    // vy faces
    M[2][1] += two * exy10 * hey0 * hvx;  M[2][0] -= two * exy00 * hey0 * hvx;
    M[2][5] += two * eyz01 * hey0 * hvz;  M[2][4] -= two * eyz00 * hey0 * hvz;
    M[3][1] -= two * exy11 * hey1 * hvx;  M[3][0] += two * exy01 * hey1 * hvx;
    M[3][5] -= two * eyz11 * hey1 * hvz;  M[3][4] += two * eyz10 * hey1 * hvz;
    // vz faces
    M[4][1] += two * exz10 * hez0 * hvx;  M[4][0] -= two * exz00 * hez0 * hvx;
    M[4][3] += two * eyz10 * hez0 * hvy;  M[4][2] -= two * eyz00 * hez0 * hvy;
    M[5][1] -= two * exz11 * hez1 * hvx;  M[5][0] += two * exz01 * hez1 * hvx;
    M[5][3] -= two * eyz11 * hez1 * hvy;  M[5][2] += two * eyz01 * hez1 * hvy;
}

template <typename T>
__global__ void __launch_bounds__(128) k_vanka_full(LevelView<T> L, T *P, Vec4<T> vin, Vec4<T> vout, Vec4<T> b,
                                                    T omega, int col)
{
    pdl_enter();
    int half = (L.ny) / 2;
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long lines = (long)(L.nx - 1) * (L.nz - 1);
    if (t >= lines * half) return;
    int jj = (int)(t % half);
    long line = t / half;
    int i = 1 + (int)(line % (L.nx - 1)), k = 1 + (int)(line / (L.nx - 1));
    int j0 = (((1 + i + k) & 1) == col) ? 1 : 2;
    int j = j0 + 2 * jj;
    if (j > L.ny - 1) return;
    Fields<T, T> x{P, vin.c[1], vin.c[2], vin.c[3]};
    int u = P2IDX(L, i, j, k);
    const bool pact = (L.bcm[u] & BC_P) == 0;
    int fi[6];
    const int fc[6] = {1, 1, 2, 2, 3, 3};
    T g[6], cc[6], r[6];
    bool act[6];
    fi[0] = P2IDX(L, i - 1, j - 1, k - 1); g[0] = -L.ax.ihc[i - 1]; cc[0] = -L.ax.ih[i];
    fi[1] = P2IDX(L, i, j - 1, k - 1);     g[1] = L.ax.ihc[i];      cc[1] = L.ax.ih[i];
    fi[2] = P2IDX(L, i - 1, j - 1, k - 1); g[2] = -L.ay.ihc[j - 1]; cc[2] = -L.ay.ih[j];
    fi[3] = P2IDX(L, i - 1, j, k - 1);     g[3] = L.ay.ihc[j];      cc[3] = L.ay.ih[j];
    fi[4] = P2IDX(L, i - 1, j - 1, k - 1); g[4] = -L.az.ihc[k - 1]; cc[4] = -L.az.ih[k];
    fi[5] = P2IDX(L, i - 1, j - 1, k);     g[5] = L.az.ihc[k];      cc[5] = L.az.ih[k];
    const int ofs[6][3] = {{-1, -1, -1}, {0, -1, -1}, {-1, -1, -1}, {-1, 0, -1}, {-1, -1, -1}, {-1, -1, 0}};
    T M[6][6];
    face_block(L, i, j, k, M);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        int a = i + ofs[q][0], bb = j + ofs[q][1], c = k + ofs[q][2];
        T d = 0;
        act[q] = !(L.bcm[fi[q]] & (1 << fc[q]));
        r[q] = 0;
        if (act[q]) {
            T ax;
            if (fc[q] == 1) ax = row_vx(L, x, a, bb, c, &d);
            else if (fc[q] == 2) ax = row_vy(L, x, a, bb, c, &d);
            else ax = row_vz(L, x, a, bb, c, &d);
            r[q] = b.c[fc[q]][fi[q]] - ax;
        }
        M[q][q] = d;
    }
    // masked system: held faces become identity rows / zero columns
    T y1[6], y2[6];
#pragma unroll
    for (int a = 0; a < 6; a++) {
#pragma unroll
        for (int c = 0; c < 6; c++)
            if (!(act[a] && act[c])) M[a][c] = a == c ? (T)1 : (T)0;
        y1[a] = act[a] ? r[a] : (T)0;
        y2[a] = act[a] ? g[a] : (T)0;
    }
    // constant trip counts so that M, y1, y2 stay in registers
#pragma unroll
    for (int c = 0; c < 6; c++) {
        const T ip = (T)1 / M[c][c];
#pragma unroll
        for (int a = 0; a < 6; a++) {
            if (a > c) {
                const T f = M[a][c] * ip;
#pragma unroll
                for (int e = 0; e < 6; e++)
                    if (e > c) M[a][e] -= f * M[c][e];
                y1[a] -= f * y1[c];
                y2[a] -= f * y2[c];
            }
        }
    }
#pragma unroll
    for (int cc5 = 0; cc5 < 6; cc5++) {
        const int c = 5 - cc5;
#pragma unroll
        for (int e = 0; e < 6; e++) {
            if (e > c) {
                y1[c] -= M[c][e] * y1[e];
                y2[c] -= M[c][e] * y2[e];
            }
        }
        const T ip = (T)1 / M[c][c];
        y1[c] *= ip;
        y2[c] *= ip;
    }
    T dp = 0;
    if (pact) {
        T num = -(b.c[0][u] - row_p(L, x, i, j, k)), den = 0;
#pragma unroll
        for (int q = 0; q < 6; q++) {
            num += cc[q] * y1[q];
            den += cc[q] * y2[q];
        }
        if (den != (T)0) {
            dp = num / den;
            P[u] += omega * dp;
        }
    }
#pragma unroll
    for (int q = 0; q < 6; q++)
        if (act[q]) vout.c[fc[q]][fi[q]] = vin.c[fc[q]][fi[q]] + omega * (y1[q] - dp * y2[q]);
}

// Viscosities a cell's rows use, in the order of cell_eta_offset: the cell
// itself, its six neighbours (low, high x; y; z), its four edges of each
// orientation.
constexpr int kCellEta = 19;

// Field (0 ec, 1 exy, 2 exz, 3 eyz) and node offset from the cell's low corner
// F = (i-1, j-1, k-1) of viscosity q (y stride 1, x stride sy, z stride sz).
__device__ __forceinline__ int cell_eta_offset(int q, int sy, int sz, int &field)
{
    field = q < 7 ? 0 : (q - 7) / 4 + 1;
    const int u = sz + sy + 1, e = (q - 7) & 3;
    switch (q) {
    case 0: return u;
    case 1: return u - sy;
    case 2: return u + sy;
    case 3: return u - 1;
    case 4: return u + 1;
    case 5: return u - sz;
    case 6: return u + sz;
    default: break;
    }
    // edge (lo, hi) along the two axes across it: xy 00 01 (y) 10 (x) 11, xz 00 01 (z) 10 (x) 11, yz 00 01 (z) 10 (y) 11
    const int first = field == 3 ? 1 : sy, second = field == 1 ? 1 : sz;
    return (e & 2 ? first : 0) + (e & 1 ? second : 0);
}

// Viscosities of a cell from the level's fields.
template <typename T>
struct LevelEta {
    const LevelView<T> &L;
    int F;
    __device__ __forceinline__ T operator()(int q) const
    {
        int f;
        const int o = F + cell_eta_offset(q, L.ny, L.nx * L.ny, f);
        return eta_at(L, f == 0 ? L.ec : (f == 1 ? L.exy : (f == 2 ? L.exz : L.eyz)), o);
    }
};
// Unknowns that no thread of the launch writes.
struct LoadConst {
    template <typename T>
    __device__ __forceinline__ T operator()(const T *p) const { return __ldg(p); }
};

// Momentum parts (A v + grad p) of the six face rows of cell (i, j, k) from
// shared stresses, and the cell's divergence: the cell's three normal
// stresses from one set of strain rates, the six neighbour cells' normal
// stresses along their face normals, the twelve edge shear stresses once
// each.  Every velocity, viscosity and pressure is loaded once, addressed
// from the cell's low corner F = (i-1, j-1, k-1) (y stride 1, x stride ny, z
// stride nx*ny); the deviatoric third is a multiplication by 1/3.  The same
// terms as row_vx/row_vy/row_vz up to rounding.  kDiag: also the rows'
// diagonals (diag_vx .. diag_vz) in d.
template <typename T, bool kDiag, typename Eta, typename Load>
__device__ __forceinline__ void cell_rows(const Axis<T> &AX, const Axis<T> &AY, const Axis<T> &AZ, int sy, int sz,
                                          const Fields<T, T> &x, int i, int j, int k, int F, const Eta &eta,
                                          const Load &load, T ax[6], T &div, T *d)
{
    const T *vx = x.vx + F, *vy = x.vy + F, *vz = x.vz + F;
    // velocities around the cell (offsets from F)
    const T vx0 = load(vx), vxX = load(vx + sy), vxXX = load(vx + 2 * sy), vxm = load(vx - sy);
    const T vxY = load(vx + 1), vxy_ = load(vx - 1), vxXY = load(vx + sy + 1), vxXy = load(vx + sy - 1);
    const T vxZ = load(vx + sz), vxz_ = load(vx - sz), vxXZ = load(vx + sy + sz), vxXz = load(vx + sy - sz);
    const T vy0 = load(vy), vyY = load(vy + 1), vyYY = load(vy + 2), vym = load(vy - 1);
    const T vyX = load(vy + sy), vyx_ = load(vy - sy), vyXY = load(vy + sy + 1), vyxY = load(vy - sy + 1);
    const T vyZ = load(vy + sz), vyz_ = load(vy - sz), vyYZ = load(vy + 1 + sz), vyYz = load(vy + 1 - sz);
    const T vz0 = load(vz), vzZ = load(vz + sz), vzZZ = load(vz + 2 * sz), vzm = load(vz - sz);
    const T vzX = load(vz + sy), vzx_ = load(vz - sy), vzXZ = load(vz + sy + sz), vzxZ = load(vz - sy + sz);
    const T vzY = load(vz + 1), vzy_ = load(vz - 1), vzYZ = load(vz + 1 + sz), vzyZ = load(vz - 1 + sz);
    const T third = (T)(1.0 / 3.0), two = (T)2.0;
    const T hx0 = AX.ih[i - 1], hx1 = AX.ih[i], hx2 = AX.ih[i + 1];
    const T hy0 = AY.ih[j - 1], hy1 = AY.ih[j], hy2 = AY.ih[j + 1];
    const T hz0 = AZ.ih[k - 1], hz1 = AZ.ih[k], hz2 = AZ.ih[k + 1];
    // In FP32 the viscosities and pressures are loaded here too, so that all of a
    // cell's loads are in flight together; in FP64 that costs too many registers.
    constexpr bool kAhead = sizeof(T) == 4;
    const T *pp = x.p + F + sz + sy + 1;
    T en[kAhead ? kCellEta : 1], pn[kAhead ? 7 : 1];
    const int po[7] = {0, -sy, sy, -1, 1, -sz, sz};
    if constexpr (kAhead) {
#pragma unroll
        for (int q = 0; q < 7; q++) pn[q] = load(pp + po[q]);
#pragma unroll
        for (int q = 0; q < kCellEta; q++) en[q] = eta(q);
    }
    auto E = [&](int q) {
        if constexpr (kAhead) return en[q];
        else return eta(q);
    };
    auto PR = [&](int q) {
        if constexpr (kAhead) return pn[q];
        else return load(pp + po[q]);
    };
    // own cell
    const T exx = (vxX - vx0) * hx1, eyy = (vyY - vy0) * hy1, ezz = (vzZ - vz0) * hz1;
    div = exx + eyy + ezz;
    const T E2 = two * E(0);
    const T s0 = E2 * (exx - div * third), s1 = E2 * (eyy - div * third), s2 = E2 * (ezz - div * third);
    // neighbour cells: normal stress along the shared face's normal
    T sL, sR, sF, sB, sD, sU;
    {   // cell (i-1, j, k): faces vx[F-sy], vx[F]; vy[F-sy], vy[F-sy+1]; vz[F-sy], vz[F-sy+sz]
        const T a = (vx0 - vxm) * hx0, b = (vyxY - vyx_) * hy1, c = (vzxZ - vzx_) * hz1;
        sL = two * E(1) * (a - (a + b + c) * third);
    }
    {   // cell (i+1, j, k)
        const T a = (vxXX - vxX) * hx2, b = (vyXY - vyX) * hy1, c = (vzXZ - vzX) * hz1;
        sR = two * E(2) * (a - (a + b + c) * third);
    }
    {   // cell (i, j-1, k)
        const T a = (vxXy - vxy_) * hx1, b = (vy0 - vym) * hy0, c = (vzyZ - vzy_) * hz1;
        sF = two * E(3) * (b - (a + b + c) * third);
    }
    {   // cell (i, j+1, k)
        const T a = (vxXY - vxY) * hx1, b = (vyYY - vyY) * hy2, c = (vzYZ - vzY) * hz1;
        sB = two * E(4) * (b - (a + b + c) * third);
    }
    {   // cell (i, j, k-1)
        const T a = (vxXz - vxz_) * hx1, b = (vyYz - vyz_) * hy1, c = (vz0 - vzm) * hz0;
        sD = two * E(5) * (c - (a + b + c) * third);
    }
    {   // cell (i, j, k+1)
        const T a = (vxXZ - vxZ) * hx1, b = (vyYZ - vyZ) * hy1, c = (vzZZ - vzZ) * hz2;
        sU = two * E(6) * (c - (a + b + c) * third);
    }
    // edge shear stresses (sxy, sxz, syz at the cell's twelve edges)
    const T ex0 = AX.ihe[i - 1], ex1 = AX.ihe[i], ey0 = AY.ihe[j - 1], ey1 = AY.ihe[j];
    const T ez0 = AZ.ihe[k - 1], ez1 = AZ.ihe[k];
    const T xy00 = two * E(7) * ((vx0 - vxy_) * ey0 + (vy0 - vyx_) * ex0);
    const T xy01 = two * E(8) * ((vxY - vx0) * ey1 + (vyY - vyxY) * ex0);
    const T xy10 = two * E(9) * ((vxX - vxXy) * ey0 + (vyX - vy0) * ex1);
    const T xy11 = two * E(10) * ((vxXY - vxX) * ey1 + (vyXY - vyY) * ex1);
    const T xz00 = two * E(11) * ((vx0 - vxz_) * ez0 + (vz0 - vzx_) * ex0);
    const T xz01 = two * E(12) * ((vxZ - vx0) * ez1 + (vzZ - vzxZ) * ex0);
    const T xz10 = two * E(13) * ((vxX - vxXz) * ez0 + (vzX - vz0) * ex1);
    const T xz11 = two * E(14) * ((vxXZ - vxX) * ez1 + (vzXZ - vzZ) * ex1);
    const T yz00 = two * E(15) * ((vy0 - vyz_) * ez0 + (vz0 - vzy_) * ey0);
    const T yz01 = two * E(16) * ((vyZ - vy0) * ez1 + (vzZ - vzyZ) * ey0);
    const T yz10 = two * E(17) * ((vyY - vyYz) * ez0 + (vzY - vz0) * ey1);
    const T yz11 = two * E(18) * ((vyYZ - vyY) * ez1 + (vzYZ - vzZ) * ey1);
    const T p0 = PR(0), pL = PR(1), pR = PR(2), pF = PR(3), pB = PR(4), pD = PR(5), pU = PR(6);
    const T cx0 = AX.ihc[i - 1], cx1 = AX.ihc[i], cy0 = AY.ihc[j - 1], cy1 = AY.ihc[j];
    const T cz0 = AZ.ihc[k - 1], cz1 = AZ.ihc[k];
    const T wx = AX.ihv[i - 1], wy = AY.ihv[j - 1], wz = AZ.ihv[k - 1];
    ax[0] = (s0 - sL) * cx0 + (xy01 - xy00) * wy + (xz01 - xz00) * wz - (p0 - pL) * cx0;
    ax[1] = (sR - s0) * cx1 + (xy11 - xy10) * wy + (xz11 - xz10) * wz - (pR - p0) * cx1;
    ax[2] = (s1 - sF) * cy0 + (xy10 - xy00) * wx + (yz01 - yz00) * wz - (p0 - pF) * cy0;
    ax[3] = (sB - s1) * cy1 + (xy11 - xy01) * wx + (yz11 - yz10) * wz - (pB - p0) * cy1;
    ax[4] = (s2 - sD) * cz0 + (xz10 - xz00) * wx + (yz10 - yz00) * wy - (p0 - pD) * cz0;
    ax[5] = (sU - s2) * cz1 + (xz11 - xz01) * wx + (yz11 - yz01) * wy - (pU - p0) * cz1;
    if (kDiag) {
        const T t43 = (T)(4.0 / 3.0);
        const T eC = E(0), eL = E(1), eR = E(2), eF = E(3), eB = E(4), eD = E(5), eU = E(6);
        const T nxy00 = E(7), nxy01 = E(8), nxy10 = E(9), nxy11 = E(10);
        const T nxz00 = E(11), nxz01 = E(12), nxz10 = E(13), nxz11 = E(14);
        const T nyz00 = E(15), nyz01 = E(16), nyz10 = E(17), nyz11 = E(18);
        d[0] = -(cx0 * t43 * (eC * hx1 + eL * hx0) + wy * two * (nxy01 * ey1 + nxy00 * ey0) + wz * two * (nxz01 * ez1 + nxz00 * ez0));
        d[1] = -(cx1 * t43 * (eR * hx2 + eC * hx1) + wy * two * (nxy11 * ey1 + nxy10 * ey0) + wz * two * (nxz11 * ez1 + nxz10 * ez0));
        d[2] = -(cy0 * t43 * (eC * hy1 + eF * hy0) + wx * two * (nxy10 * ex1 + nxy00 * ex0) + wz * two * (nyz01 * ez1 + nyz00 * ez0));
        d[3] = -(cy1 * t43 * (eB * hy2 + eC * hy1) + wx * two * (nxy11 * ex1 + nxy01 * ex0) + wz * two * (nyz11 * ez1 + nyz10 * ez0));
        d[4] = -(cz0 * t43 * (eC * hz1 + eD * hz0) + wx * two * (nxz10 * ex1 + nxz00 * ex0) + wy * two * (nyz10 * ey1 + nyz00 * ey0));
        d[5] = -(cz1 * t43 * (eU * hz2 + eC * hz1) + wx * two * (nxz11 * ex1 + nxz01 * ex0) + wy * two * (nyz11 * ey1 + nyz01 * ey0));
    }
}

// The same on a level's own fields.
template <typename T>
__device__ __forceinline__ void cell_rows(const LevelView<T> &L, const Fields<T, T> &x, int i, int j, int k,
                                          const int fi[6], T ax[6], T &div)
{
    cell_rows<T, false>(L.ax, L.ay, L.az, L.ny, L.nx * L.ny, x, i, j, k, fi[0], LevelEta<T>{L, fi[0]}, LoadConst{}, ax,
                        div, (T *)nullptr);
}

// Cell of thread t in colour col (cells with (i + j + k) of one parity), or
// false when the slot is past the last cell of its line.
template <typename T>
__device__ __forceinline__ bool colour_cell(const LevelView<T> &L, int col, long t, int &i, int &j, int &k)
{
    const int half = L.ny / 2;
    const long lines = (long)(L.nx - 1) * (L.nz - 1);
    if (t >= lines * half) return false;
    const int jj = (int)(t % half);
    const long line = t / half;
    i = 1 + (int)(line % (L.nx - 1));
    k = 1 + (int)(line / (L.nx - 1));
    j = ((((1 + i + k) & 1) == col) ? 1 : 2) + 2 * jj;
    return j <= L.ny - 1;
}

// the six faces of cell (i, j, k): low and high x, y, z faces
template <typename T>
__device__ __forceinline__ void cell_faces(const LevelView<T> &L, int i, int j, int k, int fi[6])
{
    fi[0] = P2IDX(L, i - 1, j - 1, k - 1);
    fi[1] = P2IDX(L, i, j - 1, k - 1);
    fi[2] = fi[0];
    fi[3] = P2IDX(L, i - 1, j, k - 1);
    fi[4] = fi[0];
    fi[5] = P2IDX(L, i - 1, j - 1, k);
}

// ---------------------------------------------------------------------------
// One colour pass of the cell-block smoother with a diagonal velocity block
// (diagonal Vanka / SCGS) over the cells with (i+j+k)&1 == col.  Each cell
// corrects its six face velocities and its pressure together with the velocity
// block replaced by its diagonal:
//   d_v dv_v + g_v dp = r_v,  sum_v c_v dv_v = r_p.
// Every cell of the colour reads the state from before the pass: velocities
// are read from vin and written to vout (each face belongs to exactly one
// cell of each colour), the pressure is updated in place (a cell's pressure is
// read only by its own face rows among the cells of one colour).  Residuals
// and diagonals come from one set of loads (cell_rows); evaluated row by row
// the FP32 pass took 133 us at 129^3, now 96 us, and 17 us, now 12 us, at 36^3.
template <typename T>
__device__ __forceinline__ void vanka_item(const LevelView<T> &L, T *P, const Vec4<T> &vin, const Vec4<T> &vout,
                                           const Vec4<T> &b, T omega, int col, long t)
{
    int i, j, k;
    if (!colour_cell(L, col, t, i, j, k)) return;
    Fields<T, T> x{P, vin.c[1], vin.c[2], vin.c[3]};
    const int u = P2IDX(L, i, j, k);
    const bool pbc = (L.bcm[u] & BC_P) != 0;
    int fi[6];
    const int fc[6] = {1, 1, 2, 2, 3, 3};
    cell_faces(L, i, j, k, fi);
    bool act[6];
#pragma unroll
    for (int q = 0; q < 6; q++) act[q] = !(L.bcm[fi[q]] & (1 << fc[q]));
    T ax[6], d[6], div;
    cell_rows<T, true>(L.ax, L.ay, L.az, L.ny, L.nx * L.ny, x, i, j, k, fi[0], LevelEta<T>{L, fi[0]}, LoadConst{}, ax,
                       div, d);
    const T g[6] = {-L.ax.ihc[i - 1], L.ax.ihc[i], -L.ay.ihc[j - 1], L.ay.ihc[j], -L.az.ihc[k - 1], L.az.ihc[k]};
    const T hx = L.ax.ih[i], hy = L.ay.ih[j], hz = L.az.ih[k];
    const T cc[6] = {-hx, hx, -hy, hy, -hz, hz};
    T num = 0, den = 0, r[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        r[q] = act[q] ? b.c[fc[q]][fi[q]] - ax[q] : (T)0;
        if (act[q]) {
            num += cc[q] * r[q] / d[q];
            den += cc[q] * g[q] / d[q];
        }
    }
    T dp = 0;
    if (!pbc && den != (T)0) {
        dp = (num - (b.c[0][u] - div)) / den;
        P[u] += omega * dp;
    }
#pragma unroll
    for (int q = 0; q < 6; q++)
        if (act[q] && d[q] != (T)0)
            vout.c[fc[q]][fi[q]] = vin.c[fc[q]][fi[q]] + omega * (r[q] - g[q] * dp) / d[q];
}
template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 4 : 3) k_vanka(LevelView<T> L, T *P, Vec4<T> vin, Vec4<T> vout, Vec4<T> b, T omega,
                                               int col)
{
    pdl_enter();
    vanka_item(L, P, vin, vout, b, omega, col, (long)blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// k_vanka_full with the six momentum residuals from cell_rows (shared
// stresses): same terms as row_vx/row_vy/row_vz, about half the loads and
// arithmetic.  The cell system is built and eliminated on every sweep.
template <typename T>
__global__ void __launch_bounds__(128) k_vanka_fast(LevelView<T> L, T *P, Vec4<T> vin, Vec4<T> vout, Vec4<T> b,
                                                    T omega, int col)
{
    pdl_enter();
    int i, j, k;
    if (!colour_cell(L, col, (long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    Fields<T, T> x{P, vin.c[1], vin.c[2], vin.c[3]};
    const int u = P2IDX(L, i, j, k);
    const bool pact = (L.bcm[u] & BC_P) == 0;
    int fi[6];
    const int fc[6] = {1, 1, 2, 2, 3, 3};
    cell_faces(L, i, j, k, fi);
    const T g[6] = {-L.ax.ihc[i - 1], L.ax.ihc[i], -L.ay.ihc[j - 1], L.ay.ihc[j], -L.az.ihc[k - 1], L.az.ihc[k]};
    const T hx = L.ax.ih[i], hy = L.ay.ih[j], hz = L.az.ih[k];
    const T cc[6] = {-hx, hx, -hy, hy, -hz, hz};
    T ax[6], div;
    cell_rows(L, x, i, j, k, fi, ax, div);
    T M[6][6];
    face_block(L, i, j, k, M);
    M[0][0] = diag_vx(L, i - 1, j - 1, k - 1);
    M[1][1] = diag_vx(L, i, j - 1, k - 1);
    M[2][2] = diag_vy(L, i - 1, j - 1, k - 1);
    M[3][3] = diag_vy(L, i - 1, j, k - 1);
    M[4][4] = diag_vz(L, i - 1, j - 1, k - 1);
    M[5][5] = diag_vz(L, i - 1, j - 1, k);
    bool act[6];
    T y1[6], y2[6];
#pragma unroll
    for (int q = 0; q < 6; q++) act[q] = !(L.bcm[fi[q]] & (1 << fc[q]));
#pragma unroll
    for (int a = 0; a < 6; a++) {
#pragma unroll
        for (int c = 0; c < 6; c++)
            if (!(act[a] && act[c])) M[a][c] = a == c ? (T)1 : (T)0;
        y1[a] = act[a] ? b.c[fc[a]][fi[a]] - ax[a] : (T)0;
        y2[a] = act[a] ? g[a] : (T)0;
    }
#pragma unroll
    for (int c = 0; c < 6; c++) {
        const T ip = (T)1 / M[c][c];
#pragma unroll
        for (int a = 0; a < 6; a++) {
            if (a > c) {
                const T f = M[a][c] * ip;
#pragma unroll
                for (int e = 0; e < 6; e++)
                    if (e > c) M[a][e] -= f * M[c][e];
                y1[a] -= f * y1[c];
                y2[a] -= f * y2[c];
            }
        }
    }
#pragma unroll
    for (int cc5 = 0; cc5 < 6; cc5++) {
        const int c = 5 - cc5;
#pragma unroll
        for (int e = 0; e < 6; e++) {
            if (e > c) {
                y1[c] -= M[c][e] * y1[e];
                y2[c] -= M[c][e] * y2[e];
            }
        }
        const T ip = (T)1 / M[c][c];
        y1[c] *= ip;
        y2[c] *= ip;
    }
    T dp = 0;
    if (pact) {
        T num = -(b.c[0][u] - div), den = 0;
#pragma unroll
        for (int q = 0; q < 6; q++) {
            num += cc[q] * y1[q];
            den += cc[q] * y2[q];
        }
        if (den != (T)0) {
            dp = num / den;
            P[u] += omega * dp;
        }
    }
#pragma unroll
    for (int q = 0; q < 6; q++)
        if (act[q]) vout.c[fc[q]][fi[q]] = vin.c[fc[q]][fi[q]] + omega * (y1[q] - dp * y2[q]);
}

// ---------------------------------------------------------------------------
// Full cell-block smoother with stored cell factors.  The masked cell system
// of k_vanka_full depends on the viscosities and the grid only, so once per
// solve k_vanka_factor inverts the 6x6 face block M of every cell of one
// colour (Gauss-Jordan without pivoting: -M is diagonally dominant; in FP64,
// also for the FP32 cycle, whose factors are stored rounded to float).
// Scaled by the faces' control volumes the block is symmetric: with
// V'_a = ih / ihc along face a's normal (the face's control volume over the
// cell's), S = diag(V') M = S^T, so M^-1 = S^-1 diag(V') with S^-1 symmetric,
// and V'_a g_a = cc_a (the continuity coefficients).  Stored per cell,
// entry-major so that a warp's loads are coalesced:
//   entries 0..20  the upper triangle of S^-1 row by row (rows and columns
//                  of held faces zero);
//   entry 21       1/den, den = cc . S^-1 cc (0 where the cell pressure is a
//                  boundary unknown or den = 0, which holds the pressure).
// The sweep (k_vanka_stored) assembles the residuals with cell_rows and
// applies the stored factors: y1 = S^-1 (V' r), y2 = S^-1 cc,
// dp = (cc . y1 - r_p) / den, v += omega (y1 - dp y2), p += omega dp; the
// same update as k_vanka_full up to rounding, without building and
// eliminating the 6x6 block on every sweep.
constexpr int kBlkEntries = 22;
// packed upper-triangle index of (a, c), a <= c
__host__ __device__ constexpr int tri_index(int a, int c) { return a * 6 - a * (a - 1) / 2 + (c - a); }

template <typename T>
__device__ __forceinline__ T face_ratio(T ih, T ihc) { return ih / ihc; }
template <>
__device__ __forceinline__ float face_ratio<float>(float ih, float ihc) { return __fdividef(ih, ihc); }

template <typename T>
__device__ __forceinline__ void face_volumes(const LevelView<T> &L, int i, int j, int k, T v[6])
{
    const T hx = L.ax.ih[i], hy = L.ay.ih[j], hz = L.az.ih[k];
    v[0] = face_ratio(hx, L.ax.ihc[i - 1]);
    v[1] = face_ratio(hx, L.ax.ihc[i]);
    v[2] = face_ratio(hy, L.ay.ihc[j - 1]);
    v[3] = face_ratio(hy, L.ay.ihc[j]);
    v[4] = face_ratio(hz, L.az.ihc[k - 1]);
    v[5] = face_ratio(hz, L.az.ihc[k]);
}

template <typename T, typename S>
__global__ void __launch_bounds__(128) k_vanka_factor(LevelView<T> L, int col, S *blk, long stride)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (!colour_cell(L, col, t, i, j, k)) return;
    const int u = P2IDX(L, i, j, k);
    int fi[6];
    const int fc[6] = {1, 1, 2, 2, 3, 3};
    cell_faces(L, i, j, k, fi);
    const T hx = L.ax.ih[i], hy = L.ay.ih[j], hz = L.az.ih[k];
    const T cc[6] = {-hx, hx, -hy, hy, -hz, hz};
    T M[6][6];
    face_block(L, i, j, k, M);
    M[0][0] = diag_vx(L, i - 1, j - 1, k - 1);
    M[1][1] = diag_vx(L, i, j - 1, k - 1);
    M[2][2] = diag_vy(L, i - 1, j - 1, k - 1);
    M[3][3] = diag_vy(L, i - 1, j, k - 1);
    M[4][4] = diag_vz(L, i - 1, j - 1, k - 1);
    M[5][5] = diag_vz(L, i - 1, j - 1, k);
    bool act[6];
#pragma unroll
    for (int q = 0; q < 6; q++) act[q] = !(L.bcm[fi[q]] & (1 << fc[q]));
#pragma unroll
    for (int a = 0; a < 6; a++)
#pragma unroll
        for (int c = 0; c < 6; c++)
            if (!(act[a] && act[c])) M[a][c] = a == c ? (T)1 : (T)0;
    // in-place Gauss-Jordan inverse
#pragma unroll
    for (int c = 0; c < 6; c++) {
        const T ip = (T)1 / M[c][c];
        M[c][c] = (T)1;
#pragma unroll
        for (int e = 0; e < 6; e++) M[c][e] *= ip;
#pragma unroll
        for (int a = 0; a < 6; a++) {
            if (a != c) {
                const T f = M[a][c];
                M[a][c] = (T)0;
#pragma unroll
                for (int e = 0; e < 6; e++) M[a][e] -= f * M[c][e];
            }
        }
    }
    // S^-1 = M^-1 diag(V')^-1, symmetrised; held rows and columns zero
    T v[6];
    face_volumes(L, i, j, k, v);
#pragma unroll
    for (int a = 0; a < 6; a++)
#pragma unroll
        for (int c = 0; c < 6; c++)
            M[a][c] = (act[a] && act[c]) ? M[a][c] / v[c] : (T)0;
    T den = 0;
#pragma unroll
    for (int a = 0; a < 6; a++) {
        T y2 = 0;
#pragma unroll
        for (int c = 0; c < 6; c++) y2 += (T)0.5 * (M[a][c] + M[c][a]) * cc[c];
        den += cc[a] * y2;
    }
#pragma unroll
    for (int a = 0; a < 6; a++)
#pragma unroll
        for (int c = a; c < 6; c++) blk[(long)tri_index(a, c) * stride + t] = to_factor<S>((T)0.5 * (M[a][c] + M[c][a]));
    const bool pact = (L.bcm[u] & BC_P) == 0;
    blk[21L * stride + t] = to_factor<S>((pact && den != (T)0) ? (T)1 / den : (T)0);
}

template <typename T>
__device__ __forceinline__ void vanka_stored_item(const LevelView<T> &L, T *P, const Vec4<T> &vin,
                                                  const Vec4<T> &vout, const Vec4<T> &b, T omega, int col,
                                                  const factor_t<T> *__restrict__ blk, long stride, long t)
{
    int i, j, k;
    if (!colour_cell(L, col, t, i, j, k)) return;
    Fields<T, T> x{P, vin.c[1], vin.c[2], vin.c[3]};
    const int u = P2IDX(L, i, j, k);
    int fi[6];
    const int fc[6] = {1, 1, 2, 2, 3, 3};
    cell_faces(L, i, j, k, fi);
    T ax[6], div;
    cell_rows(L, x, i, j, k, fi, ax, div);
    const T hx = L.ax.ih[i], hy = L.ay.ih[j], hz = L.az.ih[k];
    const T cc[6] = {-hx, hx, -hy, hy, -hz, hz};
    T v[6];
    face_volumes(L, i, j, k, v);
    bool act[6];
    T vr[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        act[q] = !(L.bcm[fi[q]] & (1 << fc[q]));
        vr[q] = act[q] ? (b.c[fc[q]][fi[q]] - ax[q]) * v[q] : (T)0;
    }
    T y1[6] = {0, 0, 0, 0, 0, 0}, y2[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int a = 0; a < 6; a++) {
#pragma unroll
        for (int c = a; c < 6; c++) {
            const T m = ld_factor(blk + (long)tri_index(a, c) * stride + t);
            y1[a] += m * vr[c];
            y2[a] += m * cc[c];
            if (c != a) {
                y1[c] += m * vr[a];
                y2[c] += m * cc[a];
            }
        }
    }
    const T inv = ld_factor(blk + 21L * stride + t);
    T dp = 0;
    if (inv != (T)0) {
        T num = -(b.c[0][u] - div);
#pragma unroll
        for (int q = 0; q < 6; q++) num += cc[q] * y1[q];
        dp = num * inv;
        P[u] += omega * dp;
    }
#pragma unroll
    for (int q = 0; q < 6; q++)
        if (act[q]) vout.c[fc[q]][fi[q]] = vin.c[fc[q]][fi[q]] + omega * (y1[q] - dp * y2[q]);
}
// Latency-bound: what counts is how many of a cell's about 70 loads are in
// flight.  FP32: 128 registers, with the viscosities and pressures loaded ahead
// (cell_rows): 72 / 16.4 / 10.3 / 8.8 us a pass on the levels of 129^3 where 72
// registers with seven blocks an SM took 74 / 20.7 / 12.4 / 12.3 us.  FP64: 168
// registers, loads where they are used: 176 us against 199 us, and 205 us with
// the loads ahead.
template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 4 : 3) k_vanka_stored(
    LevelView<T> L, T *P, Vec4<T> vin, Vec4<T> vout, Vec4<T> b, T omega, int col,
    const factor_t<T> *__restrict__ blk, long stride)
{
    pdl_enter();
    vanka_stored_item(L, P, vin, vout, b, omega, col, blk, stride, (long)blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Transfers.  Per-axis tables (host-built from the reference's index rules,
// move3mgNew.c:3562-3575 and the corresponding blocks of vprestrict and
// vpprolong): for a fine index m, the coarse interval lo[m] and the weights
// w0 (coarse lo) and w1 (coarse lo+1).  Restriction uses the inverse lists.
__device__ __forceinline__ int ax_type(int comp, int axis)
{
    if (comp == 0) return 2;
    return (comp == axis + 1) ? 0 : 1;
}

__device__ __forceinline__ double block_sum(double v, double *sh);  // below (norms)

// tv.m[axis][type] for a runtime type without copying the parameter struct
__device__ __forceinline__ AxisMap pick_map(const AxisMap (&m)[3], int type)
{
    return type == 0 ? m[0] : (type == 1 ? m[1] : m[2]);
}

// Restriction (vprestrict, move3mgNew.c:3965-4353): b_c = sum_f w r_f / sum_f w
// over the non-boundary fine rows (pressure residuals scaled by eta_f/eta_c,
// 4308), for non-boundary coarse rows (0 otherwise); x_c = 0 (4351).  The
// residual is 0 on boundary rows, so the numerator needs no mask; the weights'
// sums without them are fixed by the tables (k_restrict_weights).  A block
// takes 256 / kSplit consecutive (component, coarse node) pairs, components
// outermost, and its kSplit groups of threads take the entries of the z lists
// in turn.  Without the mask loads and the weight sums 257^3 -> 131^3 takes 0.63
// ms (0.94 with them, 0.05 of the HBM rate: bound by its gathers' instructions),
// 20^3 -> 12^3 14.5 us with four threads a pair (23.5 us).  Fused with the first half of the coarse
// right-hand-side compatibility shift: every block with pressure rows adds its
// volume-weighted continuity rows into partial[block]; the last of them to
// finish (ticket counter, reset by that block) sums the partials in block order
// and writes sums[0] = sum of vol * b_P and sums[1] = vol_total (fixed per
// level).
constexpr int kRestrictList = 5;   // longest inverse list of one axis (host-checked)
constexpr int kRestrictStride = 8; // entries reserved per coarse index in the padded lists
constexpr int kRestrictThreads = 256;

// Padded inverse lists of one axis: fine index and weight e of coarse index I
// at [I * kRestrictStride + e]; unused entries repeat a valid index with
// weight 0.
template <typename T>
__device__ __forceinline__ void restrict_lists(const AxisMap &m, int I, int idx[kRestrictList], T w[kRestrictList])
{
#pragma unroll
    for (int e = 0; e < kRestrictList; e++) {
        idx[e] = __ldg(m.pidx + I * kRestrictStride + e);
        w[e] = (T)__ldg(m.pw + I * kRestrictStride + e);
    }
}

// ws[c * n + v]: sum of the weights of the regular fine rows of coarse row (v, c)
template <typename T>
__global__ void k_restrict_weights(LevelView<T> F, LevelView<T> Cl, TransferView tv, T *ws)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4L * Cl.n) return;
    const int c = (int)(t / Cl.n), v = (int)(t % Cl.n);
    const int J = v % Cl.ny, I = (v / Cl.ny) % Cl.nx, K = v / (Cl.nx * Cl.ny);
    int xi[kRestrictList], yi[kRestrictList], zi[kRestrictList];
    T xw[kRestrictList], yw[kRestrictList], zw[kRestrictList];
    restrict_lists(pick_map(tv.m[0], ax_type(c, 0)), I, xi, xw);
    restrict_lists(pick_map(tv.m[1], ax_type(c, 1)), J, yi, yw);
    restrict_lists(pick_map(tv.m[2], ax_type(c, 2)), K, zi, zw);
    T s = 0;
    for (int a = 0; a < kRestrictList; a++)
        for (int d = 0; d < kRestrictList; d++)
            for (int e = 0; e < kRestrictList; e++) {
                const int f = zi[a] * (F.nx * F.ny) + xi[d] * F.ny + yi[e];
                if (!(F.bcm[f] & (1 << c))) s += zw[a] * xw[d] * yw[e];
            }
    ws[t] = s;
}

template <typename T, int kSplit>
__global__ void __launch_bounds__(kRestrictThreads) k_restrict_compat(
    LevelView<T> F, Vec4<T> rf, LevelView<T> Cl, Vec4<T> bc, Vec4<T> xc, TransferView tv, int scale_p,
    const T *__restrict__ wsum, double vol_total, double *partial, unsigned *ticket, double *sums)
{
    pdl_enter();
    constexpr int kPairs = kRestrictThreads / kSplit;
    __shared__ double sh[32];
    __shared__ T part[kSplit][kPairs];
    __shared__ bool last;
    const int n = Cl.n, pair = threadIdx.x % kPairs, zs = threadIdx.x / kPairs;
    const long t = (long)blockIdx.x * kPairs + pair;
    double contrib = 0;
    bool row = false;
    int c = 0, v = 0, I = 0, J = 0, K = 0;
    T acc = 0;
    if (t < 4L * n) {
        c = (int)(t / n);
        v = (int)(t % n);
        J = v % Cl.ny;
        I = (v / Cl.ny) % Cl.nx;
        K = v / (Cl.nx * Cl.ny);
        row = valid_pos(c, I, J, K, Cl.nx, Cl.ny, Cl.nz) && !(Cl.bcm[v] & (1 << c));
    }
    if (row) {
        const T *rfc = c == 0 ? rf.c[0] : (c == 1 ? rf.c[1] : (c == 2 ? rf.c[2] : rf.c[3]));
        const AxisMap mz = pick_map(tv.m[2], ax_type(c, 2));
        int xi[kRestrictList], yi[kRestrictList];
        T xw[kRestrictList], yw[kRestrictList];
        restrict_lists(pick_map(tv.m[0], ax_type(c, 0)), I, xi, xw);
        restrict_lists(pick_map(tv.m[1], ax_type(c, 1)), J, yi, yw);
#pragma unroll
        for (int q0 = 0; q0 < kRestrictList; q0 += kSplit) {
            const int q = q0 + zs;
            if (q >= kRestrictList) break;
            const T wz = (T)__ldg(mz.pw + K * kRestrictStride + q);
            const int base = __ldg(mz.pidx + K * kRestrictStride + q) * (F.nx * F.ny);
            if (wz == (T)0) continue;
            T line = 0;
#pragma unroll
            for (int ax = 0; ax < kRestrictList; ax++) {
                if (xw[ax] == (T)0) continue;
                const int f = base + xi[ax] * F.ny;
                T s = 0;
#pragma unroll
                for (int ay = 0; ay < kRestrictList; ay++) {
                    if (ay == kRestrictList - 1 && yw[ay] == (T)0) continue;
                    T val = __ldg(rfc + f + yi[ay]);
                    if (c == 0 && scale_p) val *= (T)__ldg(F.ec + f + yi[ay]);
                    s += val * yw[ay];
                }
                line += s * xw[ax];
            }
            acc += line * wz;
        }
    }
    if (kSplit > 1) {
        if (zs > 0) part[zs][pair] = acc;
        __syncthreads();
    }
    if (zs == 0 && t < 4L * n) {
#pragma unroll
        for (int e = 1; e < kSplit; e++) acc += part[e][pair];
        T out = 0;
        if (row) {
            const T ws = wsum[t];
            // the pressure residuals' viscosity ratio eta_f / eta_c: eta_f per fine node above, the division here
            if (c == 0 && scale_p) acc /= (T)Cl.ec[v];
            out = ws != (T)0 ? acc / ws : (T)0;
            if (c == 0 && I > 0 && J > 0 && K > 0)
                contrib = (double)out / ((double)Cl.ax.ih[I] * (double)Cl.ay.ih[J] * (double)Cl.az.ih[K]);
        }
        (c == 0 ? xc.c[0] : (c == 1 ? xc.c[1] : (c == 2 ? xc.c[2] : xc.c[3])))[v] = 0;
        (c == 0 ? bc.c[0] : (c == 1 ? bc.c[1] : (c == 2 ? bc.c[2] : bc.c[3])))[v] = out;
    }
    const unsigned pblocks = (unsigned)((n + kPairs - 1) / kPairs);
    if (blockIdx.x >= pblocks) return;
    const double bsum = block_sum(contrib, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = bsum;
        __threadfence();
        last = atomicAdd(ticket, 1u) == pblocks - 1;
    }
    __syncthreads();
    if (last) {
        __threadfence();
        double s = 0;
        for (int q = threadIdx.x; q < (int)pblocks; q += blockDim.x) s += ((volatile double *)partial)[q];
        s = block_sum(s, sh);
        if (threadIdx.x == 0) {
            sums[0] = s;
            sums[1] = vol_total;
            *ticket = 0;
        }
    }
}
inline unsigned restrict_blocks(long n, int split)
{
    const long pairs = kRestrictThreads / split;
    return (unsigned)((4 * n + pairs - 1) / pairs);
}

// x_f += sum_c w x_c * (p1koef | v1koef) over every fine unknown position.
template <typename T>
__device__ __forceinline__ void prolong_item(const LevelView<T> &F, const Vec4<T> &xf, const LevelView<T> &Cl,
                                             const Vec4<T> &xc, const TransferView &tv, T p1, T v1, int u)
{
    if (u >= F.n) return;
    int j = u % F.ny, i = (u / F.ny) % F.nx, k = u / (F.nx * F.ny);
    for (int c = 0; c < 4; c++) {
        if (!valid_pos(c, i, j, k, F.nx, F.ny, F.nz)) continue;
        const AxisMap &mx = tv.m[0][ax_type(c, 0)], &my = tv.m[1][ax_type(c, 1)], &mz = tv.m[2][ax_type(c, 2)];
        int lx = mx.lo[i], ly = my.lo[j], lz = mz.lo[k];
        T wx0 = (T)mx.w0[i], wx1 = (T)mx.w1[i], wy0 = (T)my.w0[j], wy1 = (T)my.w1[j];
        T wz0 = (T)mz.w0[k], wz1 = (T)mz.w1[k];
        T s = 0;
#pragma unroll
        for (int d = 0; d < 2; d++)
#pragma unroll
            for (int a = 0; a < 2; a++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    T w = (d ? wz1 : wz0) * (a ? wx1 : wx0) * (e ? wy1 : wy0);
                    s += xc.c[c][P2IDX(Cl, lx + a, ly + e, lz + d)] * w;
                }
        xf.c[c][u] += s * (c == 0 ? p1 : v1);
    }
}
template <typename T>
__global__ void k_prolong(LevelView<T> F, Vec4<T> xf, LevelView<T> Cl, Vec4<T> xc, TransferView tv, T p1, T v1)
{
    pdl_enter();
    prolong_item(F, xf, Cl, xc, tv, p1, v1, blockIdx.x * blockDim.x + threadIdx.x);
}

// ronurestrict (move3mgNew.c:3386-3527): coarse nu, ro as weighted averages
// of the fine node values (nu averaged as nu, log nu or 1/nu per viscmod).
__global__ void k_ronurestrict(int fnx, int fny, int fnz, const float *fnu, const float *fro, int cnx, int cny,
                               int cnz, float *cnu, float *cro, AxisMap mx, AxisMap my, AxisMap mz, int viscmod)
{
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= cnx * cny * cnz) return;
    int J = v % cny, I = (v / cny) % cnx, K = v / (cnx * cny);
    double sn = 0, sr = 0, sw = 0;
    for (int qz = mz.ptr[K]; qz < mz.ptr[K + 1]; qz++)
        for (int qx = mx.ptr[I]; qx < mx.ptr[I + 1]; qx++)
            for (int qy = my.ptr[J]; qy < my.ptr[J + 1]; qy++) {
                int f = mz.idx[qz] * fnx * fny + mx.idx[qx] * fny + my.idx[qy];
                double w = mz.w[qz] * mx.w[qx] * my.w[qy];
                double nv = fnu[f];
                double fv = viscmod == 0 ? nv : (viscmod == 1 ? log(nv) : 1.0 / nv);
                sn += fv * w;
                sr += (double)fro[f] * w;
                sw += w;
            }
    double nv = sn / sw;
    if (viscmod == 1) nv = exp(nv);
    if (viscmod == 2) nv = 1.0 / nv;
    cnu[v] = (float)nv;
    cro[v] = (float)(sr / sw);
}

__device__ __forceinline__ double vmean(int viscmod, const double *v, int n)
{
    double s = 0;
    if (viscmod == 0) {
        for (int i = 0; i < n; i++) s += v[i];
        return s / n;
    }
    if (viscmod == 1) {
        for (int i = 0; i < n; i++) s += log(v[i]);
        return exp(s / n);
    }
    for (int i = 0; i < n; i++) s += 1.0 / v[i];
    return 1.0 / (s / n);
}

__device__ __forceinline__ double clampd(double v, double lo, double hi)
{
    if (v > hi) v = hi;
    if (v < lo) v = lo;
    return v;
}

// Per-stencil viscosities of one level, clamped to [nubeg, nuend]: level 0
// from nxx..nyz (sxxcalc:36-38, sxycalc:433-435, ...); coarse levels from the
// 8 cell-corner (sxx) or 2 edge-end (sxy, sxz, syz) nu values (41-47, 438-444).
__global__ void k_level_eta(int nx, int ny, int nz, const float *nu, const float *nxx, const float *nxy,
                            const float *nxz, const float *nyz, float *ec, float *exy, float *exz, float *eyz,
                            double lo, double hi, int viscmod, int level0)
{
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nx * ny * nz) return;
    if (level0) {
        ec[u] = (float)clampd(nxx[u], lo, hi);
        exy[u] = (float)clampd(nxy[u], lo, hi);
        exz[u] = (float)clampd(nxz[u], lo, hi);
        eyz[u] = (float)clampd(nyz[u], lo, hi);
        return;
    }
    int j = u % ny, i = (u / ny) % nx, k = u / (nx * ny);
    int xy = nx * ny;
    if (i > 0 && j > 0 && k > 0) {
        double v[8] = {nu[u - xy - ny - 1], nu[u - xy - ny], nu[u - xy - 1], nu[u - xy],
                       nu[u - ny - 1],      nu[u - ny],      nu[u - 1],      nu[u]};
        ec[u] = (float)clampd(vmean(viscmod, v, 8), lo, hi);
    } else {
        ec[u] = (float)lo;
    }
    double v2[2];
    v2[0] = nu[u];
    v2[1] = k + 1 < nz ? nu[u + xy] : nu[u];
    exy[u] = (float)clampd(vmean(viscmod, v2, 2), lo, hi);
    v2[1] = j + 1 < ny ? nu[u + 1] : nu[u];
    exz[u] = (float)clampd(vmean(viscmod, v2, 2), lo, hi);
    v2[1] = i + 1 < nx ? nu[u + ny] : nu[u];
    eyz[u] = (float)clampd(vmean(viscmod, v2, 2), lo, hi);
}

// Level-0 right-hand sides of the Stokes rows (xstokserr:845, ystokserr:1060,
// zstokserr:1279): -g * (sum of 4 float densities, summed in float) / 4.
template <typename T>
__global__ void k_rhs0(int nx, int ny, int nz, const float *ro, const uint8_t *bcm, Vec4<T> b, double gxk, double gyk,
                       double gzk)
{
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nx * ny * nz) return;
    int j = u % ny, i = (u / ny) % nx, k = u / (nx * ny);
    int xy = nx * ny;
    uint8_t m = bcm[u];
    b.c[0][u] = 0;
    T vx = 0, vy = 0, vz = 0;
    if (valid_pos(1, i, j, k, nx, ny, nz) && !(m & BC_VX)) {
        float s = ro[u] + ro[u + 1] + ro[u + xy] + ro[u + xy + 1];
        vx = (T)(-gxk * (double)s / 4.0);
    }
    if (valid_pos(2, i, j, k, nx, ny, nz) && !(m & BC_VY)) {
        float s = ro[u] + ro[u + ny] + ro[u + xy] + ro[u + xy + ny];
        vy = (T)(-gyk * (double)s / 4.0);
    }
    if (valid_pos(3, i, j, k, nx, ny, nz) && !(m & BC_VZ)) {
        float s = ro[u] + ro[u + 1] + ro[u + ny] + ro[u + ny + 1];
        vz = (T)(-gzk * (double)s / 4.0);
    }
    b.c[1][u] = vx;
    b.c[2][u] = vy;
    b.c[3][u] = vz;
}

// Boundary-row constants into the level-0 right-hand side.
template <typename T>
__global__ void k_bc_consts(int nbc, const int *bu, const float *bconst, Vec4<T> b)
{
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nbc) return;
    int uc = bu[q];
    b.c[uc & 3][uc >> 2] = (T)bconst[q];
}

// ---------------------------------------------------------------------------
// Deterministic reductions: a block tree; partials are summed in block order.

__device__ __forceinline__ double block_sum(double v, double *sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double s = 0;
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    }
    __syncthreads();
    return s;
}

// Sum of volume * b_P over continuity rows and of the volumes (compatibility).
template <typename T>
__device__ __forceinline__ void compat_apply_item(const LevelView<T> &L, T *bp, double s0, double s1, int u)
{
    if (u >= L.n || s1 <= 0) return;
    int j = u % L.ny, i = (u / L.ny) % L.nx, k = u / (L.nx * L.ny);
    if (i == 0 || j == 0 || k == 0 || (L.bcm[u] & BC_P)) return;
    bp[u] -= (T)(s0 / s1);
}
template <typename T>
__global__ void k_compat_apply(LevelView<T> L, T *bp, const double *sums)
{
    pdl_enter();
    compat_apply_item(L, bp, sums[0], sums[1], blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Small vector kernels.
__global__ void k_f32_to_f64(int n, Vec4<float> a, Vec4<double> b)
{
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
#pragma unroll
    for (int c = 0; c < 4; c++) b.c[c][u] = (double)a.c[c][u];
}

// Pressure shift so that the pinned cell holds pin_value (move3mgNew.c:2834-2855).
__global__ void k_pressure_shift_value(const double *p, int pin, double pin_value, double *shift)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) shift[0] = pin >= 0 ? pin_value - p[pin] : 0.0;
}
__global__ void k_pressure_shift(int nx, int ny, int nz, double *p, const double *shift)
{
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nx * ny * nz) return;
    int j = u % ny, i = (u / ny) % nx, k = u / (nx * ny);
    if (i > 0 && j > 0 && k > 0) p[u] += shift[0];
}

}  // namespace p2
