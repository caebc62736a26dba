// All smoothing sweeps of a small level in one launch.
//
// On a level of up to about 43^3 nodes a colour pass as a launch of its own,
// followed by a launch for the boundary rows, is all latency: it waits for one
// chain of loads and for two launches.  Here every cell of both colours has a
// thread for the whole call.  What does not change between sweeps (the cell's
// factors or diagonals, viscosities, right-hand side, the spacings) is read
// once into shared memory; a pass loads the cell's 36 velocities and 7
// pressures, relaxes it, and writes its faces, its pressure and the boundary
// rows that copy them.  All four fields alternate between two buffers, so one
// barrier per pass is enough: nothing written in a pass is read in it.
// Levels of at most kResSlots slots per colour a block on 16 blocks (about
// 20^3) run as one cluster with the hardware's cluster barrier; larger ones as
// a cooperative grid, one block per SM, with a counter in global memory.
// A pass takes 3.0 / 3.5 / 3.9 us (FP32, stored factors) on 12^3 / 20^3 / 36^3:
// the barrier, one round of loads from L2 and one cell's chain of about 600
// instructions.  V-cycles: 33^3 0.260 -> 0.231 ms, 129^3 with doubling sweeps
// 4.03 -> 3.26 ms, 257^3 11.76 -> 11.15 ms.  The grid form keeps every SM for its
// launch, so concurrent solves take passes where those give the same bits
// (Solver::passes_in_batch).
#pragma once

#include "p2_barrier.cuh"
#include "p2_kernels.cuh"

namespace p2 {

constexpr int kResThreads = 512;              // two colours of kResSlots cells
constexpr int kResSlots = kResThreads / 2;
constexpr int kResCluster = 16;

// Boundary rows for the resident sweeps: the rows' chains as for
// k_bc_set_chain, and per colour and slot the rows that follow one of the
// cell's unknowns: {unknown * 8 + face (0..5, 6 for the pressure), row, bits of the
// product of the chain's coefficients}: a float's, or the two halves of a double
// where no float holds it (the first entry then has its top bit set).
struct ResidentBC {
    int nbc;
    const int *bu, *bt, *bnext;
    const float *bk;
    const int *ptr;
    const int4 *dep;
    int cap;  // most entries of one block
};

struct LoadPlain {
    template <typename T>
    __device__ __forceinline__ T operator()(const T *p) const { return *p; }
};
struct SharedEta {
    const float *e;
    int stride;
    __device__ __forceinline__ float operator()(int q) const { return e[q * stride]; }
};

// values stored per cell besides the right-hand side: the 22 factor entries,
// or 1/d of the six rows and 1/den of the diagonal block
template <bool kFull>
__host__ __device__ constexpr int res_values() { return kFull ? kBlkEntries : 7; }
// a row that follows an unknown of the block's cells: its constant part, coefficient, unknown and face
template <typename T>
struct ResDep {
    T c;
    float k;
    int what;  // as in ResidentBC::dep
};
constexpr size_t kResSmemMax = 227 * 1024 - 64;
template <typename T, bool kFull>
__host__ __device__ constexpr size_t res_smem(int threads, int tab, int cap)
{
    return (sizeof(T) * (res_values<kFull>() + 7) + sizeof(float) * kCellEta) * (size_t)threads +
           sizeof(T) * 12 * (size_t)tab + sizeof(ResDep<T>) * (size_t)cap;
}

template <typename T, bool kFull, bool kCluster>
__global__ void __launch_bounds__(kResThreads, 1) k_smooth_resident(LevelView<T> L, Vec4<T> x, Vec4<T> y, Vec4<T> b,
                                                                    T omega, int passes,
                                                                    const factor_t<T> *__restrict__ blk, long stride,
                                                                    ResidentBC R, int tabn, const T *tab,
                                                                    GridBarrier B)
{
    constexpr int kV = res_values<kFull>();
    extern __shared__ unsigned char res_sm[];
    __shared__ bool ok;
    const int nt = blockDim.x, tid = threadIdx.x, S = nt / 2;
    T *val = (T *)res_sm + tid;                         // [kV][nt]
    T *rhs = (T *)res_sm + (size_t)kV * nt + tid;       // [7][nt]
    T *tabs = (T *)res_sm + (size_t)(kV + 7) * nt;      // 12 tables
    ResDep<T> *deps = (ResDep<T> *)(tabs + 12 * tabn);  // [cap]
    float *eta = (float *)(deps + R.cap) + tid;         // [kCellEta][nt]
    const int col = tid >= S;
    const long slot = (long)blockIdx.x * S + (tid - col * S);
    const long slots = (long)(L.nx - 1) * (L.nz - 1) * (L.ny / 2);
    int i = 1, j = 1, k = 1;
    const bool valid = colour_cell(L, col, slot, i, j, k);
    for (int q = tid; q < 12 * tabn; q += nt) tabs[q] = tab[q];
    const Axis<T> AX{tabs, tabs + tabn, tabs + 2 * tabn, tabs + 3 * tabn};
    const Axis<T> AY{tabs + 4 * tabn, tabs + 5 * tabn, tabs + 6 * tabn, tabs + 7 * tabn};
    const Axis<T> AZ{tabs + 8 * tabn, tabs + 9 * tabn, tabs + 10 * tabn, tabs + 11 * tabn};
    const int sy = L.ny, sz = L.nx * L.ny;
    const int F = valid ? P2IDX(L, i - 1, j - 1, k - 1) : 0, u = F + sz + sy + 1;
    int fi[6];
    const int fc[6] = {1, 1, 2, 2, 3, 3};
    fi[0] = fi[2] = fi[4] = F;
    fi[1] = F + sy;
    fi[3] = F + 1;
    fi[5] = F + sz;
    unsigned act = 0;       // bit q: face q is a regular row
    bool pown = false;      // the cell's pressure is no boundary row
    int d0 = 0, d1 = 0;
    if (valid) {
#pragma unroll
        for (int q = 0; q < 6; q++) act |= (L.bcm[fi[q]] & (1 << fc[q])) ? 0u : 1u << q;
        pown = !(L.bcm[u] & BC_P);
#pragma unroll
        for (int q = 0; q < kCellEta; q++) eta[q * nt] = (float)LevelEta<T>{L, F}(q);
        if (kFull) {
            const factor_t<T> *f = blk + (size_t)col * kBlkEntries * stride + slot;
#pragma unroll
            for (int q = 0; q < kBlkEntries; q++) val[q * nt] = ld_factor(f + q * stride);
        }
        d0 = R.ptr[col * slots + slot];
        d1 = R.ptr[col * slots + slot + 1];
    }
    // the block's entries of both colours, one range after the other; its thread's own become local indices
    const long s0 = min((long)blockIdx.x * S, slots), s1 = min(s0 + S, slots);
    const int e0 = R.ptr[s0], n0 = R.ptr[s1] - e0, e1 = R.ptr[slots + s0], n1 = R.ptr[slots + s1] - e1;
    d0 -= col ? e1 - n0 : e0;
    d1 -= col ? e1 - n0 : e0;
    // everything above is constant over the solve; below, the previous kernel's results
    asm volatile("griddepcontrol.wait;" ::: "memory");
    T p = 0;
    if (valid) {
        p = x.c[0][u];
        rhs[6 * nt] = b.c[0][u];
#pragma unroll
        for (int q = 0; q < 6; q++) rhs[q * nt] = b.c[fc[q]][fi[q]];
    }
    // boundary rows of both buffers from the incoming state, as k_bc_set_chain evaluates them
    auto row_value = [&](int r0, bool constant) {
        int chain[kMaxBcChain], m = 0, r = r0;
        chain[m++] = r;
        while (R.bnext[r] >= 0 && m < kMaxBcChain) {
            r = R.bnext[r];
            chain[m++] = r;
        }
        const int t = R.bt[r];
        int uc = R.bu[r];
        T v = b.c[uc & 3][uc >> 2];
        if (!constant && t >= 0) v += (T)R.bk[r] * x.c[t & 3][t >> 2];
        for (int s = m - 2; s >= 0; s--) {
            const int rr = chain[s];
            uc = R.bu[rr];
            v = b.c[uc & 3][uc >> 2] + (T)R.bk[rr] * v;
        }
        return v;
    };
    for (int r = blockIdx.x * nt + tid; r < R.nbc; r += gridDim.x * nt) {
        const int uc = R.bu[r];
        const T v = row_value(r, false);
        x.c[uc & 3][uc >> 2] = v;
        y.c[uc & 3][uc >> 2] = v;
    }
    for (int e = tid; e < n0 + n1; e += nt) {
        const int4 D = R.dep[e < n0 ? e0 + e : e1 + e - n0];
        deps[e] = ResDep<T>{row_value(D.y, true), D.x < 0 ? (float)__hiloint2double(D.w, D.z) : __int_as_float(D.z), D.x};
    }
    __syncthreads();  // the tables and entries
    if (!kFull && valid) {
        T ax[6], div, d[6];
        const Fields<T, T> f{x.c[0], x.c[1], x.c[2], x.c[3]};
        cell_rows<T, true>(AX, AY, AZ, sy, sz, f, i, j, k, F, SharedEta{eta, nt}, LoadPlain{}, ax, div, d);
        const T g[6] = {-AX.ihc[i - 1], AX.ihc[i], -AY.ihc[j - 1], AY.ihc[j], -AZ.ihc[k - 1], AZ.ihc[k]};
        const T cc[6] = {-AX.ih[i], AX.ih[i], -AY.ih[j], AY.ih[j], -AZ.ih[k], AZ.ih[k]};
        T den = 0;
#pragma unroll
        for (int q = 0; q < 6; q++) {
            const T di = (act >> q & 1) && d[q] != (T)0 ? (T)1 / d[q] : (T)0;
            val[q * nt] = di;
            den += cc[q] * g[q] * di;
        }
        val[6 * nt] = pown && den != (T)0 ? (T)1 / den : (T)0;
    }
    unsigned target = 0;
    bool go = res_sync<kCluster>(B, target, &ok);
    // the buffers of this pass's input and output
    T *i0 = x.c[0], *i1 = x.c[1], *i2 = x.c[2], *i3 = x.c[3], *o0 = y.c[0], *o1 = y.c[1], *o2 = y.c[2], *o3 = y.c[3];
    auto swap = [](T *&a, T *&c) { T *t = a; a = c; c = t; };
    for (int s = 0; go && s < passes; s++) {
        const bool odd = s & 1;
        if (s + 1 == passes) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        if (valid) {
            const bool mine = col == (int)odd;
            T vn[6];
            if (mine) {
                const Fields<T, T> f{i0, i1, i2, i3};
                T ax[6], div;
                cell_rows<T, false>(AX, AY, AZ, sy, sz, f, i, j, k, F, SharedEta{eta, nt}, LoadPlain{}, ax, div,
                                    (T *)nullptr);
                const T hx = AX.ih[i], hy = AY.ih[j], hz = AZ.ih[k];
                const T cc[6] = {-hx, hx, -hy, hy, -hz, hz};
                T dv[6], dp = 0;
                if (kFull) {
                    const T vol[6] = {face_ratio(hx, AX.ihc[i - 1]), face_ratio(hx, AX.ihc[i]),
                                      face_ratio(hy, AY.ihc[j - 1]), face_ratio(hy, AY.ihc[j]),
                                      face_ratio(hz, AZ.ihc[k - 1]), face_ratio(hz, AZ.ihc[k])};
                    T vr[6], y1[6] = {0, 0, 0, 0, 0, 0}, y2[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
                    for (int q = 0; q < 6; q++) vr[q] = act >> q & 1 ? (rhs[q * nt] - ax[q]) * vol[q] : (T)0;
#pragma unroll
                    for (int a = 0; a < 6; a++) {
#pragma unroll
                        for (int c = a; c < 6; c++) {
                            const T m = val[tri_index(a, c) * nt];
                            y1[a] += m * vr[c];
                            y2[a] += m * cc[c];
                            if (c != a) {
                                y1[c] += m * vr[a];
                                y2[c] += m * cc[a];
                            }
                        }
                    }
                    const T inv = val[21 * nt];
                    if (inv != (T)0) {
                        T num = -(rhs[6 * nt] - div);
#pragma unroll
                        for (int q = 0; q < 6; q++) num += cc[q] * y1[q];
                        dp = num * inv;
                    }
#pragma unroll
                    for (int q = 0; q < 6; q++) dv[q] = y1[q] - dp * y2[q];
                } else {
                    const T g[6] = {-AX.ihc[i - 1], AX.ihc[i], -AY.ihc[j - 1], AY.ihc[j], -AZ.ihc[k - 1], AZ.ihc[k]};
                    T num = -(rhs[6 * nt] - div), r[6];
#pragma unroll
                    for (int q = 0; q < 6; q++) {
                        r[q] = act >> q & 1 ? (rhs[q * nt] - ax[q]) * val[q * nt] : (T)0;
                        num += cc[q] * r[q];
                    }
                    if (val[6 * nt] != (T)0) dp = num * val[6 * nt];
#pragma unroll
                    for (int q = 0; q < 6; q++) dv[q] = r[q] - g[q] * dp * val[q * nt];
                }
                p += omega * dp;
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    if (!(act >> q & 1)) continue;
                    vn[q] = (fc[q] == 1 ? i1 : fc[q] == 2 ? i2 : i3)[fi[q]] + omega * dv[q];
                    (fc[q] == 1 ? o1 : fc[q] == 2 ? o2 : o3)[fi[q]] = vn[q];
                }
            }
            if (pown) o0[u] = p;
            for (int e = d0; e < d1; e++) {
                const ResDep<T> D = deps[e];
                const int face = D.what & 7, uc = (D.what & 0x7fffffff) >> 3;
                if (!mine && face != 6) continue;
                T dk = (T)D.k;
                if (sizeof(T) == 8 && D.what < 0) {
                    const int4 X = R.dep[e < n0 ? e0 + e : e1 + e - n0];
                    dk = (T)__hiloint2double(X.w, X.z);
                }
                const T v = face == 0 ? vn[0] : face == 1 ? vn[1] : face == 2 ? vn[2] : face == 3 ? vn[3]
                          : face == 4 ? vn[4] : face == 5 ? vn[5] : p;
                T *o = (uc & 3) == 0 ? o0 : ((uc & 3) == 1 ? o1 : ((uc & 3) == 2 ? o2 : o3));
                o[uc >> 2] = D.c + dk * v;
            }
        }
        swap(i0, o0); swap(i1, o1); swap(i2, o2); swap(i3, o3);
        if (s + 1 < passes) go = res_sync<kCluster>(B, target, &ok);
    }
    if (!kCluster) res_leave(B);
}

}  // namespace p2
