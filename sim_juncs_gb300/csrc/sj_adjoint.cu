// Discrete adjoint of the stepper's step, and the objective DFT.
//
// The step is linear in the fields with coefficients that do not depend on
// them (S, eps_inf^{-1}, the CPML b and c, the ADE's A, B and C sigma), so
// its adjoint is the reverse sequence of the transposed sub-updates, with the
// same coefficients: for step n, first the transpose of the E update
// (eps_inf^{-1}, the polarisation ADE, the E-side psi, the backward
// differences of H), then the transpose of the H update (the H-side psi and
// the forward differences of E).  Each is a gather, one thread per cell, so no
// two threads write one value:
//   k_adj_e  completes dF/dE^{n+1} with what the H update's differences of
//            step n+1 read from E here (hb and its psi adjoints, here and at
//            the -1 neighbours), then transposes the E update; it leaves
//            cv = S eps^{-1} dF/dE, the adjoint of each curl, for k_adj_h;
//   k_adj_h  gathers the E update's differences (cv and the E-side psi
//            adjoints, here and at the +1 neighbours) into dF/dH and
//            transposes the H update's psi.
// What the H update's differences read is -S hb, so nothing has to be handed
// from k_adj_h to the next k_adj_e.  A psi adjoint is kept as T, the value
// before its factor b: the difference's adjoint is cv + c T, and b T enters
// the next T, so neighbours need no arrays of their own for either.
// The objective's dF/dE^n source is added to eb between the steps, by blocks
// of k_adj_h's launch of their own (its cells do not touch eb).  The gradient with respect to a
// design voxel's inverse eps is sum_n dF/dE^{n+1} * acc^n, acc^n being the E
// update's bracket at step n, recorded while the segment is run forward.
//
// A thread takes a column (FP32: a pair of columns) of a z segment, neighbours
// in z carried; a plane's columns are dealt out by their linear index (no idle
// lanes on odd rows).  Bound: HBM, per step and plain FP32 cell 85 bytes (hb
// read, eb read and written, cv written, the material byte; cv read, hb read
// and written) against the 145 of passes that store the adjoints of all twelve
// differences.  160^3 FP32: 116 us per step (about 300 before), 463 MB with
// the psi at 4.0 TB/s; 4 x 192^3 on quartz 0.82 ms (1.6 before) at 4.6 TB/s.
// One launch per kernel and instance; the descriptor travels as a kernel
// parameter (several in one, indexed by the block, cost an indexed constant
// load per pointer: 38 against 31.5 M warp instructions).
#include <algorithm>
#include <cstring>

#include "sj_physics.cuh"

namespace sj {

namespace {

// Small blocks end their marches independently (160^3 gradient of 200 steps:
// 76.2 ms with 64 threads, 77.3 with 256), and twelve of them per SM (80
// registers) beat sixteen with spills.
constexpr int ADJ_THREADS = 64;
template <typename real>
constexpr int adj_minb() { return sizeof(real) == 4 ? 12 : 6; }
// Columns per thread: two in FP32 (addresses, branches and constant loads of a
// plane are shared: 24.0 against 31.5 M warp instructions per E transpose of
// 160^3), one in FP64, whose pair would not fit the registers.
template <typename real>
constexpr int adj_cols() { return sizeof(real) == 4 ? 2 : 1; }

template <typename real>
__device__ __forceinline__ real prof_at(const InstDev<real>& I, int a, int q, int which) {
    // which: 0 = b (integer points), 1 = c (integer), 2 = b (half), 3 = c (half)
    return __ldg(I.prof[a] + which * dim_of(I, a) + q);
}

template <typename real>
__device__ __forceinline__ long long design_index(const InstDev<real>& I, int i, int j, int k) {
    if (!I.dinv) return -1;
    const int u = i - I.des_lo[0], v = j - I.des_lo[1], w = k - I.des_lo[2];
    if ((unsigned)u >= (unsigned)I.des_n[0] || (unsigned)v >= (unsigned)I.des_n[1] ||
        (unsigned)w >= (unsigned)I.des_n[2])
        return -1;
    return ((long long)w * I.des_n[1] + v) * I.des_n[0] + u;
}

// W neighbouring cells of a row (one: W = 1), moved as one access
template <typename real, int W>
struct Vec {
    real v[W];
};
template <typename real, int W>
struct alignas(W * sizeof(real)) VecMem {
    real v[W];
};
template <int W, typename real>
__device__ __forceinline__ Vec<real, W> vld(const real* p, unsigned o) {
    Vec<real, W> r;
    const VecMem<real, W> m = *reinterpret_cast<const VecMem<real, W>*>(p + o);
#pragma unroll
    for (int w = 0; w < W; ++w) r.v[w] = m.v[w];
    return r;
}
// read-only for the launch
template <int W, typename real>
__device__ __forceinline__ Vec<real, W> vldg(const real* p, unsigned o) {
    Vec<real, W> r;
    if constexpr (W == 2) {
        const float2 m = __ldg(reinterpret_cast<const float2*>(p + o));
        r.v[0] = m.x, r.v[1] = m.y;
    } else {
        r.v[0] = __ldg(p + o);
    }
    return r;
}
template <int W, typename real>
__device__ __forceinline__ void vst(real* p, unsigned o, const Vec<real, W>& x) {
    VecMem<real, W> m;
#pragma unroll
    for (int w = 0; w < W; ++w) m.v[w] = x.v[w];
    *reinterpret_cast<VecMem<real, W>*>(p + o) = m;
}

// The psi adjoints a thread's cells read of one axis: the two their
// differences' adjoints take (p, q) and the two they update (u, v).  0 where
// no cell is in the slab; the factors of a cell outside it are 0.
template <typename real, int W>
struct PsiIn {
    Vec<real, W> p, q, u, v;
};
// any: some lane of the warp is in the slab, else no load is issued at all (a
// predicated one costs its issue slots)
template <typename real, int W>
__device__ __forceinline__ PsiIn<real, W> psi_in(bool any, bool on, const real* T, const real* U, unsigned o,
                                                 unsigned vol) {
    PsiIn<real, W> r = {};
    if (any && on) {
        r.p = vldg<W>(T, o), r.q = vldg<W>(T, o + vol);
        r.u = vld<W>(U, o), r.v = vld<W>(U, o + vol);
    }
    return r;
}
// T' = b T +- c of the two, in the cells of the slab
template <typename real, int W>
__device__ __forceinline__ void psi_next(bool on, const bool* cell, real* U, unsigned o, unsigned vol, const real* b,
                                         const PsiIn<real, W>& r, const real* c0, real s0, const real* c1, real s1) {
    if (!on) return;
    Vec<real, W> x, y;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        x.v[w] = cell[w] ? b[w] * r.u.v[w] + s0 * c0[w] : real(0);
        y.v[w] = cell[w] ? b[w] * r.v.v[w] + s1 * c1[w] : real(0);
    }
    vst<W>(U, o, x);
    vst<W>(U, o + vol, y);
}

// L2 prefetch: each warp asks for its cells of the next plane of every array it
// reads (4 x 192^3 gradient of 60 steps: 140.6 -> 136.0 ms; two planes ahead
// 139.8), one 128-byte line per lane (a warp's cells are two lines of an
// array: lanes 2a and 2a + 1 take those of array a).  Arrays: three fields
// read, three updated, the material bytes, then the psi pairs of the x and y
// axes where the warp reads them.
template <typename real>
__device__ __forceinline__ const char* prefetch_line(unsigned act, real* const* F, real* const* G, const uint8_t* combo,
                                                     real* const* T, real* const* U, bool ux, bool uy, unsigned o,
                                                     unsigned vol, unsigned& step) {
    const int l = threadIdx.x & 31, a = l >> 1;
    const unsigned lo = __shfl_sync(act, o, 0), hi = __shfl_sync(act, o, 16);
    const unsigned at = (l & 1) ? hi : lo;
    step = sizeof(real);
    if (a < 3) return (const char*)(F[a] + at);
    if (a < 6) return (const char*)(G[a - 3] + at);
    if (a == 6 && combo) {
        step = 1;
        return (const char*)(combo + at);
    }
    if (a >= 7 && a < 15) {
        const int m = a - 7, ax = m >> 2;
        if (!(ax ? uy : ux) || !T[ax]) return nullptr;
        return (const char*)(((m & 2) ? U[ax] : T[ax]) + ((m & 1) ? vol : 0u) + at);
    }
    return nullptr;
}
__device__ __forceinline__ void prefetch_l2(const char* p, bool on) {
    if (on && p) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// A thread's place: its column(s) of the plane, slab membership, factors
template <typename real, int W>
struct Place {
    int i, j;
    bool in[W], xs[W], xany, ys;
    bool ycell[W];
};
template <typename real, int W>
__device__ __forceinline__ bool place(const InstDev<real>& I, Place<real, W>& P) {
    const unsigned gx = ((unsigned)I.nx + W - 1) / W;
    const unsigned p = blockIdx.x * ADJ_THREADS + threadIdx.x;
    if (p >= gx * (unsigned)I.ny) return false;
    P.j = (int)(p / gx), P.i = (int)(p - (unsigned)P.j * gx) * W;
    P.xany = false;
    P.ys = in_slab(I, 1, P.j);
#pragma unroll
    for (int w = 0; w < W; ++w) {
        P.in[w] = P.i + w < I.nx;
        P.xs[w] = P.in[w] && in_slab(I, 0, P.i + w);
        P.xany |= P.xs[w];
        P.ycell[w] = true;
    }
    return true;
}

// Transpose of the E update.  eb holds dF/dE^{n+1} without the gather from
// step n+1's H update on entry, the E update's share of dF/dE^n on exit.
// Offsets within the instance are 32-bit (sj_adjoint_gradient admits grids of
// fewer than 2^31 voxels).
template <typename real, int W>
__global__ void __launch_bounds__(ADJ_THREADS, adj_minb<real>())
k_adj_e(const __grid_constant__ AdjDev<real> A, long long n, int zs) {
    const InstDev<real>& I = A.I;
    Place<real, W> P;
    if (!place<real, W>(I, P)) return;
    const int k0 = (int)blockIdx.y * zs, k1 = min(I.nz, k0 + zs), i = P.i, j = P.j;
    const unsigned px = (unsigned)I.px, plane = (unsigned)I.plane, vol = (unsigned)I.vol;
    const bool xm = i > 0, ym = j > 0;
    const bool xsm = xm && in_slab(I, 0, i - 1), ysm = ym && in_slab(I, 1, j - 1);
    const real S = I.S;
    // H-side c here and at the -1 neighbours, E-side b here
    real cx[W], bx[W], by[W];
#pragma unroll
    for (int w = 0; w < W; ++w)
        cx[w] = P.xs[w] ? prof_at(I, 0, i + w, 3) : real(0), bx[w] = P.xs[w] ? prof_at(I, 0, i + w, 0) : real(0);
    const real cxm = xsm ? prof_at(I, 0, i - 1, 3) : real(0);
    const real cy = P.ys ? prof_at(I, 1, j, 3) : real(0), cym = ysm ? prof_at(I, 1, j - 1, 3) : real(0);
    by[0] = P.ys ? prof_at(I, 1, j, 0) : real(0);
    if (W == 2) by[W - 1] = by[0];
    const unsigned act = __activemask();
    const bool ux = __any_sync(act, P.xany || xsm), uy = __any_sync(act, P.ys || ysm);
    const bool des = I.dinv && (unsigned)(j - I.des_lo[1]) < (unsigned)I.des_n[1] && i + W > I.des_lo[0] &&
                     i < I.des_lo[0] + I.des_n[0];
    unsigned o = (unsigned)k0 * plane + (unsigned)j * px + (unsigned)i;
    // t4 of Hx and t3 of Hy at the plane below
    Vec<real, W> t4xz = {}, t3yz = {};
    if (k0 > 0) {
        const unsigned om = o - plane;
        const Vec<real, W> h0 = vldg<W>(A.hb[0], om), h1 = vldg<W>(A.hb[1], om);
        const bool zsm = in_slab(I, 2, k0 - 1);
        const real c = zsm ? prof_at(I, 2, k0 - 1, 3) : real(0);
        Vec<real, W> p = {}, q = {};
        if (zsm) p = vldg<W>(A.psHb[2], om), q = vldg<W>(A.psHb[2], om + vol);
#pragma unroll
        for (int w = 0; w < W; ++w) t4xz.v[w] = c * p.v[w] + S * h0.v[w], t3yz.v[w] = c * q.v[w] - S * h1.v[w];
    }
    unsigned pstep = 0;
    const char* pf = nullptr;
    if (act == 0xffffffffu) {
        pf = prefetch_line<real>(act, A.hb, A.eb, I.combo, A.psHb, A.psEb, ux, uy, o, vol, pstep);
        if (pf) pf += (size_t)plane * pstep;
    }
    for (int k = k0; k < k1; ++k, o += plane) {
        if (pf) {
            prefetch_l2(pf, k + 1 < k1);
            pf += (size_t)plane * pstep;
        }
        const bool zsl = in_slab(I, 2, k);
        real cz = 0, bz[W];
        bz[0] = 0;
        if (zsl) cz = prof_at(I, 2, k, 3), bz[0] = prof_at(I, 2, k, 0);
        if (W == 2) bz[W - 1] = bz[0];
        unsigned char cb[W];
        if constexpr (W == 2) {
            const uchar2 c2 = __ldg(reinterpret_cast<const uchar2*>(I.combo + o));
            cb[0] = c2.x, cb[1] = c2.y;
        } else {
            cb[0] = __ldg(I.combo + o);
        }
        const Vec<real, W> h0 = vldg<W>(A.hb[0], o), h1 = vldg<W>(A.hb[1], o), h2 = vldg<W>(A.hb[2], o);
        const real h1x = xm ? __ldg(A.hb[1] + o - 1) : real(0), h2x = xm ? __ldg(A.hb[2] + o - 1) : real(0);
        Vec<real, W> h0y = {}, h2y = {};
        if (ym) h0y = vldg<W>(A.hb[0], o - px), h2y = vldg<W>(A.hb[2], o - px);
        Vec<real, W> e[3] = {vld<W>(A.eb[0], o), vld<W>(A.eb[1], o), vld<W>(A.eb[2], o)};
        const PsiIn<real, W> X = psi_in<real, W>(ux, P.xany, A.psHb[0], A.psEb[0], o, vol);
        const PsiIn<real, W> Y = psi_in<real, W>(uy, P.ys, A.psHb[1], A.psEb[1], o, vol);
        const PsiIn<real, W> Z = psi_in<real, W>(zsl, zsl, A.psHb[2], A.psEb[2], o, vol);
        real Xpm = 0, Xqm = 0;
        Vec<real, W> Ypm = {}, Yqm = {};
        if (ux && xsm) Xpm = __ldg(A.psHb[0] + o - 1), Xqm = __ldg(A.psHb[0] + o - 1 + vol);
        if (uy && ysm) Ypm = vldg<W>(A.psHb[1], o - px), Yqm = vldg<W>(A.psHb[1], o - px + vol);
        unsigned mask[W];
        real ab[3][W], cv[3][W];
        // t4 of Hy and t3 of Hz at the -1 column
        real t4ym = cxm * Xpm + S * h1x, t3zm = cxm * Xqm - S * h2x;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const real g0 = S * h0.v[w], g1 = S * h1.v[w], g2 = S * h2.v[w];
            // t3, t4 of the H update's differences (t3 = -S hb + c T, t4 = S hb + c T)
            const real t3x = cy * Y.p.v[w] - g0, t4x = cz * Z.p.v[w] + g0;
            const real t3y = cz * Z.q.v[w] - g1, t4y = cx[w] * X.p.v[w] + g1;
            const real t3z = cx[w] * X.q.v[w] - g2, t4z = cy * Y.q.v[w] + g2;
            const real t3xm = cym * Ypm.v[w] - S * h0y.v[w], t4zm = cym * Yqm.v[w] + S * h2y.v[w];
            real e0 = e[0].v[w], e1 = e[1].v[w], e2 = e[2].v[w];
            e2 += t3xm - t3x;
            e1 += t4xz.v[w] - t4x;
            e0 += t3yz.v[w] - t3y;
            e2 += t4ym - t4y;
            e1 += t3zm - t3z;
            e0 += t4zm - t4z;
            t4xz.v[w] = t4x;
            t3yz.v[w] = t3y;
            t4ym = t4y;
            t3zm = t3z;
            const bool in = W == 1 || P.in[w];  // a row's last pair may end beyond the grid
            e[0].v[w] = in ? e0 : real(0), e[1].v[w] = in ? e1 : real(0), e[2].v[w] = in ? e2 : real(0);
            const real* cf = I.coef + cb[w] * I.ncoef;
            mask[w] = in ? __ldg(I.pmask + cb[w]) : 0u;
            ab[0][w] = __ldg(cf), ab[1][w] = __ldg(cf + 1), ab[2][w] = __ldg(cf + 2);
        }
        if (des)
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const long long d = design_index(I, i + w, j, k);
                if (d < 0) continue;
                const long long nd = (long long)I.des_n[0] * I.des_n[1] * I.des_n[2];
                ab[0][w] = ab[1][w] = ab[2][w] = I.dinv[d];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    A.g[d * 3 + c] += (double)e[c].v[w] * (double)A.rec[((n - A.rec_t0) * nd + d) * 3 + c];
            }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            Vec<real, W> x;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                ab[c][w] *= e[c].v[w];  // adjoint of the bracket acc
                x.v[w] = cv[c][w] = S * ab[c][w];
            }
            vst<W>(A.cv[c], o, x);
        }
        if (ux)
            psi_next<real, W>(P.xany, P.xs, A.psEb[0], o, vol, bx, X, cv[1], real(-1), cv[2], real(1));
        if (uy)
            psi_next<real, W>(P.ys, P.ycell, A.psEb[1], o, vol, by, Y, cv[0], real(1), cv[2], real(-1));
        if (zsl)
            psi_next<real, W>(true, P.ycell, A.psEb[2], o, vol, bz, Z, cv[0], real(-1), cv[1], real(1));
#pragma unroll
        for (int w = 0; w < W; ++w) {
            if (!mask[w]) continue;
            const real* cf = I.coef + cb[w] * I.ncoef;
            const unsigned u = ((unsigned)(k - I.dlo[2]) * (unsigned)I.dn[1] + (unsigned)(j - I.dlo[1])) *
                                   (unsigned)I.dn[0] + (unsigned)(i + w - I.dlo[0]);
            const size_t dvol = (size_t)I.dvol;
            // the first pole of every component together, then the others
            real q0[3], q1[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const unsigned m = (mask[w] >> (8 * c)) & 255u;
                const real* x = A.pb + (size_t)((m ? __ffs(m) - 1 : 0) * 6 + c) * dvol + u;
                q0[c] = m ? x[0] : real(0), q1[c] = m ? x[3 * dvol] : real(0);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                bool first = true;
                for (unsigned m = (mask[w] >> (8 * c)) & 255u; m; m &= m - 1, first = false) {
                    // one pole's ADE transpose: (dF/dP^{n+1}, dF/dP^n) -> (dF/dP^n, dF/dP^{n-1})
                    const int pl = __ffs(m) - 1;
                    real* x = A.pb + (size_t)(pl * 6 + c) * dvol + u;
                    const real pnb = (first ? q0[c] : x[0]) - ab[c][w];
                    const real pn = (first ? q1[c] : x[3 * dvol]) + ab[c][w] + I.A[pl] * pnb;
                    x[3 * dvol] = I.B[pl] * pnb;
                    x[0] = pn;
                    e[c].v[w] += __ldg(cf + 3 + 3 * pl + c) * pnb;
                }
            }
        }
        vst<W>(A.eb[0], o, e[0]);
        vst<W>(A.eb[1], o, e[1]);
        vst<W>(A.eb[2], o, e[2]);
    }
}

// dF/dH^{n+1/2} += what the E update's differences read from H at this cell,
// then the transpose of the H update's psi; hb itself carries over to
// H^{n-1/2}.  The block columns from cell_blocks on add the objective's
// dF/dE^n to eb, a thread per cell and component.
template <typename real, int W>
__global__ void __launch_bounds__(ADJ_THREADS, adj_minb<real>())
k_adj_h(const __grid_constant__ AdjDev<real> A, long long n, int zs, unsigned cell_blocks) {
    const InstDev<real>& I = A.I;
    if (blockIdx.x >= cell_blocks) {
        const unsigned t = ((blockIdx.x - cell_blocks) * gridDim.y + blockIdx.y) * ADJ_THREADS + threadIdx.x;
        const unsigned q = t / 3, c = t % 3;
        if (q >= (unsigned)A.n_cells || !((A.comp_mask >> c) & 1)) return;
        double sn, cs;
        sincospi(2.0 * A.freq * ((double)n * I.dt), &sn, &cs);
        const int* x = A.cells + 3 * q;
        const double2 v = A.D[t];
        A.eb[c][(long long)x[2] * I.plane + (long long)x[1] * I.px + x[0]] +=
            (real)(2.0 * I.dt * (v.x * cs + v.y * sn));
        return;
    }
    Place<real, W> P;
    if (!place<real, W>(I, P)) return;
    const int k0 = (int)blockIdx.y * zs, k1 = min(I.nz, k0 + zs), i = P.i, j = P.j;
    const unsigned px = (unsigned)I.px, plane = (unsigned)I.plane, vol = (unsigned)I.vol;
    const bool xp = i + W < I.nx, yp = j + 1 < I.ny;
    const bool xsp = xp && in_slab(I, 0, i + W), ysp = yp && in_slab(I, 1, j + 1);
    const real S = I.S;
    // E-side c here and at the +1 neighbours, H-side b here
    real cx[W], bx[W], by[W];
#pragma unroll
    for (int w = 0; w < W; ++w)
        cx[w] = P.xs[w] ? prof_at(I, 0, i + w, 1) : real(0), bx[w] = P.xs[w] ? prof_at(I, 0, i + w, 2) : real(0);
    const real cxp = xsp ? prof_at(I, 0, i + W, 1) : real(0);
    const real cy = P.ys ? prof_at(I, 1, j, 1) : real(0), cyp = ysp ? prof_at(I, 1, j + 1, 1) : real(0);
    by[0] = P.ys ? prof_at(I, 1, j, 2) : real(0);
    if (W == 2) by[W - 1] = by[0];
    const unsigned act = __activemask();
    const bool ux = __any_sync(act, P.xany || xsp), uy = __any_sync(act, P.ys || ysp);
    unsigned o = (unsigned)k0 * plane + (unsigned)j * px + (unsigned)i;
    // cv of Ex and Ey at the plane, with their z terms (t2 of Ex, t1 of Ey)
    Vec<real, W> cv0 = vldg<W>(A.cv[0], o), cv1 = vldg<W>(A.cv[1], o), t2x, t1y;
    {
        const bool zsl = in_slab(I, 2, k0);
        const real c = zsl ? prof_at(I, 2, k0, 1) : real(0);
        Vec<real, W> p = {}, q = {};
        if (zsl) p = vldg<W>(A.psEb[2], o), q = vldg<W>(A.psEb[2], o + vol);
#pragma unroll
        for (int w = 0; w < W; ++w) t2x.v[w] = c * p.v[w] - cv0.v[w], t1y.v[w] = c * q.v[w] + cv1.v[w];
    }
    unsigned pstep = 0;
    const char* pf = nullptr;
    if (act == 0xffffffffu) {
        pf = prefetch_line<real>(act, A.cv, A.hb, nullptr, A.psEb, A.psHb, ux, uy, o, vol, pstep);
        if (pf) pf += (size_t)plane * pstep;
    }
    for (int k = k0; k < k1; ++k, o += plane) {
        if (pf) {
            prefetch_l2(pf, k + 1 < k1);
            pf += (size_t)plane * pstep;
        }
        const bool kp = k + 1 < I.nz;
        const bool zsl = in_slab(I, 2, k), zsp = kp && in_slab(I, 2, k + 1);
        real czp = 0, bz[W];
        bz[0] = 0;
        if (zsp) czp = prof_at(I, 2, k + 1, 1);
        if (zsl) bz[0] = prof_at(I, 2, k, 2);
        if (W == 2) bz[W - 1] = bz[0];
        Vec<real, W> cv0n = {}, cv1n = {}, c0y = {}, c2y = {};
        if (kp) cv0n = vldg<W>(A.cv[0], o + plane), cv1n = vldg<W>(A.cv[1], o + plane);
        const Vec<real, W> cv2 = vldg<W>(A.cv[2], o);
        if (yp) c0y = vldg<W>(A.cv[0], o + px), c2y = vldg<W>(A.cv[2], o + px);
        const real c1x = xp ? __ldg(A.cv[1] + o + W) : real(0), c2x = xp ? __ldg(A.cv[2] + o + W) : real(0);
        Vec<real, W> h0 = vld<W>(A.hb[0], o), h1 = vld<W>(A.hb[1], o), h2 = vld<W>(A.hb[2], o);
        const PsiIn<real, W> X = psi_in<real, W>(ux, P.xany, A.psEb[0], A.psHb[0], o, vol);
        const PsiIn<real, W> Y = psi_in<real, W>(uy, P.ys, A.psEb[1], A.psHb[1], o, vol);
        PsiIn<real, W> Z = {};
        if (zsl) Z.u = vld<W>(A.psHb[2], o), Z.v = vld<W>(A.psHb[2], o + vol);
        if (zsp) Z.p = vldg<W>(A.psEb[2], o + plane), Z.q = vldg<W>(A.psEb[2], o + plane + vol);
        real Xpp = 0, Xqp = 0;
        Vec<real, W> Ypp = {}, Yqp = {};
        if (ux && xsp) Xpp = __ldg(A.psEb[0] + o + W), Xqp = __ldg(A.psEb[0] + o + W + vol);
        if (uy && ysp) Ypp = vldg<W>(A.psEb[1], o + px), Yqp = vldg<W>(A.psEb[1], o + px + vol);
        real g[3][W];  // adjoint of the curl of E
        // t2 of Ey and t1 of Ez at the +1 column (the pair's second column beyond the grid: none)
        real t2yp = cxp * Xpp - c1x, t1zp = cxp * Xqp + c2x;
#pragma unroll
        for (int w = W - 1; w >= 0; --w) {
            // t1, t2 of the E update's differences (t1 = cv + c T, t2 = -cv + c T)
            const real t1x = cy * Y.p.v[w] + cv0.v[w], t2y = cx[w] * X.p.v[w] - cv1.v[w];
            const real t1z = cx[w] * X.q.v[w] + cv2.v[w], t2z = cy * Y.q.v[w] - cv2.v[w];
            const real t1xp = cyp * Ypp.v[w] + c0y.v[w], t2zp = cyp * Yqp.v[w] - c2y.v[w];
            const real t2xn = czp * Z.p.v[w] - cv0n.v[w], t1yn = czp * Z.q.v[w] + cv1n.v[w];
            real a0 = h0.v[w], a1 = h1.v[w], a2 = h2.v[w];
            a2 += t1x - t1xp;
            a1 += t2x.v[w] - t2xn;
            a0 += t1y.v[w] - t1yn;
            a2 += t2y - t2yp;
            a1 += t1z - t1zp;
            a0 += t2z - t2zp;
            const bool in = W == 1 || P.in[w];
            h0.v[w] = in ? a0 : real(0), h1.v[w] = in ? a1 : real(0), h2.v[w] = in ? a2 : real(0);
            t2yp = in ? t2y : real(0);
            t1zp = in ? t1z : real(0);
            t2x.v[w] = t2xn;
            t1y.v[w] = t1yn;
            g[0][w] = -S * h0.v[w], g[1][w] = -S * h1.v[w], g[2][w] = -S * h2.v[w];
        }
        vst<W>(A.hb[0], o, h0);
        vst<W>(A.hb[1], o, h1);
        vst<W>(A.hb[2], o, h2);
        if (ux)
            psi_next<real, W>(P.xany, P.xs, A.psHb[0], o, vol, bx, X, g[1], real(-1), g[2], real(1));
        if (uy)
            psi_next<real, W>(P.ys, P.ycell, A.psHb[1], o, vol, by, Y, g[0], real(1), g[2], real(-1));
        if (zsl)
            psi_next<real, W>(true, P.ycell, A.psHb[2], o, vol, bz, Z, g[0], real(-1), g[1], real(1));
        cv0 = cv0n;
        cv1 = cv1n;
    }
}

template <typename real>
struct ObjParams {
    ObjDev<real> o[OBJ_MAX];
};

// D[q][c] += dt E_c^n(cell q) e^{i 2 pi f n dt}, one thread per (objective
// cell, E component in the mask), blockIdx.y = instance
template <typename real>
__global__ void k_objective(const __grid_constant__ ObjParams<real> P, int cur, long long n) {
    const ObjDev<real>& O = P.o[blockIdx.y];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int q = t / 3, c = t % 3;
    if (q >= O.n_cells || !((O.comp_mask >> c) & 1)) return;
    const int* x = O.cells + 3 * q;
    double sn, cs;
    sincospi(2.0 * O.freq * ((double)n * O.dt), &sn, &cs);
    const double e = (double)O.E[cur][c][(long long)x[2] * O.plane + (long long)x[1] * O.px + x[0]] * O.dt;
    double2 v = O.D[t];
    v.x += e * cs;
    v.y += e * sn;
    O.D[t] = v;
}

// Planes per thread: 8 where the device stays full of blocks (1, 2, 16 and 32 are
// 9%, 2%, 1% and 1% slower on 160^3), fewer on small grids.
int adj_segment(long long plane_blocks, int nz) {
    int zs = 8;
    while (zs > 1 && plane_blocks * ((nz + zs - 1) / zs) < 12 * 152) zs >>= 1;
    return zs;
}

}  // namespace

template <typename real>
cudaError_t launch_adjoint_step(const AdjDev<real>& a, long long n, cudaStream_t s) {
    const InstDev<real>& I = a.I;
    constexpr int W = adj_cols<real>();
    const long long blocks = ((long long)((I.nx + W - 1) / W) * I.ny + ADJ_THREADS - 1) / ADJ_THREADS;
    const int zs = adj_segment(blocks, I.nz);
    const unsigned segs = (unsigned)((I.nz + zs - 1) / zs);
    k_adj_e<real, W><<<dim3((unsigned)blocks, segs), ADJ_THREADS, 0, s>>>(a, n, zs);
    // the objective's blocks: a patch of 25 cells fills two; a plane of 192^2 cells, in
    // one block a loop longer than the step (40 steps of 192^3: 79.0 ms), 1728 (15.9)
    const long long src = (3ll * a.n_cells + ADJ_THREADS - 1) / ADJ_THREADS;
    const unsigned cols = (unsigned)blocks + (unsigned)((src + segs - 1) / segs);
    k_adj_h<real, W><<<dim3(cols, segs), ADJ_THREADS, 0, s>>>(a, n, zs, (unsigned)blocks);
    return cudaGetLastError();
}

template <typename real>
cudaError_t launch_objective(const ObjDev<real>* o, int n_inst, int cur, long long n, cudaStream_t s) {
    for (int q0 = 0; q0 < n_inst; q0 += OBJ_MAX) {
        const int m = std::min(OBJ_MAX, n_inst - q0);
        ObjParams<real> P;
        memset(&P, 0, sizeof(P));
        int threads = 0;
        for (int q = 0; q < m; ++q) P.o[q] = o[q0 + q], threads = std::max(threads, 3 * P.o[q].n_cells);
        if (threads == 0) continue;
        k_objective<real><<<dim3((unsigned)(threads + 127) / 128, (unsigned)m), 128, 0, s>>>(P, cur, n);
    }
    return cudaGetLastError();
}

template cudaError_t launch_adjoint_step<float>(const AdjDev<float>&, long long, cudaStream_t);
template cudaError_t launch_adjoint_step<double>(const AdjDev<double>&, long long, cudaStream_t);
template cudaError_t launch_objective<float>(const ObjDev<float>*, int, int, long long, cudaStream_t);
template cudaError_t launch_objective<double>(const ObjDev<double>*, int, int, long long, cudaStream_t);
}  // namespace sj
