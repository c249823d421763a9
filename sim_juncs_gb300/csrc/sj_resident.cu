// Small grids: many steps of the fused schedule in one cooperative launch.
//
// A 64^3 step is 262k cells, a few microseconds of work from L2, but as tile
// launches it costs ten launches on forked streams, and its 64 tiles of 16
// planes are a serial march on 64 of the 152 SMs.  Here a grid of resident
// blocks (one per SM) runs a whole run of steps: per step an H phase
// and an E phase over every cell of every instance, in place, with a grid
// barrier after each.  In the E phase a cell's sources and polarisations
// follow its curl directly (they are separate passes after the tile kernels).
// The cell's arithmetic is the tile kernels', operation for operation, so
// the bits are theirs (this file too is compiled with contraction off).
//
// FP32 is bound by latency up to about 64^3 (36^3 7.9 us per step, 64^3 9.1: two
// L2 round trips and two barriers; 72 us as tile launches) and by L2 above.
// FP64 is bound by the FP64 pipe (19 cycles per warp instruction and SM):
// 64^3 26 us per step (124 as tile launches), of which 17 are its 35 FP64
// operations per cell; 256 x 256 x 192 802 us, of which 720.
//
// Cells are dealt out by their linear index over nx*ny*nz, so odd rows leave
// no idle lanes.  Probes have blocks of their own: E probes of step n are
// read during its H phase, which does not write E, and H probes of step n
// (H^{n-1/2}) during the E phase of step n-1, which does not write H.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>

#include "sj_physics.cuh"

namespace sj {

namespace {

constexpr int RES_MAXF = 256;
// Threads of a block, by the cells of the launch.  More warps hide more latency
// and keep the FP64 pipe busier at a phase's ends, on few cells they only add
// to the barrier: us per step of 36^3, 48^3, 64^3, 128^3, 192^3
//   FP64  512 threads  13.2 15.0 27.4 168 537;  768  16.8 16.6 26.4 165 512
//         (256 x 256 x 192 bowtie 875 and 802)
//   FP32  512 threads  7.9 7.6 11.2 63.8 249;  1024  8.6 8.3 9.2 44.7 166
template <typename real>
constexpr int res_threads(bool few) { return few ? 512 : (sizeof(real) == 4 ? 1024 : 768); }
constexpr long long RES_FEW_CELLS = 1 << 18;  // fewer cells than this: the small blocks

// A block takes its cells in chunks of this many consecutive ones, dealt out
// over the blocks in turn.  FP64 is bound by the FP64 pipe of each SM, so its
// chunks are one warp's (the SMs' shares differ by one: 64^3 27.3 us per step,
// 29.9 with 256); FP32's are the block's, whose rows share L1 lines.
template <typename real, int T>
constexpr int res_chunk() { return sizeof(real) == 4 ? T : 32; }

// What a block knows of one instance besides its descriptor.  FP64 deals the
// columns between the x slabs first and the slabs' columns after them: a
// warp then seldom mixes the two, and only the slabs' warps pay for the x
// terms (all warps of a 64-cell row would).
struct ResGrid {
    Div dx, dxs, dy;             // columns between the x slabs (FP32: all), columns of the slabs, rows
    unsigned inner, cells;       // cells of the former, of all
    unsigned start;              // this block's first cell
    int lo;                      // first column between the slabs
    int hsrc, esrc;              // any H / E source
};

struct Cell {
    int i, j, k;
};
template <typename real>
__device__ __forceinline__ Cell res_cell(const ResGrid& G, unsigned t) {
    Cell c;
    if (sizeof(real) == 4) {
        const unsigned q = G.dx.div(t), kk = G.dy.div(q);
        c.i = (int)(t - q * G.dx.d), c.j = (int)(q - kk * G.dy.d), c.k = (int)kk;
        return c;
    }
    const bool in = t < G.inner;
    const Div& D = in ? G.dx : G.dxs;
    t -= in ? 0u : G.inner;
    const unsigned q = D.div(t), kk = G.dy.div(q);
    c.i = (int)(t - q * D.d), c.j = (int)(q - kk * G.dy.d), c.k = (int)kk;
    c.i += in ? G.lo : (c.i >= G.lo ? (int)G.dx.d : 0);
    return c;
}

// Grid barrier: every block arrives with release, waits for `target`
// arrivals with acquire.  A wait that does not end within `limit` ns records
// SJ_E_TIMEOUT and ends the launch (false, block-uniform).
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, unsigned long long limit, DevState* st) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned long long t0 = 0;
        for (unsigned spin = 0;; ++spin) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if ((spin & 1023u) == 1023u) {
                unsigned long long t;
                asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
                if (!t0) t0 = t;
                if (t - t0 > limit) {
                    st->status = SJ_E_TIMEOUT;
                    ok = 0;
                    break;
                }
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

// Does this lane run the terms of an axis its cell lies (on) or not in the
// slab of?  FP64: when some lane of the warp does, by select (a branch per
// lane has the compiler emit the common FP64 work once for each side).
template <typename real>
__device__ __forceinline__ bool res_any(bool on) {
    return sizeof(real) == 8 ? __any_sync(__activemask(), on) : on;
}

// One CPML term: psi = fma(b, psi, c d), added to or subtracted from the curl
// where the cell is in the slab; any: some lane of the warp is
template <bool ADD, typename real>
__device__ __forceinline__ void res_term(real& cv, bool any, bool on, real b, real c, real d, real po, real* p) {
    if (!any) return;
    const real ps = fma(b, po, c * d);
    if (on) *p = ps;
    cv = ADD ? cv + (on ? ps : real(-0.0)) : cv - (on ? ps : real(0));
}

template <typename real>
__device__ __forceinline__ bool src_hit(const SrcDev<real>& s, int i, int j, int k) {
    return (unsigned)(i - s.lo[0]) < (unsigned)s.n[0] && (unsigned)(j - s.lo[1]) < (unsigned)s.n[1] &&
           (unsigned)(k - s.lo[2]) < (unsigned)s.n[2];
}

// dt J of the H sources of component comp at the cell
template <typename real>
__device__ __forceinline__ real res_hsrc(const InstDev<real>& I, int comp, int i, int j, int k, long long n, real h) {
    real acc = 0;
    bool hit = false;
    for (int s = 0; s < I.n_src; ++s) {
        const SrcDev<real>& v = I.src[s];
        if (v.comp != comp || !src_hit(v, i, j, k)) continue;
        acc += (real)v.tab[n] * v.w[0][i - v.lo[0]] * v.w[1][j - v.lo[1]] * v.w[2][k - v.lo[2]];
        hit = true;
    }
    return hit ? h - acc : h;
}

// H^{n+1/2} of one cell, in place
template <typename real>
__device__ __forceinline__ void res_h(const InstDev<real>& I, const ResGrid& G, int cur, unsigned t, long long n) {
    const Cell c3 = res_cell<real>(G, t);
    const int i = c3.i, j = c3.j, k = c3.k;
    const int nx = I.nx, ny = I.ny, nz = I.nz;
    const unsigned px = (unsigned)I.px, plane = (unsigned)I.plane, vol = (unsigned)I.vol;
    const unsigned o = (unsigned)k * plane + (unsigned)j * px + (unsigned)i;
    const real* eX = I.F[cur][0];
    const real* eY = I.F[cur][1];
    const real* eZ = I.F[cur][2];
    real* const hX = I.F[cur][3] + o;
    real* const hY = I.F[cur][4] + o;
    real* const hZ = I.F[cur][5] + o;
    const bool xp = i + 1 < nx, yp = j + 1 < ny, zp = k + 1 < nz;
    const bool xo = in_slab(I, 0, i), yo = in_slab(I, 1, j), zo = in_slab(I, 2, k);
    const real ex = eX[o], ey = eY[o], ez = eZ[o];
    const real ex_y = yp ? eX[o + px] : real(0), ex_z = zp ? eX[o + plane] : real(0);
    const real ey_x = xp ? eY[o + 1] : real(0), ey_z = zp ? eY[o + plane] : real(0);
    const real ez_x = xp ? eZ[o + 1] : real(0), ez_y = yp ? eZ[o + px] : real(0);
    const real hx0 = *hX, hy0 = *hY, hz0 = *hZ;
    const bool ax = res_any<real>(xo), ay = res_any<real>(yo), az = res_any<real>(zo);
    real *pX = nullptr, *pY = nullptr, *pZ = nullptr;
    real qx0 = 0, qx1 = 0, qy0 = 0, qy1 = 0, qz0 = 0, qz1 = 0;
    real bx = 1, cx = 0, by = 1, cy = 0, bz = 1, cz = 0;
    if (xo) {
        pX = I.psiH[cur][0] + o;
        qx0 = pX[0], qx1 = pX[vol];
        bx = __ldg(I.prof[0] + 2 * nx + i), cx = __ldg(I.prof[0] + 3 * nx + i);
    }
    if (yo) {
        pY = I.psiH[cur][1] + o;
        qy0 = pY[0], qy1 = pY[vol];
        by = __ldg(I.prof[1] + 2 * ny + j), cy = __ldg(I.prof[1] + 3 * ny + j);
    }
    if (zo) {
        pZ = I.psiH[cur][2] + o;
        qz0 = pZ[0], qz1 = pZ[vol];
        bz = __ldg(I.prof[2] + 2 * nz + k), cz = __ldg(I.prof[2] + 3 * nz + k);
    }
    real hx, hy, hz;
    {
        const real d1 = ez_y - ez, d2 = ey_z - ey;
        real cv = d1 - d2;
        res_term<true>(cv, ay, yo, by, cy, d1, qy0, pY);
        res_term<false>(cv, az, zo, bz, cz, d2, qz0, pZ);
        hx = fma(-I.S, cv, hx0);
    }
    {
        const real d1 = ex_z - ex, d2 = ez_x - ez;
        real cv = d1 - d2;
        res_term<true>(cv, az, zo, bz, cz, d1, qz1, pZ + vol);
        res_term<false>(cv, ax, xo, bx, cx, d2, qx0, pX);
        hy = fma(-I.S, cv, hy0);
    }
    {
        const real d1 = ey_x - ey, d2 = ex_y - ex;
        real cv = d1 - d2;
        res_term<true>(cv, ax, xo, bx, cx, d1, qx1, pX + vol);
        res_term<false>(cv, ay, yo, by, cy, d2, qy1, pY + vol);
        hz = fma(-I.S, cv, hz0);
    }
    if (G.hsrc) {
        hx = res_hsrc(I, 3, i, j, k, n, hx);
        hy = res_hsrc(I, 4, i, j, k, n, hy);
        hz = res_hsrc(I, 5, i, j, k, n, hz);
    }
    *hX = hx;
    *hY = hy;
    *hZ = hz;
}

// E^{n+1} of one cell, in place: curl, then the E sources in order, then the
// polarisations of the cell's material.  DES: a cell of the design region
// scales by its own eps^-1 and, while a segment is recorded, its bracket
// S curl H - dt J - dP is stored.
template <bool DES, typename real>
__device__ __forceinline__ void res_e(const InstDev<real>& I, const ResGrid& G, int cur, unsigned t, long long n) {
    const Cell c3 = res_cell<real>(G, t);
    const int i = c3.i, j = c3.j, k = c3.k;
    const int nx = I.nx, ny = I.ny, nz = I.nz;
    const unsigned px = (unsigned)I.px, plane = (unsigned)I.plane, vol = (unsigned)I.vol;
    const unsigned o = (unsigned)k * plane + (unsigned)j * px + (unsigned)i;
    const real* hX = I.F[cur][3];
    const real* hY = I.F[cur][4];
    const real* hZ = I.F[cur][5];
    const int cb = __ldg(I.combo + o);
    const unsigned mask = __ldg(I.pmask + cb);
    const real* cf = I.coef + cb * I.ncoef;
    const real* sv = cf + I.ncoef - 3;
    const bool xm = i > 0, ym = j > 0, zm = k > 0;
    const bool xo = in_slab(I, 0, i), yo = in_slab(I, 1, j), zo = in_slab(I, 2, k);
    const real hx = hX[o], hy = hY[o], hz = hZ[o];
    const real hx_y = ym ? hX[o - px] : real(0), hx_z = zm ? hX[o - plane] : real(0);
    const real hy_x = xm ? hY[o - 1] : real(0), hy_z = zm ? hY[o - plane] : real(0);
    const real hz_x = xm ? hZ[o - 1] : real(0), hz_y = ym ? hZ[o - px] : real(0);
    real* const E[3] = {I.F[cur][0] + o, I.F[cur][1] + o, I.F[cur][2] + o};
    const real e0[3] = {*E[0], *E[1], *E[2]};
    const bool ax = res_any<real>(xo), ay = res_any<real>(yo), az = res_any<real>(zo);
    real *pX = nullptr, *pY = nullptr, *pZ = nullptr;
    real qx0 = 0, qx1 = 0, qy0 = 0, qy1 = 0, qz0 = 0, qz1 = 0;
    real bx = 1, cx = 0, by = 1, cy = 0, bz = 1, cz = 0;
    if (xo) {
        pX = I.psiE[0] + o;
        qx0 = pX[0], qx1 = pX[vol];
        bx = __ldg(I.prof[0] + i), cx = __ldg(I.prof[0] + nx + i);
    }
    if (yo) {
        pY = I.psiE[1] + o;
        qy0 = pY[0], qy1 = pY[vol];
        by = __ldg(I.prof[1] + j), cy = __ldg(I.prof[1] + ny + j);
    }
    if (zo) {
        pZ = I.psiE[2] + o;
        qz0 = pZ[0], qz1 = pZ[vol];
        bz = __ldg(I.prof[2] + k), cz = __ldg(I.prof[2] + nz + k);
    }
    real sinv[3] = {__ldg(sv), __ldg(sv + 1), __ldg(sv + 2)}, dinv = 0, acc[3];
    long long d = -1;
    if (DES && I.dinv) {
        const int u = i - I.des_lo[0], v = j - I.des_lo[1], w = k - I.des_lo[2];
        if ((unsigned)u < (unsigned)I.des_n[0] && (unsigned)v < (unsigned)I.des_n[1] &&
            (unsigned)w < (unsigned)I.des_n[2]) {
            d = ((long long)w * I.des_n[1] + v) * I.des_n[0] + u;
            dinv = I.dinv[d];
            sinv[0] = sinv[1] = sinv[2] = I.S * dinv;
        }
    }
    real e[3];
    {
        const real d1 = hz - hz_y, d2 = hy - hy_z;
        real cv = d1 - d2;
        res_term<true>(cv, ay, yo, by, cy, d1, qy0, pY);
        res_term<false>(cv, az, zo, bz, cz, d2, qz0, pZ);
        e[0] = fma(sinv[0], cv, e0[0]);
        if (DES) acc[0] = I.S * cv;
    }
    {
        const real d1 = hx - hx_z, d2 = hz - hz_x;
        real cv = d1 - d2;
        res_term<true>(cv, az, zo, bz, cz, d1, qz1, pZ + vol);
        res_term<false>(cv, ax, xo, bx, cx, d2, qx0, pX);
        e[1] = fma(sinv[1], cv, e0[1]);
        if (DES) acc[1] = I.S * cv;
    }
    {
        const real d1 = hy - hy_x, d2 = hx - hx_y;
        real cv = d1 - d2;
        res_term<true>(cv, ax, xo, bx, cx, d1, qx1, pX + vol);
        res_term<false>(cv, ay, yo, by, cy, d2, qy1, pY + vol);
        e[2] = fma(sinv[2], cv, e0[2]);
        if (DES) acc[2] = I.S * cv;
    }
    if (G.esrc)
        for (int s = 0; s < I.n_src; ++s) {
            const SrcDev<real>& v = I.src[s];
            if (v.comp >= 3 || !src_hit(v, i, j, k)) continue;
            const real J = (real)v.tab[n] * v.w[0][i - v.lo[0]] * v.w[1][j - v.lo[1]] * v.w[2][k - v.lo[2]];
            const real c = DES && d >= 0 ? dinv : __ldg(cf + v.comp);
#pragma unroll
            for (int a = 0; a < 3; ++a)
                if (a == v.comp) {
                    e[a] = fma(-c, J, e[a]);
                    if (DES) acc[a] -= J;
                }
        }
    if (mask) {
        const unsigned u = ((unsigned)(k - I.dlo[2]) * (unsigned)I.dn[1] + (unsigned)(j - I.dlo[1])) *
                               (unsigned)I.dn[0] + (unsigned)(i - I.dlo[0]);
        const long long lv = 3 * I.dvol;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const unsigned mc = (mask >> (8 * c)) & 255u;
            if (!mc) continue;
            real corr = 0;
            for (unsigned m = mc; m; m &= m - 1) {
                const int p = __ffs(m) - 1;
                real* pp = I.P + ((long long)p * 6 + c) * I.dvol + u;
                const real pn = *pp, pq = pp[lv];
                const real pnew = I.A[p] * pn + I.B[p] * pq + __ldg(cf + 3 + 3 * p + c) * e0[c];
                corr += pnew - pn;
                pp[lv] = pn;
                *pp = pnew;
            }
            e[c] = fma(-(DES && d >= 0 ? dinv : __ldg(cf + c)), corr, e[c]);
            if (DES) acc[c] -= corr;
        }
    }
    if (DES && d >= 0 && I.rec_acc && n >= I.rec_t0 && n < I.rec_t0 + I.rec_len) {
        const long long nd = (long long)I.des_n[0] * I.des_n[1] * I.des_n[2];
        real* r = I.rec_acc + ((n - I.rec_t0) * nd + d) * 3;
        r[0] = acc[0], r[1] = acc[1], r[2] = acc[2];
    }
    *E[0] = e[0];
    *E[1] = e[1];
    *E[2] = e[2];
}

// dt e^{i 2 pi f t} of every DFT frequency for the E (h = 0) or H (h = 1)
// probes of step n
template <typename real>
__device__ __forceinline__ void res_phases(const InstDev<real>& I, long long n, int h, double2* ph) {
    const double tt = h ? ((double)n - 0.5) * I.dt : (double)n * I.dt;
    for (int f = threadIdx.x; f < I.n_freq; f += blockDim.x) {
        double s, c;
        sincospi(2.0 * I.freqs[f] * tt, &s, &c);
        ph[f] = make_double2(c * I.dt, s * I.dt);
    }
}

// What a thread keeps of a probe through a run of steps.
template <typename real>
struct Probe {
    const real* F[8];   // stencil points, null outside the grid
    double w[8];
    double2* row;       // DFT sums, null without
    int comp, mon;
};
template <typename real>
__device__ __forceinline__ Probe<real> res_probe(const InstDev<real>& I, int cur, int p) {
    Probe<real> r;
    r.comp = I.probe_comp[p];
    r.mon = I.probe_mon[p];
    const int ds = I.probe_dft[p];
    r.row = ds >= 0 ? I.dft + (long long)ds * I.n_freq : nullptr;
    const real* F = I.F[cur][r.comp];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const long long idx = I.probe_idx[8 * p + m];
        r.F[m] = idx >= 0 ? F + idx : nullptr;
        r.w[m] = I.probe_w[8 * p + m];
    }
    return r;
}

// Sample a probe at step n: its monitor value (at save points) and its DFT
// sums, as the tile path's probe blocks form them.
template <typename real>
__device__ __forceinline__ void res_sample(const InstDev<real>& I, const Probe<real>& r, long long n, bool save,
                                           int n_freq, DevState* st, const double2* ph) {
    const bool mon = r.mon >= 0 && save;
    if (!mon && !r.row) return;
    double2 a[4];
    if (r.row)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (u < n_freq) a[u] = r.row[u];
    double v = 0.0;
#pragma unroll
    for (int m = 0; m < 8; ++m)
        if (r.F[m]) v += r.w[m] * (double)*r.F[m];
    if (mon) monitor_store(I, n, r.mon, v, st);
    if (!r.row) return;
    for (int f0 = 0; f0 < n_freq; f0 += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (f0 && f0 + u < n_freq) a[u] = r.row[f0 + u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (f0 + u < n_freq) {
                a[u].x += v * ph[f0 + u].x;
                a[u].y += v * ph[f0 + u].y;
                r.row[f0 + u] = a[u];
            }
    }
}

// The E or H probes (h) of every instance at step n.  Block b of nb takes
// every nb-th chunk of `per` probes.
template <typename real>
__device__ __forceinline__ void res_probes(const InstDev<real>* tab, int n_inst, int cur, long long n, int h, int b,
                                           int nb, int per, DevState* st, double2* ph) {
    int item = 0;
    for (int q = 0; q < n_inst; ++q) {
        const InstDev<real>& I = tab[q];
        const bool save = n % I.save_span == 0;
        const int chunks = (I.n_probe + per - 1) / per;
        if (!chunks || (!save && !I.n_dft)) {
            item += chunks;
            continue;
        }
        bool have = false;
        for (int c = 0; c < chunks; ++c, ++item) {
            if (item % nb != b) continue;
            if (!have && I.n_dft) {
                __syncthreads();
                res_phases(I, n, h, ph);
                __syncthreads();
            }
            have = true;
            const int p = c * per + (int)threadIdx.x;
            if ((int)threadIdx.x >= per || p >= I.n_probe || (I.probe_comp[p] >= 3) != (h != 0)) continue;
            res_sample(I, res_probe(I, cur, p), n, save, I.n_freq, st, ph);
        }
    }
}

// A block that keeps the objective's DFT sums of an instance (one chunk of its
// cells and components) through a run of steps, sampling E^n during the H phase.
template <typename real>
__device__ __noinline__ void res_objective_block(const ObjDev<real>& O, int cur, int chunk, long long n0, int n_steps,
                                                 int h_probes, unsigned* bar, unsigned long long limit, DevState* st) {
    __shared__ double2 ph;
    const int t = chunk * (int)blockDim.x + (int)threadIdx.x, q = t / 3, c = t % 3;
    const bool on = q < O.n_cells && ((O.comp_mask >> c) & 1);
    const real* E = nullptr;
    double2 v = make_double2(0.0, 0.0);
    if (on) {
        const int* x = O.cells + 3 * q;
        E = O.E[cur][c] + ((long long)x[2] * O.plane + (long long)x[1] * O.px + x[0]);
        v = O.D[t];
    }
    const double dt = O.dt;
    auto phase = [&](long long n) {
        if (threadIdx.x == 0) sincospi(2.0 * O.freq * ((double)n * dt), &ph.y, &ph.x);
    };
    unsigned target = 0;
    phase(n0);
    __syncthreads();
    if (h_probes && !grid_barrier(bar, target += gridDim.x, limit, st)) return;
    for (int s = 0; s < n_steps; ++s) {
        const bool more = s + 1 < n_steps;
        if (on) {
            const double e = (double)*E * dt;
            v.x = fma(e, ph.x, v.x);
            v.y = fma(e, ph.y, v.y);
        }
        if (!grid_barrier(bar, target += gridDim.x, limit, st)) return;
        phase(n0 + s + 1);
        if (more && !grid_barrier(bar, target += gridDim.x, limit, st)) return;
    }
    if (on) O.D[t] = v;
}

// A probe block's run of steps.  one_chunk: every block has at most one
// chunk, so a thread keeps its probe, and the phases of its next samples are
// formed while the cells of the phase before are updated.
template <typename real>
__device__ __noinline__ void res_probe_block(const InstDev<real>* tab, int n_inst, int cur, long long n0, int n_steps,
                                             int b, int nb, int per, int h_probes, int one_chunk, unsigned* bar,
                                             unsigned long long limit, DevState* st) {
    __shared__ double2 ph[2][RES_MAXF];
    unsigned target = 0;
    if (!one_chunk) {
        if (h_probes) {
            res_probes<real>(tab, n_inst, cur, n0, 1, b, nb, per, st, ph[1]);
            if (!grid_barrier(bar, target += gridDim.x, limit, st)) return;
        }
        for (int s = 0; s < n_steps; ++s) {
            const bool more = s + 1 < n_steps;
            res_probes<real>(tab, n_inst, cur, n0 + s, 0, b, nb, per, st, ph[0]);
            if (!grid_barrier(bar, target += gridDim.x, limit, st)) return;
            if (h_probes && more) res_probes<real>(tab, n_inst, cur, n0 + s + 1, 1, b, nb, per, st, ph[1]);
            if (more && !grid_barrier(bar, target += gridDim.x, limit, st)) return;
        }
        return;
    }
    int item = 0, q = 0, chunk = 0;
    for (; q < n_inst; ++q) {
        const int chunks = (tab[q].n_probe + per - 1) / per;
        chunk = b - item;
        item += chunks;
        if (b < item) break;
    }
    const InstDev<real>& I = tab[q];
    const int p = chunk * per + (int)threadIdx.x, n_freq = I.n_freq;
    Probe<real> r;
    r.comp = -1;
    if ((int)threadIdx.x < per && p < I.n_probe) r = res_probe(I, cur, p);
    const int kind = r.comp < 0 ? -1 : r.comp >= 3;  // 0: an E probe, 1: an H probe
    const bool dft = I.n_dft > 0;
    long long until = n0 % I.save_span;              // steps to the next save point
    until = until ? I.save_span - until : 0;
    if (dft) {
        res_phases(I, n0, 0, ph[0]);
        res_phases(I, n0, 1, ph[1]);
    }
    __syncthreads();
    if (h_probes) {
        if (kind == 1) res_sample(I, r, n0, until == 0, n_freq, st, ph[1]);
        if (!grid_barrier(bar, target += gridDim.x, limit, st)) return;
    }
    for (int s = 0; s < n_steps; ++s) {
        const long long n = n0 + s;
        const bool more = s + 1 < n_steps;
        if (kind == 0) res_sample(I, r, n, until == 0, n_freq, st, ph[0]);
        until = until ? until - 1 : I.save_span - 1;
        if (dft && h_probes) res_phases(I, n + 1, 1, ph[1]);
        if (!grid_barrier(bar, target += gridDim.x, limit, st)) return;
        if (dft) res_phases(I, n + 1, 0, ph[0]);
        if (kind == 1 && more) res_sample(I, r, n + 1, until == 0, n_freq, st, ph[1]);
        if (more && !grid_barrier(bar, target += gridDim.x, limit, st)) return;
    }
}

// ONE: a single instance, its descriptor in the parameter space; else the
// descriptors are copied to shared memory.  The fields' buffer `cur` is
// stepped in place.
template <typename real, int T, bool ONE, bool DES>
__global__ void __launch_bounds__(T, 1)
k_resident(const __grid_constant__ InstDev<real> one, const InstDev<real>* __restrict__ tab, int n_inst, int cur,
           int n_steps, int workers, int probe_blocks, int per, int h_probes, int one_chunk, const ObjDev<real>* __restrict__ obj,
           unsigned* bar, unsigned long long limit, int stall, DevState* st) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ ResGrid grids[RES_MAX_INST];
    constexpr unsigned CH = res_chunk<real, T>(), SLOTS = T / CH;
    const long long n0 = st->step;
    if ((int)blockIdx.x >= workers) {
        if (stall && blockIdx.x == gridDim.x - 1) return;  // sj_set_test_stall: never arrives at a barrier
        int b = (int)blockIdx.x - workers;
        if (b < probe_blocks) {
            res_probe_block<real>(tab, n_inst, cur, n0, n_steps, b, probe_blocks, per, h_probes, one_chunk, bar, limit,
                                  st);
            return;
        }
        if constexpr (DES) {
            b -= probe_blocks;
            int q = 0;
            for (;; ++q) {
                const int c = (3 * obj[q].n_cells + (int)blockDim.x - 1) / (int)blockDim.x;
                if (b < c) break;
                b -= c;
            }
            res_objective_block<real>(obj[q], cur, b, n0, n_steps, h_probes, bar, limit, st);
        }
        return;
    }
    InstDev<real>* sh = reinterpret_cast<InstDev<real>*>(smem);
    if (!ONE) {
        const int* s = reinterpret_cast<const int*>(tab);
        int* d = reinterpret_cast<int*>(sh);
        const int nw = n_inst * (int)(sizeof(InstDev<real>) / sizeof(int));
        for (int w = threadIdx.x; w < nw; w += blockDim.x) d[w] = s[w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        unsigned first = 0;
        for (int q = 0; q < n_inst; ++q) {
            const InstDev<real>& I = ONE ? one : sh[q];
            ResGrid& g = grids[q];
            const unsigned rows = (unsigned)I.ny * (unsigned)I.nz;
            const unsigned ws = sizeof(real) == 8 ? (unsigned)(I.pl[0] + I.ph[0]) : 0u;
            g.dx.set(max(1u, (unsigned)I.nx - ws));
            g.dxs.set(max(1u, ws));
            g.dy.set((unsigned)I.ny);
            g.inner = ((unsigned)I.nx - ws) * rows;
            g.cells = (unsigned)I.nx * rows;
            g.lo = ws ? I.pl[0] : 0;
            // this block's first cell: chunks go to the blocks in turn, instance after instance
            g.start = (blockIdx.x + (unsigned)workers - first) % (unsigned)workers * CH;
            first = (first + (g.cells + CH - 1) / CH) % (unsigned)workers;
            g.hsrc = g.esrc = 0;
            for (int s = 0; s < I.n_src; ++s) (I.src[s].comp >= 3 ? g.hsrc : g.esrc) = 1;
        }
    }
    __syncthreads();
    const unsigned at = threadIdx.x / CH * ((unsigned)workers * CH) + threadIdx.x % CH;
    const unsigned stride = (unsigned)workers * CH * SLOTS;
    unsigned target = 0;
    if (h_probes && !grid_barrier(bar, target += gridDim.x, limit, st)) return;
    for (int s = 0; s < n_steps; ++s) {
        const long long n = n0 + s;
        for (int q = 0; q < n_inst; ++q) {
            const ResGrid& G = grids[q];
            for (unsigned t = G.start + at; t < G.cells; t += stride) res_h<real>(ONE ? one : sh[q], G, cur, t, n);
        }
        if (!grid_barrier(bar, target += gridDim.x, limit, st)) return;
        for (int q = 0; q < n_inst; ++q) {
            const ResGrid& G = grids[q];
            for (unsigned t = G.start + at; t < G.cells; t += stride) res_e<DES>(ONE ? one : sh[q], G, cur, t, n);
        }
        if (s + 1 < n_steps && !grid_barrier(bar, target += gridDim.x, limit, st)) return;
    }
    // every block read st->step before the first barrier
    if (blockIdx.x == 0 && threadIdx.x == 0) st->step = n0 + n_steps;
}

}  // namespace

namespace {
template <typename real, int T>
const void* res_kernel_t(int n_inst, bool des) {
    if (n_inst > 1)
        return des ? (const void*)k_resident<real, T, false, true> : (const void*)k_resident<real, T, false, false>;
    return des ? (const void*)k_resident<real, T, true, true> : (const void*)k_resident<real, T, true, false>;
}
template <typename real>
const void* res_kernel(bool few, int n_inst, bool des) {
    return few ? res_kernel_t<real, res_threads<real>(true)>(n_inst, des)
               : res_kernel_t<real, res_threads<real>(false)>(n_inst, des);
}
template <typename real>
bool res_few(const InstDev<real>* h_insts, int n_inst) {
    long long cells = 0;
    for (int q = 0; q < n_inst; ++q) cells += (long long)h_insts[q].nx * h_insts[q].ny * h_insts[q].nz;
    return cells < RES_FEW_CELLS;
}

// How the probes of a launch are dealt out, and ns per step of the cells and
// of the probes (E probes ride on the H phase, H probes on the E phase).
// Fitted to runs with 1000 to 200000 probes of 5 to 256 frequencies on 64^3 and
// 128^3: a block takes 18 ns for a probe (its stencil, indexes and weights from
// L2) and 2.6 ns for each of its DFT sums (a row is its own thread's: 32-byte
// sectors read and written by one SM), at least 250 ns per frequency (a
// thread's sums go through L2 four at a time).  So the probes' blocks are as
// many as keep them within half a step of the cells, at most an eighth of the
// grid: every thread takes a probe where that gives as many, else fewer do
// (64^3 FP32, 1000 probes of 50 frequencies: 141 us per step in one block, 33
// in eleven; 10000 of 5: 34 and 22).
struct ProbePlan {
    int blocks, per;         // probe blocks, probes per chunk
    long long chunks;
    double cells, probes[2]; // ns
};
template <typename real>
ProbePlan probe_plan(const InstDev<real>* h_insts, int n_inst, int max_blocks) {
    const int T = res_threads<real>(res_few(h_insts, n_inst)), most = std::max(1, max_blocks / 8);
    ProbePlan P = {};
    double cells = 0, ns[2] = {0, 0}, chain = 0;
    long long total = 0;
    for (int q = 0; q < n_inst; ++q) {
        const InstDev<real>& I = h_insts[q];
        cells += (double)I.nx * I.ny * I.nz;
        total += I.n_probe;
        const double each = I.n_probe ? 18.0 / (I.n_dft ? 1 : I.save_span) + 2.6 * I.n_dft * I.n_freq / I.n_probe : 0.0;
        ns[0] += each * (I.n_probe - I.n_hprobe);
        ns[1] += each * I.n_hprobe;
        if (I.n_dft) chain = std::max(chain, 250.0 * I.n_freq);
    }
    P.cells = sizeof(real) == 4 ? 5000 + 0.021 * cells : 9000 + 0.066 * cells;
    const auto chunks = [&](int per) {
        long long c = 0;
        for (int q = 0; q < n_inst; ++q) c += (h_insts[q].n_probe + per - 1) / per;
        return c;
    };
    P.per = T;
    const double want = std::min<double>(most, std::ceil(2 * std::max(ns[0], ns[1]) / P.cells));
    if (want > (double)chunks(T)) {
        P.per = std::min(T, ((int)std::ceil(total / want) + 31) / 32 * 32);
        while (P.per < T && chunks(P.per) > most) P.per += 32;
        P.per = std::min(P.per, T);
    }
    P.chunks = chunks(P.per);
    P.blocks = (int)std::min<long long>(P.chunks, most);
    if (P.chunks) {
        const double rounds = (double)((P.chunks + P.blocks - 1) / P.blocks);
        for (int h = 0; h < 2; ++h)
            P.probes[h] = std::max(ns[h] ? chain : 0.0, ns[h] / total * std::min<double>(rounds * P.per, (double)total));
    }
    return P;
}
}  // namespace

// Does a run of steps with these probes take less time here than as tile
// launches, whose probes are spread over the whole device?  us per step of the
// tile launches, without probes: FP32 64^3 41, 128^3 77, 160^3 102; FP64 64^3
// 71, 128^3 240, 256 x 256 x 192 974.  64^3 FP32 with 10000 probes of 50
// frequencies: 142 us here, 45 there; 50000: 432 and 50; 128^3 FP64 with 200000:
// 1441 and 370.
template <typename real>
bool resident_pays(const InstDev<real>* h_insts, int n_inst, int max_blocks) {
    const ProbePlan P = probe_plan(h_insts, n_inst, max_blocks);
    if (!P.chunks) return true;
    double cells = 0;
    for (int q = 0; q < n_inst; ++q) cells += (double)h_insts[q].nx * h_insts[q].ny * h_insts[q].nz;
    const double tiles = sizeof(real) == 4 ? 35000 + 0.0165 * cells : 50000 + 0.075 * cells;
    return std::max(P.cells / 2, P.probes[0]) + std::max(P.cells / 2, P.probes[1]) <= tiles;
}
template bool resident_pays<float>(const InstDev<float>*, int, int);
template bool resident_pays<double>(const InstDev<double>*, int, int);

template <typename real>
int resident_grid(const InstDev<real>* h_insts, int n_inst) {
    int dev = 0, sms = 0, coop = 0, least = INT_MAX;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (!coop) return 0;
    const bool few = res_few(h_insts, n_inst);
    const size_t smem = n_inst > 1 ? (size_t)n_inst * sizeof(InstDev<real>) : 0;
    for (int des = 0; des < 2; ++des) {
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, res_kernel<real>(few, n_inst, des), res_threads<real>(few),
                                                          smem) != cudaSuccess)
            return 0;
        least = std::min(least, nb);
    }
    return least * sms;
}

template <typename real>
int resident_objective_blocks(const InstDev<real>* h_insts, const ObjDev<real>* o, int n_inst) {
    const int T = res_threads<real>(res_few(h_insts, n_inst));
    int b = 0;
    for (int q = 0; q < n_inst; ++q) b += (3 * o[q].n_cells + T - 1) / T;
    return b;
}

template <typename real>
cudaError_t launch_resident(const InstDev<real>* h_insts, const InstDev<real>* d_insts, int n_inst, int cur,
                            int n_steps, int max_blocks, const ObjDev<real>* d_obj, int obj_blocks, unsigned* d_bar,
                            unsigned long long limit_ns, int stall, DevState* st, cudaStream_t s) {
    long long cells = 0;
    int h_probes = 0;
    bool des = d_obj != nullptr;
    const bool few = res_few(h_insts, n_inst);
    const int T = res_threads<real>(few);
    for (int q = 0; q < n_inst; ++q) {
        const InstDev<real>& I = h_insts[q];
        cells += (long long)I.nx * I.ny * I.nz;
        h_probes |= I.n_hprobe > 0;
        des |= I.dinv != nullptr;
    }
    ProbePlan plan = probe_plan(h_insts, n_inst, max_blocks);
    int probe = plan.blocks;
    stall = stall ? 1 : 0;  // one block more
    int w = (int)std::min<long long>((cells + T - 1) / T, max_blocks - probe - obj_blocks - stall);
    if (w < 1) return cudaErrorInvalidValue;
    // The barrier's counter starts at 0.  After a time-out it starts above any target:
    // the status's low byte over three zero bytes (cur is 0 or 1), so that launches
    // queued behind, which have no state to step on, do not wait either.  (1.2 us more
    // than a memset per launch; the status read in the kernel instead moved the step
    // loop's time by 1-2%, registers and spills the same.)
    static_assert(offsetof(DevState, status) == offsetof(DevState, cur) + sizeof(int) && SJ_E_TIMEOUT < 0, "layout");
    cudaError_t e = cudaMemcpyAsync(d_bar, reinterpret_cast<const char*>(st) + offsetof(DevState, status) - 3,
                                    sizeof(unsigned), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    InstDev<real> one = h_insts[0];
    int one_chunk = plan.chunks <= probe;
    void* args[] = {&one,      &d_insts,   &n_inst, &cur,   &n_steps,  &w,     &probe, &plan.per,
                    &h_probes, &one_chunk, &d_obj,  &d_bar, &limit_ns, &stall, &st};
    const size_t smem = n_inst > 1 ? (size_t)n_inst * sizeof(InstDev<real>) : 0;
    return cudaLaunchCooperativeKernel(res_kernel<real>(few, n_inst, des), dim3(w + probe + obj_blocks + stall), dim3(T), args,
                                       smem, s);
}

template int resident_grid<float>(const InstDev<float>*, int);
template int resident_grid<double>(const InstDev<double>*, int);
template int resident_objective_blocks<float>(const InstDev<float>*, const ObjDev<float>*, int);
template int resident_objective_blocks<double>(const InstDev<double>*, const ObjDev<double>*, int);
template cudaError_t launch_resident<float>(const InstDev<float>*, const InstDev<float>*, int, int, int, int,
                                            const ObjDev<float>*, int, unsigned*, unsigned long long, int,
                                            DevState*, cudaStream_t);
template cudaError_t launch_resident<double>(const InstDev<double>*, const InstDev<double>*, int, int, int, int,
                                             const ObjDev<double>*, int, unsigned*, unsigned long long, int,
                                             DevState*, cudaStream_t);

}  // namespace sj
