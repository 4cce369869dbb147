// k_dsm64.cu -- the dynamic Smagorinsky pass (subgrid.f90:376-538) of the
// FP64 path, as two kernels without shared memory or barriers.
//
// An SM issues one FP64 warp instruction per 19 clocks (each of its four
// sub-partitions one per 64-76), whatever the number of resident warps, so
// the pass costs its FP64 instructions and nothing else: about 240 a cell
// here, in 4.7 M cells 2.1 ms, against 0.25 ms for the 300 bytes a cell that
// go through memory.  (A one-pass tile kernel took
// 539: the halo of its tiles is computed 1.4 times over, its strain rates
// take every difference by itself, and its filters a multiply for each
// weight; 7.0 ms per pass at 192 x 128 x 192 cells, where its tiles also
// filled 63 % of the block slots.  The two kernels: 0.84 + 1.52 ms.)
//
// A warp owns a segment of W = 32 or 16 adjacent columns of one row j and
// marches along z over a chunk of planes; W = 16 packs two rows into a warp
// where that leaves fewer idle columns.  x neighbours come from the
// neighbouring lanes by shuffles; the values of the two columns next to a
// segment are formed by its first lanes, one quantity and side each, so that
// a row's edges cost the instructions of one quantity.  y neighbours are
// loaded (or summed) again per row, z neighbours are carried up the march.
//
// Scales: every filter is taken with the weights 1, 4, 1 (a + c, then one
// multiply-add with 4), a factor 6 per direction, 216 in all; the one-sided
// rule of the end rows (2/3, 1/3) is 4 and 2, i.e. the neighbour inside
// taken for both.  Centre velocities enter as sums of two faces (u2 = 2 u)
// and the mixed strain rates as the sums over their four edges (t = 8 S_ij).
// All of it is undone once per warp, in the plane partials.
//
//   k_dsm64_q   at every canonical cell from U, V, W at actual indices
//               (subgrid.f90:390-428): u2_i u2_j, |S| S_ij (t for the mixed
//               ones), |S|; and 216 Uf, Vf, Wf on the canonical elements
//               (subgrid.f90:429-445)
//   k_dsm64_lm  their filters, L, M and the plane partials of L.M and M.M
//               (subgrid.f90:447-513), everything through the periodic wrap
//               (the reference's periodic fills, subgrid.f90:448-458)
//
// hat(u_i) is taken from the filtered velocities (the mean of two faces and
// the filter commute) except in the rows 2 and nyg-1, where the reference's
// one-sided filter of the centre velocities does not read the ghost rows that
// Uf uses: there the centre velocities are stored and filtered themselves.
#include <algorithm>

#include "cf_internal.cuh"

namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr int D64_T = 128;  // threads per block: one warp per sub-partition

// canonical arrays of dsm_q: the 12 filtered quantities, the centre
// velocities (rows 2, 3, nyg-2, nyg-1 only), |S| (slot 15, where every
// reader of the lazily formed nu_t expects it)
enum { D_U2 = 0, D_V2, D_W2, D_Q0, D_S = 15 };

struct D64 {
    Fld<double> U, V, W, Uf, Vf, Wf;  // state and (canonical elements of) the filtered velocities
    RcpT<double> rc;
    double *q;                        // canonical arrays, n apart
    int ng;  // groups of components
    double *part;
    long n;
    int nx, ny, nz, nxg, nyg, nxp, nym, nzp, nseg, kc_len, nkc;
};

template <int W>
struct Seg {
    int l, s, j, i0, i;  // lane in the segment, segment, row, first and own column
    bool act;            // the segment exists
    __device__ __forceinline__ Seg(int nrows, int j0, int nseg) {
        constexpr int SPW = 32 / W;
        const long tot = (long)nrows * nseg;
        long g = ((long)blockIdx.x * (D64_T / 32) + (threadIdx.x >> 5)) * SPW + (threadIdx.x & 31) / W;
        act = g < tot;
        g = act ? g : tot - 1;
        l = threadIdx.x & (W - 1);
        s = (int)(g / nrows);  // rows fastest: the warps of a block share their rows' neighbours
        j = j0 + (int)(g % nrows);
        i0 = 2 + s * W;
        i = i0 + l;
    }
    // the value of the lane to the left / right; from `edge` of lane el at the segment's ends
    __device__ __forceinline__ double left(double v, double edge, int el) const {
        const double a = __shfl_up_sync(FULLM, v, 1, W), b = __shfl_sync(FULLM, edge, el, W);
        return l == 0 ? b : a;
    }
    __device__ __forceinline__ double right(double v, double edge, int el) const {
        const double a = __shfl_down_sync(FULLM, v, 1, W), b = __shfl_sync(FULLM, edge, el, W);
        return l == W - 1 ? b : a;
    }
};

// |S| from the diagonal components and t = 8 x the mixed ones
__device__ __forceinline__ double s_mag(double d0, double d1, double d2, double t12, double t13, double t23) {
    const double a = d0 * d0 + d1 * d1 + d2 * d2, b = t12 * t12 + t13 * t13 + t23 * t23;
    const double x = fma(b, 1.0 / 32.0, a);
    return sqrt(x + x);
}

template <int W>
__global__ void __launch_bounds__(D64_T) k_dsm64_q(const __grid_constant__ D64 a) {
    const Seg<W> sg(a.nyg, 1, a.nseg);
    const int nx = a.nx, ny = a.ny, nyg = a.nyg, j = sg.j, l = sg.l;
    const int kb = 2 + blockIdx.y * a.kc_len, ke = min(kb + a.kc_len - 1, a.nz - 1);
    const int i = min(sg.i, nx);  // the last column read: the right neighbour of nx-1
    const bool cell = j >= 2 && j <= nyg - 1;
    const bool own = sg.act && sg.i <= nx - 1, ownq = own && cell;
    // rows: the neighbours of j, reflected at the ends of the arrays (the
    // filter's one-sided rule); for cells they are j-1 and j+1.  V has ny rows
    const int ja = j == 1 ? 2 : j - 1, jc = j == nyg ? nyg - 1 : j + 1;
    const int jv = min(j, ny), jva = jv == 1 ? 2 : jv - 1, jvc = jv == ny ? ny - 1 : jv + 1;
    const long uo = a.U.idx(i, j, 0), uoa = a.U.idx(i, ja, 0), uoc = a.U.idx(i, jc, 0);
    const long vo = a.V.idx(i, jv, 0), voa = a.V.idx(i, jva, 0), voc = a.V.idx(i, jvc, 0);
    const long wo = a.W.idx(i, j, 0), woa = a.W.idx(i, ja, 0), woc = a.W.idx(i, jc, 0);
    // edge lanes: field l / 2 (U, V, W), side l % 2
    const int ef = l < 6 ? l >> 1 : 0;
    const Fld<double> E = ef == 0 ? a.U : (ef == 1 ? a.V : a.W);
    const int ei = (l & 1) ? min(sg.i0 + W, nx) : sg.i0 - 1;
    const long eo = E.idx(ei, ef == 1 ? jv : j, 0), eoa = E.idx(ei, ef == 1 ? jva : ja, 0),
               eoc = E.idx(ei, ef == 1 ? jvc : jc, 0);
    const bool edge = l < 6;
    const int ig = min(sg.i, nx - 1), jg = min(max(j, 2), nyg - 1);
    const double rx = a.rc.dx[ig], rx0 = a.rc.dxg[ig], rx1 = a.rc.dxg[ig + 1];
    const double ry = a.rc.dy[jg], ry0 = a.rc.dyg[jg], ry1 = a.rc.dyg[jg + 1];
    const bool keepu = j <= 3 || j >= nyg - 2;  // centre velocities stored
    const bool anyc = __any_sync(FULLM, cell);
    double u2l = 0, v2l = 0, wl0 = 0, wla = 0, wlc = 0, el = 0;                        // plane p-1
    double t12 = 0, p13 = 0, p23 = 0, d0 = 0, d1 = 0, d2 = 0, u2o = 0, v2o = 0, w2o = 0;  // pending cell at p-1
    double h0[3] = {0, 0, 0}, h1[3] = {0, 0, 0};                                       // x-y filtered planes p-2, p-1
    const long plane = (long)a.nxp * a.nym;
    double *qp = a.q + (long)(ig - 2) + (long)a.nxp * (jg - 2) + plane * (kb - 2);
    for (int p = kb - 1; p <= ke + 1; p++) {
        const long uz = (long)a.U.sz * p, vz = (long)a.V.sz * p, wz = (long)a.W.sz * p;
        const double *U = a.U.p + uz, *V = a.V.p + vz, *Wp = a.W.p + wz;
        const double u1 = U[uo], ua = U[uoa], uc = U[uoc];
        const double v1 = V[vo], va = V[voa], vc = V[voc];
        const double w1 = Wp[wo], wa = Wp[woa], wc = Wp[woc];
        const double um1 = U[uo - 1], uma = U[uoa - 1], umc = U[uoc - 1];
        double x0 = 0, x1 = 0, x2 = 0;
        if (edge) {
            const double *Ep = E.p + (long)E.sz * p;
            x0 = Ep[eoa];
            x1 = Ep[eo];
            x2 = Ep[eoc];
        }
        // filtered velocities: y, x, then z from the two planes below
        const double ey = fma(4.0, x1, x0 + x2);
        const double fy[3] = {fma(4.0, u1, ua + uc), fma(4.0, v1, va + vc), fma(4.0, w1, wa + wc)};
        double fo[3];
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const double fx = fma(4.0, fy[f], sg.left(fy[f], ey, 2 * f) + sg.right(fy[f], ey, 2 * f + 1));
            fo[f] = fma(4.0, h1[f], h0[f] + fx);
            h0[f] = h1[f];
            h1[f] = fx;
        }
        if (p >= kb + 1 && own) {
            a.Uf.p[a.Uf.idx(sg.i, j, p - 1)] = fo[0];
            if (j <= ny) a.Vf.p[a.Vf.idx(sg.i, j, p - 1)] = fo[1];
            a.Wf.p[a.Wf.idx(sg.i, j, p - 1)] = fo[2];
        }
        if (anyc) {
            const double u2 = um1 + u1, v2 = va + v1;
            if (p >= kb) {
                const double dzr = a.rc.dzg[p], du = (u2 - u2l) * dzr, dv = (v2 - v2l) * dzr;
                if (p >= kb + 1) {  // the cell at p-1 is complete
                    const double t13 = p13 + du, t23 = p23 + dv;
                    const double S = s_mag(d0, d1, d2, t12, t13, t23);
                    if (ownq) {
                        const long n = a.n;
                        qp[(D_Q0 + 0) * n] = u2o * u2o;
                        qp[(D_Q0 + 1) * n] = v2o * v2o;
                        qp[(D_Q0 + 2) * n] = w2o * w2o;
                        qp[(D_Q0 + 3) * n] = u2o * v2o;
                        qp[(D_Q0 + 4) * n] = u2o * w2o;
                        qp[(D_Q0 + 5) * n] = v2o * w2o;
                        qp[(D_Q0 + 6) * n] = S * d0;
                        qp[(D_Q0 + 7) * n] = S * d1;
                        qp[(D_Q0 + 8) * n] = S * d2;
                        qp[(D_Q0 + 9) * n] = S * t12;
                        qp[(D_Q0 + 10) * n] = S * t13;
                        qp[(D_Q0 + 11) * n] = S * t23;
                        qp[D_S * n] = S;
                        if (keepu) {
                            qp[D_U2 * n] = u2o;
                            qp[D_V2 * n] = v2o;
                            qp[D_W2 * n] = w2o;
                        }
                    }
                    qp += plane;
                }
                if (p <= ke) {
                    const double u2a = uma + ua, u2c = umc + uc;
                    const double w2 = wl0 + w1, w2a = wla + wa, w2c = wlc + wc;
                    const double es = (ef == 1 ? x0 : el) + x1;  // v2 and w2 of the edge columns
                    const double vL = sg.left(v2, es, 2), vR = sg.right(v2, es, 3);
                    const double wL = sg.left(w2, es, 4), wR = sg.right(w2, es, 5);
                    t12 = (u2 - u2a) * ry0 + (u2c - u2) * ry1 + (v2 - vL) * rx0 + (vR - v2) * rx1;
                    p13 = du + (w2 - wL) * rx0 + (wR - w2) * rx1;
                    p23 = dv + (w2 - w2a) * ry0 + (w2c - w2) * ry1;
                    d0 = (u1 - um1) * rx;
                    d1 = (v1 - va) * ry;
                    d2 = (w1 - wl0) * a.rc.dz[p];
                    u2o = u2;
                    v2o = v2;
                    w2o = w2;
                }
            }
            u2l = u2;
            v2l = v2;
        }
        wl0 = w1;
        wla = wa;
        wlc = wc;
        el = x1;
    }
}

// Components C0 .. C0+NC-1 of L and M (11, 22, 33, 12, 13, 23); `group` is
// the slot of their partials among a.ng.
template <int W, int C0, int NC>
__device__ __forceinline__ void lm_march(const D64 &a, int group) {
    constexpr int NQ = 2 * NC;  // filtered quantities: u_i u_j, then |S| S_ij
    auto qid = [](int q) { return q < NC ? C0 + q : 6 + C0 + q - NC; };
    const Seg<W> sg(a.nym, 2, a.nseg);
    const int nx = a.nx, nyg = a.nyg, nxp = a.nxp, nzp = a.nzp, j = sg.j, l = sg.l;
    const int kb = 2 + blockIdx.y * a.kc_len, ke = min(kb + a.kc_len - 1, a.nz - 1);
    const bool own = sg.act && sg.i <= nx - 1;
    const int i = wrapn(min(sg.i, nx), nxp), im = wrapn(i - 1, nxp);
    const int iL = wrapn(sg.i0 - 1, nxp), iR = wrapn(min(sg.i0 + W, nx), nxp);
    // canonical offsets of this column in rows j-1, j, j+1 (reflected at rows 2 and nyg-1)
    const int ja = j == 2 ? 3 : j - 1, jc = j == nyg - 1 ? nyg - 2 : j + 1;
    const int q1 = (i - 2) + nxp * (j - 2), qa = (i - 2) + nxp * (ja - 2), qc = (i - 2) + nxp * (jc - 2);
    const long plane = (long)nxp * a.nym, n = a.n;
    // edge lanes of the quantities' y filter: quantity eq, side; W = 32 both
    // sides at once (lanes 0-15 left, 16-31 right), W = 16 one after the other
    const int eq = qid(min(l & 15, NQ - 1));
    const int e0 = (W == 32 && l >= 16 ? iR : iL) - 2;
    const double *const EQ = a.q + (D_Q0 + eq) * n + e0 + nxp * (j - 2);
    const int eda = nxp * (ja - j), edc = nxp * (jc - j), edr = iR - iL;
    // edge lanes of v2, w2 of the filtered velocities: lanes 0, 1 V, 2, 3 W
    const Fld<double> E = l < 2 ? a.Vf : a.Wf;
    const long eo = E.idx((l & 1) ? iR : iL, j, 0);
    const long uo = a.Uf.idx(i, j, 0), uom = a.Uf.idx(im, j, 0), vo = a.Vf.idx(i, j, 0), wo = a.Wf.idx(i, j, 0);
    const long usy = a.Uf.sy, vsy = a.Vf.sy, wsy = a.Wf.sy;
    const int ig = min(sg.i, nx - 1);
    const double rx = a.rc.dx[ig], rx0 = a.rc.dxg[ig], rx1 = a.rc.dxg[ig + 1];
    const double ry = a.rc.dy[j], ry0 = a.rc.dyg[j], ry1 = a.rc.dyg[j + 1];
    const bool wrow = j == 2 || j == nyg - 1, anyw = __any_sync(FULLM, wrow);
    double h0[NQ], h1[NQ], g0[3] = {0, 0, 0}, g1[3] = {0, 0, 0};
#pragma unroll
    for (int q = 0; q < NQ; q++) h0[q] = h1[q] = 0;
    double u2l = 0, v2l = 0, wl0 = 0, wla = 0, wlc = 0, el = 0;
    double t12 = 0, p13 = 0, p23 = 0, d0 = 0, d1 = 0, d2 = 0, w2o = 0;
    double lmd = 0, lmo = 0, mmd = 0, mmo = 0;
    for (int r = kb - 1; r <= ke + 1; r++) {
        const int k = wrapn(r, nzp);
        const double *Q = a.q + D_Q0 * n + plane * (k - 2);
        // filtered velocities of plane r
        const double *U = a.Uf.p + (long)a.Uf.sz * k, *V = a.Vf.p + (long)a.Vf.sz * k, *Wp = a.Wf.p + (long)a.Wf.sz * k;
        const double u1 = U[uo], ua = U[uo - usy], uc = U[uo + usy];
        const double um1 = U[uom], uma = U[uom - usy], umc = U[uom + usy];
        const double v1 = V[vo], va = V[vo - vsy];
        const double w1 = Wp[wo], wa = Wp[wo - wsy], wc = Wp[wo + wsy];
        double x0 = 0, x1 = 0;
        if (l < 4) {
            const double *Ep = E.p + (long)E.sz * k;
            x1 = Ep[eo];
            if (l < 2) x0 = Ep[eo - E.sy];
        }
        // y filter at the two columns next to the segment
        const double *Eq = EQ + plane * (k - 2);
        const double yL = fma(4.0, Eq[0], Eq[eda] + Eq[edc]);
        double yR = yL;
        if constexpr (W == 16) yR = fma(4.0, Eq[edr], Eq[edr + eda] + Eq[edr + edc]);
        double H[NQ];
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const long qo = qid(q) * n;
            const double y = fma(4.0, Q[q1 + qo], Q[qa + qo] + Q[qc + qo]);
            const double x = fma(4.0, y, sg.left(y, yL, q) + sg.right(y, yR, W == 32 ? 16 + q : q));
            H[q] = fma(4.0, h1[q], h0[q] + x);
            h0[q] = h1[q];
            h1[q] = x;
        }
        double hw[3] = {0, 0, 0};
        if (anyw) {  // the centre velocities filtered one-sided (every lane for its neighbours' sake)
            const double *C = a.q + plane * (k - 2);
#pragma unroll
            for (int f = 0; f < 3; f++) {
                auto yf = [&](int o) { return fma(4.0, C[o + nxp * (j - 2) + f * n], C[o + nxp * (ja - 2) + f * n] + C[o + nxp * (jc - 2) + f * n]); };
                const double y = yf(i - 2), e = yf(((l & 1) ? iR : iL) - 2);
                const double x = fma(4.0, y, sg.left(y, e, 0) + sg.right(y, e, 1));
                hw[f] = fma(4.0, g1[f], g0[f] + x);
                g0[f] = g1[f];
                g1[f] = x;
            }
        }
        const double u2 = um1 + u1, v2 = va + v1;
        if (r >= kb) {
            const double dzr = a.rc.dzg[r], du = (u2 - u2l) * dzr, dv = (v2 - v2l) * dzr;
            if (r >= kb + 1) {  // plane r-1 is complete
                const double t13 = p13 + du, t23 = p23 + dv;
                const double c = s_mag(d0, d1, d2, t12, t13, t23) * (1.0 / 54.0);
                const double fu = wrow ? hw[0] : u2l, fv = wrow ? hw[1] : v2l, fw = wrow ? hw[2] : w2o;
                const double f[3] = {fu, fv, fw}, S[6] = {d0, d1, d2, t12, t13, t23};
                const int reps = r - 1 == 2 ? 2 : 1;  // plane 2 stands for its duplicate too
#pragma unroll
                for (int q = 0; q < NC; q++) {
                    constexpr int IA[6] = {0, 1, 2, 0, 0, 1}, IB[6] = {0, 1, 2, 1, 2, 2};
                    const double L = fma(-f[IA[C0 + q]], f[IB[C0 + q]] * (1.0 / 216.0), H[q]), M = fma(c, S[C0 + q], -H[NC + q]);
                    double &lm = C0 + q < 3 ? lmd : lmo, &mm = C0 + q < 3 ? mmd : mmo;
                    for (int t = 0; t < reps; t++) {
                        lm = fma(L, M, lm);
                        mm = fma(M, M, mm);
                    }
                }
            }
            if (r <= ke) {
                const double u2a = uma + ua, u2c = umc + uc;
                const double w2 = wl0 + w1, w2a = wla + wa, w2c = wlc + wc;
                const double es = (l < 2 ? x0 : el) + x1;
                const double vL = sg.left(v2, es, 0), vR = sg.right(v2, es, 1);
                const double wL = sg.left(w2, es, 2), wR = sg.right(w2, es, 3);
                t12 = (u2 - u2a) * ry0 + (u2c - u2) * ry1 + (v2 - vL) * rx0 + (vR - v2) * rx1;
                p13 = du + (w2 - wL) * rx0 + (wR - w2) * rx1;
                p23 = dv + (w2 - w2a) * ry0 + (w2c - w2) * ry1;
                d0 = (u1 - um1) * rx;
                d1 = (v1 - va) * ry;
                d2 = (w1 - wl0) * a.rc.dz[r];
                w2o = w2;
            }
        }
        u2l = u2;
        v2l = v2;
        wl0 = w1;
        wla = wa;
        wlc = wc;
        el = x1;
    }
    // undo the scales; column 2 stands for its duplicate too
    const double wx = own ? (sg.i == 2 ? 2.0 : 1.0) : 0.0;
    double sl = wx * fma(0.25, lmo, lmd) * (1.0 / (864.0 * 216.0)), sm = wx * fma(1.0 / 32.0, mmo, mmd) * (1.0 / (216.0 * 216.0));
    if (!own) sl = sm = 0.0;
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
        sl += __shfl_down_sync(FULLM, sl, o, W);
        sm += __shfl_down_sync(FULLM, sm, o, W);
    }
    if (l == 0 && sg.act) {
        const long slot = ((long)(j - 2) * (a.nseg * a.nkc) + sg.s * a.nkc + blockIdx.y) * a.ng + group;
        a.part[2 * slot] = sl;
        a.part[2 * slot + 1] = sm;
    }
}

template <int W>
__global__ void __launch_bounds__(D64_T) k_dsm64_lm(const __grid_constant__ D64 a) {
    lm_march<W, 0, 6>(a, 0);
}
// two components a warp (blockIdx.z): the strain rates of the filtered
// velocities are formed by three warps instead of one
template <int W>
__global__ void __launch_bounds__(D64_T) k_dsm64_lm3(const __grid_constant__ D64 a) {
    if (blockIdx.z == 0) lm_march<W, 0, 2>(a, 0);
    else if (blockIdx.z == 1) lm_march<W, 2, 2>(a, 1);
    else lm_march<W, 4, 2>(a, 2);
}

// lanes per segment: 16 where a row then has fewer idle columns (a warp
// instruction costs the same with idle lanes)
int d64_w(int nxp) { return cdiv(nxp, 16) * 16 < cdiv(nxp, 32) * 32 ? 16 : 32; }

}  // namespace

// z-chunk length (192 x 128 x 192: 28 planes, whose last wave is nearly
// empty, 2.55 ms a pass; 18 to 24 planes 2.36)
int dsm64_plan(int nxp, int nym, int nzp, int sms) {
    const int w = d64_w(nxp), nseg = cdiv(nxp, w);
    return fp64_chunk_len(cdiv((long)nseg * nym, (32 / w) * (D64_T / 32)), sms, nzp, 1, 0.9);
}

// (three per segment and chunk where its components are split)
int dsm64_slots(int nxp, int nzp, int kc) { return 3 * cdiv(nxp, d64_w(nxp)) * cdiv(nzp, kc); }

// |S| into the canonical scratch, the plane partials into dsm_part
int launch_dsm64(cf_ctx *ctx, int b, int *nchunk) {
    D64 a;
    a.U = make_fld<double>(ctx->U[b], ctx->nx, ctx->nyg);
    a.V = make_fld<double>(ctx->V[b], ctx->nxg, ctx->ny);
    a.W = make_fld<double>(ctx->W[b], ctx->nxg, ctx->nyg);
    a.Uf = make_fld<double>(ctx->Uf, ctx->nx, ctx->nyg);
    a.Vf = make_fld<double>(ctx->Vf, ctx->nxg, ctx->ny);
    a.Wf = make_fld<double>(ctx->Wf, ctx->nxg, ctx->nyg);
    a.rc = rcp_of<double>(ctx);
    a.q = (double *)ctx->dsm_q;
    a.part = ctx->dsm_part;
    a.n = (long)ctx->nCan;
    a.nx = ctx->nx; a.ny = ctx->ny; a.nz = ctx->nz; a.nxg = ctx->nxg; a.nyg = ctx->nyg;
    a.nxp = ctx->nxp; a.nym = ctx->nym; a.nzp = ctx->nzp;
    const int w = d64_w(ctx->nxp);
    a.nseg = cdiv(ctx->nxp, w);
    a.kc_len = ctx->dsm_kc;
    a.nkc = cdiv(ctx->nzp, ctx->dsm_kc);
    // Three warps for one where even so every quarter of an SM has at most one
    // (the smallest grids): about 90 FP64 instructions a plane of the march
    // instead of 165; 16^3 48 -> 34 us a launch (5 of them the launch).
    const long warps = cdiv((long)a.nseg * ctx->nym, 32 / w) * (long)a.nkc;
    a.ng = 3 * warps <= 4L * ctx->sms ? 3 : 1;
    *nchunk = a.nseg * a.nkc * a.ng;
    if ((size_t)*nchunk > ctx->dsm_part_nch) return cf_fail(ctx, CF_ERR_INVALID, "plane-partial slots");
    const int per = (32 / w) * (D64_T / 32);
    const dim3 gq(cdiv((long)a.nseg * ctx->nyg, per), a.nkc), gl(cdiv((long)a.nseg * ctx->nym, per), a.nkc);
    if (w == 32) k_dsm64_q<32><<<gq, D64_T, 0, ctx->st>>>(a);
    else k_dsm64_q<16><<<gq, D64_T, 0, ctx->st>>>(a);
    count_launch(ctx, "k_dsm64_q");
    const dim3 gl3(gl.x, gl.y, 3);
    if (a.ng == 3) {
        if (w == 32) k_dsm64_lm3<32><<<gl3, D64_T, 0, ctx->st>>>(a);
        else k_dsm64_lm3<16><<<gl3, D64_T, 0, ctx->st>>>(a);
    } else {
        if (w == 32) k_dsm64_lm<32><<<gl, D64_T, 0, ctx->st>>>(a);
        else k_dsm64_lm<16><<<gl, D64_T, 0, ctx->st>>>(a);
    }
    count_launch(ctx, "k_dsm64_lm");
    CF_CUDA(cudaGetLastError());
    return 0;
}
