// k_dsm32.cu -- the dynamic Smagorinsky pass (subgrid.f90:376-538) of the
// split path (FP32), as two kernels without shared memory or barriers.
//
//   k_dsm32_q   at every canonical cell from U, V, W at actual indices
//               (subgrid.f90:390-428): the centre velocities, |S| S_ij and
//               |S|; and 216 Uf, Vf, Wf (subgrid.f90:429-445)
//   k_dsm32_lm  the filters of u_i u_j and |S| S_ij, L, M and the plane
//               partials of L.M and M.M (subgrid.f90:447-513), everything
//               through the periodic wrap (the reference's periodic fills,
//               subgrid.f90:448-458)
//
// 112 bytes a cell go through memory (12 + 52 and 48), 80 us at 192 x 128 x
// 192 cells and the measured 6.75 TB/s; a one-pass tile kernel moved 16 but
// issued 860 instructions and 270 shared-memory wavefronts a cell with two
// barriers a plane (200 us).  Here a warp owns a segment of 2 LS columns of
// one row j and marches along z over a chunk of planes; a lane holds two
// adjacent columns, so that loads and stores of the canonical arrays are 8
// bytes a lane, the arithmetic is packed FP32x2, and the x filter needs one
// shuffle per side and quantity for two cells.  LS = 16 and 8 put two and
// four rows into a warp where that leaves fewer idle columns.  y neighbours
// are loaded again per row (L1), z neighbours are carried up the march.
//
// U, V, W are read at their actual indices, so the pass needs no periodic
// ghosts: it serves every state and either wall treatment.
//
// Scales: filters are taken with the weights 1, 4, 1, a factor 216 in all
// (the one-sided rule of the end rows, 2/3 and 1/3, is the neighbour inside
// taken for both); the centre velocities are stored as (sum of two faces)/32
// and |S| S_ij times 2^-11, the mixed components as sums over their four
// edges (8 S_ij), which keeps the sums of squares near their unscaled size.
// All powers of two but the 216, undone once per warp in the partials.
// Velocity differences are always taken between neighbours before anything
// is summed, as the reference does (a difference of sums would round the
// sums first).
//
// hat(u_i) is the mean of two faces' filtered velocities (the mean and the
// filter commute).  In the rows 2 and nyg-1 the reference's one-sided filter
// of the centre velocities does not read the ghost rows that Uf uses: two
// extra rows of k_dsm32_q filter U, V, W with that rule for them.
#include <algorithm>

#include "cf_internal.cuh"

namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr int D32_T = 128;  // threads per block

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 sp(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, sp(-1.f), a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg2(float2 a) { return f2(-a.x, -a.y); }
// a + 4 b + c
__device__ __forceinline__ float2 w141(float2 a, float2 b, float2 c) { return fma2(sp(4.f), b, add2(a, c)); }
__device__ __forceinline__ float w141(float a, float b, float c) { return fmaf(4.f, b, a + c); }

// canonical arrays of dsm_q: centre velocities, |S| S_ij, |S| (slot 15,
// where every reader of the lazily formed nu_t expects it)
// S_E..S_E+2: the one-sided rows of the filtered velocities, [k][2][nxp]
enum { S_U2 = 0, S_V2, S_W2, S_Q = 3, S_E = 9, S_S = 15 };
constexpr float SC_U = 1.f / 32.f, SC_S = 1.f / 2048.f;

struct D32 {
    Fld<float> U, V, W;
    RcpT<float> rc;
    float *q;                // canonical arrays, n apart
    float *uf, *vf, *wf;     // 216 Uf, Vf, Wf on canonical elements, rows 1..nyg (V: ny): [k][row][nxp]
    float4 *part;
    long n;
    int nx, ny, nz, nyg, nxp, nym, nzp, nseg, kc_len, nkc;
};

template <int LS>
struct Seg2 {
    int l, s, j, i0, i;  // lane in the segment, segment, row, first column, the lane's first column
    bool act;            // the segment exists
    __device__ __forceinline__ Seg2(int nrows, int j0, int nseg) {
        constexpr int SPW = 32 / LS;
        const long tot = (long)nrows * nseg;
        long g = ((long)blockIdx.x * (D32_T / 32) + (threadIdx.x >> 5)) * SPW + (threadIdx.x & 31) / LS;
        act = g < tot;
        g = act ? g : tot - 1;
        l = threadIdx.x & (LS - 1);
        s = (int)(g / nrows);  // rows fastest: the warps of a block share their rows' neighbours
        j = j0 + (int)(g % nrows);
        i0 = 2 + s * 2 * LS;
        i = i0 + 2 * l;
    }
};

// |S| of two cells from the diagonal components and t = 8 x the mixed ones
__device__ __forceinline__ float2 s_mag(float2 d0, float2 d1, float2 d2, float2 t12, float2 t13, float2 t23) {
    const float2 a = fma2(d2, d2, fma2(d1, d1, mul2(d0, d0))), b = fma2(t23, t23, fma2(t13, t13, mul2(t12, t12)));
    const float2 x = fma2(b, sp(1.f / 32.f), a), y = add2(x, x);
    return f2(sqrtf(y.x), sqrtf(y.y));
}

// strain rates of two cells in the march: what plane p of the velocities
// gives, and the terms that wait for plane p+1
struct Strain {
    float2 u0, um, v1, va, w0, x, y;     // plane p-1: velocities; x and y differences of W over their spacings
    float2 t12, p13, p23, d0, d1, d2;    // the cell at p-1, t13 and t23 without their upper z part
    float2 du, dv;                       // z differences of U and V through the face below p
};

// columns i-1, i, i+1, i+2 of one row as two pairs
struct Quad {
    float2 p, q;
    __device__ __forceinline__ float2 c() const { return f2(p.y, q.x); }  // columns i, i+1
};

struct SGeo {
    float2 rx, rx0, rx1;
    float ry, ry0, ry1;
};

// Plane p: U (rows j-1, j, j+1), V (j-1, j), W (j-1, j, j+1; at the
// neighbours in x only row j).  strain_z first, with the cell at p-1 still
// in s; then strain_plane (store: p is a cell's plane).
__device__ __forceinline__ void strain_z(Strain &s, float2 u0, float2 um, float2 v1, float2 va, float dzr) {
    s.du = mul2(add2(sub2(u0, s.u0), sub2(um, s.um)), sp(dzr));
    s.dv = mul2(add2(sub2(v1, s.v1), sub2(va, s.va)), sp(dzr));
}
__device__ __forceinline__ void strain_plane(Strain &s, const SGeo &g, const Quad &ua, const Quad &u, const Quad &uc,
                                             const Quad &va, const Quad &v, float2 wa, const Quad &w, float2 wc,
                                             float dzw, bool store) {
    const float2 u0 = u.c(), v1 = v.c(), w0 = w.c(), v0a = va.c();
    const float2 x = fma2(sub2(w0, w.p), g.rx0, mul2(sub2(w.q, w0), g.rx1)),
                 y = fma2(sub2(w0, wa), sp(g.ry0), mul2(sub2(wc, w0), sp(g.ry1)));
    if (store) {
        const float2 up = add2(sub2(uc.c(), u0), sub2(uc.p, u.p)), lo = add2(sub2(u0, ua.c()), sub2(u.p, ua.p));
        const float2 vr = add2(sub2(v.q, v1), sub2(va.q, v0a)), vl = add2(sub2(v1, v.p), sub2(v0a, va.p));
        s.t12 = fma2(vl, g.rx0, fma2(vr, g.rx1, fma2(lo, sp(g.ry0), mul2(up, sp(g.ry1)))));
        s.p13 = add2(add2(x, s.x), s.du);
        s.p23 = add2(add2(y, s.y), s.dv);
        s.d0 = mul2(sub2(u0, u.p), g.rx);
        s.d1 = mul2(sub2(v1, v0a), sp(g.ry));
        s.d2 = mul2(sub2(w0, s.w0), sp(dzw));
    }
    s.u0 = u0;
    s.um = u.p;
    s.v1 = v1;
    s.va = v0a;
    s.w0 = w0;
    s.x = x;
    s.y = y;
}

template <int LS>
__global__ void __launch_bounds__(D32_T, 4) k_dsm32_q(const __grid_constant__ D32 a) {
    // rows 1..nyg, then the two one-sided rows of the filtered velocities
    const Seg2<LS> sg(a.nyg + 2, 1, a.nseg);
    const int ny = a.ny, nyg = a.nyg, nxp = a.nxp;
    const int ext = sg.j - nyg;  // 1, 2: the one-sided rows of j = 2 and nyg-1
    const int j = ext <= 0 ? sg.j : (ext == 1 ? 2 : nyg - 1);
    const int kb = 2 + blockIdx.y * a.kc_len, ke = min(kb + a.kc_len - 1, a.nz - 1);
    const int i = min(sg.i, nxp);  // lanes past the last pair repeat it
    const bool cell = ext <= 0 && j >= 2 && j <= nyg - 1;
    const bool own = sg.act && sg.i <= nxp, ownq = own && cell;
    // rows: the neighbours of j, reflected at the ends of the arrays (of the
    // interior for the one-sided rows); for cells they are j-1 and j+1.  V
    // has ny rows; for the one-sided rows its three rows from the wall in
    int ja = j - 1, jc = j + 1, jv = min(j, ny);
    if (j == 1 || ext == 1) ja = j + 1;
    if (j == nyg || ext == 2) jc = j - 1;
    int jva = jv == 1 ? 2 : jv - 1, jvc = jv == ny ? ny - 1 : jv + 1;
    if (ext == 1) { jva = 1; jv = 2; jvc = 3; }
    if (ext == 2) { jva = ny; jv = ny - 1; jvc = ny - 2; }
    const int uo = a.U.idx(i - 1, j, 1), uoa = a.U.idx(i - 1, ja, 1), uoc = a.U.idx(i - 1, jc, 1);
    const int vo = a.V.idx(i - 1, jv, 1), voa = a.V.idx(i - 1, jva, 1), voc = a.V.idx(i - 1, jvc, 1);
    const int wo = a.W.idx(i - 1, j, 1), woa = a.W.idx(i - 1, ja, 1), woc = a.W.idx(i - 1, jc, 1);
    const int jg = min(max(j, 2), nyg - 1);
    SGeo g;
    g.rx = f2(a.rc.dx[i], a.rc.dx[i + 1]);
    g.rx0 = f2(a.rc.dxg[i], a.rc.dxg[i + 1]);
    g.rx1 = f2(a.rc.dxg[i + 1], a.rc.dxg[i + 2]);
    g.ry = a.rc.dy[jg];
    g.ry0 = a.rc.dyg[jg];
    g.ry1 = a.rc.dyg[jg + 1];
    const bool anyc = __any_sync(FULLM, cell);
    Strain s = {};
    float2 h0[3], h1[3], u2o = sp(0.f), v2o = sp(0.f), w2o = sp(0.f);
#pragma unroll
    for (int f = 0; f < 3; f++) h0[f] = h1[f] = sp(0.f);
    const int plane = nxp * a.nym, fpu = nxp * nyg, fpv = nxp * ny;
    float *qp = a.q + (i - 2) + (long)nxp * (jg - 2) + (long)plane * (kb - 2);
    float *uf, *vf, *wf;
    int su = fpu, sv = fpv;  // their plane strides
    if (ext <= 0) {
        uf = a.uf + (i - 2) + (long)nxp * (j - 1) + (long)fpu * (kb - 2);
        vf = a.vf + (i - 2) + (long)nxp * (jv - 1) + (long)fpv * (kb - 2);
        wf = a.wf + (i - 2) + (long)nxp * (j - 1) + (long)fpu * (kb - 2);
    } else {
        su = sv = 2 * nxp;
        uf = a.q + S_E * a.n + (i - 2) + (long)nxp * (ext - 1) + (long)su * (kb - 2);
        vf = uf + a.n;
        wf = vf + a.n;
    }
    for (int p = kb - 1; p <= ke + 1; p++) {
        const float *U = a.U.p + (long)a.U.sz * (p - 1), *V = a.V.p + (long)a.V.sz * (p - 1),
                    *Wp = a.W.p + (long)a.W.sz * (p - 1);
        // U: columns i-1.. start at an even offset of rows of even length
        auto ldu = [&](int o) {
            Quad r;
            r.p = *(const float2 *)(U + o);
            r.q = *(const float2 *)(U + o + 2);
            return r;
        };
        auto ld = [](const float *F, int o) {
            Quad r;
            r.p = f2(F[o], F[o + 1]);
            r.q = f2(F[o + 2], F[o + 3]);
            return r;
        };
        const Quad ua = ldu(uoa), u = ldu(uo), uc = ldu(uoc);
        Quad va = ld(V, voa), v = ld(V, vo), vc = ld(V, voc);
        if (ext > 0) {  // the centre velocities of rows j and its inner neighbour
            v.p = add2(v.p, va.p);
            v.q = add2(v.q, va.q);
            const Quad r1 = ld(V, vo);
            va.p = vc.p = add2(r1.p, vc.p);
            va.q = vc.q = add2(r1.q, vc.q);
        }
        const Quad wa = ld(Wp, woa), w = ld(Wp, wo), wc = ld(Wp, woc);
        // filtered velocities: y, x, then z from the two planes below
        auto fxy = [](const Quad &a, const Quad &b, const Quad &c) {
            const float2 P = w141(a.p, b.p, c.p), Q = w141(a.q, b.q, c.q);
            return fma2(sp(4.f), f2(P.y, Q.x), add2(P, Q));
        };
        const float2 fx[3] = {fxy(ua, u, uc), fxy(va, v, vc), fxy(wa, w, wc)};
        float2 fo[3];
#pragma unroll
        for (int f = 0; f < 3; f++) {
            fo[f] = w141(h0[f], h1[f], fx[f]);
            h0[f] = h1[f];
            h1[f] = fx[f];
        }
        if (p >= kb + 1) {
            if (own) {
                *(float2 *)uf = fo[0];
                if (j <= ny) *(float2 *)vf = fo[1];
                *(float2 *)wf = fo[2];
            }
            uf += su;
            vf += sv;
            wf += su;
        }
        if (anyc) {
            if (p >= kb) {
                strain_z(s, u.c(), u.p, v.c(), va.c(), a.rc.dzg[p]);
                if (p >= kb + 1) {  // the cell at p-1 is complete
                    const float2 t13 = add2(s.p13, s.du), t23 = add2(s.p23, s.dv);
                    const float2 S = s_mag(s.d0, s.d1, s.d2, s.t12, t13, t23), Ss = mul2(S, sp(SC_S));
                    if (ownq) {
                        const long n = a.n;
                        *(float2 *)(qp + S_U2 * n) = u2o;
                        *(float2 *)(qp + S_V2 * n) = v2o;
                        *(float2 *)(qp + S_W2 * n) = w2o;
                        *(float2 *)(qp + (S_Q + 0) * n) = mul2(Ss, s.d0);
                        *(float2 *)(qp + (S_Q + 1) * n) = mul2(Ss, s.d1);
                        *(float2 *)(qp + (S_Q + 2) * n) = mul2(Ss, s.d2);
                        *(float2 *)(qp + (S_Q + 3) * n) = mul2(Ss, s.t12);
                        *(float2 *)(qp + (S_Q + 4) * n) = mul2(Ss, t13);
                        *(float2 *)(qp + (S_Q + 5) * n) = mul2(Ss, t23);
                        *(float2 *)(qp + S_S * n) = S;
                    }
                    qp += plane;
                }
                u2o = mul2(add2(u.c(), u.p), sp(SC_U));
                v2o = mul2(add2(v.c(), va.c()), sp(SC_U));
                w2o = mul2(add2(w.c(), s.w0), sp(SC_U));
            }
            const bool in = p >= kb && p <= ke;
            strain_plane(s, g, ua, u, uc, va, v, wa.c(), w, wc.c(), in ? a.rc.dz[p] : 0.f, in);
        }
    }
}

// quantity q of the 12 filtered ones: u_a u_b (q < 6) or |S| S_ij
__device__ __forceinline__ constexpr int pa_of(int q) { return q < 3 ? q : (q == 5 ? 1 : 0); }
__device__ __forceinline__ constexpr int pb_of(int q) { return q < 3 ? q : (q == 3 ? 1 : 2); }

template <int LS>
__global__ void __launch_bounds__(D32_T, 3) k_dsm32_lm(const __grid_constant__ D32 a) {
    constexpr int NQ = 12, NR = (2 * NQ + LS - 1) / LS;  // edge values: rounds of LS lanes
    const Seg2<LS> sg(a.nym, 2, a.nseg);
    const int nyg = a.nyg, nxp = a.nxp, nzp = a.nzp, j = sg.j, l = sg.l;
    const int kb = 2 + blockIdx.y * a.kc_len, ke = min(kb + a.kc_len - 1, a.nz - 1);
    const bool own = sg.act && sg.i <= nxp;
    // 0-based canonical columns: the lane's pair (past the last one: the
    // first, its right neighbour through the wrap) and its neighbours
    const int c0 = sg.i <= nxp ? sg.i - 2 : 0, cm = c0 == 0 ? nxp - 1 : c0 - 1, cp = c0 + 2 == nxp ? 0 : c0 + 2;
    const int cL = sg.i0 == 2 ? nxp - 1 : sg.i0 - 3, cR = sg.i0 - 2 + 2 * LS >= nxp ? 0 : sg.i0 - 2 + 2 * LS;
    // rows j-1, j, j+1 (reflected at rows 2 and nyg-1)
    const int ja = j == 2 ? 3 : j - 1, jc = j == nyg - 1 ? nyg - 2 : j + 1;
    const int r1 = nxp * (j - 2), ra = nxp * (ja - 2), rcr = nxp * (jc - 2);
    const long plane = (long)nxp * a.nym, n = a.n;
    // edge lanes: value id = r LS + l is quantity id % 12 at the column left
    // (id < 12) or right of the segment
    long eA[NR], eB[NR];  // eB < 0: not a product
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int id = min(r * LS + l, 2 * NQ - 1), q = id % NQ, c = id < NQ ? cL : cR;
        eA[r] = (q < 6 ? pa_of(q) : S_Q + q - 6) * n + c;
        eB[r] = q < 6 ? pb_of(q) * n + c : -1;
    }
    const int fpu = nxp * nyg, fpv = nxp * a.ny, fr = nxp * (j - 1);
    const int ig = min(sg.i, nxp);
    SGeo g;
    g.rx = f2(a.rc.dx[ig], a.rc.dx[ig + 1]);
    g.rx0 = f2(a.rc.dxg[ig], a.rc.dxg[ig + 1]);
    g.rx1 = f2(a.rc.dxg[ig + 1], a.rc.dxg[ig + 2]);
    g.ry = a.rc.dy[j];
    g.ry0 = a.rc.dyg[j];
    g.ry1 = a.rc.dyg[j + 1];
    const bool wrow = j == 2 || j == nyg - 1;
    const int fe = j == 2 ? 0 : nxp;  // its one-sided row
    float2 h0[NQ], h1[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) h0[q] = h1[q] = sp(0.f);
    Strain s = {};
    float2 fw = sp(0.f);
    float2 lmd = sp(0.f), lmo = sp(0.f), mmd = sp(0.f), mmo = sp(0.f);
    for (int r = kb - 1; r <= ke + 1; r++) {
        const int k = wrapn(r, nzp) - 2;
        const bool out = r >= kb + 1;  // plane r-1 is complete
        // 4 |Sf| Sf_ij (scaled like the filtered |S| S_ij) and hat(u_i) at plane r-1, from plane r
        float2 m[6], fu, fv, fwk;
        {
            const float *U = a.uf + fpu * k + fr, *V = a.vf + fpv * k + fr, *Wp = a.wf + fpu * k + fr;
            auto ldq = [&](const float *F) {  // columns i-1 .. i+2
                Quad t;
                const float2 c = *(const float2 *)(F + c0);
                t.p = f2(F[cm], c.x);
                t.q = f2(c.y, F[cp]);
                return t;
            };
            auto ldp = [&](const float *F) {  // columns i-1, i, i+1
                Quad t;
                const float2 c = *(const float2 *)(F + c0);
                t.p = f2(F[cm], c.x);
                t.q = f2(c.y, 0.f);
                return t;
            };
            const Quad ua = ldp(U - nxp), u = ldp(U), uc = ldp(U + nxp);
            const Quad va = ldq(V - nxp), v = ldq(V), w = ldq(Wp);
            const float2 wa = *(const float2 *)(Wp - nxp + c0), wc = *(const float2 *)(Wp + nxp + c0);
            if (r >= kb) strain_z(s, u.c(), u.p, v.c(), va.c(), a.rc.dzg[r]);
            if (out) {
                const float2 t13 = add2(s.p13, s.du), t23 = add2(s.p23, s.dv);
                const float2 c = mul2(s_mag(s.d0, s.d1, s.d2, s.t12, t13, t23), sp(SC_S / 54.f));
                m[0] = mul2(c, s.d0);
                m[1] = mul2(c, s.d1);
                m[2] = mul2(c, s.d2);
                m[3] = mul2(c, s.t12);
                m[4] = mul2(c, t13);
                m[5] = mul2(c, t23);
                fu = add2(s.u0, s.um);
                fv = add2(s.v1, s.va);
                fwk = fw;
                if (wrow) {
                    const int k1 = wrapn(r - 1, nzp) - 2, k0 = wrapn(r - 2, nzp) - 2;
                    const float *E = a.q + S_E * n + fe + 2 * nxp * k1;
                    const float2 e = *(const float2 *)(E + c0);
                    fu = add2(e, f2(E[cm], e.x));
                    fv = *(const float2 *)(E + n + c0);
                    fwk = add2(*(const float2 *)(E + 2 * n + c0),
                               *(const float2 *)(a.q + (S_E + 2) * n + fe + 2 * nxp * k0 + c0));
                }
            }
            fw = add2(w.c(), s.w0);
            const bool in = r >= kb && r <= ke;
            strain_plane(s, g, ua, u, uc, va, v, wa, w, wc, in ? a.rc.dz[r] : 0.f, in);
        }
        const float *Q = a.q + (int)plane * k;
        // y filter at the two columns next to the segment
        float ev[NR];
#pragma unroll
        for (int t = 0; t < NR; t++) {
            const float *A = Q + eA[t];
            float x0 = A[ra], x1 = A[r1], x2 = A[rcr];
            if (eB[t] >= 0) {
                const float *B = Q + eB[t];
                x0 *= B[ra];
                x1 *= B[r1];
                x2 *= B[rcr];
            }
            ev[t] = w141(x0, x1, x2);
        }
        // the filter of quantity q from its y-filtered plane r: x, then z; returns plane r-1's
        auto filt = [&](int q, float2 y) {
            const float eL = __shfl_sync(FULLM, ev[q / LS], q % LS, LS),
                        eR = __shfl_sync(FULLM, ev[(NQ + q) / LS], (NQ + q) % LS, LS);
            const float yl = __shfl_up_sync(FULLM, y.y, 1, LS), yr = __shfl_down_sync(FULLM, y.x, 1, LS);
            const float l0 = l == 0 ? eL : yl, q0 = l == LS - 1 ? eR : yr;
            const float2 x = fma2(sp(4.f), y, add2(f2(l0, y.x), f2(y.y, q0)));
            const float2 H = w141(h0[q], h1[q], x);
            h0[q] = h1[q];
            h1[q] = x;
            return H;
        };
        float2 L[6];
        {
            float2 cu[3][3];
#pragma unroll
            for (int f = 0; f < 3; f++) {
                const float *C = Q + f * n + c0;
                cu[f][0] = *(const float2 *)(C + ra);
                cu[f][1] = *(const float2 *)(C + r1);
                cu[f][2] = *(const float2 *)(C + rcr);
            }
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const int x = pa_of(q), y = pb_of(q);
                L[q] = filt(q, w141(mul2(cu[x][0], cu[y][0]), mul2(cu[x][1], cu[y][1]), mul2(cu[x][2], cu[y][2])));
            }
        }
        if (out) {
            // L_ij times 864 SC_U^2
            const float2 sc = sp(-SC_U * SC_U / 216.f), f[3] = {fu, fv, fwk};
#pragma unroll
            for (int q = 0; q < 6; q++) L[q] = fma2(f[pa_of(q)], mul2(f[pb_of(q)], sc), L[q]);
        }
        const float wz = r - 1 == 2 ? 2.f : 1.f;  // plane 2 stands for its duplicate too
#pragma unroll
        for (int q = 6; q < NQ; q++) {
            const float *C = Q + (S_Q + q - 6) * n + c0;
            const float2 H = filt(q, w141(*(const float2 *)(C + ra), *(const float2 *)(C + r1), *(const float2 *)(C + rcr)));
            if (out) {
                const float2 M = sub2(m[q - 6], H), Mw = mul2(M, sp(wz));
                if (q < 9) {
                    lmd = fma2(L[q - 6], Mw, lmd);
                    mmd = fma2(M, Mw, mmd);
                } else {
                    lmo = fma2(L[q - 6], Mw, lmo);
                    mmo = fma2(M, Mw, mmo);
                }
            }
        }
    }
    // undo the scales; column 2 stands for its duplicate too
    const float wx = sg.i == 2 ? 2.f : 1.f;
    constexpr float SL = 864.f * SC_U * SC_U * 216.f * SC_S, SM = 216.f * 216.f * SC_S * SC_S;
    const float2 lm = fma2(sp(0.25f), lmo, lmd), mm = fma2(sp(1.f / 32.f), mmo, mmd);
    float ah = 0.f, al = 0.f, bh = 0.f, bl = 0.f;
    if (own) {
        two_sum(wx * lm.x, lm.y, ah, al);
        two_sum(wx * mm.x, mm.y, bh, bl);
    }
#pragma unroll
    for (int o = LS / 2; o > 0; o >>= 1) {
        const float a1 = __shfl_down_sync(FULLM, ah, o, LS), a2 = __shfl_down_sync(FULLM, al, o, LS);
        const float b1 = __shfl_down_sync(FULLM, bh, o, LS), b2 = __shfl_down_sync(FULLM, bl, o, LS);
        ff_add2(ah, al, a1, a2);
        ff_add2(bh, bl, b1, b2);
    }
    if (l == 0 && sg.act) {
        // float-float times the inverse scales, the products' rounding recovered
        auto scale = [](float h, float lo, float f, float &oh, float &ol) {
            const float p = h * f, e = fmaf(h, f, -p) + lo * f;
            oh = p;
            ol = e;
        };
        float4 v;
        scale(ah, al, 1.f / SL, v.x, v.y);
        scale(bh, bl, 1.f / SM, v.z, v.w);
        a.part[(long)(j - 2) * (a.nseg * a.nkc) + sg.s * a.nkc + blockIdx.y] = v;
    }
}

// lanes per segment: the width that leaves the fewest idle columns, the
// widest of them
int d32_ls(int nxp) {
    int best = 32;
    for (int ls : {16, 8})
        if (cdiv(nxp, 2 * ls) * ls < cdiv(nxp, 2 * best) * best) best = ls;
    return best;
}

}  // namespace

// z-chunk length and plane-partial slots per row: the count that minimises
// (waves of resident blocks of the filter kernel) x (planes per chunk + 1.5
// for the halo planes)
void dsm32_plan(int nxp, int nym, int nzp, int sms, int *kc, size_t *nchunk) {
    const int ls = d32_ls(nxp), nseg = cdiv(nxp, 2 * ls);
    int per = 1;
    if (ls == 32) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_dsm32_lm<32>, D32_T, 0);
    else if (ls == 16) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_dsm32_lm<16>, D32_T, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_dsm32_lm<8>, D32_T, 0);
    const long blocks = cdiv((long)nseg * nym, (32 / ls) * (D32_T / 32)), res = (long)std::max(per, 1) * sms;
    double best_cost = 1e300;
    int best = 1;
    for (int n = 1; n <= nzp; n++) {
        const int len = cdiv(nzp, n);
        const double cost = (double)cdiv(blocks * cdiv(nzp, len), res) * (len + 1.5);
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = len;
        }
    }
    *kc = best;
    *nchunk = (size_t)nseg * cdiv(nzp, best);
}

int dsm32_slots(int nxp, int nzp, int kc) { return cdiv(nxp, 2 * d32_ls(nxp)) * cdiv(nzp, kc); }

// |S| into the canonical scratch, the plane partials into dsm_part
int launch_dsm32(cf_ctx *ctx, int b, int *nchunk) {
    D32 a;
    a.U = make_fld<float>(ctx->U[b], ctx->nx, ctx->nyg);
    a.V = make_fld<float>(ctx->V[b], ctx->nxg, ctx->ny);
    a.W = make_fld<float>(ctx->W[b], ctx->nxg, ctx->nyg);
    a.rc = rcp_of<float>(ctx);
    a.q = (float *)ctx->dsm_q;
    a.uf = (float *)ctx->Uf;
    a.vf = (float *)ctx->Vf;
    a.wf = (float *)ctx->Wf;
    a.part = (float4 *)ctx->dsm_part;
    a.n = (long)ctx->nCan;
    a.nx = ctx->nx; a.ny = ctx->ny; a.nz = ctx->nz; a.nyg = ctx->nyg;
    a.nxp = ctx->nxp; a.nym = ctx->nym; a.nzp = ctx->nzp;
    const int ls = d32_ls(ctx->nxp);
    a.nseg = cdiv(ctx->nxp, 2 * ls);
    a.kc_len = ctx->dsm_kc;
    a.nkc = cdiv(ctx->nzp, ctx->dsm_kc);
    *nchunk = a.nseg * a.nkc;
    if ((size_t)*nchunk > ctx->dsm_part_nch) return cf_fail(ctx, CF_ERR_INVALID, "plane-partial slots");
    const int per = (32 / ls) * (D32_T / 32);
    const dim3 gq(cdiv((long)a.nseg * (ctx->nyg + 2), per), a.nkc), gl(cdiv((long)a.nseg * ctx->nym, per), a.nkc);
    if (ls == 32) k_dsm32_q<32><<<gq, D32_T, 0, ctx->st>>>(a);
    else if (ls == 16) k_dsm32_q<16><<<gq, D32_T, 0, ctx->st>>>(a);
    else k_dsm32_q<8><<<gq, D32_T, 0, ctx->st>>>(a);
    count_launch(ctx, "k_dsm32_q");
    if (ls == 32) k_dsm32_lm<32><<<gl, D32_T, 0, ctx->st>>>(a);
    else if (ls == 16) k_dsm32_lm<16><<<gl, D32_T, 0, ctx->st>>>(a);
    else k_dsm32_lm<8><<<gl, D32_T, 0, ctx->st>>>(a);
    count_launch(ctx, "k_dsm32_lm");
    CF_CUDA(cudaGetLastError());
    return 0;
}
