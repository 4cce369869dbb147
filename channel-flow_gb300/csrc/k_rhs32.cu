// k_rhs32.cu -- right-hand sides of u, v and w with the RK update
// (equations.f90:24-498, time_integration.f90:108-145) of the split path
// (FP32), one launch per substep.
//
// Per cell 64 bytes go through memory (velocities, u^n in two words, the
// stored right-hand side, |S|, the new state), 45 us at 192 x 128 x 192 cells
// and the measured 6.75 TB/s.  A kernel of one cell per thread, with every
// flux of a cell formed by its own thread, issued 470 instructions a cell and
// took 96 us there (in a replayed graph, a launch's 5 us included) and 119 us
// at 256 x 96 x 256; this one 300 per two cells, 75 and 96 us.
//
// A block of 128 threads owns a tile of 2 LS columns x R = 128 / LS rows and
// marches along z over a chunk of planes.  A lane holds two adjacent columns
// and forms their fluxes as packed FP32x2 from columns i-1 .. i+2 of a row
// (two 8-byte reads of shared memory): the fluxes on upper x faces and edges
// of both cells and by itself the one left of the pair, the upper and lower
// ones in y, and the upper ones in z, which are the lower ones of the next
// plane.  The planes of U, V, W and nu_t (or |S|) with one halo cell are
// copied to shared memory asynchronously, three ahead of the lowest one read;
// one barrier a plane.  The body has no branch before the stores (planes
// below the chunk and idle lanes only skip those).  Four blocks of 128
// registers per SM instead of three of 168 spill: 85 and 110 us.
//
// The reference divides the cross-derivative of a viscous flux by another
// spacing where the flux is a cell's upper face than where it is its lower
// one (equations.f90:108-163, 276-331, 435-493; the same on uniform grids),
// so some fluxes have two values.
//
// Scales: normal fluxes times 4, xy and yz edges times 2, xz edges times 4
// (the interpolations' halves left out, exact powers of two), undone in the
// divergence's coefficients.
#include <algorithm>

#include "cf_internal.cuh"
#include "f32x2.cuh"

namespace {

constexpr int R32_T = 128;  // threads per block
constexpr int R32_NB = 4;   // planes in shared memory: k and k+1, two on their way

// nu_t: its field, or held as |S| on canonical cells and the plane
// coefficient C(j): nu_t(i,j,k) = max(-C(jj)|S|(wrap i, jj, wrap k)/2, 0),
// jj = j clamped to the interior, negated on the wall ghost rows for
// Dirichlet_nu_t (subgrid.f90:521-536).
struct Nut32 {
    Fld<float> nt;
    const float *S, *C;  // C: 1-based rows
    int nxp, nym, nzp, dirichlet;
};

struct R32 {
    Fld<float> U, V, W;
    Nut32 ns;
    Trio<float> out, F1, Uo, Uolo, Unlo;
    const float *w0, *w1;
    RcpT<float> rc;
    const DevScal *ds;
    float nu, Om, ca, cb;
    int rot, nxp, nyg, ny, klim, kc_len, ls, nbx, nby, nbz;
};

template <int LS>
using RTile = HaloTile<LS, R32_T>;
constexpr int R32_NPMAX = 396;  // largest of RTile<32>, <16>, <8>::NP

// The RK update of a point for substep S (time_integration.f90:108-145), u^n =
// uo + lo: S = 1 stores the right-hand side as F1; substep 3 stores the new
// state as hi + lo, the others the rounded sum.
template <int S>
__device__ __forceinline__ void rk_put(float r, float inc, float uo, float lo, int o, const Fld<float> &out,
                                       const Fld<float> &F1, const Fld<float> &Unlo) {
    if constexpr (S == 1) F1.p[o] = r;
    if constexpr (S == 3) {
        ff_add(uo, lo, inc);
        out.p[o] = uo;
        Unlo.p[o] = lo;
    } else {
        out.p[o] = uo + (lo + inc);
    }
}

// The tile (bx, by, bz) of one channel, substep S.  LAZY: nu_t from |S| and C.
template <int LS, int S, bool LAZY>
__device__ __forceinline__ void rhs32_tile(const R32 &a, float (*st)[4][R32_NPMAX], int bx, int by, int bz) {
    typedef RTile<LS> TL;
    constexpr int SX = TL::SX, NP = TL::NP, NL = TL::NL, R = TL::R, NB = R32_NB;
    static_assert(NP <= R32_NPMAX, "tile");
    const int ny = a.ny, nyg = a.nyg, nxp = a.nxp;
    const int l = threadIdx.x % LS, ty = TL::row();
    const int i0 = 2 + bx * TL::WS, i = min(i0 + 2 * l, nxp), j0 = 2 + by * R, j = min(j0 + ty, nyg - 1);
    const int kb = 2 + bz * a.kc_len, ke = min(kb + a.kc_len - 1, a.klim);
    const bool own = i0 + 2 * l <= nxp && j0 + ty <= nyg - 1, ownv = own && j <= ny - 1;
    const Nut32 &ns = a.ns;
    // this thread's elements of a plane: the same tile position in every field
    int eU[NL], eV[NL], eW[NL], eN[NL];
#pragma unroll
    for (int q = 0; q < NL; q++) {
        const int e = threadIdx.x + q * R32_T, sy = e / SX, sx = e - sy * SX;
        // past the last neighbours: not read
        const int c = min(i0 - 1 + sx, nxp + 2), r = min(j0 - 1 + sy, nyg), rv = min(r, ny);
        eU[q] = a.U.idx(c, r, 1);
        eV[q] = a.V.idx(c, rv, 1);
        eW[q] = a.W.idx(c, r, 1);
        eN[q] = LAZY ? wrapn(c, ns.nxp) - 2 + ns.nxp * (min(max(r, 2), nyg - 1) - 2) : ns.nt.idx(c, r, 1);
    }
    auto fetch = [&](int k, int b) {
        const float *U = a.U.p + (long)a.U.sz * (k - 1), *V = a.V.p + (long)a.V.sz * (k - 1),
                    *Wp = a.W.p + (long)a.W.sz * (k - 1),
                    *N = LAZY ? ns.S + (long)ns.nxp * ns.nym * (wrapn(k, ns.nzp) - 2) : ns.nt.p + (long)ns.nt.sz * (k - 1);
#pragma unroll
        for (int q = 0; q < NL; q++) {
            const int e = threadIdx.x + q * R32_T;
            if (NP % R32_T == 0 || e < NP) {
                copy_async<4>(&st[b][0][e], U + eU[q]);
                copy_async<4>(&st[b][1][e], V + eV[q]);
                copy_async<4>(&st[b][2][e], Wp + eW[q]);
                copy_async<4>(&st[b][3][e], N + eN[q]);
            }
        }
        copy_commit();
    };
#pragma unroll
    for (int d = 0; d < NB - 1; d++) fetch(kb - 1 + d, d);
    const float nu = a.nu, nu2 = nu + nu, nu4 = nu2 + nu2;
    const float w0 = a.w0[min(j, ny)], w1 = a.w1[min(j, ny)], w0m = a.w0[j - 1], w1m = a.w1[j - 1];
    const float ryg0 = a.rc.dyg[j], ryg1 = a.rc.dyg[j + 1], ry = a.rc.dy[j], ry1 = j + 1 <= ny ? a.rc.dy[j + 1] : 0.f;
    const float2 rx = f2(a.rc.dx[i], a.rc.dx[i + 1]), rx1 = f2(rx.y, a.rc.dx[i + 2]);
    const float2 rxg0 = f2(a.rc.dxg[i], a.rc.dxg[i + 1]), rxg1 = f2(rxg0.y, a.rc.dxg[i + 2]);
    const float dt = ds_dt<float>(a.ds), dPdx = ds_dpdx<float>(a.ds), dPdz = ds_dpdz<float>(a.ds);
    // |S| to nu_t: coefficients of rows j-1, j, j+1 and the ghost rows' sign
    float ca = 0.f, cb = 0.f, cc = 0.f, ga = 1.f, gc = 1.f;
    if constexpr (LAZY) {
        ca = -0.5f * ns.C[max(j - 1, 2)];
        cb = -0.5f * ns.C[j];
        cc = -0.5f * ns.C[min(j + 1, nyg - 1)];
        if (ns.dirichlet) {
            if (j == 2) ga = -1.f;
            if (j == nyg - 1) gc = -1.f;
        }
    }
    auto nut = [](Quad v, float c, float g) {
        if constexpr (LAZY) {
            v.p = mul2(v.p, sp(c));
            v.q = mul2(v.q, sp(c));
            v.p = mul2(f2(fmaxf(v.p.x, 0.f), fmaxf(v.p.y, 0.f)), sp(g));
            v.q = mul2(f2(fmaxf(v.q.x, 0.f), fmaxf(v.q.y, 0.f)), sp(g));
        }
        return v;
    };
    const int o1 = (ty + 1) * SX + 2 * l, oa = o1 - SX, oc = o1 + SX;
    int iu = a.out.u.idx(i, j, kb - 1), iv = a.out.v.idx(i, min(j, ny), kb - 1), iw = a.out.w.idx(i, j, kb - 1);
    copy_wait<NB - 2>();
    __syncthreads();  // plane kb-1 is in
    Quad na = nut(quad(st[0][3] + oa), ca, ga), nb = nut(quad(st[0][3] + o1), cb, 1.f), nc = nut(quad(st[0][3] + oc), cc, gc);
    float2 zu_l = sp(0.f), zv_l = sp(0.f), zw_l = sp(0.f);  // fluxes through the z faces below plane k
    float dz0 = kb - 1 >= 2 ? a.rc.dz[kb - 1] : 0.f, dz1 = a.rc.dz[kb], dzg1 = a.rc.dzg[kb];
    for (int k = kb - 1, b = 0; k <= ke; k++, b = (b + 1) & (NB - 1)) {
        // operands of the update, in flight during the stencils
        auto two = [](const Fld<float> &F, int o) { return f2(F.p[o], F.p[o + 1]); };
        const float2 uo = two(a.Uo.u, iu), vo = two(a.Uo.v, iv), wo = two(a.Uo.w, iw);
        const float2 ul = two(a.Uolo.u, iu), vl = two(a.Uolo.v, iv), wl = two(a.Uolo.w, iw);
        float2 fu = sp(0.f), fv = sp(0.f), fw = sp(0.f);
        if constexpr (S > 1) {
            fu = two(a.F1.u, iu);
            fv = two(a.F1.v, iv);
            fw = two(a.F1.w, iw);
        }
        copy_wait<NB - 3>();
        __syncthreads();  // plane k+1 is in; the buffer of k-1 is no longer read
        if (k + NB - 1 <= ke + 1) fetch(k + NB - 1, (b + NB - 1) & (NB - 1));
        else copy_commit();
        const float z1 = dz0, z2 = dz1, z3 = dzg1;  // of planes k and k+1
        dz0 = dz1;
        dz1 = a.rc.dz[min(k + 2, ke + 1)];
        dzg1 = a.rc.dzg[min(k + 2, ke + 1)];
        const float(*T)[R32_NPMAX] = st[b], (*Tn)[R32_NPMAX] = st[(b + 1) & (NB - 1)];
        const Quad nna = nut(quad(Tn[3] + oa), ca, ga), nnb = nut(quad(Tn[3] + o1), cb, 1.f), nnc = nut(quad(Tn[3] + oc), cc, gc);
        const Quad ua = quad(T[0] + oa), ub = quad(T[0] + o1), uc = quad(T[0] + oc), un = quad(Tn[0] + o1);
        const Quad va = quad(T[1] + oa), vb = quad(T[1] + o1), vc = quad(T[1] + oc), vna = quad(Tn[1] + oa), vnb = quad(Tn[1] + o1);
        const Quad wa = quad(T[2] + oa), wb = quad(T[2] + o1), wc = quad(T[2] + oc), wn = quad(Tn[2] + o1);
        const float2 u0 = ub.c(), v0 = vb.c(), w_0 = wb.c(), u1 = un.c(), v1 = vnb.c(), w1c = wc.c(), wac = wa.c();
        const float2 nbc = nb.c(), nnbc = nnb.c();
        const float2 sb = add2(nbc, nb.q), sn = add2(nnbc, nnb.q);     // nu_t of both cells of an x face
        const float2 zb = add2(nbc, nnbc);                             // of a z face
        auto flux = [](float2 ne, float2 g, float2 A) { return fma2(ne, g, mul2(A, sp(-1.f))); };
        // difference of two products in x: a b of the pair less those one cell to
        // the left (aL bL, a.x b.x); in y: a b + c d with c negated.  One of the
        // two products is not rounded.
        auto dx = [](float2 a, float2 b, float aL, float bL) {
            return f2(fmaf(a.x, b.x, -(aL * bL)), fmaf(a.y, b.y, -(a.x * b.x)));
        };
        auto dy = [](float2 a, float2 b, float2 c, float2 d) { return fma2(a, b, mul2(c, d)); };
        const float2 uac = ua.c(), vac = va.c();
        // minus the quantities of the edges and faces below (nu_t, velocities)
        const float2 zna = add2(na.c(), nna.c());
        float2 ru, rv, rw;
        {  // xy edge (i+1/2, j+1/2): u through the y face, v through the x face
            const float2 ne = fma2(sp(w1), add2(nc.c(), nc.q), fma2(sp(w0), sb, sp(nu2)));
            const float2 ucc = uc.c(), P = fma2(sp(w1), ucc, mul2(sp(w0), u0)), Q = add2(v0, vb.q);
            const float2 gr = mul2(sub2(ucc, u0), sp(ryg1)), dV = sub2(vb.q, v0), gx = fma2(dV, rxg1, gr);
            // v through the face left of the pair
            const float neL = fmaf(w1, nc.p.x + nc.p.y, fmaf(w0, nb.p.x + nb.p.y, nu2));
            const float PL = fmaf(w1, uc.p.x, w0 * ub.p.x), QL = vb.p.x + vb.p.y;
            const float gL = fmaf(vb.p.y - vb.p.x, rxg0.x, (uc.p.x - ub.p.x) * ryg1);
            rv = mul2(mul2(rx, sp(0.5f)), sub2(dx(ne, gx, neL, gL), dx(P, Q, PL, QL)));
            // (j-1/2): u through the y face below
            const float2 nea = fma2(sp(-w1m), sb, fma2(sp(-w0m), add2(na.c(), na.q), sp(-nu2)));
            const float2 Pa = fma2(sp(-w1m), u0, mul2(sp(-w0m), uac)), Qa = add2(vac, va.q);
            const float2 gy = fma2(dV, rx1, gr), ga = fma2(sub2(va.q, vac), rx, mul2(sub2(u0, uac), sp(ryg0)));
            ru = mul2(sub2(dy(ne, gy, nea, ga), dy(P, Q, Pa, Qa)), sp(0.5f * ry));
            // v through the centres of rows j+1 and j
            const float2 vcc = vc.c(), s1 = add2(v0, vcc), s0 = add2(vac, v0);
            const float2 m1 = mul2(add2(nc.c(), sp(nu)), sp(8.f * ry1)), m0 = mul2(add2(nbc, sp(nu)), sp(-8.f * ry));
            rv = fma2(sub2(dy(m1, sub2(vcc, v0), m0, sub2(v0, vac)), dy(s1, s1, mul2(s0, sp(-1.f)), s0)), sp(0.25f * ryg1), rv);
        }
        {  // u through the centres of columns i+1 (both cells') and i
            const float2 s1 = add2(u0, ub.q), m1 = mul2(add2(nb.q, sp(nu)), mul2(rx1, sp(8.f)));
            const float s0 = ub.p.x + ub.p.y, m0 = (nu + nb.p.y) * (8.f * rx.x);
            ru = fma2(mul2(rxg1, sp(0.25f)), sub2(dx(m1, sub2(ub.q, u0), m0, ub.p.y - ub.p.x), dx(s1, s1, s0, s0)), ru);
        }
        float2 zu, zv, zw;
        {  // xz edge (i+1/2, k+1/2): u through the z face, w through the x face
            const float2 ne = add2(sp(nu4), add2(sb, sn)), P = add2(u0, u1), Q = add2(w_0, wb.q), A = mul2(P, Q);
            const float2 dU = sub2(u1, u0), dW = sub2(wb.q, w_0), gz = mul2(dU, sp(z3)), gx = mul2(dW, rxg1);
            const float2 zup = flux(ne, fma2(dW, rx1, gz), A);
            zu = flux(ne, fma2(dW, rx, gz), A);
            const float2 g = fma2(dU, sp(z2), gx);
            const float neL = nu4 + ((nb.p.x + nb.p.y) + (nnb.p.x + nnb.p.y));
            const float PL = ub.p.x + un.p.x, QL = wb.p.x + wb.p.y;
            const float gL = fmaf(un.p.x - ub.p.x, z1, (wb.p.y - wb.p.x) * rxg0.x);
            const float2 v = f2(fmaf(ne.x, g.x, -(neL * gL)), fmaf(ne.y, g.y, -(ne.x * fmaf(dU.x, z1, gx.x))));
            ru = fma2(sub2(zup, zu_l), sp(0.25f * z1), ru);
            rw = mul2(mul2(rx, sp(0.25f)), sub2(v, dx(P, Q, PL, QL)));
        }
        {  // yz edges (j+1/2, k+1/2) and (j-1/2, k+1/2): v through the z face, w through the y face
            const float2 ne = fma2(sp(w1), add2(nc.c(), nnc.c()), fma2(sp(w0), zb, sp(nu2)));
            const float2 P = add2(v0, v1), Q = fma2(sp(w1), w1c, mul2(sp(w0), w_0));
            const float2 dV = sub2(v1, v0), gW = mul2(sub2(w1c, w_0), sp(ryg1));
            zv = flux(ne, fma2(dV, sp(z3), gW), mul2(P, Q));
            const float2 nea = fma2(sp(-w1m), zb, fma2(sp(-w0m), zna, sp(-nu2)));
            const float2 vnac = vna.c(), Pa = add2(vac, vnac), Qa = fma2(sp(-w1m), w_0, mul2(sp(-w0m), wac));
            const float2 ga = fma2(sub2(vnac, vac), sp(z1), mul2(sub2(w_0, wac), sp(ryg0)));
            rv = fma2(sub2(zv, zv_l), sp(0.5f * z1), rv);
            rw = fma2(sub2(dy(ne, fma2(dV, sp(z2), gW), nea, ga), dy(P, Q, Pa, Qa)), sp(0.5f * ry), rw);
        }
        {  // w through the centre of plane k+1
            const float2 wnc = wn.c(), s = add2(w_0, wnc);
            zw = flux(mul2(add2(nnbc, sp(nu)), sp(8.f * z2)), sub2(wnc, w_0), mul2(s, s));
            rw = fma2(sub2(zw, zw_l), sp(0.25f * z3), rw);
        }
        ru = add2(ru, sp(dPdx));
        rw = add2(rw, sp(dPdz));
        zu_l = zu;
        zv_l = zv;
        zw_l = zw;
        na = nna;
        nb = nnb;
        nc = nnc;
        if (a.rot) {
            // equations.f90:169-177, 334-342
            const float2 h = sp(0.25f), m = sp(2.f * a.Om);
            ru = fma2(m, mul2(h, add2(add2(vac, v0), add2(va.q, vb.q))), ru);
            const float2 q = fma2(sp(w0), add2(ub.p, u0), mul2(sp(w1), add2(uc.p, uc.c())));
            rv = fma2(mul2(m, sp(-0.5f)), q, rv);
        }
        auto inc = [&](float2 r, float2 f) {
            if constexpr (S == 1) return mul2(sp(dt * a.ca), r);
            else return mul2(sp(dt), fma2(sp(a.cb), r, mul2(sp(a.ca), f)));
        };
        const float2 du = inc(ru, fu), dv = inc(rv, fv), dw = inc(rw, fw);
        if (own && k >= kb) {
            rk_put<S>(ru.x, du.x, uo.x, ul.x, iu, a.out.u, a.F1.u, a.Unlo.u);
            rk_put<S>(ru.y, du.y, uo.y, ul.y, iu + 1, a.out.u, a.F1.u, a.Unlo.u);
            rk_put<S>(rw.x, dw.x, wo.x, wl.x, iw, a.out.w, a.F1.w, a.Unlo.w);
            rk_put<S>(rw.y, dw.y, wo.y, wl.y, iw + 1, a.out.w, a.F1.w, a.Unlo.w);
            if (ownv) {
                rk_put<S>(rv.x, dv.x, vo.x, vl.x, iv, a.out.v, a.F1.v, a.Unlo.v);
                rk_put<S>(rv.y, dv.y, vo.y, vl.y, iv + 1, a.out.v, a.F1.v, a.Unlo.v);
            }
        }
        iu += a.out.u.sz;
        iv += a.out.v.sz;
        iw += a.out.w.sz;
    }
}

template <int LS, int S, bool LAZY>
__global__ void __launch_bounds__(R32_T, 3) k_rhs32(const __grid_constant__ R32 a) {
    __shared__ __align__(16) float st[R32_NB][4][R32_NPMAX];
    rhs32_tile<LS, S, LAZY>(a, st, blockIdx.x, blockIdx.y, blockIdx.z);
}

// One launch over the tiles of several channels (an ensemble): member m owns
// blocks first[m] .. first[m+1]-1, in the order of its own launch's grid.
struct R32Batch {
    int n;
    int first[CF_ENS_MAXM + 1];
    R32 a[CF_ENS_MAXM];
};

template <int LS, int S, bool LAZY>
__device__ __noinline__ void rhs32_batch_tile(const R32 &a, float (*st)[4][R32_NPMAX], int b) {
    rhs32_tile<LS, S, LAZY>(a, st, b % a.nbx, (b / a.nbx) % a.nby, b / (a.nbx * a.nby));
}

template <int S>
__global__ void __launch_bounds__(R32_T, 3) k_rhs32_batch(const __grid_constant__ R32Batch B) {
    __shared__ __align__(16) float st[R32_NB][4][R32_NPMAX];
    const int bid = blockIdx.x;
    int m = 0;
    while (m + 1 < B.n && bid >= B.first[m + 1]) m++;
    const R32 &a = B.a[m];
    const int b = bid - B.first[m];
    if (a.ns.S) {
        if (a.ls == 32) rhs32_batch_tile<32, S, true>(a, st, b);
        else if (a.ls == 16) rhs32_batch_tile<16, S, true>(a, st, b);
        else rhs32_batch_tile<8, S, true>(a, st, b);
    } else {
        if (a.ls == 32) rhs32_batch_tile<32, S, false>(a, st, b);
        else if (a.ls == 16) rhs32_batch_tile<16, S, false>(a, st, b);
        else rhs32_batch_tile<8, S, false>(a, st, b);
    }
}

R32 rhs32_args(cf_ctx *ctx, int s, int src, int dst) {
    R32 a;
    auto trio = [&](void *u, void *v, void *w) {
        Trio<float> t;
        t.u = make_fld<float>(u, ctx->nx, ctx->nyg);
        t.v = make_fld<float>(v, ctx->nxg, ctx->ny);
        t.w = make_fld<float>(w, ctx->nxg, ctx->nyg);
        return t;
    };
    const Trio<float> in = trio(ctx->U[src], ctx->V[src], ctx->W[src]);
    a.U = in.u; a.V = in.v; a.W = in.w;
    const int o = ctx->old;
    a.out = trio(ctx->U[dst], ctx->V[dst], ctx->W[dst]);
    a.F1 = trio(ctx->F[0][0], ctx->F[0][1], ctx->F[0][2]);
    a.Uo = trio(ctx->U[o], ctx->V[o], ctx->W[o]);
    a.Uolo = trio(ctx->Ulo[o], ctx->Vlo[o], ctx->Wlo[o]);
    a.Unlo = s == 3 ? trio(ctx->Ulo[dst], ctx->Vlo[dst], ctx->Wlo[dst]) : trio(nullptr, nullptr, nullptr);
    Nut32 &ns = a.ns;
    ns.nt = make_fld<float>(ctx->nut, ctx->nxg, ctx->nyg);
    ns.S = ctx->nut_lazy ? (const float *)ctx->dsm_q + 15 * ctx->nCan : nullptr;  // |S| slot of the canonical scratch
    ns.C = (const float *)(ctx->avg_nu_t + ctx->nyg + 2);
    ns.nxp = ctx->nxp; ns.nym = ctx->nym; ns.nzp = ctx->nzp;
    ns.dirichlet = ctx->prm.Dirichlet_nu_t == 1;
    const GeoT<float> g = geo_of<float>(ctx);
    a.w0 = g.w0; a.w1 = g.w1;
    a.rc = rcp_of<float>(ctx);
    a.ds = ctx->ds;
    a.nu = (float)ctx->prm.nu;
    a.Om = (float)ctx->omega_z;
    a.rot = fabs(ctx->omega_z) > 1e-6 ? 1 : 0;
    const RkCoef rk = rk_coefs();  // weights of F1 (of the right-hand side itself in substep 1) and of the right-hand side
    a.ca = (float)rk.c[s][1];
    a.cb = s == 1 ? 0.f : (float)(s == 2 ? rk.c[2][2] : rk.c[3][3]);
    // canonical cells only (i <= nxp+1, k <= nzp+1): the periodic duplicate
    // column of V, W and plane of U, V are rewritten by the boundary
    // conditions after the projection and read by nothing before them
    a.nxp = ctx->nxp; a.nyg = ctx->nyg; a.ny = ctx->ny;
    a.klim = ctx->nzp + 1;
    const int nkc = std::max(std::max(ctx->rhs_nkc, 1), cdiv(ctx->nzp, RHS_ZMAX_HOST));
    a.kc_len = cdiv(ctx->nzp, nkc);
    a.ls = tile_lanes(ctx->nxp);
    a.nbx = cdiv(ctx->nxp, 2 * a.ls);
    a.nby = cdiv(ctx->nym, R32_T / a.ls);
    a.nbz = cdiv(ctx->nzp, a.kc_len);
    return a;
}

template <int LS, bool LAZY>
void rhs32_run(cf_ctx *ctx, const R32 &a, int s) {
    const dim3 grd(a.nbx, a.nby, a.nbz);
    if (s == 1) k_rhs32<LS, 1, LAZY><<<grd, R32_T, 0, ctx->st>>>(a);
    else if (s == 2) k_rhs32<LS, 2, LAZY><<<grd, R32_T, 0, ctx->st>>>(a);
    else k_rhs32<LS, 3, LAZY><<<grd, R32_T, 0, ctx->st>>>(a);
}

template <bool LAZY>
void rhs32_ls(cf_ctx *ctx, const R32 &a, int s) {
    if (a.ls == 32) rhs32_run<32, LAZY>(ctx, a, s);
    else if (a.ls == 16) rhs32_run<16, LAZY>(ctx, a, s);
    else rhs32_run<8, LAZY>(ctx, a, s);
}

}  // namespace

// z chunks
int rhs32_plan(int nxp, int nym, int nzp, int sms) {
    const int ls = tile_lanes(nxp);
    int per = 1;
    if (ls == 32) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rhs32<32, 2, true>, R32_T, 0);
    else if (ls == 16) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rhs32<16, 2, true>, R32_T, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rhs32<8, 2, true>, R32_T, 0);
    return cdiv(nzp, chunk_len((long)cdiv(nxp, 2 * ls) * cdiv(nym, R32_T / ls), per, sms, nzp));
}

int launch_rhs32(cf_ctx *ctx, int s, int src, int dst) {
    const R32 a = rhs32_args(ctx, s, src, dst);
    if (a.ns.S) rhs32_ls<true>(ctx, a, s);
    else rhs32_ls<false>(ctx, a, s);
    count_launch(ctx, "k_rhs32");
    CF_CUDA(cudaGetLastError());
    return 0;
}

// The right-hand sides + RK update of substep s of n split-path channels
// (state buffers src[q] -> dst[q]) in one launch: per channel exactly the
// arithmetic of launch_rhs32.
int launch_rhs32_batch(cudaStream_t st, cf_ctx *const *m, int s, const int *src, const int *dst, int n) {
    if (n < 1 || n > CF_ENS_MAXM) return CF_ERR_INVALID;
    R32Batch B;
    B.n = n;
    B.first[0] = 0;
    for (int q = 0; q < n; q++) {
        B.a[q] = rhs32_args(m[q], s, src[q], dst[q]);
        B.first[q + 1] = B.first[q] + B.a[q].nbx * B.a[q].nby * B.a[q].nbz;
    }
    if (s == 1) k_rhs32_batch<1><<<B.first[n], R32_T, 0, st>>>(B);
    else if (s == 2) k_rhs32_batch<2><<<B.first[n], R32_T, 0, st>>>(B);
    else k_rhs32_batch<3><<<B.first[n], R32_T, 0, st>>>(B);
    return cudaGetLastError() == cudaSuccess ? 0 : CF_ERR_CUDA;
}
