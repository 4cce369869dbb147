// k_rhs64.cu -- right-hand sides of u, v and w with the RK update
// (equations.f90:24-498, time_integration.f90:108-145) of the FP64 path, and
// each right-hand side by itself for the call-by-call interface (the same
// arithmetic, without the fluxes the other components need).
//
// What bounds it is the count of FP64 instructions (an SM issues one per 19
// clocks, see k_dsm64.cu), so every flux is formed once: the three normal
// fluxes at the cell centres and, at each edge, the product of the two
// interpolated velocities, the edge viscosity and the two velocity
// differences for both components that use them -- about 105 instructions a
// cell instead of 191 of a tile kernel that forms the x and y fluxes in both
// neighbouring cells (1691 -> 1075 us a launch at 192 x 128 x 192).
//
// A warp owns a segment of W = 32 or 16 columns of one row and marches along
// z.  Fluxes on a cell's upper faces and edges are formed by its own lane;
// the lower ones come from the lane to the left (a shuffle; at a segment's
// first column from its first three lanes, which form one of the left
// column's three fluxes each, in one instruction sequence), from the row
// below (through shared memory, double-buffered, one barrier per plane; the
// block's first row only forms what the next one needs) and from the plane
// below (carried).
//
// The reference divides the cross-derivative of a viscous flux by another
// spacing where the flux is a cell's upper face than where it is its lower
// one (equations.f90:108-163, 276-331, 435-493; the same on uniform grids),
// so an edge has up to two values per component: suffix _l below is the one
// the next cell takes as its lower face.
//
// Scales: normal fluxes times 4, xy and yz edges times 2, xz edges times 4
// (the interpolations' halves left out, exact powers of two), undone in the
// divergence's coefficients.
#include <algorithm>

#include "cf_internal.cuh"

namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr int R64_WARPS = 8;   // warps per block at most
constexpr int R64_ZMAX = 64;   // planes per chunk at most (their spacings sit in shared memory)

struct R64 {
    Fld<double> U, V, W, nt;
    Trio<double> out, F1, Uo;
    GeoT<double> g;
    RcpT<double> rc;
    const DevScal *ds;
    double nu, Om, ca, cb;
    // ilim, klim: last column and plane; rb: rows per block (one more row
    // forms only the lower fluxes)
    int rot, nyg, ny, ilim, klim, rb, kc_len;
};

// COMP 3: u, v and w with the update of substep S; 0, 1, 2: the right-hand
// side of u, v or w stored in out.
template <int W, int S, int COMP>
__global__ void __launch_bounds__(R64_WARPS * 32, 2) k_rhs64(const __grid_constant__ R64 a) {
    constexpr int SPW = 32 / W;
    constexpr bool CU = COMP == 0 || COMP == 3, CV = COMP == 1 || COMP == 3, CW = COMP == 2 || COMP == 3;
    __shared__ double xch[2][R64_WARPS * SPW][3][W];
    // per plane k of the chunk (and the one below it): 8 rdz[k+1], rdz[k],
    // rdz[k+1], rdzg[k+1], rdz[k]/4, rdz[k]/2, rdzg[k+1]/4
    __shared__ double zt[R64_ZMAX + 1][7];
    const int ny = a.ny, nyg = a.nyg, ilim = a.ilim;
    const int kb = 2 + blockIdx.z * a.kc_len, ke = min(kb + a.kc_len - 1, a.klim);
    for (int t = threadIdx.x; t < ke - kb + 2; t += blockDim.x) {
        const int k = kb - 1 + t;
        const double z0 = k >= 2 ? a.rc.dz[k] : 0.0, z1 = a.rc.dz[k + 1], zg = a.rc.dzg[k + 1];
        zt[t][0] = 8.0 * z1;
        zt[t][1] = z0;
        zt[t][2] = z1;
        zt[t][3] = zg;
        zt[t][4] = 0.25 * z0;
        zt[t][5] = 0.5 * z0;
        zt[t][6] = 0.25 * zg;
    }
    __syncthreads();
    const int l = threadIdx.x & (W - 1), row = threadIdx.x / W;  // row 0: the row below the block's rows
    const int i0 = 2 + blockIdx.x * W, ii = i0 + l, i = min(ii, ilim);
    const int jj = 1 + (int)blockIdx.y * a.rb + row, j = min(jj, nyg - 1);
    const bool active = row <= a.rb && jj <= nyg - 1, own = active && row > 0 && ii <= ilim;
    const bool full = __any_sync(FULLM, row > 0);  // some row of the warp is one of the block's
    const double nu = a.nu, nu2 = nu + nu, nu4 = nu2 + nu2;
    const double w0 = a.g.w0[min(j, ny)], w1 = a.g.w1[min(j, ny)];
    const double rx = a.rc.dx[i], rx1 = a.rc.dx[i + 1], rxg1 = a.rc.dxg[i + 1];
    const double ryg1 = a.rc.dyg[j + 1], ry1_8 = j + 1 <= ny ? 8.0 * a.rc.dy[j + 1] : 0.0, rx1_8 = 8.0 * rx1;
    const double ryh = j >= 2 ? 0.5 * a.rc.dy[j] : 0.0, rxh = 0.5 * rx, rxq = 0.25 * rx, rxgq = 0.25 * rxg1, rygq = 0.25 * ryg1;
    // this column's offsets (row j+1 of V clamped: read by rows without a v cell)
    const long ou = a.U.idx(i, j, 0), ov = a.V.idx(i, min(j, ny), 0), ow = a.W.idx(i, j, 0), on = a.nt.idx(i, j, 0);
    const int vup = j + 1 <= ny ? a.V.sy : 0;
    // lanes 0, 1, 2 of a segment: the left column's normal u flux, xy-edge
    // v flux and xz-edge w flux, as nu_e (c1 (X1 - X0) + c2 (Y1 - Y0)) -
    // (wa X0 + wb X1) (Y0 + Y1) with nu_e = base + wa nA + wb nB
    const int el = min(l, 2), iL = i0 - 1;
    const Fld<double> EY = el == 0 ? a.U : (el == 1 ? a.V : a.W);
    const long eX0 = a.U.idx(iL, j, 0), eX1 = el == 0 ? a.U.idx(i0, j, 0) : (el == 1 ? a.U.idx(iL, j + 1, 0) : a.U.idx(iL, j, 1));
    const long eY0 = EY.idx(iL, el == 1 ? min(j, ny) : j, 0), eY1 = eY0 + 1;
    const long eA0 = a.nt.idx(el == 0 ? i0 : iL, j, 0), eA1 = a.nt.idx(i0, j, 0);
    const long eB0 = el == 1 ? a.nt.idx(iL, j + 1, 0) : a.nt.idx(iL, j, 1), eB1 = eB0 + 1;
    const double ewa = el == 1 ? w0 : 1.0, ewb = el == 1 ? w1 : 1.0, ebase = el == 0 ? nu : (el == 1 ? nu2 : nu4);
    const double ec2 = el == 0 ? 0.0 : a.rc.dxg[i0], ec1f = el == 0 ? 8.0 * a.rc.dx[i0] : ryg1;
    const double dt = a.ds->dt, ca = dt * a.ca, cb = dt * a.cb, dPdx = a.ds->dPdx, dPdz = a.ds->dPdz;
    const int NT = blockDim.x;
    auto left = [&](double v, double edge, int e) {
        const double p = __shfl_up_sync(FULLM, v, 1, W), q = __shfl_sync(FULLM, edge, e, W);
        return l == 0 ? q : p;
    };
    double zu_l = 0, zv_l = 0, zw_l = 0;  // fluxes through the z faces below plane k
    // values of plane k that were plane k+1's before
    long pk = kb - 1;
    double U0 = a.U.p[ou + a.U.sz * pk], V0 = a.V.p[ov + a.V.sz * pk], W0 = a.W.p[ow + a.W.sz * pk];
    double n00 = a.nt.p[on + a.nt.sz * pk], n01 = a.nt.p[on + a.nt.sz * pk + a.nt.sy];
    double sx = n00 + a.nt.p[on + a.nt.sz * pk + 1];
    for (int k = kb - 1; k <= ke; k++) {
        const bool head = k < kb;  // the plane below the chunk: only the fluxes up from it
        const double *z = zt[k - kb + 1];
        const long ku = (long)a.U.sz * k, kv = (long)a.V.sz * k, kw = (long)a.W.sz * k, kn = (long)a.nt.sz * k;
        const double *U = a.U.p + ou + ku, *V = a.V.p + ov + kv, *Wp = a.W.p + ow + kw, *N = a.nt.p + on + kn;
        // (u and v go one plane further than W's planes reach)
        const double Un = U[a.U.sz], Vn = V[a.V.sz], Wn = CW ? Wp[a.W.sz] : 0.0;
        if (!CW) W0 = Wp[0];
        const double nn00 = N[a.nt.sz], nn10 = N[a.nt.sz + 1], nn01 = N[a.nt.sz + a.nt.sy];
        const double Uup = U[a.U.sy], Vr = V[1], Vup = V[vup], Wr = Wp[1], Wup = Wp[a.W.sy];
        const double n11 = N[a.nt.sy + 1];
        double uo = 0, vo = 0, wo = 0, fu = 0, fv = 0, fw = 0;
        if (COMP == 3 && !head && own) {
            const long o = a.out.u.idx(i, j, k);
            uo = a.Uo.u.p[o];
            if constexpr (S > 1) fu = a.F1.u.p[o];
            const long ww = a.out.w.idx(i, j, k);
            wo = a.Uo.w.p[ww];
            if constexpr (S > 1) fw = a.F1.w.p[ww];
            if (j <= ny - 1) {
                const long vv = a.out.v.idx(i, j, k);
                vo = a.Uo.v.p[vv];
                if constexpr (S > 1) fv = a.F1.v.p[vv];
            }
        }
        const double sxn = nn00 + nn10;
        // yz edge (j+1/2, k+1/2): v through the z face, w through the y face
        double zv = 0, yw = 0, yw_l = 0;
        if (CV || CW) {
            const double ne = fma(w1, n01 + nn01, fma(w0, n00 + nn00, nu2));
            const double A = (V0 + Vn) * fma(w1, Wup, w0 * W0), dV = Vn - V0, gW = (Wup - W0) * ryg1;
            if (CV) zv = fma(ne, fma(dV, z[3], gW), -A);
            if (CW) {
                yw = fma(ne, fma(dV, z[2], gW), -A);
                yw_l = fma(ne, fma(dV, z[1], gW), -A);
            }
        }
        double zu = 0, zu_up = 0, xw = 0, xw_l = 0, zw = 0;
        if ((CU || CW) && full) {
            // xz edge (i+1/2, k+1/2): u through the z face, w through the x face
            const double ne = nu4 + (sx + sxn), A = (U0 + Un) * (W0 + Wr), dU = Un - U0, dW = Wr - W0;
            if (CU) {
                const double gz = dU * z[3];
                zu_up = fma(ne, fma(dW, rx1, gz), -A);
                zu = fma(ne, fma(dW, rx, gz), -A);
            }
            if (CW) {
                const double gx = dW * rxg1;
                xw = fma(ne, fma(dU, z[2], gx), -A);
                xw_l = fma(ne, fma(dU, z[1], gx), -A);
                // w through the centre of plane k+1
                const double s = W0 + Wn;
                zw = fma((nu + nn00) * z[0], Wn - W0, -(s * s));
            }
        }
        if (!head) {
            // xy edge (i+1/2, j+1/2): u through the y face, v through the x face
            double yu = 0, yu_l = 0, xv = 0;
            if (CU || CV) {
                const double ne = fma(w1, n01 + n11, fma(w0, sx, nu2));
                const double A = fma(w1, Uup, w0 * U0) * (V0 + Vr), g = (Uup - U0) * ryg1, dV = Vr - V0;
                if (CU) {
                    yu = fma(ne, fma(dV, rx1, g), -A);
                    yu_l = fma(ne, fma(dV, rx, g), -A);
                }
                if (CV) xv = fma(ne, fma(dV, rxg1, g), -A);
            }
            double yv = 0;
            if (CV) {  // v through the centre of row j+1
                const double sv = V0 + Vup;
                yv = fma((nu + n01) * ry1_8, Vup - V0, -(sv * sv));
            }
            double(*xb)[3][W] = xch[k & 1];
            if (CU) xb[row][0][l] = yu_l;
            if (CW) xb[row][1][l] = yw_l;
            if (CV) xb[row][2][l] = yv;
            double xu = 0, ef = 0;
            if (full) {
                if (CU) {  // u through the centre of column i+1
                    const double Ur = U[1], s = U0 + Ur;
                    xu = fma((nu + N[1]) * rx1_8, Ur - U0, -(s * s));
                }
                // the left column's three fluxes
                if (l < 3) {
                    const double *X = a.U.p + ku, *Y = EY.p + (long)EY.sz * k, *E = a.nt.p + kn;
                    const double X0 = X[eX0], X1 = X[eX1], Y0 = Y[eY0], Y1 = Y[eY1];
                    const double A1 = el == 0 ? 0.0 : E[eA1], B0 = el == 0 ? 0.0 : E[eB0], B1 = el == 0 ? 0.0 : E[eB1];
                    const double ne = fma(ewb, B0 + B1, fma(ewa, E[eA0] + A1, ebase));
                    const double A = fma(ewb, X1, ewa * X0) * (Y0 + Y1);
                    ef = fma(ne, fma(Y1 - Y0, ec2, (X1 - X0) * (el == 2 ? z[1] : ec1f)), -A);
                }
            }
            asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
            if (full) {
                const int rl = max(row - 1, 0);
                double ru = 0, rv = 0, rw = 0;
                if (CU) {
                    ru = fma(rxgq, xu - left(xu, ef, 0), dPdx);
                    ru = fma(ryh, yu - xb[rl][0][l], ru);
                    ru = fma(z[4], zu_up - zu_l, ru);
                }
                if (CV) {
                    rv = rxh * (xv - left(xv, ef, 1));
                    rv = fma(rygq, yv - xb[rl][2][l], rv);
                    rv = fma(z[5], zv - zv_l, rv);
                }
                if (CW) {
                    rw = fma(rxq, xw - left(xw_l, ef, 2), dPdz);
                    rw = fma(ryh, yw - xb[rl][1][l], rw);
                    rw = fma(z[6], zw - zw_l, rw);
                }
                if (a.rot && own) {
                    // equations.f90:169-177, 334-342
                    const double h = 0.5;
                    if (CU) ru += 2.0 * a.Om * (h * (h * (V[-a.V.sy] + V0) + h * (V[1 - a.V.sy] + Vr)));
                    if (CV && j <= ny - 1) rv -= 2.0 * a.Om * (w0 * (h * (U[-1] + U0)) + w1 * (h * (U[a.U.sy - 1] + Uup)));
                }
                if (COMP < 3) {
                    const Fld<double> F = COMP == 0 ? a.out.u : (COMP == 1 ? a.out.v : a.out.w);
                    if (own && (COMP != 1 || j <= ny - 1)) F.p[F.idx(i, j, k)] = COMP == 0 ? ru : (COMP == 1 ? rv : rw);
                } else if (own) {
                    const long o = a.out.u.idx(i, j, k), ww = a.out.w.idx(i, j, k), vv = a.out.v.idx(i, j, k);
                    if constexpr (S == 1) {
                        a.F1.u.p[o] = ru;
                        a.F1.w.p[ww] = rw;
                        a.out.u.p[o] = fma(ca, ru, uo);
                        a.out.w.p[ww] = fma(ca, rw, wo);
                    } else {
                        a.out.u.p[o] = fma(ca, fu, fma(cb, ru, uo));
                        a.out.w.p[ww] = fma(ca, fw, fma(cb, rw, wo));
                    }
                    if (j <= ny - 1) {
                        if constexpr (S == 1) {
                            a.F1.v.p[vv] = rv;
                            a.out.v.p[vv] = fma(ca, rv, vo);
                        } else {
                            a.out.v.p[vv] = fma(ca, fv, fma(cb, rv, vo));
                        }
                    }
                }
            }
        }
        zu_l = zu;
        zv_l = zv;
        zw_l = zw;
        U0 = Un;
        V0 = Vn;
        W0 = Wn;
        n00 = nn00;
        n01 = nn01;
        sx = sxn;
    }
}

struct R64Plan {
    int w, rb, warps;
};

// segments of 16 lanes where a row then has fewer idle columns; rows per
// block: at most 8 warps, one row of them the halo, the fewest warps in all
R64Plan r64_shape(int nxp, int nym) {
    R64Plan p;
    p.w = cdiv(nxp, 16) * 16 < cdiv(nxp, 32) * 32 ? 16 : 32;
    const int spw = 32 / p.w;
    long best = -1;
    p.rb = 1;
    p.warps = 1;
    for (int rb = 1; rb <= R64_WARPS * spw - 1; rb++) {
        const int warps = cdiv(rb + 1, spw);
        const long cost = (long)cdiv(nym, rb) * warps;
        if (best < 0 || cost <= best) {
            best = cost;
            p.rb = rb;
            p.warps = warps;
        }
    }
    return p;
}

}  // namespace

// z chunks (64 x 48 x 64: 10 chunks, one block an SM, 66 us; 22 chunks 60)
int rhs64_plan(int nxp, int nym, int nzp, int sms) {
    const R64Plan p = r64_shape(nxp, nym);
    const long blocks = (long)cdiv(nxp, p.w) * cdiv(nym, p.rb);
    return cdiv(nzp, fp64_chunk_len(blocks, sms, nzp, cdiv(nzp, R64_ZMAX), 0.5));
}

static R64 r64_args(cf_ctx *ctx, int src, const R64Plan &p) {
    R64 a;
    a.U = make_fld<double>(ctx->U[src], ctx->nx, ctx->nyg);
    a.V = make_fld<double>(ctx->V[src], ctx->nxg, ctx->ny);
    a.W = make_fld<double>(ctx->W[src], ctx->nxg, ctx->nyg);
    a.nt = make_fld<double>(ctx->nut, ctx->nxg, ctx->nyg);
    a.g = ctx->geo;
    a.rc = rcp_of<double>(ctx);
    a.ds = ctx->ds;
    a.nu = ctx->prm.nu;
    a.Om = ctx->omega_z;
    a.rot = fabs(ctx->omega_z) > 1e-6 ? 1 : 0;  // equations.f90:169, 334
    a.ny = ctx->ny; a.nyg = ctx->nyg;
    a.rb = p.rb;
    a.kc_len = cdiv(ctx->nzp, std::max(ctx->rhs_nkc, cdiv(ctx->nzp, R64_ZMAX)));
    a.ca = a.cb = 0.0;
    return a;
}

static Trio<double> r64_trio(cf_ctx *ctx, void *u, void *v, void *w) {
    Trio<double> t;
    t.u = make_fld<double>(u, ctx->nx, ctx->nyg);
    t.v = make_fld<double>(v, ctx->nxg, ctx->ny);
    t.w = make_fld<double>(w, ctx->nxg, ctx->nyg);
    return t;
}

// Right-hand sides of buffer src and the update of substep s into buffer dst
// (canonical cells: the boundary conditions after the projection rewrite the
// periodic duplicates, and nothing reads them before), on stream st.
int launch_rhs64(cf_ctx *ctx, cudaStream_t st, int s, int src, int dst) {
    const R64Plan p = r64_shape(ctx->nxp, ctx->nym);
    R64 a = r64_args(ctx, src, p);
    void *nt;
    if (int rc = launch_nut_rhs64(ctx, st, &nt)) return rc;
    a.nt = make_fld<double>(nt, ctx->nxg, ctx->nyg);
    a.out = r64_trio(ctx, ctx->U[dst], ctx->V[dst], ctx->W[dst]);
    a.F1 = r64_trio(ctx, ctx->F[0][0], ctx->F[0][1], ctx->F[0][2]);
    a.Uo = r64_trio(ctx, ctx->U[ctx->old], ctx->V[ctx->old], ctx->W[ctx->old]);
    // rk_coef (initialization.f90:408-416)
    a.ca = s == 1 ? 8.0 / 15.0 : 1.0 / 4.0;
    a.cb = s == 2 ? 5.0 / 12.0 : 3.0 / 4.0;
    a.ilim = ctx->nx - 1;
    a.klim = ctx->nz - 1;
    const dim3 grd(cdiv(ctx->nxp, p.w), cdiv(ctx->nym, p.rb), cdiv(ctx->nzp, a.kc_len));
#define CF_R64(WW, SS) k_rhs64<WW, SS, 3><<<grd, p.warps * 32, 0, st>>>(a)
    if (p.w == 32) {
        if (s == 1) CF_R64(32, 1); else if (s == 2) CF_R64(32, 2); else CF_R64(32, 3);
    } else {
        if (s == 1) CF_R64(16, 1); else if (s == 2) CF_R64(16, 2); else CF_R64(16, 3);
    }
#undef CF_R64
    return cudaGetLastError() == cudaSuccess ? 0 : cf_fail(ctx, CF_ERR_CUDA, "k_rhs64");
}

// The right-hand side of component comp of the current state into slot, on
// the ranges of equations.f90 (periodic duplicates included).
int launch_rhs64_comp(cf_ctx *ctx, int comp, int slot) {
    const R64Plan p = r64_shape(ctx->nxp, ctx->nym);
    R64 a = r64_args(ctx, ctx->cur, p);
    a.out = r64_trio(ctx, ctx->F[slot][0], ctx->F[slot][1], ctx->F[slot][2]);
    a.F1 = a.Uo = a.out;
    a.ilim = comp == 0 ? ctx->nx - 1 : ctx->nxg - 1;
    a.klim = comp == 2 ? ctx->nz - 1 : ctx->nzg - 1;
    const dim3 grd(cdiv(a.ilim - 1, p.w), cdiv(ctx->nym, p.rb), cdiv(a.klim - 1, a.kc_len));
#define CF_R64(WW, CC) k_rhs64<WW, 0, CC><<<grd, p.warps * 32, 0, ctx->st>>>(a)
    if (p.w == 32) {
        if (comp == 0) CF_R64(32, 0); else if (comp == 1) CF_R64(32, 1); else CF_R64(32, 2);
    } else {
        if (comp == 0) CF_R64(16, 0); else if (comp == 1) CF_R64(16, 1); else CF_R64(16, 2);
    }
#undef CF_R64
    count_launch(ctx, "k_rhs64");
    CF_CUDA(cudaGetLastError());
    return 0;
}
