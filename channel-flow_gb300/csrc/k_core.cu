// k_core.cu -- boundary conditions, momentum right-hand sides, RK3 update,
// mass-flow forcing, time-step and divergence reductions.
#include <algorithm>


#include "cf_internal.cuh"

// ---------------------------------------------------------------------------
// apply_boundary_conditions (boundary_conditions.f90:20-75).
// One thread per ghost element.  The reference first copies the x-periodic
// planes, then the z-periodic planes (including x ghosts), then overwrites the
// two wall rows for every (i,k); the composed result at a ghost element is
// therefore a copy from the canonical position (wrap(i), j, wrap(k)), and the
// wall rows are built from row 2 / row nyg-1 at (wrap(i), wrap(k)).
// ---------------------------------------------------------------------------
// ybc: 0 = Dirichlet at centres (ghost = -interior), 1 = zero at faces,
//      2 = nonzero Neumann at centres (ghost = interior - dy*alpha(i,wall,k))
struct BcField {
    void *p, *plo;
    int n1, n2, n3, xc, zc, ybc;
    const double *alpha;
    int n;  // ghost elements of this field
};
struct BcSet {
    BcField f[3];
    int nxp, nzp;
    double dyb, dyt;
};

template <typename T>
__device__ __forceinline__ void bc_elem(const BcField &d, int nxp, int nzp, double dyb, double dyt, int t) {
    const Fld<T> F = make_fld<T>(d.p, d.n1, d.n2), Flo = make_fld<T>(d.plo, d.n1, d.n2);
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3, xc = d.xc, zc = d.zc, ybc = d.ybc;
    const int gx = xc ? 3 : 2, gz = zc ? 3 : 2;
    const int nY = 2 * n1 * n3;
    const int nX = gx * (n2 - 2) * n3;
    int i, j, k;
    if (t < nY) {
        i = t % n1 + 1;
        int r = t / n1;
        k = r % n3 + 1;
        j = (r / n3) == 0 ? 1 : n2;
        int is = wrapc(i, nxp), ks = wrapc(k, nzp);
        if (ybc == 1) {
            F(i, j, k) = T(0);
            if (Flo.p) Flo(i, j, k) = T(0);
        } else {
            int jsrc = (j == 1) ? 2 : n2 - 1;
            T v = F(is, jsrc, ks);
            if (ybc == 0) {
                F(i, j, k) = -v;
                if (Flo.p) Flo(i, j, k) = -Flo(is, jsrc, ks);
            } else {
                int w = (j == 1) ? 0 : 1;
                double a = d.alpha[(i - 1) + (long)n1 * (w + 2L * (k - 1))];
                double dy = (j == 1) ? dyb : dyt;
                if (Flo.p) {
                    double hv = (double)v + (double)Flo(is, jsrc, ks) - dy * a;
                    T hi = (T)hv;
                    F(i, j, k) = hi;
                    Flo(i, j, k) = (T)(hv - (double)hi);
                } else {
                    F(i, j, k) = (T)((double)v - dy * a);
                }
            }
        }
        return;
    }
    t -= nY;
    if (t < nX) {
        int g = t % gx;
        int r = t / gx;
        j = r % (n2 - 2) + 2;
        k = r / (n2 - 2) + 1;
        i = (g == 0) ? 1 : (xc ? (g == 1 ? n1 - 1 : n1) : n1);
    } else {
        t -= nX;
        int g = t % gz;
        int r = t / gz;
        j = r % (n2 - 2) + 2;
        i = r / (n2 - 2) + 2;  // non-ghost x: 2 .. n1-gx+1
        k = (g == 0) ? 1 : (zc ? (g == 1 ? n3 - 1 : n3) : n3);
    }
    int is = wrapc(i, nxp), ks = wrapc(k, nzp);
    F(i, j, k) = F(is, j, ks);
    if (Flo.p) Flo(i, j, k) = Flo(is, j, ks);
}

// The ghost shells of U, V and W in one launch: thread t belongs to the
// field whose element range contains it.
template <typename T>
__global__ void k_bc(BcSet s) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (t < s.f[q].n) {
            bc_elem<T>(s.f[q], s.nxp, s.nzp, s.dyb, s.dyt, t);
            return;
        }
        t -= s.f[q].n;
    }
}

static BcField bc_field(void *p, void *plo, int n1, int n2, int n3, int xc, int zc, int ybc, const double *alpha) {
    BcField f;
    int gx = xc ? 3 : 2, gz = zc ? 3 : 2;
    f.p = p;
    f.plo = plo;
    f.n1 = n1;
    f.n2 = n2;
    f.n3 = n3;
    f.xc = xc;
    f.zc = zc;
    f.ybc = ybc;
    f.alpha = alpha;
    f.n = 2 * n1 * n3 + gx * (n2 - 2) * n3 + gz * (n2 - 2) * (n1 - gx);
    return f;
}

template <typename T>
int launch_bc(cf_ctx *ctx, int b, bool lo) {
    int wm = ctx->prm.iwall_model;
    BcSet s;
    // U: x faces, y centres, z centres
    s.f[0] = bc_field(ctx->U[b], lo ? ctx->Ulo[b] : nullptr, ctx->nx, ctx->nyg, ctx->nzg, 0, 1, wm == 3 ? 2 : 0, ctx->alpha_x);
    // V: x centres, y faces, z centres
    s.f[1] = bc_field(ctx->V[b], lo ? ctx->Vlo[b] : nullptr, ctx->nxg, ctx->ny, ctx->nzg, 1, 1, 1, nullptr);
    // W: x centres, y centres, z faces
    s.f[2] = bc_field(ctx->W[b], lo ? ctx->Wlo[b] : nullptr, ctx->nxg, ctx->nyg, ctx->nz, 1, 0, wm == 3 ? 2 : 0, ctx->alpha_z);
    s.nxp = ctx->nxp;
    s.nzp = ctx->nzp;
    s.dyb = ctx->hyg[2] - ctx->hyg[1];
    s.dyt = ctx->hyg[ctx->nyg] - ctx->hyg[ctx->nyg - 1];
    const int tot = s.f[0].n + s.f[1].n + s.f[2].n;
    ctx->nut_renew = false;
    k_bc<T><<<cdiv(tot, 256), 256, 0, ctx->st>>>(s);
    count_launch(ctx, "k_bc");
    CF_CUDA(cudaGetLastError());
    return 0;
}

// ---------------------------------------------------------------------------
// Momentum right-hand sides, equations.f90:24-498, one thread per point.
// ---------------------------------------------------------------------------
// The spacings enter as reciprocals (rc): 1/(xg(i+1)-xg(i)) = rc.dxg[i+1],
// 1/(x(i)-x(i-1)) = rc.dx[i], and so on.
template <typename T, typename A, typename RC>
__device__ __forceinline__ T rhs_u_point(const GeoT<T> &g, const RC &rc, const A &U, const A &V, const A &W,
                                         const A &nt, T nu, T dPdx, T Om, bool rot, int i, int j, int k) {
    const T *w0 = g.w0, *w1 = g.w1;
    const T h = T(0.5), q = T(0.25);
    const T rdx1 = rc.dx[i], rdx2 = rc.dx[i + 1], rdx3 = rc.dxg[i + 1];
    const T rdy3 = rc.dy[j];
    const T rdz1 = rc.dzg[k], rdz2 = rc.dzg[k + 1], rdz3 = rc.dz[k];
    // 1) -du^2/dx  (equations.f90:43-57)
    T a = h * (U(i, j, k) + U(i + 1, j, k));
    T b = h * (U(i - 1, j, k) + U(i, j, k));
    T r = -(a * a - b * b) * rdx3;
    // 2) -duv/dy   (:62-79)
    T uy1 = w0[j] * U(i, j, k) + w1[j] * U(i, j + 1, k);
    T uy0 = w0[j - 1] * U(i, j - 1, k) + w1[j - 1] * U(i, j, k);
    T vx1 = h * (V(i, j, k) + V(i + 1, j, k));
    T vx0 = h * (V(i, j - 1, k) + V(i + 1, j - 1, k));
    r += -(uy1 * vx1 - uy0 * vx0) * rdy3;
    // 3) -duw/dz   (:84-101)
    T uz1 = h * (U(i, j, k) + U(i, j, k + 1));
    T wx1 = h * (W(i, j, k) + W(i + 1, j, k));
    T uz0 = h * (U(i, j, k - 1) + U(i, j, k));
    T wx0 = h * (W(i, j, k - 1) + W(i + 1, j, k - 1));
    r += -(uz1 * wx1 - uz0 * wx0) * rdz3;
    // 4) viscous   (:108-163)
    T t2j = (U(i, j + 1, k) - U(i, j, k)) * rc.dyg[j + 1];
    T t2jm = (U(i, j, k) - U(i, j - 1, k)) * rc.dyg[j];
    T nu_x1 = nu + nt(i, j, k);
    T nu_x2 = nu + nt(i + 1, j, k);
    T nu_y1 = nu + h * (w0[j - 1] * nt(i, j - 1, k) + w1[j - 1] * nt(i, j, k) + w0[j - 1] * nt(i + 1, j - 1, k) +
                        w1[j - 1] * nt(i + 1, j, k));
    T nu_y2 = nu + h * (w0[j] * nt(i, j, k) + w1[j] * nt(i, j + 1, k) + w0[j] * nt(i + 1, j, k) + w1[j] * nt(i + 1, j + 1, k));
    T nu_z2 = nu + q * (nt(i, j, k) + nt(i, j, k + 1) + nt(i + 1, j, k) + nt(i + 1, j, k + 1));
    T visc = T(2) * rdx3 * (nu_x2 * (U(i + 1, j, k) - U(i, j, k)) * rdx2 - nu_x1 * (U(i, j, k) - U(i - 1, j, k)) * rdx1) +
             rdy3 * (nu_y2 * (t2j + (V(i + 1, j, k) - V(i, j, k)) * rdx2) -
                     nu_y1 * (t2jm + (V(i + 1, j - 1, k) - V(i, j - 1, k)) * rdx1));
    T nu_z1 = nu + q * (nt(i, j, k) + nt(i, j, k - 1) + nt(i + 1, j, k) + nt(i + 1, j, k - 1));
    visc += rdz3 * (nu_z2 * ((U(i, j, k + 1) - U(i, j, k)) * rdz2 + (W(i + 1, j, k) - W(i, j, k)) * rdx2) -
                    nu_z1 * ((U(i, j, k) - U(i, j, k - 1)) * rdz1 + (W(i + 1, j, k - 1) - W(i, j, k - 1)) * rdx1));
    r += visc;
    r += dPdx;  // :166
    if (rot) {  // |Om| > 1e-6, :169-177
        T tv0 = h * (V(i, j - 1, k) + V(i, j, k));
        T tv1 = h * (V(i + 1, j - 1, k) + V(i + 1, j, k));
        r += T(2) * Om * (h * (tv0 + tv1));
    }
    return r;
}

template <typename T, typename A, typename RC>
__device__ __forceinline__ T rhs_v_point(const GeoT<T> &g, const RC &rc, const A &U, const A &V, const A &W,
                                         const A &nt, T nu, T Om, bool rot, int i, int j, int k) {
    const T *w0 = g.w0, *w1 = g.w1;
    const T h = T(0.5);
    const T rdx1 = rc.dxg[i], rdx2 = rc.dxg[i + 1], rdx3 = rc.dx[i];
    const T rdy1 = rc.dy[j], rdy2 = rc.dy[j + 1], rdy3 = rc.dyg[j + 1];
    const T rdz1 = rc.dzg[k], rdz2 = rc.dzg[k + 1], rdz3 = rc.dz[k];
    // 1) -dv^2/dy (equations.f90:205-223)
    T a = h * (V(i, j, k) + V(i, j + 1, k));
    T b = h * (V(i, j - 1, k) + V(i, j, k));
    T r = -(a * a - b * b) * rdy3;
    // 2) -duv/dx (:228-245)
    T uy1 = w0[j] * U(i, j, k) + w1[j] * U(i, j + 1, k);
    T uy0 = w0[j] * U(i - 1, j, k) + w1[j] * U(i - 1, j + 1, k);
    T vx1 = h * (V(i, j, k) + V(i + 1, j, k));
    T vx0 = h * (V(i - 1, j, k) + V(i, j, k));
    r += -(uy1 * vx1 - uy0 * vx0) * rdx3;
    // 3) -dvw/dz (:250-267)
    T vz1 = h * (V(i, j, k) + V(i, j, k + 1));
    T wy1 = w0[j] * W(i, j, k) + w1[j] * W(i, j + 1, k);
    T vz0 = h * (V(i, j, k - 1) + V(i, j, k));
    T wy0 = w0[j] * W(i, j, k - 1) + w1[j] * W(i, j + 1, k - 1);
    r += -(vz1 * wy1 - vz0 * wy0) * rdz3;
    // 4) viscous (:276-331)
    T nu_x1 = nu + h * (w0[j] * nt(i - 1, j, k) + w1[j] * nt(i - 1, j + 1, k) + w0[j] * nt(i, j, k) + w1[j] * nt(i, j + 1, k));
    T nu_x2 = nu + h * (w0[j] * nt(i, j, k) + w1[j] * nt(i, j + 1, k) + w0[j] * nt(i + 1, j, k) + w1[j] * nt(i + 1, j + 1, k));
    T nu_y1 = nu + nt(i, j, k);
    T nu_y2 = nu + nt(i, j + 1, k);
    T nu_z2 = nu + h * (w0[j] * nt(i, j, k) + w1[j] * nt(i, j + 1, k) + w0[j] * nt(i, j, k + 1) + w1[j] * nt(i, j + 1, k + 1));
    T visc = rdx3 * (nu_x2 * ((V(i + 1, j, k) - V(i, j, k)) * rdx2 + (U(i, j + 1, k) - U(i, j, k)) * rdy3) -
                     nu_x1 * ((V(i, j, k) - V(i - 1, j, k)) * rdx1 + (U(i - 1, j + 1, k) - U(i - 1, j, k)) * rdy3)) +
             T(2) * rdy3 * (nu_y2 * (V(i, j + 1, k) - V(i, j, k)) * rdy2 - nu_y1 * (V(i, j, k) - V(i, j - 1, k)) * rdy1);
    T nu_z1 = nu + h * (w0[j] * nt(i, j, k - 1) + w1[j] * nt(i, j + 1, k - 1) + w0[j] * nt(i, j, k) + w1[j] * nt(i, j + 1, k));
    visc += rdz3 * (nu_z2 * ((V(i, j, k + 1) - V(i, j, k)) * rdz2 + (W(i, j + 1, k) - W(i, j, k)) * rdy3) -
                    nu_z1 * ((V(i, j, k) - V(i, j, k - 1)) * rdz1 + (W(i, j + 1, k - 1) - W(i, j, k - 1)) * rdy3));
    r += visc;
    if (rot) {  // :334-342
        T tu0 = h * (U(i - 1, j, k) + U(i, j, k));
        T tu1 = h * (U(i - 1, j + 1, k) + U(i, j + 1, k));
        r -= T(2) * Om * (w0[j] * tu0 + w1[j] * tu1);
    }
    return r;
}

template <typename T, typename A, typename RC>
__device__ __forceinline__ T rhs_w_point(const GeoT<T> &g, const RC &rc, const A &U, const A &V, const A &W,
                                         const A &nt, T nu, T dPdz, int i, int j, int k) {
    const T *w0 = g.w0, *w1 = g.w1;
    const T h = T(0.5), q = T(0.25);
    const T rdx1 = rc.dxg[i], rdx2 = rc.dxg[i + 1], rdx3 = rc.dx[i];
    const T rdy3 = rc.dy[j];
    const T rdz1 = rc.dz[k], rdz2 = rc.dz[k + 1], rdz3 = rc.dzg[k + 1];
    // 1) -dw^2/dz (equations.f90:370-384)
    T a = h * (W(i, j, k) + W(i, j, k + 1));
    T r = T(0);
    T b = h * (W(i, j, k - 1) + W(i, j, k));
    r = -(a * a - b * b) * rdz3;
    // 2) -duw/dx (:389-406)
    T uz1 = h * (U(i, j, k) + U(i, j, k + 1));
    T uz0 = h * (U(i - 1, j, k) + U(i - 1, j, k + 1));
    T wx1 = h * (W(i, j, k) + W(i + 1, j, k));
    T wx0 = h * (W(i - 1, j, k) + W(i, j, k));
    r += -(uz1 * wx1 - uz0 * wx0) * rdx3;
    // 3) -dvw/dy (:411-428)
    T vz1 = h * (V(i, j, k) + V(i, j, k + 1));
    T vz0 = h * (V(i, j - 1, k) + V(i, j - 1, k + 1));
    T wy1 = w0[j] * W(i, j, k) + w1[j] * W(i, j + 1, k);
    T wy0 = w0[j - 1] * W(i, j - 1, k) + w1[j - 1] * W(i, j, k);
    r += -(vz1 * wy1 - vz0 * wy0) * rdy3;
    // 4) viscous (:435-493)
    T t2j = (W(i, j + 1, k) - W(i, j, k)) * rc.dyg[j + 1];
    T t2jm = (W(i, j, k) - W(i, j - 1, k)) * rc.dyg[j];
    T nu_x1 = nu + q * (nt(i, j, k) + nt(i, j, k + 1) + nt(i - 1, j, k) + nt(i - 1, j, k + 1));
    T nu_x2 = nu + q * (nt(i, j, k) + nt(i, j, k + 1) + nt(i + 1, j, k) + nt(i + 1, j, k + 1));
    T nu_y1 = nu + h * (w0[j - 1] * nt(i, j - 1, k) + w1[j - 1] * nt(i, j, k) + w0[j - 1] * nt(i, j - 1, k + 1) +
                        w1[j - 1] * nt(i, j, k + 1));
    T nu_y2 = nu + h * (w0[j] * nt(i, j, k) + w1[j] * nt(i, j + 1, k) + w0[j] * nt(i, j, k + 1) + w1[j] * nt(i, j + 1, k + 1));
    T nu_z2 = nu + nt(i, j, k + 1);
    T visc = rdx3 * (nu_x2 * ((W(i + 1, j, k) - W(i, j, k)) * rdx2 + (U(i, j, k + 1) - U(i, j, k)) * rdz2) -
                     nu_x1 * ((W(i, j, k) - W(i - 1, j, k)) * rdx1 + (U(i - 1, j, k + 1) - U(i - 1, j, k)) * rdz1)) +
             rdy3 * (nu_y2 * (t2j + (V(i, j, k + 1) - V(i, j, k)) * rdz2) -
                     nu_y1 * (t2jm + (V(i, j - 1, k + 1) - V(i, j - 1, k)) * rdz1));
    T nu_z1 = nu + nt(i, j, k);
    visc += T(2) * rdz3 * (nu_z2 * (W(i, j, k + 1) - W(i, j, k)) * rdz2 - nu_z1 * (W(i, j, k) - W(i, j, k - 1)) * rdz1);
    r += visc;
    r += dPdz;  // :496
    return r;
}

// one right-hand side into its slot
template <typename T, int COMP>
__global__ void k_rhs(GeoT<T> g, RcpT<T> rc, Fld<T> U, Fld<T> V, Fld<T> W, Fld<T> nt, const DevScal *ds, T nu, T Om, int rot,
                      Fld<T> out, int i1, int j1, int k1) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
    int k = blockIdx.z + 2;
    if (i > i1 || j > j1 || k > k1) return;
    T r;
    if (COMP == 0) r = rhs_u_point<T, Fld<T>>(g, rc, U, V, W, nt, nu, ds_dpdx<T>(ds), Om, rot, i, j, k);
    else if (COMP == 1) r = rhs_v_point<T, Fld<T>>(g, rc, U, V, W, nt, nu, Om, rot, i, j, k);
    else r = rhs_w_point<T, Fld<T>>(g, rc, U, V, W, nt, nu, ds_dpdz<T>(ds), i, j, k);
    out(i, j, k) = r;
}

template <typename T>
static int rhs_launch(cf_ctx *ctx, int comp, int slot) {
    if (int rc = launch_nut_materialize<T>(ctx)) return rc;
    const GeoT<T> g = geo_of<T>(ctx);
    const int b = ctx->cur;
    const Fld<T> U = make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg), V = make_fld<T>(ctx->V[b], ctx->nxg, ctx->ny),
                 W = make_fld<T>(ctx->W[b], ctx->nxg, ctx->nyg), nt = make_fld<T>(ctx->nut, ctx->nxg, ctx->nyg);
    int i1, j1, k1, n1, n2;
    if (comp == 0) { i1 = ctx->nx - 1; j1 = ctx->nyg - 1; k1 = ctx->nzg - 1; n1 = ctx->nx; n2 = ctx->nyg; }
    else if (comp == 1) { i1 = ctx->nxg - 1; j1 = ctx->ny - 1; k1 = ctx->nzg - 1; n1 = ctx->nxg; n2 = ctx->ny; }
    else { i1 = ctx->nxg - 1; j1 = ctx->nyg - 1; k1 = ctx->nz - 1; n1 = ctx->nxg; n2 = ctx->nyg; }
    // F arrays use the full field extents (interior written)
    const Fld<T> out = make_fld<T>(ctx->F[slot][comp], n1, n2);
    const dim3 blk(32, 4, 1), grd(cdiv(i1 - 1, 32), cdiv(j1 - 1, 4), k1 - 1);
    const T nu = (T)ctx->prm.nu, Om = (T)ctx->omega_z;
    const int rot = fabs(ctx->omega_z) > 1e-6;  // equations.f90:169, 334
    const RcpT<T> rc = rcp_of<T>(ctx);
    if (comp == 0) k_rhs<T, 0><<<grd, blk, 0, ctx->st>>>(g, rc, U, V, W, nt, ctx->ds, nu, Om, rot, out, i1, j1, k1);
    else if (comp == 1) k_rhs<T, 1><<<grd, blk, 0, ctx->st>>>(g, rc, U, V, W, nt, ctx->ds, nu, Om, rot, out, i1, j1, k1);
    else k_rhs<T, 2><<<grd, blk, 0, ctx->st>>>(g, rc, U, V, W, nt, ctx->ds, nu, Om, rot, out, i1, j1, k1);
    count_launch(ctx, "k_rhs");
    CF_CUDA(cudaGetLastError());
    return 0;
}

template <typename T>
int launch_rhs(cf_ctx *ctx, int comp, int slot) {
    if constexpr (sizeof(T) == 8) {
        if (int rc = launch_nut_materialize<double>(ctx)) return rc;
        return launch_rhs64_comp(ctx, comp, slot);
    } else {
        return rhs_launch<T>(ctx, comp, slot);
    }
}

template <typename T>
int launch_rhs_update(cf_ctx *ctx, int s, int src, int dst) {
    if constexpr (sizeof(T) == 8) {
        if (int rc = launch_rhs64(ctx, ctx->st, s, src, dst)) return rc;
        count_launch(ctx, "k_rhs64");
        return 0;
    } else {
        return launch_rhs32(ctx, s, src, dst);
    }
}

// RK update from stored slots (time_integration.f90:108-146), U = Uo + dt*sum
template <typename T>
__global__ void k_rk_update(Fld<T> U, Fld<T> Uo, Fld<T> F1, Fld<T> F2, Fld<T> F3, const DevScal *ds, int s, RkCoef rk,
                            int i1, int j1, int k1) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
    int k = blockIdx.z + 2;
    if (i > i1 || j > j1 || k > k1) return;
    // rk_coef(3,2) = 0 (initialization.f90:416); the order of the fused update
    const double dt = ds->dt, uo = (double)Uo(i, j, k), f1 = (double)F1(i, j, k);
    double u;
    if (s == 1) u = fma(dt * rk.c[1][1], f1, uo);
    else if (s == 2) u = fma(dt * rk.c[2][1], f1, fma(dt * rk.c[2][2], (double)F2(i, j, k), uo));
    else u = fma(dt * rk.c[3][1], f1, fma(dt * rk.c[3][3], (double)F3(i, j, k), uo));
    U(i, j, k) = (T)u;
}

template <typename T>
int launch_rk_update(cf_ctx *ctx, int s) {
    RkCoef rk = rk_coefs();
    for (int comp = 0; comp < 3; comp++) {
        int i1, j1, k1, n1, n2;
        if (comp == 0) { i1 = ctx->nx - 1; j1 = ctx->nyg - 1; k1 = ctx->nzg - 1; n1 = ctx->nx; n2 = ctx->nyg; }
        else if (comp == 1) { i1 = ctx->nxg - 1; j1 = ctx->ny - 1; k1 = ctx->nzg - 1; n1 = ctx->nxg; n2 = ctx->ny; }
        else { i1 = ctx->nxg - 1; j1 = ctx->nyg - 1; k1 = ctx->nz - 1; n1 = ctx->nxg; n2 = ctx->nyg; }
        void **cur = comp == 0 ? ctx->U : comp == 1 ? ctx->V : ctx->W;
        Fld<T> U = make_fld<T>(cur[ctx->cur], n1, n2), Uo = make_fld<T>(cur[ctx->old], n1, n2);
        Fld<T> F1 = make_fld<T>(ctx->F[0][comp], n1, n2), F2 = make_fld<T>(ctx->F[1][comp], n1, n2),
               F3 = make_fld<T>(ctx->F[2][comp], n1, n2);
        dim3 blk(32, 4, 1), grd(cdiv(i1 - 1, 32), cdiv(j1 - 1, 4), k1 - 1);
        k_rk_update<T><<<grd, blk, 0, ctx->st>>>(U, Uo, F1, F2, F3, ctx->ds, s, rk, i1, j1, k1);
        count_launch(ctx, "k_rk_update");
    }
    CF_CUDA(cudaGetLastError());
    return 0;
}

template <typename T>
__global__ void k_copy(const T *a, T *b, long n) {
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) b[t] = a[t];
}

template <typename T>
int launch_copy_state(cf_ctx *ctx, int src, int dst) {
    size_t n[3] = {ctx->nU, ctx->nV, ctx->nW};
    void **f[3] = {ctx->U, ctx->V, ctx->W};
    void **lo[3] = {ctx->Ulo, ctx->Vlo, ctx->Wlo};
    for (int c = 0; c < 3; c++) {
        CF_CUDA(cudaMemcpyAsync(f[c][dst], f[c][src], n[c] * sizeof(T), cudaMemcpyDeviceToDevice, ctx->st));
        if (lo[c][src] && lo[c][dst])
            CF_CUDA(cudaMemcpyAsync(lo[c][dst], lo[c][src], n[c] * sizeof(T), cudaMemcpyDeviceToDevice, ctx->st));
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Mass flow, mass_flow.f90.  Block partial sums + a fixed-order final sum so
// the result does not depend on scheduling.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffff, v, o);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) r += sh[q];
    __syncthreads();
    return r;
}

// mode 1: trapezoid of U (mass_flow.f90:116-123):
//   sum_{j=3}^{nyg-1} (U_j + U_{j-1}) (yg_j - yg_{j-1})/2 = sum_j c_j sum_i U_ij
// with c_j the two adjacent half-intervals.  Block (k plane, MASS_JR rows),
// one warp per row at a time: the row sum over i is accumulated
// compensated (hi + lo TwoSum) in the state's precision, so that the FP64
// work is one multiply-add per row.
constexpr int MASS_JR = 16;
template <typename T>
__global__ void __launch_bounds__(256) k_mass_partial(Fld<T> U, const double *yg, int nx, int nyg, double *part) {
    __shared__ double sh[8];
    const int k = blockIdx.x + 2, j0 = 2 + blockIdx.y * MASS_JR;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double acc = 0.0;
    for (int r = wp; r < MASS_JR; r += nw) {
        const int j = j0 + r;
        if (j > nyg - 1) break;
        double rsum;
        if constexpr (sizeof(T) == 4) {
            // lanes and the warp tree in float-float: no FP64 per element or per lane
            float hi = 0.f, lo = 0.f;
#pragma unroll 8
            for (int i = lane + 2; i <= nx - 1; i += 32) ff_add(hi, lo, U(i, j, k));
            for (int o = 16; o > 0; o >>= 1) {
                const float oh = __shfl_down_sync(0xffffffffu, hi, o), ol = __shfl_down_sync(0xffffffffu, lo, o);
                ff_add(hi, lo, oh);
                lo += ol;
            }
            rsum = (double)hi + (double)lo;
        } else {
            rsum = 0.0;
#pragma unroll 8
            for (int i = lane + 2; i <= nx - 1; i += 32) rsum += U(i, j, k);
            for (int o = 16; o > 0; o >>= 1) rsum += __shfl_down_sync(0xffffffffu, rsum, o);
        }
        if (lane == 0) {
            const double c = (j >= 3 ? 0.5 * (yg[j] - yg[j - 1]) : 0.0) + (j <= nyg - 2 ? 0.5 * (yg[j + 1] - yg[j]) : 0.0);
            acc += c * rsum;
        }
    }
    if (lane == 0) sh[wp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < nw; q++) s += sh[q];
        part[blockIdx.x * gridDim.y + blockIdx.y] = s;
    }
}

// mode 1 in the split path, with no FP64 instruction per row or warp (each
// is dozens of times the cost of an FP32 one on this part): the row sum over
// i in float-float, times c_j held as float hi + lo, accumulated per warp and
// per block in float-float; one float-float partial per block.
__global__ void __launch_bounds__(256) k_mass_partial_ff(Fld<float> U, const float2 *cj, int nx, int nyg, float2 *part) {
    __shared__ float2 sh[8];
    const int k = blockIdx.x + 2, j0 = 2 + blockIdx.y * MASS_JR;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float ah = 0.f, al = 0.f;
    for (int r = wp; r < MASS_JR; r += nw) {
        const int j = j0 + r;
        if (j > nyg - 1) break;
        float hi = 0.f, lo = 0.f;
        // the row's loads issued MP at a time before they are summed (a
        // dependent sum per load would wait out the memory latency each time)
        constexpr int MP = 8;
        for (int i0 = lane + 2; i0 <= nx - 1; i0 += 32 * MP) {
            float v[MP];
#pragma unroll
            for (int q = 0; q < MP; q++) v[q] = i0 + 32 * q <= nx - 1 ? U(i0 + 32 * q, j, k) : 0.f;
#pragma unroll
            for (int q = 0; q < MP; q++)
                if (i0 + 32 * q <= nx - 1) ff_add(hi, lo, v[q]);
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float oh = __shfl_down_sync(0xffffffffu, hi, o), ol = __shfl_down_sync(0xffffffffu, lo, o);
            ff_add(hi, lo, oh);
            lo += ol;
        }
        // lane 0: (hi + lo) * (c.x + c.y), the product's rounding error
        // recovered by an FMA
        const float2 c = cj[j];
        const float p = c.x * hi;
        const float e = fmaf(c.x, hi, -p) + (c.x * lo + c.y * hi);
        ff_add2(ah, al, p, e);
    }
    if (lane == 0) sh[wp] = make_float2(ah, al);
    __syncthreads();
    if (threadIdx.x == 0) {
        float h = 0.f, l = 0.f;
        for (int q = 0; q < nw; q++) ff_add2(h, l, sh[q].x, sh[q].y);
        part[blockIdx.x * gridDim.y + blockIdx.y] = make_float2(h, l);
    }
}

// its final: the float-float partials summed in a fixed order (lane-strided,
// warp tree, block tree), the correction of mode 1 in FP64 by one thread
__global__ void __launch_bounds__(256) k_mass_final_ff(const float2 *part, int n, DevScal *ds, double norm) {
    __shared__ float2 sh[8];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float h = 0.f, l = 0.f;
    for (int q = threadIdx.x; q < n; q += blockDim.x) ff_add2(h, l, part[q].x, part[q].y);
    for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_down_sync(0xffffffffu, h, o), ol = __shfl_down_sync(0xffffffffu, l, o);
        ff_add2(h, l, oh, ol);
    }
    if (lane == 0) sh[wp] = make_float2(h, l);
    __syncthreads();
    if (threadIdx.x != 0) return;
    h = 0.f;
    l = 0.f;
    for (int q = 0; q < nw; q++) ff_add2(h, l, sh[q].x, sh[q].y);
    const double s = (double)h + (double)l;
    ds->mass_sum = s;
    const double corr = ds->Qflow_x_0 - s / norm;
    ds->lmax[2] = corr;  // scratch slot: correction before division by dt
    ds->corrf = (float)corr;
}

// mode 2: centre-line sum (mass_flow.f90:203-204), planes k = 1..nzg-2
template <typename T>
__global__ void k_ucl_partial(Fld<T> U, int nx, int jc, double *part) {
    __shared__ double sh[32];
    int k = blockIdx.x + 1;
    double s = 0.0;
    for (int i = threadIdx.x + 1; i <= nx - 2; i += blockDim.x) s += (double)U(i, jc, k);
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// mode 3: trapezoid of V (mass_flow.f90:160-167)
template <typename T>
__global__ void k_massv_partial(Fld<T> V, const double *y, int nxg, int ny, double *part) {
    __shared__ double sh[32];
    int k = blockIdx.x + 2;
    double s = 0.0;
    int ni = nxg - 2, nj = ny - 1;
    for (int t = threadIdx.x; t < ni * nj; t += blockDim.x) {
        int i = t % ni + 2, j = t / ni + 2;
        s += ((double)V(i, j, k) + (double)V(i, j - 1, k)) * 0.5 * (y[j] - y[j - 1]);
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// final: the correction into ds (mass_flow.f90:130, 174, 209); the
// partials are summed in a fixed order (lane-strided, then the block tree)
__global__ void __launch_bounds__(256) k_mass_final(const double *part, int n, DevScal *ds, int mode, double norm) {
    __shared__ double sh[32];
    double s = 0.0;
    for (int q = threadIdx.x; q < n; q += blockDim.x) s += part[q];
    s = block_sum(s, sh);
    if (threadIdx.x != 0) return;
    ds->mass_sum = s;
    double corr;
    if (mode == 1) corr = ds->Qflow_x_0 - s / norm;
    else if (mode == 2) corr = ds->Ucenterline_x - s / norm;
    else corr = ds->Qflow_y_0 - s / norm;
    ds->lmax[2] = corr;  // scratch slot: correction before division by dt
    ds->corrf = (float)corr;
}

// add the correction to the interior and store dPdx = corr/dt
// (time_integration.f90:154-156, 159-161, 167-169)
// KP planes per thread, every load issued before the first store
constexpr int MASS_KP = 4;
// i0 = 2: interior only (i0..i1, i0..j1, i0..k1).  i0 = 1: the whole array,
// ghosts included, as apply_boundary_conditions would leave it afterwards:
// +c on the rows 2..j1 (periodic copies included) and wsign*c on the wall
// ghost rows 1 and j1+1 (-1: no-slip ghosts of U, 0: the wall faces of V).
template <typename T>
__global__ void __launch_bounds__(128) k_mass_apply(Fld<T> F, Fld<T> Flo, DevScal *ds, int i1, int j1, int k1, int mode,
                                                    int i0, int wsign) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + i0;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + i0;
    const int k0 = blockIdx.z * MASS_KP + i0;
    if (i == i0 && j == i0 && k0 == i0) {
        double corr = ds->lmax[2];
        if (mode == 3) ds->dPdy = corr / ds->dt;
        else {
            ds->dPdx = corr / ds->dt;
            ds->dPdxf = (float)ds->dPdx;
        }
    }
    if (i > i1 || j > j1) return;
    const bool wall = i0 == 1 && (j == 1 || j == j1);
    if (wall && wsign == 0) return;
    T h[MASS_KP], l[MASS_KP];
    const bool lo = Flo.p != nullptr;
#pragma unroll
    for (int q = 0; q < MASS_KP; q++) {
        const int k = k0 + q;
        h[q] = k <= k1 ? F(i, j, k) : T(0);
        l[q] = (lo && k <= k1) ? Flo(i, j, k) : T(0);
    }
    if constexpr (sizeof(T) == 4) {
        const float c = wall ? -ds->corrf : ds->corrf;
#pragma unroll
        for (int q = 0; q < MASS_KP; q++) {
            const int k = k0 + q;
            if (k > k1) break;
            if (lo) {
                float hi = h[q], lw = l[q];
                ff_add(hi, lw, c);
                F(i, j, k) = hi;
                Flo(i, j, k) = lw;
            } else {
                F(i, j, k) = h[q] + c;
            }
        }
    } else {
        const double c = wall ? -ds->lmax[2] : ds->lmax[2];
#pragma unroll
        for (int q = 0; q < MASS_KP; q++)
            if (k0 + q <= k1) F(i, j, k0 + q) = h[q] + c;
    }
}

template <typename T>
static int mass_partial(cf_ctx *ctx, int b, int mode) {
    double *part = ctx->d_red;
    int nb = ctx->nzg - 2;
    double norm;
    if (mode == 1 && sizeof(T) == 4) {
        const int njc = cdiv(ctx->nyg - 2, MASS_JR);
        k_mass_partial_ff<<<dim3(nb, njc), 256, 0, ctx->st>>>(make_fld<float>(ctx->U[b], ctx->nx, ctx->nyg),
                                                               ctx->d_mass_c, ctx->nx, ctx->nyg, (float2 *)part);
        count_launch(ctx, "k_mass_partial");
        k_mass_final_ff<<<1, 256, 0, ctx->st>>>((const float2 *)part, nb * njc, ctx->ds, ctx->mass_norm);
        count_launch(ctx, "k_mass_final");
        CF_CUDA(cudaGetLastError());
        return 0;
    }
    if (mode == 1) {
        const int njc = cdiv(ctx->nyg - 2, MASS_JR);
        k_mass_partial<T><<<dim3(nb, njc), 256, 0, ctx->st>>>(make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg), ctx->geo.yg,
                                                               ctx->nx, ctx->nyg, part);
        nb *= njc;
        norm = ctx->mass_norm;
    } else if (mode == 2) {
        int jc = ctx->ny / 2 + 1;
        k_ucl_partial<T><<<nb, 256, 0, ctx->st>>>(make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg), ctx->nx, jc, part);
        norm = (double)(ctx->nx - 2) * (double)(ctx->nzg - 2);
    } else {
        k_massv_partial<T><<<nb, 256, 0, ctx->st>>>(make_fld<T>(ctx->V[b], ctx->nxg, ctx->ny), ctx->geo.y, ctx->nxg,
                                                     ctx->ny, part);
        norm = ctx->mass_norm_vv;
    }
    count_launch(ctx, "k_mass_partial");
    k_mass_final<<<1, 256, 0, ctx->st>>>(part, nb, ctx->ds, mode, norm);
    count_launch(ctx, "k_mass_final");
    CF_CUDA(cudaGetLastError());
    return 0;
}

template <typename T>
int launch_mass_value(cf_ctx *ctx, int b, int mode) {
    return mass_partial<T>(ctx, b, mode);
}

template <typename T>
int launch_mass_flow(cf_ctx *ctx, int b, int mode, bool ghosts) {
    int rc = mass_partial<T>(ctx, b, mode);
    if (rc) return rc;
    return launch_mass_apply<T>(ctx, b, mode, ghosts);
}

template <typename T>
int launch_mass_apply(cf_ctx *ctx, int b, int mode, bool ghosts) {
    dim3 blk(32, 4, 1);
    if (mode == 3) {
        if (ghosts) {
            int i1 = ctx->nxg, j1 = ctx->ny, k1 = ctx->nzg;
            k_mass_apply<T><<<dim3(cdiv(i1, 32), cdiv(j1, 4), cdiv(k1, MASS_KP)), blk, 0, ctx->st>>>(
                make_fld<T>(ctx->V[b], ctx->nxg, ctx->ny), make_fld<T>(ctx->Vlo[b], ctx->nxg, ctx->ny), ctx->ds, i1, j1,
                k1, mode, 1, 0);
        } else {
            int i1 = ctx->nxg - 1, j1 = ctx->ny - 1, k1 = ctx->nzg - 1;
            k_mass_apply<T><<<dim3(cdiv(i1 - 1, 32), cdiv(j1 - 1, 4), cdiv(k1 - 1, MASS_KP)), blk, 0, ctx->st>>>(
                make_fld<T>(ctx->V[b], ctx->nxg, ctx->ny), make_fld<T>(ctx->Vlo[b], ctx->nxg, ctx->ny), ctx->ds, i1, j1,
                k1, mode, 2, 0);
        }
    } else {
        if (ghosts) {
            int i1 = ctx->nx, j1 = ctx->nyg, k1 = ctx->nzg;
            k_mass_apply<T><<<dim3(cdiv(i1, 32), cdiv(j1, 4), cdiv(k1, MASS_KP)), blk, 0, ctx->st>>>(
                make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg), make_fld<T>(ctx->Ulo[b], ctx->nx, ctx->nyg), ctx->ds, i1, j1,
                k1, mode, 1, -1);
        } else {
            int i1 = ctx->nx - 1, j1 = ctx->nyg - 1, k1 = ctx->nzg - 1;
            k_mass_apply<T><<<dim3(cdiv(i1 - 1, 32), cdiv(j1 - 1, 4), cdiv(k1 - 1, MASS_KP)), blk, 0, ctx->st>>>(
                make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg), make_fld<T>(ctx->Ulo[b], ctx->nx, ctx->nyg), ctx->ds, i1, j1,
                k1, mode, 2, 0);
        }
    }
    count_launch(ctx, "k_mass_apply");
    CF_CUDA(cudaGetLastError());
    return 0;
}

// ---------------------------------------------------------------------------
// compute_dt, time_integration.f90:179-227.  max over (i,j,k) of dx_i/|U| is
// dx_i / min_{j,k}|U| exactly (division by a positive number is monotone), so
// the kernel reduces min|U| per x index, min|V| per y index, min|W| per z
// index and a second kernel forms the maxima.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void atomic_min_pos(double *a, double v) {
    // non-negative doubles order like their bit patterns
    atomicMin((unsigned long long *)a, (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ void atomic_max_pos(double *a, double v) {
    atomicMax((unsigned long long *)a, (unsigned long long)__double_as_longlong(v));
}

// CORR: the corrected convective limit of cf_params.cfl_corrected, which
// needs the maxima of |u| per index instead (same blocks and atomics).  The
// extrema are kept in the state's precision: FP32 ones as the bit patterns of
// non-negative floats (which order like unsigned integers) with 32-bit
// atomics, FP64 ones as 64-bit patterns; widening a float to double is exact,
// so the quotients of the finaliser do not depend on the storage.
template <typename T, bool CORR>
__global__ void __launch_bounds__(256) k_dt_min(Fld<T> U, Fld<T> V, Fld<T> W, int nxg, int nyg, int nzg, T *mu, T *mv,
                                                T *mw) {
    // block (x: up to 256 x indices, y: JR rows, z: KR planes), thread = x index i:
    // min |U| per i over the block's rows
    // and planes, min |V| per row, min |W| per plane; all loads of a plane's
    // rows are issued together.  One global atomic per index per block.
    constexpr int JR = 16, KR = 2;
    __shared__ T vsm[8][JR];
    __shared__ T wsm[8][KR];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int i = 2 + blockIdx.x * blockDim.x + threadIdx.x, j0 = 2 + blockIdx.y * JR, k0 = 2 + blockIdx.z * KR;
    const T init = CORR ? T(0) : T(INFINITY);
    auto ext = [](T a, T b) { return CORR ? fmax(a, b) : fmin(a, b); };
    T umin = init;
    T vmin[JR];
#pragma unroll
    for (int r = 0; r < JR; r++) vmin[r] = init;
#pragma unroll
    for (int kk = 0; kk < KR; kk++) {
        const int k = k0 + kk;
        T wmin = init;
        if (k <= nzg - 1 && i <= nxg - 1) {
            T u[JR], v[JR], w[JR];
#pragma unroll
            for (int r = 0; r < JR; r++) {
                const int j = min(j0 + r, nyg - 1);  // clamped rows repeat row nyg-1
                u[r] = U(i, j, k);
                v[r] = V(i, j, k);
                w[r] = W(i, j, k);
            }
#pragma unroll
            for (int r = 0; r < JR; r++) {
                umin = ext(umin, fabs(u[r]));
                vmin[r] = ext(vmin[r], fabs(v[r]));
                wmin = ext(wmin, fabs(w[r]));
            }
        }
        for (int o = 16; o > 0; o >>= 1) wmin = ext(wmin, __shfl_down_sync(0xffffffff, wmin, o));
        if (lane == 0) wsm[wp][kk] = wmin;
    }
#pragma unroll
    for (int r = 0; r < JR; r++) {
        T v = vmin[r];
        for (int o = 16; o > 0; o >>= 1) v = ext(v, __shfl_down_sync(0xffffffff, v, o));
        if (lane == 0) vsm[wp][r] = v;
    }
    auto put = [](T *a, T v) {
        if constexpr (sizeof(T) == 4) {
            if (CORR) atomicMax((unsigned *)a, __float_as_uint(v));
            else atomicMin((unsigned *)a, __float_as_uint(v));
        } else {
            if (CORR) atomic_max_pos(a, v);
            else atomic_min_pos(a, v);
        }
    };
    if (i <= nxg - 1) put(&mu[i], umin);
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (threadIdx.x < JR) {
        const int j = j0 + threadIdx.x;
        if (j <= nyg - 1) {
            T m = vsm[0][threadIdx.x];
            for (int q = 1; q < nw; q++) m = ext(m, vsm[q][threadIdx.x]);
            put(&mv[j], m);
        }
    } else if (threadIdx.x < JR + KR) {  // JR + KR <= 32: present in a one-warp block too
        const int kk = threadIdx.x - JR, k = k0 + kk;
        if (k <= nzg - 1) {
            T m = wsm[0][kk];
            for (int q = 1; q < nw; q++) m = ext(m, wsm[q][kk]);
            put(&mw[k], m);
        }
    }
}


// The maxima dx/min|u| per direction (one FP64 quotient per thread), dt, and
// the minima reset to +inf for the next call.  corr: the minima dx/max|u|
// instead, the maxima reset to 0.  The quotients are non-negative, so their
// extrema are taken on the 64-bit patterns with integer compares (FP64
// max/min chains are slow on this part); a NaN quotient is skipped like
// fmax/fmin skip it.
template <typename T>
__global__ void __launch_bounds__(1024) k_dt_final(T *mu, T *mv, T *mw, Geo g, DevScal *ds, double CFL, double dt_vis,
                                                   int corr, int advance_t) {
    typedef unsigned long long u64;
    __shared__ u64 sh[3][32];
    const int nxi = g.nxg - 2, nyi = g.nyg - 2, nzi = g.nzg - 2;
    const u64 pinf = 0x7FF0000000000000ull;
    const u64 init = corr ? pinf : 0ull;
    auto ext = [corr](u64 a, u64 b) { return corr ? (a < b ? a : b) : (a > b ? a : b); };
    auto key = [init, pinf](double q) {
        const u64 b = (u64)__double_as_longlong(q);
        return b > pinf ? init : b;
    };
    u64 l[3] = {init, init, init};
    for (int t = threadIdx.x; t < nxi + nyi + nzi; t += blockDim.x) {
        if (t < nxi) {
            const int i = t + 2;
            l[0] = ext(l[0], key((g.xg[i + 1] - g.xg[i]) / (double)mu[i]));
        } else if (t < nxi + nyi) {
            const int j = t - nxi + 2;
            l[1] = ext(l[1], key((g.yg[j + 1] - g.yg[j]) / (double)mv[j]));
        } else {
            const int k = t - nxi - nyi + 2;
            l[2] = ext(l[2], key((g.zg[k + 1] - g.zg[k]) / (double)mw[k]));
        }
    }
#pragma unroll
    for (int d = 0; d < 3; d++)
        for (int o = 16; o > 0; o >>= 1) l[d] = ext(l[d], __shfl_down_sync(0xffffffff, l[d], o));
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { sh[0][w] = l[0]; sh[1][w] = l[1]; sh[2][w] = l[2]; }
    __syncthreads();
    const T reset = corr ? T(0) : T(INFINITY);
    for (int t = threadIdx.x; t < g.nxg + 2; t += blockDim.x) mu[t] = reset;
    for (int t = threadIdx.x; t < g.nyg + 2; t += blockDim.x) mv[t] = reset;
    for (int t = threadIdx.x; t < g.nzg + 2; t += blockDim.x) mw[t] = reset;
    if (w != 0) return;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        u64 x = lane < nw ? sh[d][lane] : init;
        for (int o = 16; o > 0; o >>= 1) x = ext(x, __shfl_down_sync(0xffffffff, x, o));
        l[d] = x;
    }
    if (lane != 0) return;
    const double lU = __longlong_as_double((long long)l[0]), lV = __longlong_as_double((long long)l[1]),
                 lW = __longlong_as_double((long long)l[2]);
    double du = CFL * lU, dv = CFL * lV, dw = CFL * lW;
    double dt_conv = fmin(du, fmin(dv, dw));
    double dt = fmin(dt_conv, dt_vis);
    dt = fmin(dt, 5e-3);
    if (CFL < 0) dt = -CFL;
    if (ds->fixed_dt > 0) dt = ds->fixed_dt;
    ds->dt = dt;
    ds->dtf = (float)dt;
    // the step's t = to + rk_t(3) dt, rk_t(3) = 1 (time_integration.f90:146);
    // nothing in the step reads t
    if (advance_t) ds->t = ds->t + dt;
    ds->lmax[0] = lU;
    ds->lmax[1] = lV;
}

template <typename T>
int launch_dt(cf_ctx *ctx, int b, bool advance_t) {
    // extrema start at +inf (0 for the corrected rule): set at context
    // creation and reset by k_dt_final; stored in the state's precision
    T *mu = (T *)ctx->d_dtmin, *mv = mu + ctx->nxg + 2, *mw = mv + ctx->nyg + 2;
    // blocks as wide as the x range (whole warps, at most 256 threads): no
    // idle threads, and more of the small blocks resident at once
    const int bx = std::min(256, 32 * cdiv(ctx->nxg - 2, 32));
    const dim3 grd(cdiv(ctx->nxg - 2, bx), cdiv(ctx->nyg - 2, 16), cdiv(ctx->nzg - 2, 2));
    const Fld<T> U = make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg), V = make_fld<T>(ctx->V[b], ctx->nxg, ctx->ny),
                 W = make_fld<T>(ctx->W[b], ctx->nxg, ctx->nyg);
    if (ctx->prm.cfl_corrected) k_dt_min<T, true><<<grd, bx, 0, ctx->st>>>(U, V, W, ctx->nxg, ctx->nyg, ctx->nzg, mu, mv, mw);
    else k_dt_min<T, false><<<grd, bx, 0, ctx->st>>>(U, V, W, ctx->nxg, ctx->nyg, ctx->nzg, mu, mv, mw);
    count_launch(ctx, "k_dt_min");
    double CFL = ctx->prm.CFL;
    double vu = CFL * pow(ctx->dxmin, 2.0) / ctx->prm.nu, vv = CFL * pow(ctx->dymin, 2.0) / ctx->prm.nu,
           vw = CFL * pow(ctx->dzmin, 2.0) / ctx->prm.nu;
    double dt_vis = fmin(vu, fmin(vv, vw));
    k_dt_final<T><<<1, 1024, 0, ctx->st>>>(mu, mv, mw, ctx->geo, ctx->ds, CFL, dt_vis, ctx->prm.cfl_corrected ? 1 : 0,
                                           advance_t ? 1 : 0);
    count_launch(ctx, "k_dt_final");
    CF_CUDA(cudaGetLastError());
    return 0;
}

// ---------------------------------------------------------------------------
// check_divergence, projection.f90:234-256 (signed max from 0, and max |div|)
// ---------------------------------------------------------------------------

// A NaN divergence in any cell makes both results NaN (a blown-up field is
// reported as such; fmax alone would drop it).  The NaN is the positive
// quiet one, whose bit pattern orders above +Inf for atomic_max_pos.
__device__ __forceinline__ double nan_max(double a, double b) {
    return (isnan(a) || isnan(b)) ? __longlong_as_double(0x7FF8000000000000LL) : fmax(a, b);
}

template <typename T>
__global__ void k_div(Fld<T> U, Fld<T> V, Fld<T> W, Geo g, double *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
    int k = blockIdx.z + 2;
    double d = 0.0, a = 0.0;
    if (i <= g.nxg - 1 && j <= g.nyg - 1) {
        d = ((double)U(i, j, k) - (double)U(i - 1, j, k)) / (g.x[i] - g.x[i - 1]) +
            ((double)V(i, j, k) - (double)V(i, j - 1, k)) / (g.y[j] - g.y[j - 1]) +
            ((double)W(i, j, k) - (double)W(i, j, k - 1)) / (g.z[k] - g.z[k - 1]);
        a = nan_max(fabs(d), 0.0);
        d = nan_max(d, 0.0);
    }
    for (int o = 16; o > 0; o >>= 1) {
        d = nan_max(d, __shfl_down_sync(0xffffffff, d, o));
        a = nan_max(a, __shfl_down_sync(0xffffffff, a, o));
    }
    if (((threadIdx.x + threadIdx.y * blockDim.x) & 31) == 0) {
        atomic_max_pos(&out[0], d);
        atomic_max_pos(&out[1], a);
    }
}

template <typename T>
int launch_div_check(cf_ctx *ctx, int b, double *d_out) {
    CF_CUDA(cudaMemsetAsync(d_out, 0, 2 * sizeof(double), ctx->st));
    dim3 blk(32, 4, 1), grd(cdiv(ctx->nxg - 2, 32), cdiv(ctx->nyg - 2, 4), ctx->nzg - 2);
    k_div<T><<<grd, blk, 0, ctx->st>>>(make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg), make_fld<T>(ctx->V[b], ctx->nxg, ctx->ny),
                                       make_fld<T>(ctx->W[b], ctx->nxg, ctx->nyg), ctx->geo, d_out);
    count_launch(ctx, "k_div");
    CF_CUDA(cudaGetLastError());
    return 0;
}

#define INST(T)                                                      \
    template int launch_bc<T>(cf_ctx *, int, bool);                  \
    template int launch_rhs<T>(cf_ctx *, int, int);                  \
    template int launch_rhs_update<T>(cf_ctx *, int, int, int);      \
    template int launch_rk_update<T>(cf_ctx *, int);                 \
    template int launch_copy_state<T>(cf_ctx *, int, int);           \
    template int launch_mass_flow<T>(cf_ctx *, int, int, bool);      \
    template int launch_mass_value<T>(cf_ctx *, int, int);           \
    template int launch_mass_apply<T>(cf_ctx *, int, int, bool);     \
    template int launch_dt<T>(cf_ctx *, int, bool);                  \
    template int launch_div_check<T>(cf_ctx *, int, double *);
INST(double)
INST(float)
