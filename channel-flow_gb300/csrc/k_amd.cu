// k_amd.cu -- anisotropic minimum dissipation eddy viscosity,
// subgrid.f90:639-881, in one pass (FP64; the split path's is in k_amd32.cu).
//
// The reference builds the model from whole-array and array-section
// operations on the temporaries term, term_1..term_4 (squared or plain
// velocity differences, each moved to the cell centre by two or three
// interpolate_x/_y/_z calls of interpolation.f90:24-105).  At a canonical
// centre (i = 2..nx-1, j = 2..nyg-1, k = 2..nz-1) every one of those
// operations reduces to 27 differences of U, V, W in the cell's 3x3x3
// neighbourhood, combined with weights 1/2; the kernel evaluates that
// reduced form per cell in the order the reference accumulates it.  The
// values the reference computes outside the canonical cells are all
// overwritten by its periodic copies and the wall rule (subgrid.f90:873-876),
// so each canonical value is also written to the duplicate and ghost
// positions that copy it.
//
// A block owns a TX x TY tile of (i, j) columns and marches along z over a
// chunk of planes with planes k, k+1 of U, V, W (tile plus one halo cell) in
// a shared-memory ring of three, the third being filled; what a cell takes
// from plane k-1 is carried up the march.  Bound by its FP64 instructions:
// 6.37 ms a launch at 192 x 128 x 192 cells with 850 a cell, 1.27 ms now.
#include "cf_internal.cuh"

namespace {

constexpr int AMD_TX = 32, AMD_TY = 8;

struct AmdRing {
    static constexpr int SX = AMD_TX + 2;
    const double *b[2];  // planes k, k+1
    int i0, j0, kc;
    __device__ __forceinline__ double operator()(int i, int j, int k) const {
        return b[k - kc][(j - j0 + 1) * SX + (i - i0 + 1)];
    }
};

// What a cell takes from the plane below: sums and sums of squares of the z
// differences of U and V through the face below it, W there and its x and y
// differences.
struct AmdCarry {
    double puz, quz, pvz, qvz, w, wx[2], wy[2];
};

// Reciprocal spacings of one column and plane and their squares: faces (x, y,
// z: the cell's own spacing) and centres on its two sides (g0 below, g1 above).
struct AmdGeo {
    double x, y, z, xg[2], yg[2], zg[2];
    double x2, y2, z2, xg2[2], yg2[2], zg2[2];
};

// -C num/den at one canonical centre (subgrid.f90:658-868), clipped with
// NaN -> 0 (subgrid.f90:871).  Differences, with a, b, c in {0, 1}:
//   ux = U(i)-U(i-1);  uy[a][b] = U(i+a-1, j+b) - U(i+a-1, j+b-1);
//   uz[a][c] = U(i+a-1, k+c) - U(i+a-1, k+c-1);  vy = V(j)-V(j-1);
//   vx[a][b] = V(i+a, j+b-1) - V(i+a-1, j+b-1);  vz[b][c] = V(j+b-1, k+c) - V(j+b-1, k+c-1);
//   wz = W(k)-W(k-1);  wx[a][c] = W(i+a, k+c-1) - W(i+a-1, k+c-1);
//   wy[b][c] = W(j+b, k+c-1) - W(j+b-1, k+c-1).
// The reference only ever combines the two differences of one side (the two
// faces of their component) as their sum (p) and the sum of their squares
// (q); every term is formed from these twelve pairs:
//   8 S12 = p(uy,0) ryg0 + p(uy,1) ryg1 + p(vx,0) rxg0 + p(vx,1) rxg1 (compute_Sij, subgrid.f90:891-949),
//   den = (d r)^2 of the diagonal ones + 1/4 sum q r^2 of the others (subgrid.f90:662-763),
//   num: S11 (ux^2 + 1/4 (q(uy) + q(uz))) and its like, and
//   2 S12 (1/4 (p(vx) ux + p(uy) vy) + 1/8 (p(uz,0) p(vz,0) + p(uz,1) p(vz,1))) and its like
//   (subgrid.f90:660-866).
// About 140 operations a cell; the spacing quotients are products with
// reciprocals formed once (54 of them per cell: as FP64 divisions they were
// three quarters of the FP64 instructions, and FP64 instructions are what
// the FP64 pass is bound by).
__device__ __forceinline__ void amd_pair(double a, double b, double &p, double &q) {
    p = a + b;
    q = a * a + b * b;
}
// the carry for plane k + 1
__device__ __forceinline__ void amd_carry(const AmdRing &U, const AmdRing &V, const AmdRing &W, int i, int j, int k, AmdCarry &c) {
    amd_pair(U(i - 1, j, k + 1) - U(i - 1, j, k), U(i, j, k + 1) - U(i, j, k), c.puz, c.quz);
    amd_pair(V(i, j - 1, k + 1) - V(i, j - 1, k), V(i, j, k + 1) - V(i, j, k), c.pvz, c.qvz);
    c.w = W(i, j, k);
#pragma unroll
    for (int s = 0; s < 2; s++) {
        c.wx[s] = W(i + s, j, k) - W(i + s - 1, j, k);
        c.wy[s] = W(i, j + s, k) - W(i, j + s - 1, k);
    }
}
__device__ __forceinline__ double amd_point(const AmdGeo &g, const AmdRing &U, const AmdRing &V, const AmdRing &W, AmdCarry &c,
                                            int i, int j, int k) {
    typedef double T;
    const T q4 = T(0.25), two = T(2);
    const AmdCarry m = c;
    amd_carry(U, V, W, i, j, k, c);
    const T ux = U(i, j, k) - U(i - 1, j, k);
    const T vy = V(i, j, k) - V(i, j - 1, k);
    const T wz = c.w - m.w;
    // sums and sums of squares of the two differences of each side
    T puy[2], pvx[2], pwx[2], pwy[2], quy[2], qvx[2], qwx[2], qwy[2];
    const T puz[2] = {m.puz, c.puz}, quz[2] = {m.quz, c.quz}, pvz[2] = {m.pvz, c.pvz}, qvz[2] = {m.qvz, c.qvz};
#pragma unroll
    for (int s = 0; s < 2; s++) {
        amd_pair(U(i - 1, j + s, k) - U(i - 1, j + s - 1, k), U(i, j + s, k) - U(i, j + s - 1, k), puy[s], quy[s]);
        amd_pair(V(i + s, j - 1, k) - V(i + s - 1, j - 1, k), V(i + s, j, k) - V(i + s - 1, j, k), pvx[s], qvx[s]);
        amd_pair(m.wx[s], c.wx[s], pwx[s], qwx[s]);
        amd_pair(m.wy[s], c.wy[s], pwy[s], qwy[s]);
    }
    const T ux2 = ux * ux, vy2 = vy * vy, wz2 = wz * wz;
    T den = quy[0] * g.yg2[0] + quy[1] * g.yg2[1] + quz[0] * g.zg2[0] + quz[1] * g.zg2[1] + qvx[0] * g.xg2[0] +
            qvx[1] * g.xg2[1] + qvz[0] * g.zg2[0] + qvz[1] * g.zg2[1] + qwx[0] * g.xg2[0] + qwx[1] * g.xg2[1] +
            qwy[0] * g.yg2[0] + qwy[1] * g.yg2[1];
    den = ux2 * g.x2 + vy2 * g.y2 + wz2 * g.z2 + q4 * den;
    T num = (ux * g.x) * (ux2 + q4 * ((quy[0] + quy[1]) + (quz[0] + quz[1])));
    num += (vy * g.y) * (vy2 + q4 * ((qvx[0] + qvx[1]) + (qvz[0] + qvz[1])));
    num += (wz * g.z) * (wz2 + q4 * ((qwx[0] + qwx[1]) + (qwy[0] + qwy[1])));
    // 8 S_ij of the mixed components times 8 times their factors
    const T t12 = puy[0] * g.yg[0] + puy[1] * g.yg[1] + pvx[0] * g.xg[0] + pvx[1] * g.xg[1];
    const T t13 = puz[0] * g.zg[0] + puz[1] * g.zg[1] + pwx[0] * g.xg[0] + pwx[1] * g.xg[1];
    const T t23 = pvz[0] * g.zg[0] + pvz[1] * g.zg[1] + pwy[0] * g.yg[0] + pwy[1] * g.yg[1];
    const T sUy = puy[0] + puy[1], sUz = puz[0] + puz[1], sVx = pvx[0] + pvx[1], sVz = pvz[0] + pvz[1],
            sWx = pwx[0] + pwx[1], sWy = pwy[0] + pwy[1];
    T off = t12 * (two * (sVx * ux + sUy * vy) + (puz[0] * pvz[0] + puz[1] * pvz[1]));
    off += t13 * (two * (sWx * ux + sUz * wz) + (puy[0] * pwy[0] + puy[1] * pwy[1]));
    off += t23 * (two * (sWy * vy + sVz * wz) + (pvx[0] * pwx[0] + pvx[1] * pwx[1]));
    num += T(1.0 / 32.0) * off;
    const T v = -T(0.3) * num / den;
    return v > T(0) ? v : T(0);
}

// nu_t at the canonical cells and at every duplicate / ghost position that
// the periodic copies (boundary_conditions.f90:87-244) and the wall rule
// (subgrid.f90:866-876) fill from them; one partial sum of the canonical
// values per (row j, block) for avg_nu_t (subgrid.f90:877-879).
__global__ void __launch_bounds__(AMD_TX *AMD_TY, 2) k_amd(GeoT<double> g, RcpT<double> rc, Fld<double> U, Fld<double> V,
                                                            Fld<double> W, Fld<double> nt, int wall_rule,
                                                            const DevScal *ds, double *part, int kc_len) {
    typedef double T;
    constexpr int TX = AMD_TX, TY = AMD_TY, SX = TX + 2, SY = TY + 2, NP = SX * SY, NT = TX * TY;
    constexpr int NL = (NP + NT - 1) / NT;
    __shared__ T ring[3][3][NP];  // [plane slot][field U V W][tile]
    const int nx = g.nx, ny = g.ny, nz = g.nz, nxg = g.nxg, nyg = g.nyg, nzg = g.nzg, nxp = g.nxp, nzp = g.nzp;
    const int i0 = 2 + blockIdx.x * TX, j0 = 2 + blockIdx.y * TY;
    const int kb = 2 + blockIdx.z * kc_len, ke = min(kb + kc_len - 1, nzp + 1);
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int i = i0 + tx, j = j0 + ty;
    const bool on = i <= nxp + 1 && j <= nyg - 1;
    // this column's reciprocal spacings (the last entries of the tables stand
    // in for columns and rows past the field, whose results are not stored)
    AmdGeo ag;
    {
        const int ii = min(i, nx - 1), jj = min(j, nyg - 1);
        ag.x = rc.dx[ii];
        ag.y = rc.dy[jj];
        ag.x2 = ag.x * ag.x;
        ag.y2 = ag.y * ag.y;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            ag.xg[s] = rc.dxg[ii + s];
            ag.yg[s] = rc.dyg[jj + s];
            ag.xg2[s] = ag.xg[s] * ag.xg[s];
            ag.yg2[s] = ag.yg[s] * ag.yg[s];
        }
        ag.zg[1] = rc.dzg[kb];
        ag.zg2[1] = ag.zg[1] * ag.zg[1];
    }
    // wall rule 2: -nu_t(2) + 2 0.38 dPdx^(1/2) (y(2)-y(1))/2
    T add = T(0);
    if (wall_rule == 2) add = (T)(2.0 * 0.38 * sqrt(ds->dPdx) * ((double)g.y[2] - (double)g.y[1]) / 2.0);
    int eia[NL], eja[NL], erem[NL];
#pragma unroll
    for (int qq = 0; qq < NL; qq++) {
        const int rem = threadIdx.x + qq * NT;
        erem[qq] = rem;
        const int sy_ = rem / SX, sx_ = rem - sy_ * SX;
        eia[qq] = i0 + sx_ - 1;
        eja[qq] = j0 + sy_ - 1;
    }
    T pre[3][NL];
    auto fetch = [&](int k) {
#pragma unroll
        for (int qq = 0; qq < NL; qq++) {
            const int ia = eia[qq], ja = eja[qq];
            const bool in = erem[qq] < NP;
            pre[0][qq] = (in && ia <= nx && ja <= nyg && k <= nzg) ? U(ia, ja, k) : T(0);
            pre[1][qq] = (in && ia <= nxg && ja <= ny && k <= nzg) ? V(ia, ja, k) : T(0);
            pre[2][qq] = (in && ia <= nxg && ja <= nyg && k <= nz) ? W(ia, ja, k) : T(0);
        }
    };
    auto commit = [&](int slot) {
#pragma unroll
        for (int qq = 0; qq < NL; qq++)
            if (erem[qq] < NP) {
#pragma unroll
                for (int f = 0; f < 3; f++) ring[slot][f][erem[qq]] = pre[f][qq];
            }
    };
    fetch(kb - 1);
    commit(0);
    fetch(kb);
    commit(1);
    fetch(kb + 1);
    commit(2);
    __syncthreads();
    AmdCarry carry = {};
    if (on) amd_carry({{ring[0][0], ring[1][0]}, i0, j0, kb - 1}, {{ring[0][1], ring[1][1]}, i0, j0, kb - 1},
                      {{ring[0][2], ring[1][2]}, i0, j0, kb - 1}, i, j, kb - 1, carry);
    __syncthreads();  // plane kb-1 no longer read
    // duplicate / ghost images of this column
    const int ix1 = i + nxp <= nxp + 3 ? i + nxp : 0, ix2 = i - nxp >= 1 ? i - nxp : 0;
    const int jg = j == 2 ? 1 : (j == nyg - 1 ? nyg : 0);
    double acc = 0.0;
    int sm1 = 0, s0 = 1, sp1 = 2;
    for (int k = kb; k <= ke; k++) {
        if (k + 1 <= ke) fetch(k + 2);  // in flight during this plane's work
        // the spacings of plane k (the lower centre spacing carried)
        ag.zg[0] = ag.zg[1];
        ag.zg2[0] = ag.zg2[1];
        ag.zg[1] = rc.dzg[k + 1];
        ag.zg2[1] = ag.zg[1] * ag.zg[1];
        ag.z = rc.dz[k];
        ag.z2 = ag.z * ag.z;
        if (on) {
            const T v = amd_point(ag, {{ring[s0][0], ring[sp1][0]}, i0, j0, k}, {{ring[s0][1], ring[sp1][1]}, i0, j0, k},
                                  {{ring[s0][2], ring[sp1][2]}, i0, j0, k}, carry, i, j, k);
            acc += v;
            const T gv = wall_rule == 0 ? v : -v + add;
            const int kz1 = k + nzp <= nzp + 3 ? k + nzp : 0, kz2 = k - nzp >= 1 ? k - nzp : 0;
            const int ixs[3] = {i, ix1, ix2}, kzs[3] = {k, kz1, kz2};
#pragma unroll
            for (int a = 0; a < 3; a++) {
                if (!ixs[a]) continue;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    if (!kzs[c]) continue;
                    nt(ixs[a], j, kzs[c]) = v;
                    if (jg) nt(ixs[a], jg, kzs[c]) = gv;
                }
            }
        }
        if (k + 1 <= ke) commit(sm1);  // plane k+2 into the slot of plane k-1
        __syncthreads();               // plane k no longer read, k+2 in
        const int t0 = sm1;
        sm1 = s0;
        s0 = sp1;
        sp1 = t0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    const int nparts = gridDim.x * gridDim.z;
    if (tx == 0 && j <= nyg - 1) part[(long)(j - 2) * nparts + blockIdx.z * gridDim.x + blockIdx.x] = acc;
}

// avg_nu_t(j) = plane mean of the canonical values, rows 2..nyg-1; rows 1
// and nyg are left as they were (subgrid.f90:877-879).  One warp per row.
__global__ void k_amd_avg(const double *part, int nparts, int nyg, double norm, double *avg) {
    const int lane = threadIdx.x & 31;
    const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5) + 2;
    if (j > nyg - 1) return;
    double a = 0.0;
    for (int qq = lane; qq < nparts; qq += 32) a += part[(long)(j - 2) * nparts + qq];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) {
        const double c = a / norm;
        avg[j] = c;
        ((float *)(avg + nyg + 2))[j] = (float)c;  // FP32 copy
    }
}

}  // namespace

// z chunks of the AMD pass.  FP64: an SM works its blocks off at the FP64
// pipe's rate, so the count that minimises the mean work of an SM (0.1 plane
// extra a chunk) and half a chunk for the uneven end (120 x 81 x 96: 6 chunks
// for one full wave 337 us, 32 to 48 chunks 295 to 299).
void amd_plan(int esz, int nxp, int nym, int nzp, int sms, int *nkc, int *nparts) {
    if (esz == 4) {
        *nkc = amd32_plan(nxp, nym, nzp, sms);
        *nparts = amd32_parts(nxp, nzp, *nkc);
        return;
    }
    const double tiles = (double)cdiv(nxp, AMD_TX) * cdiv(nym, AMD_TY);
    double best_cost = 1e300;
    int best = nzp;
    for (int n = 1; n <= nzp; n++) {
        const int len = cdiv(nzp, n);
        const double cost = tiles * (nzp + 0.1 * cdiv(nzp, len)) / sms + 0.5 * (len + 0.1);
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = len;
        }
    }
    *nkc = cdiv(nzp, best);
    *nparts = cdiv(nxp, AMD_TX) * *nkc;
}

template <typename T>
int launch_amd(cf_ctx *ctx, int b) {
    ctx->nut_lazy = false;
    if constexpr (sizeof(T) == 4) {
        if (int rc = launch_amd32(ctx, b)) return rc;
    } else {
        GeoT<T> g = geo_of<T>(ctx);
        Fld<T> U = make_fld<T>(ctx->U[b], ctx->nx, ctx->nyg);
        Fld<T> V = make_fld<T>(ctx->V[b], ctx->nxg, ctx->ny);
        Fld<T> W = make_fld<T>(ctx->W[b], ctx->nxg, ctx->nyg);
        Fld<T> nt = make_fld<T>(ctx->nut, ctx->nxg, ctx->nyg);
        const int nkc = ctx->amd_nkc, kc_len = cdiv(ctx->nzp, nkc);
        const dim3 grd(cdiv(ctx->nxp, AMD_TX), cdiv(ctx->nym, AMD_TY), nkc);
        k_amd<<<grd, AMD_TX * AMD_TY, 0, ctx->st>>>(g, rcp_of<T>(ctx), U, V, W, nt, ctx->prm.Dirichlet_nu_t, ctx->ds,
                                                    ctx->dsm_part, kc_len);
        count_launch(ctx, "k_amd");
        CF_CUDA(cudaGetLastError());
    }
    // nothing in the step reads avg_nu_t of the AMD model (the reference
    // marks it "not used"): the plane means are formed from the partials of
    // the last pass when they are asked for
    ctx->amd_nparts = amd_partials_for(ctx, ctx->amd_nkc);
    ctx->amd_avg_pending = true;
    return 0;
}

int amd_partials_for(cf_ctx *ctx, int nkc) {
    if (ctx->esz == 4) return amd32_parts(ctx->nxp, ctx->nzp, nkc);
    return cdiv(ctx->nxp, AMD_TX) * cdiv(ctx->nzp, cdiv(ctx->nzp, nkc));
}

int launch_avg_nu_t_flush(cf_ctx *ctx) {
    if (!ctx->amd_avg_pending) return 0;
    k_amd_avg<<<cdiv(ctx->nym, 8), 256, 0, ctx->st>>>(ctx->dsm_part, ctx->amd_nparts, ctx->nyg,
                                                      (double)ctx->nxp * ctx->nzp, ctx->avg_nu_t);
    count_launch(ctx, "k_amd_avg");
    ctx->amd_avg_pending = false;
    CF_CUDA(cudaGetLastError());
    return 0;
}

template int launch_amd<double>(cf_ctx *, int);
template int launch_amd<float>(cf_ctx *, int);
