// k_amd32.cu -- anisotropic minimum dissipation eddy viscosity of the split
// path (FP32), subgrid.f90:639-881, in one pass; the reduced form per cell is
// described at k_amd.cu.
//
// 16 bytes a cell go through memory, 11 us at 192 x 128 x 192 cells; the
// pass is bound by its operations, about 300 instructions for two cells at 16
// warps per SM: 58 us there (in a replayed graph, a launch's 5 us included)
// against 79 for one cell per thread, with the z differences formed for both
// their cells and two barriers a plane (92 before the differences' sums were
// shared, see k_amd.cu).
//
// A block of 128 threads owns a tile of 2 LS columns x R = 128 / LS rows and
// marches along z over a chunk of planes.  A lane holds two adjacent columns:
// the arithmetic is packed FP32x2 on columns i-1 .. i+2 of a row (two 8-byte
// reads of shared memory).  The pairs of z differences of U and V on a cell's
// upper side are the next plane's on its lower side, and the differences of W
// at a cell's lower face the last plane's.  The planes of the tile and its
// halo are copied to shared memory asynchronously, three ahead; one barrier a
// plane, no branch before the stores.
#include <algorithm>

#include "cf_internal.cuh"
#include "f32x2.cuh"

namespace {

constexpr int A32_T = 128;  // threads per block
constexpr int A32_NB = 4;   // planes in shared memory: k and k+1, two on their way

struct A32 {
    Fld<float> U, V, W, nt;
    RcpT<float> rc;
    const float *y;
    const DevScal *ds;
    double *part;
    int wall_rule, nxp, nyg, ny, nzp, kc_len;
};

template <int LS>
__global__ void __launch_bounds__(A32_T, 4) k_amd32(const __grid_constant__ A32 a) {
    typedef HaloTile<LS, A32_T> TL;
    constexpr int SX = TL::SX, NP = TL::NP, NL = TL::NL, R = TL::R, NB = A32_NB;
    __shared__ __align__(16) float st[NB][3][NP];
    const int ny = a.ny, nyg = a.nyg, nxp = a.nxp, nzp = a.nzp;
    const int l = threadIdx.x % LS, ty = TL::row();
    const int i0 = 2 + blockIdx.x * TL::WS, i = min(i0 + 2 * l, nxp), j0 = 2 + blockIdx.y * R, j = min(j0 + ty, nyg - 1);
    const int kb = 2 + blockIdx.z * a.kc_len, ke = min(kb + a.kc_len - 1, nzp + 1);
    const bool rowok = j0 + ty <= nyg - 1, own = rowok && i0 + 2 * l <= nxp;
    int eU[NL], eV[NL], eW[NL];
#pragma unroll
    for (int q = 0; q < NL; q++) {
        const int e = threadIdx.x + q * A32_T, sy = e / SX, sx = e - sy * SX;
        const int c = min(i0 - 1 + sx, nxp + 2), r = min(j0 - 1 + sy, nyg);  // past the last neighbours: not read
        eU[q] = a.U.idx(c, r, 1);
        eV[q] = a.V.idx(c, min(r, ny), 1);
        eW[q] = a.W.idx(c, r, 1);
    }
    auto fetch = [&](int k, int b) {
        const float *U = a.U.p + (long)a.U.sz * (k - 1), *V = a.V.p + (long)a.V.sz * (k - 1),
                    *Wp = a.W.p + (long)a.W.sz * (k - 1);
#pragma unroll
        for (int q = 0; q < NL; q++) {
            const int e = threadIdx.x + q * A32_T;
            if (NP % A32_T == 0 || e < NP) {
                copy_async<4>(&st[b][0][e], U + eU[q]);
                copy_async<4>(&st[b][1][e], V + eV[q]);
                copy_async<4>(&st[b][2][e], Wp + eW[q]);
            }
        }
        copy_commit();
    };
#pragma unroll
    for (int d = 0; d < NB - 1; d++) fetch(kb - 1 + d, d);
    // reciprocal spacings and their squares: the cell's own and those on its two sides
    const float2 rx = f2(a.rc.dx[i], a.rc.dx[i + 1]), xg0 = f2(a.rc.dxg[i], a.rc.dxg[i + 1]), xg1 = f2(xg0.y, a.rc.dxg[i + 2]);
    const float2 rx2 = mul2(rx, rx), xg02 = mul2(xg0, xg0), xg12 = mul2(xg1, xg1);
    const float ry = a.rc.dy[j], yg0 = a.rc.dyg[j], yg1 = a.rc.dyg[j + 1], ry2 = ry * ry, yg02 = yg0 * yg0, yg12 = yg1 * yg1;
    // wall rule 2: -nu_t(2) + 2 0.38 dPdx^(1/2) (y(2)-y(1))/2
    float add = 0.f;
    if (a.wall_rule == 2) add = (float)(2.0 * 0.38 * sqrt(a.ds->dPdx) * ((double)a.y[2] - (double)a.y[1]) / 2.0);
    // cells with duplicate or ghost images: the first two columns and the last
    // one, the rows next to a wall (planes: per plane)
    const int jg = j == 2 ? 1 : (j == nyg - 1 ? nyg : 0);
    const bool edge = i <= 3 || i + 1 >= nxp + 1 || jg;
    const int o1 = (ty + 1) * SX + 2 * l, oa = o1 - SX, oc = o1 + SX;
    int on = a.nt.idx(i, j, kb - 1);
    // carried up the march: sums and sums of squares of the z differences
    // below plane k, W and its differences at plane k-1
    float2 puz0 = sp(0.f), quz0 = sp(0.f), pvz0 = sp(0.f), qvz0 = sp(0.f), w_m = sp(0.f);
    float2 wx0m = sp(0.f), wx1m = sp(0.f), wy0m = sp(0.f), wy1m = sp(0.f);
    float zg0 = 0.f, zg1 = a.rc.dzg[kb], rz = 0.f, rzn = a.rc.dz[kb];  // of planes k and k+1
    float2 acc = sp(0.f);
    for (int k = kb - 1, b = 0; k <= ke; k++, b = (b + 1) & (NB - 1)) {
        copy_wait<NB - 3>();
        __syncthreads();  // plane k+1 is in; the buffer of k-1 is no longer read
        if (k + NB - 1 <= ke + 1) fetch(k + NB - 1, (b + NB - 1) & (NB - 1));
        else copy_commit();
        const float zl = zg0, zu = zg1, z = rz, z2 = z * z, zl2 = zl * zl, zu2 = zu * zu;
        zg0 = zg1;
        rz = rzn;
        zg1 = a.rc.dzg[min(k + 2, ke + 1)];
        rzn = a.rc.dz[min(k + 2, ke + 1)];
        const float(*T)[NP] = st[b], (*Tn)[NP] = st[(b + 1) & (NB - 1)];
        const Quad ua = quad(T[0] + oa), ub = quad(T[0] + o1), uc = quad(T[0] + oc), un = quad(Tn[0] + o1);
        const Quad va = quad(T[1] + oa), vb = quad(T[1] + o1), vna = quad(Tn[1] + oa), vnb = quad(Tn[1] + o1);
        const Quad wa = quad(T[2] + oa), wb = quad(T[2] + o1), wc = quad(T[2] + oc);
        // sum and sum of squares of two differences
        auto pq = [](float2 d, float2 e, float2 &p, float2 &q) {
            p = add2(d, e);
            q = fma2(e, e, mul2(d, d));
        };
        // of differences at columns i-1, i and i, i+1: d at (i-1, i), e at i+1
        auto pqx = [](float2 d, float e, float2 &p, float2 &q) {
            p = f2(d.x + d.y, d.y + e);
            const float2 s = mul2(d, d);
            q = f2(s.x + s.y, fmaf(e, e, s.y));
        };
        const float2 u0 = ub.c(), v0 = vb.c(), w0 = wb.c(), va0 = va.c();
        const float2 ux = sub2(u0, ub.p), vy = sub2(v0, va0), wz = sub2(w0, w_m);
        float2 puy0, quy0, puy1, quy1, puz1, quz1, pvx0, qvx0, pvx1, qvx1, pvz1, qvz1;
        float2 pwx0, qwx0, pwx1, qwx1, pwy0, qwy0, pwy1, qwy1;
        pqx(sub2(ub.p, ua.p), ub.q.x - ua.q.x, puy0, quy0);
        pqx(sub2(uc.p, ub.p), uc.q.x - ub.q.x, puy1, quy1);
        pqx(sub2(un.p, ub.p), un.q.x - ub.q.x, puz1, quz1);
        pq(sub2(va0, va.p), sub2(v0, vb.p), pvx0, qvx0);
        pq(sub2(va.q, va0), sub2(vb.q, v0), pvx1, qvx1);
        pq(sub2(vna.c(), va0), sub2(vnb.c(), v0), pvz1, qvz1);
        const float2 wx0 = sub2(w0, wb.p), wx1 = sub2(wb.q, w0), wy0 = sub2(w0, wa.c()), wy1 = sub2(wc.c(), w0);
        pq(wx0m, wx0, pwx0, qwx0);
        pq(wx1m, wx1, pwx1, qwx1);
        pq(wy0m, wy0, pwy0, qwy0);
        pq(wy1m, wy1, pwy1, qwy1);
        const float2 ux2 = mul2(ux, ux), vy2 = mul2(vy, vy), wz2 = mul2(wz, wz);
        float2 den = fma2(add2(quy1, qwy1), sp(yg12), mul2(add2(quy0, qwy0), sp(yg02)));
        den = fma2(add2(quz1, qvz1), sp(zu2), fma2(add2(quz0, qvz0), sp(zl2), den));
        den = fma2(add2(qvx1, qwx1), xg12, fma2(add2(qvx0, qwx0), xg02, den));
        den = fma2(den, sp(0.25f), fma2(wz2, sp(z2), fma2(vy2, sp(ry2), mul2(ux2, rx2))));
        float2 num = mul2(mul2(ux, rx), fma2(sp(0.25f), add2(add2(quy0, quy1), add2(quz0, quz1)), ux2));
        num = fma2(mul2(vy, sp(ry)), fma2(sp(0.25f), add2(add2(qvx0, qvx1), add2(qvz0, qvz1)), vy2), num);
        num = fma2(mul2(wz, sp(z)), fma2(sp(0.25f), add2(add2(qwx0, qwx1), add2(qwy0, qwy1)), wz2), num);
        // 8 S_ij of the mixed components times 8 times their factors
        const float2 t12 = fma2(pvx1, xg1, fma2(pvx0, xg0, fma2(puy1, sp(yg1), mul2(puy0, sp(yg0)))));
        const float2 t13 = fma2(pwx1, xg1, fma2(pwx0, xg0, fma2(puz1, sp(zu), mul2(puz0, sp(zl)))));
        const float2 t23 = fma2(pwy1, sp(yg1), fma2(pwy0, sp(yg0), fma2(pvz1, sp(zu), mul2(pvz0, sp(zl)))));
        const float2 sUy = add2(puy0, puy1), sUz = add2(puz0, puz1), sVx = add2(pvx0, pvx1), sVz = add2(pvz0, pvz1),
                     sWx = add2(pwx0, pwx1), sWy = add2(pwy0, pwy1);
        float2 off = mul2(t12, fma2(sp(2.f), fma2(sUy, vy, mul2(sVx, ux)), fma2(puz1, pvz1, mul2(puz0, pvz0))));
        off = fma2(t13, fma2(sp(2.f), fma2(sUz, wz, mul2(sWx, ux)), fma2(puy1, pwy1, mul2(puy0, pwy0))), off);
        off = fma2(t23, fma2(sp(2.f), fma2(sVz, wz, mul2(sWy, vy)), fma2(pvx1, pwx1, mul2(pvx0, pwx0))), off);
        num = mul2(fma2(sp(1.f / 32.f), off, num), sp(-0.3f));
        puz0 = puz1;
        quz0 = quz1;
        pvz0 = pvz1;
        qvz0 = qvz1;
        wx0m = wx0;
        wx1m = wx1;
        wy0m = wy0;
        wy1m = wy1;
        w_m = w0;
        if (own && k >= kb) {
            const float q0 = num.x / den.x, q1 = num.y / den.y;
            const float2 v = f2(q0 > 0.f ? q0 : 0.f, q1 > 0.f ? q1 : 0.f);  // NaN -> 0
            acc = add2(acc, v);
            a.nt.p[on] = v.x;
            a.nt.p[on + 1] = v.y;
            const int kz1 = k + nzp <= nzp + 3 ? k + nzp : 0, kz2 = k - nzp >= 1 ? k - nzp : 0;
            if (edge || kz1 || kz2) {
                const int kzs[3] = {k, kz1, kz2};
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int ih = i + h;
                    const float vh = h == 0 ? v.x : v.y, gv = a.wall_rule == 0 ? vh : -vh + add;
                    const int ixs[3] = {ih, ih + nxp <= nxp + 3 ? ih + nxp : 0, ih - nxp >= 1 ? ih - nxp : 0};
#pragma unroll
                    for (int x = 0; x < 3; x++) {
                        if (!ixs[x]) continue;
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            if (!kzs[c]) continue;
                            if (x + c > 0) a.nt(ixs[x], j, kzs[c]) = vh;
                            if (jg) a.nt(ixs[x], jg, kzs[c]) = gv;
                        }
                    }
                }
            }
        }
        on += a.nt.sz;
    }
    double s = own ? (double)acc.x + (double)acc.y : 0.0;
#pragma unroll
    for (int o = LS / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LS);
    if (l == 0 && rowok) a.part[(long)(j - 2) * (gridDim.x * gridDim.z) + blockIdx.z * gridDim.x + blockIdx.x] = s;
}

}  // namespace

// z chunks
int amd32_plan(int nxp, int nym, int nzp, int sms) {
    const int ls = tile_lanes(nxp);
    int per = 1;
    if (ls == 32) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_amd32<32>, A32_T, 0);
    else if (ls == 16) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_amd32<16>, A32_T, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_amd32<8>, A32_T, 0);
    return cdiv(nzp, chunk_len((long)cdiv(nxp, 2 * ls) * cdiv(nym, A32_T / ls), per, sms, nzp));
}

// partials per row with nkc chunks
int amd32_parts(int nxp, int nzp, int nkc) { return cdiv(nxp, 2 * tile_lanes(nxp)) * cdiv(nzp, cdiv(nzp, nkc)); }

int launch_amd32(cf_ctx *ctx, int b) {
    A32 a;
    a.U = make_fld<float>(ctx->U[b], ctx->nx, ctx->nyg);
    a.V = make_fld<float>(ctx->V[b], ctx->nxg, ctx->ny);
    a.W = make_fld<float>(ctx->W[b], ctx->nxg, ctx->nyg);
    a.nt = make_fld<float>(ctx->nut, ctx->nxg, ctx->nyg);
    a.rc = rcp_of<float>(ctx);
    a.y = geo_of<float>(ctx).y;
    a.ds = ctx->ds;
    a.part = ctx->dsm_part;
    a.wall_rule = ctx->prm.Dirichlet_nu_t;
    a.nxp = ctx->nxp; a.nyg = ctx->nyg; a.ny = ctx->ny; a.nzp = ctx->nzp;
    a.kc_len = cdiv(ctx->nzp, ctx->amd_nkc);
    const int ls = tile_lanes(ctx->nxp);
    const dim3 grd(cdiv(ctx->nxp, 2 * ls), cdiv(ctx->nym, A32_T / ls), cdiv(ctx->nzp, a.kc_len));
    if (ls == 32) k_amd32<32><<<grd, A32_T, 0, ctx->st>>>(a);
    else if (ls == 16) k_amd32<16><<<grd, A32_T, 0, ctx->st>>>(a);
    else k_amd32<8><<<grd, A32_T, 0, ctx->st>>>(a);
    count_launch(ctx, "k_amd32");
    CF_CUDA(cudaGetLastError());
    return 0;
}
