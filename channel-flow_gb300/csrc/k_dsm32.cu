// k_dsm32.cu -- the dynamic Smagorinsky pass (subgrid.f90:376-538) of the
// split path (FP32), as two kernels.
//
//   k_dsm32_q   at every canonical cell from U, V, W at actual indices
//               (subgrid.f90:390-428): the centre velocities, |S| S_ij and
//               |S|; and Uf, Vf, Wf on canonical elements (subgrid.f90:429-445)
//   k_dsm32_lm  the filters of u_i u_j and |S| S_ij, L, M and the plane
//               partials of L.M and M.M (subgrid.f90:447-513), everything
//               through the periodic wrap (the reference's periodic fills,
//               subgrid.f90:448-458)
//
// 112 bytes a cell go through memory (12 + 52 and 48), 78 us at 192 x 128 x
// 192 cells and the measured 6.75 TB/s.  One kernel for all of it moved 16
// bytes but formed the first kernel's quantities 1.3 times over (tile halos)
// and took 860 instructions and 270 shared-memory wavefronts a cell: 199 us
// (in a replayed graph, a launch's 5 us included) against 66 + 96 now; 261
// against 88 + 122 at 256 x 96 x 256.  What is left above the bytes is the
// latency of 12 warps per SM: the histories of the filters take 160 registers.
//
// A block of 128 threads owns a tile of 2 LS columns x R = 128 / LS rows and
// marches along z over a chunk of planes.  A lane holds two adjacent columns:
// the arithmetic is packed FP32x2, and with columns i-1 .. i+2 of a row as
// two 8-byte reads of shared memory the x differences and filters need no
// exchange between lanes.  The planes of the tile and its halo are copied to
// shared memory asynchronously, two ahead of the one worked on (one barrier a
// plane); z neighbours are carried up the march.  The marches' bodies have no
// branches (planes and rows that give nothing have weight 0 or skip their
// stores): with them the filters did not fill the gaps of the strain rates'
// chain, 116 us instead of 96 for the second kernel.  LS = 16 and 8 take
// tiles of 32 x 8 and 16 x 16 where that leaves fewer idle columns.  In
// k_dsm32_lm the tiles start one column before their cells, so that a row's
// copies are 16 bytes (8 where nxp is not a multiple of 4) and columns i-1, i
// of a lane aligned.  A first version without shared memory, with shuffles
// for the x neighbours and neighbours loaded per row, took 73 + 136 us.
//
// U, V, W are read at their actual indices, so the pass needs no periodic
// ghosts: it serves every state and either wall treatment.
//
// Velocity differences are taken between neighbours before anything is
// summed, as the reference does (a difference of sums would round the sums
// first); the mixed strain rates are sums over their four edges (t = 8 S_ij).
// hat(u_i) is the mean of two faces' filtered velocities (the mean and the
// filter commute).  In the rows 2 and nyg-1 the reference's one-sided filter
// of the centre velocities does not read the ghost rows that Uf uses: two
// extra rows of k_dsm32_q filter U, V, W with that rule for them.
#include <algorithm>

#include "cf_internal.cuh"
#include "f32x2.cuh"

namespace {

constexpr int D32_T = 128;  // threads per block
constexpr int D32_NB = 3;   // planes of a tile in shared memory: two on their way, one worked on

// the test filter in one direction over its weight 1/6; a one-sided end
// (2/3, 1/3) is the inner neighbour taken twice
__device__ __forceinline__ float2 wf(float2 a, float2 b, float2 c) { return fma2(sp(4.f), b, add2(a, c)); }

// x direction from the pairs of columns i-1, i and i+1, i+2: cells i, i+1
__device__ __forceinline__ float2 wx(float2 p, float2 q) {
    const float2 s = add2(p, q);
    return f2(fmaf(4.f, p.y, s.x), fmaf(4.f, q.x, s.y));
}
// z direction up the march: h = plane r-2 + 4 plane r-1 and l = plane r-1;
// takes plane r, returns the filtered plane r-1
__device__ __forceinline__ float2 wz(float2 &h, float2 &l, float2 x) {
    const float2 f = add2(h, x);
    h = fma2(sp(4.f), x, l);
    l = x;
    return f;
}

// Scales.  FS: the filter's weight in three directions, from the FP32 value
// of 1/6 that the single-precision filters of this path are taken with (FP32
// 1/3 and 2/3 are its double and quadruple).  L is a small difference of
// hat(u u) and hat(u) hat(u), which those weights, 3e-8 above 1 in sum, move
// by -9e-8 u u; the factor between the two, FS / 1024, is taken as the product
// of two FP32 numbers 1.8e-8 below it (-7e-8 u u; the nearest FP32 number is
// 1.9e-8 above it: -11e-8).  Powers of two keep the filtered quantities'
// squares near their unscaled size.
constexpr double W6 = double(float(1.0 / 6.0)), FS = W6 * W6 * W6;
constexpr float SC_U = 1.f / 32.f;                // sum of two faces -> centre velocity / 16
constexpr float SC_S = 1.f / 256.f;               // |S| S_ij
constexpr float SC_M = float(4.0 * FS / 256.0);   // 4 |Sf| Sf_ij
constexpr float SC_A = 0.00212636287f, SC_B = 0.00212622364f;  // (sum of two faces' Uf)^2
constexpr float SC_P = float(65536.0 * FS * FS);  // partials

// canonical arrays of dsm_q, n apart: centre velocities, |S| S_ij, |S| (slot
// 15, where every reader of the lazily formed nu_t expects it); slots 9-14:
// Uf, Vf, Wf as [k][row][nxp] with rows 1..nyg (V: ny), then their one-sided
// rows as [k][2][nxp] (3 (nyg + 2) <= 6 nym rows from nym = 4 on)
enum { S_U = 0, S_V, S_W, S_Q = 3, S_F = 9, S_S = 15 };

struct D32 {
    Fld<float> U, V, W;
    RcpT<float> rc;
    float *q, *uf, *vf, *wf, *ue, *ve, *we;
    float4 *part;
    long n;
    int ny, nz, nyg, nxp, nym, nzp, kc_len, nkc, ntx;
};

// |S| of two cells from the diagonal components and t = 8 x the mixed ones
__device__ __forceinline__ float2 s_mag(float2 d0, float2 d1, float2 d2, float2 t12, float2 t13, float2 t23) {
    const float2 a = fma2(d2, d2, fma2(d1, d1, mul2(d0, d0))), b = fma2(t23, t23, fma2(t13, t13, mul2(t12, t12)));
    const float2 x = fma2(b, sp(1.f / 32.f), a), y = add2(x, x);
    // square root by one Newton step on rsqrtf (within 0.6 ulp, 0 for 0):
    // unlike sqrtf without a branch, which would part the march's body
    const float2 e = f2(rsqrtf(fmaxf(y.x, 1e-37f)), rsqrtf(fmaxf(y.y, 1e-37f))), r = mul2(y, e);
    return fma2(fma2(mul2(r, sp(-1.f)), r, y), mul2(e, sp(0.5f)), r);
}

// strain rates of two cells in the march: what plane p of the velocities
// gives, and the terms that wait for plane p+1
struct Strain {
    float2 u0, um, v1, va, w0, x, y;     // plane p-1: velocities; x and y differences of W over their spacings
    float2 t12, p13, p23, d0, d1, d2;    // the cell at p-1, t13 and t23 without their upper z part
    float2 du, dv;                       // z differences of U and V through the face below p
};

struct SGeo {
    float2 rx, rx0, rx1;
    float ry, ry0, ry1;
};

// Plane p: U (rows j-1, j, j+1), V (j-1, j), W (j-1, j, j+1; at the
// neighbours in x only row j).  strain_z first, with the cell at p-1 still
// in s; then strain_plane.
__device__ __forceinline__ void strain_z(Strain &s, float2 u0, float2 um, float2 v1, float2 va, float dzr) {
    s.du = mul2(add2(sub2(u0, s.u0), sub2(um, s.um)), sp(dzr));
    s.dv = mul2(add2(sub2(v1, s.v1), sub2(va, s.va)), sp(dzr));
}
__device__ __forceinline__ void strain_plane(Strain &s, const SGeo &g, const Quad &ua, const Quad &u, const Quad &uc,
                                             const Quad &va, const Quad &v, float2 wa, const Quad &w, float2 wc,
                                             float dzw) {
    const float2 u0 = u.c(), v1 = v.c(), w0 = w.c(), v0a = va.c();
    const float2 x = fma2(sub2(w0, w.p), g.rx0, mul2(sub2(w.q, w0), g.rx1)),
                 y = fma2(sub2(w0, wa), sp(g.ry0), mul2(sub2(wc, w0), sp(g.ry1)));
    const float2 up = add2(sub2(uc.c(), u0), sub2(uc.p, u.p)), lo = add2(sub2(u0, ua.c()), sub2(u.p, ua.p));
    const float2 vr = add2(sub2(v.q, v1), sub2(va.q, v0a)), vl = add2(sub2(v1, v.p), sub2(v0a, va.p));
    s.t12 = fma2(vl, g.rx0, fma2(vr, g.rx1, fma2(lo, sp(g.ry0), mul2(up, sp(g.ry1)))));
    s.p13 = add2(add2(x, s.x), s.du);
    s.p23 = add2(add2(y, s.y), s.dv);
    s.d0 = mul2(sub2(u0, u.p), g.rx);
    s.d1 = mul2(sub2(v1, v0a), sp(g.ry));
    s.d2 = mul2(sub2(w0, s.w0), sp(dzw));
    s.u0 = u0;
    s.um = u.p;
    s.v1 = v1;
    s.va = v0a;
    s.w0 = w0;
    s.x = x;
    s.y = y;
}

// tile of the first kernel
template <int LS>
using QTile = HaloTile<LS, D32_T>;

// A block's march.  The loop's body has no branch but the one around the
// copies, so that the strain rates' chain and the filters are interleaved:
// rows and planes that have no cells only skip the stores.
template <int LS, bool ext>
__device__ __forceinline__ void q_march(const D32 &a, float (*st)[3][QTile<LS>::NP]) {
    typedef QTile<LS> TL;
    constexpr int SX = TL::SX, NP = TL::NP, NL = TL::NL, R = TL::R;
    const int ny = a.ny, nyg = a.nyg, nxp = a.nxp;
    const int l = threadIdx.x % LS, ty = TL::row();
    const int i0 = 2 + blockIdx.x * TL::WS, i = i0 + 2 * l;
    const int kb = 2 + blockIdx.z * a.kc_len, ke = min(kb + a.kc_len - 1, a.nz - 1);
    const int j0 = 1 + blockIdx.y * R;
    const int j = ext ? (ty == 0 ? 2 : nyg - 1) : j0 + ty;
    const bool rowok = ext ? ty < 2 : j <= nyg, colok = i <= nxp;
    const bool cell = !ext && j >= 2 && j <= nyg - 1;
    // tile rows of the neighbours, reflected at the ends of the arrays (the
    // filter's one-sided rule); for cells they are j-1 and j+1
    int s1 = ty + 1, sa = s1 - 1, sc = s1 + 1, v1r = s1, var = sa, vcr = sc;
    if constexpr (ext) {  // U, W: row 2 and its inner neighbour; V: the three rows from the wall in
        s1 = ty == 0 ? 1 : 4;
        sa = sc = ty == 0 ? 2 : 3;
        var = ty == 0 ? 0 : 5;
        v1r = ty == 0 ? 1 : 4;
        vcr = ty == 0 ? 2 : 3;
    } else {
        if (j == 1) sa = var = s1 + 1;
        if (j == nyg) sc = s1 - 1;
        if (j == ny) vcr = s1 - 1;
    }
    // this thread's elements of a plane: the same tile position in U, V, W
    int eu[NL], evv[NL], ew[NL];
#pragma unroll
    for (int q = 0; q < NL; q++) {
        const int e = threadIdx.x + q * D32_T, sy = e / SX, sx = e - sy * SX;
        const int c = min(i0 - 1 + sx, nxp + 2);  // past the last neighbour: not read
        int ru = j0 - 1 + sy, rv = ru;
        if (ext) {
            ru = sy < 3 ? 1 + sy : nyg - 5 + sy;
            rv = sy < 3 ? 1 + sy : ny - 5 + sy;
        }
        ru = min(max(ru, 1), nyg);
        rv = min(max(rv, 1), ny);
        eu[q] = a.U.idx(c, ru, 1);
        evv[q] = a.V.idx(c, rv, 1);
        ew[q] = a.W.idx(c, ru, 1);
    }
    auto fetch = [&](int p, int b) {
        const float *U = a.U.p + (long)a.U.sz * (p - 1), *V = a.V.p + (long)a.V.sz * (p - 1),
                    *Wp = a.W.p + (long)a.W.sz * (p - 1);
#pragma unroll
        for (int q = 0; q < NL; q++) {
            const int e = threadIdx.x + q * D32_T;
            if (NP % D32_T == 0 || e < NP) {
                copy_async<4>(&st[b][0][e], U + eu[q]);
                copy_async<4>(&st[b][1][e], V + evv[q]);
                copy_async<4>(&st[b][2][e], Wp + ew[q]);
            }
        }
        copy_commit();
    };
    const int ig = min(i, nxp), jg = min(max(j, 2), nyg - 1);
    SGeo g;
    g.rx = f2(a.rc.dx[ig], a.rc.dx[ig + 1]);
    g.rx0 = f2(a.rc.dxg[ig], a.rc.dxg[ig + 1]);
    g.rx1 = f2(a.rc.dxg[ig + 1], a.rc.dxg[ig + 2]);
    g.ry = a.rc.dy[jg];
    g.ry0 = a.rc.dyg[jg];
    g.ry1 = a.rc.dyg[jg + 1];
    const bool own = rowok && colok, ownq = own && cell;
    Strain s = {};
    float2 h0[3], h1[3], uo = sp(0.f), vo = sp(0.f), wo = sp(0.f);
#pragma unroll
    for (int f = 0; f < 3; f++) h0[f] = h1[f] = sp(0.f);
    const long plane = (long)nxp * a.nym;
    const int su = ext ? 2 * nxp : nxp * nyg, sv = ext ? 2 * nxp : nxp * ny;  // plane strides of the filtered velocities
    float *qp = a.q + (ig - 2) + (long)nxp * (jg - 2) + plane * (kb - 2);
    float *uf = (ext ? a.ue + nxp * min(ty, 1) : a.uf + (long)nxp * (j - 1)) + (ig - 2) + (long)su * (kb - 2);
    float *vf = (ext ? a.ve + nxp * min(ty, 1) : a.vf + (long)nxp * (min(j, ny) - 1)) + (ig - 2) + (long)sv * (kb - 2);
    float *wfp = (ext ? a.we + nxp * min(ty, 1) : a.wf + (long)nxp * (j - 1)) + (ig - 2) + (long)su * (kb - 2);
    const int o1 = s1 * SX + 2 * l, oa = sa * SX + 2 * l, oc = sc * SX + 2 * l;
    const int ov1 = v1r * SX + 2 * l, ova = var * SX + 2 * l, ovc = vcr * SX + 2 * l;
    const bool putv = own && (ext || j <= ny);
#pragma unroll
    for (int d = 0; d < D32_NB - 1; d++) fetch(kb - 1 + d, d);
    float dzg = 0.f, dzw = 0.f;
    for (int p = kb - 1, b = 0; p <= ke + 1; p++, b = b + 1 == D32_NB ? 0 : b + 1) {
        copy_wait<D32_NB - 2>();
        __syncthreads();  // plane p is in; the buffer of p-1 is no longer read
        const int bn = b == 0 ? D32_NB - 1 : b - 1;
        if (p + D32_NB - 1 <= ke + 1) fetch(p + D32_NB - 1, bn);
        else copy_commit();
        const float dzg0 = dzg, dzw0 = dzw;  // of plane p; the next plane's on their way
        dzg = a.rc.dzg[min(p + 1, ke + 1)];
        dzw = a.rc.dz[min(p + 1, ke)];
        if (!rowok) continue;  // whole rows of the tile: no barrier below
        const float *U = st[b][0], *V = st[b][1], *Wp = st[b][2];
        const Quad ua = quad(U + oa), u = quad(U + o1), uc = quad(U + oc);
        Quad va = quad(V + ova), v = quad(V + ov1), vc = quad(V + ovc);
        const Quad wa = quad(Wp + oa), w = quad(Wp + o1), wc = quad(Wp + oc);
        if constexpr (ext) {  // twice the centre velocities of the row and its inner neighbour
            const Quad v1 = v;
            v.p = add2(va.p, v1.p);
            v.q = add2(va.q, v1.q);
            va.p = vc.p = add2(v1.p, vc.p);
            va.q = vc.q = add2(v1.q, vc.q);
        }
        // filtered velocities: y, x, then z from the two planes below
        auto fxy = [](const Quad &a, const Quad &b, const Quad &c) {
            return wx(wf(a.p, b.p, c.p), wf(a.q, b.q, c.q));
        };
        const float2 fx[3] = {fxy(ua, u, uc), fxy(va, v, vc), fxy(wa, w, wc)};
        float2 fo[3];
#pragma unroll
        for (int f = 0; f < 3; f++) fo[f] = wz(h0[f], h1[f], fx[f]);
        const bool put = p >= kb + 1;  // plane p-1 is complete
        if constexpr (!ext) {
            strain_z(s, u.c(), u.p, v.c(), va.c(), dzg0);
            const float2 t13 = add2(s.p13, s.du), t23 = add2(s.p23, s.dv);
            const float2 S = s_mag(s.d0, s.d1, s.d2, s.t12, t13, t23), Sd = mul2(S, sp(SC_S)), So = mul2(S, sp(0.125f * SC_S));
            const float2 out[10] = {uo, vo, wo, mul2(Sd, s.d0), mul2(Sd, s.d1), mul2(Sd, s.d2),
                                    mul2(So, s.t12), mul2(So, t13), mul2(So, t23), S};
            uo = mul2(add2(u.c(), u.p), sp(SC_U));
            vo = mul2(add2(v.c(), va.c()), sp(SC_U));
            wo = mul2(add2(w.c(), s.w0), sp(SC_U));
            strain_plane(s, g, ua, u, uc, va, v, wa.c(), w, wc.c(), dzw0);
            if (ownq && put) {
#pragma unroll
                for (int q = 0; q < 9; q++) *(float2 *)(qp + q * a.n) = out[q];
                *(float2 *)(qp + S_S * a.n) = out[9];
            }
            if (put) qp += plane;
        }
        if (own && put) {
            *(float2 *)uf = fo[0];
            *(float2 *)wfp = fo[2];
            if (putv) *(float2 *)vf = fo[1];
        }
        if (put) {
            uf += su;
            vf += sv;
            wfp += su;
        }
    }
}

template <int LS>
__global__ void __launch_bounds__(D32_T, 3) k_dsm32_q(const __grid_constant__ D32 a) {
    __shared__ __align__(16) float st[D32_NB][3][QTile<LS>::NP];
    // the last block row takes the two one-sided rows of the filtered
    // velocities: its tile holds rows 1-3 and nyg-2..nyg (V: ny-2..ny)
    if (blockIdx.y == gridDim.y - 1) q_march<LS, true>(a, st);
    else q_march<LS, false>(a, st);
}

// quantity q of the 12 filtered ones: u_a u_b (q < 6) or |S| S_ij
__device__ __forceinline__ constexpr int pa_of(int q) { return q < 3 ? q : (q == 5 ? 1 : 0); }
__device__ __forceinline__ constexpr int pb_of(int q) { return q < 3 ? q : (q == 3 ? 1 : 2); }

// tile of the second kernel: R + 2 rows of 2 LS + 2 columns (the first one
// before the tile's cells), 12 arrays
template <int LS>
struct LTile {
    static constexpr int WS = 2 * LS, R = D32_T / LS, SY = R + 2, PX = WS + 4, NA = 12, NP = SY * PX;
    // with LS = 8: rows 4 apart, 4 PX = 80 words or 16 banks
    static __device__ __forceinline__ int row() {
        const int t = threadIdx.x / LS;
        return LS == 8 ? (t & 3) * 4 + (t >> 2) : t;
    }
    static constexpr size_t bytes = (size_t)D32_NB * NA * NP * sizeof(float);
};

// VEC: floats per copy (4, or 2 where nxp is not a multiple of 4)
template <int LS, int VEC>
__global__ void __launch_bounds__(D32_T, 3) k_dsm32_lm(const __grid_constant__ D32 a) {
    typedef LTile<LS> TL;
    constexpr int NQ = 12, SY = TL::SY, PX = TL::PX, NP = TL::NP, R = TL::R, WS = TL::WS;
    extern __shared__ __align__(16) float st[];  // [D32_NB][NA][SY][PX]
    const int ny = a.ny, nyg = a.nyg, nxp = a.nxp, nzp = a.nzp;
    const int l = threadIdx.x % LS, ty = TL::row();
    // 0-based canonical columns: the tile's copy starts at c0, a lane's cells
    // are c0 + 2l + 1 and c0 + 2l + 2 (the last one column nxp = column 0)
    const int c0 = blockIdx.x * WS, j0 = 2 + blockIdx.y * R, j = j0 + ty;
    const int kb = 2 + blockIdx.z * a.kc_len, ke = min(kb + a.kc_len - 1, a.nz - 1);
    const bool rowok = j <= nyg - 1, own = rowok && c0 + 2 * l + 1 < nxp;
    // copies: warps 0-2 take the rows' aligned chunks, the same ones of every
    // array; warp 3 the two columns past them (through the wrap at the last tile)
    constexpr int CPR = WS / VEC, RPI = 32 / CPR, NH = VEC == 4 ? 1 : 2;  // chunks a row, rows per warp and copy
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int gq[NH], gu[NH], gv[NH], so[NH];  // offsets in a canonical plane, a plane of U / W, of V, in the tile
    bool on[NH];
#pragma unroll
    for (int h = 0; h < NH; h++) {
        int sy, c, x;
        if (warp < 3) {
            sy = (warp * NH + h) * RPI + lane / CPR;
            x = (lane % CPR) * VEC;
            c = c0 + x;
            on[h] = sy < SY && c < nxp;
        } else {
            sy = lane + 32 * h;
            x = min(WS, nxp - c0);
            c = c0 + x >= nxp ? 0 : c0 + x;
            on[h] = sy < SY;
        }
        const int r = j0 - 1 + sy;  // row
        gq[h] = c + nxp * (min(max(r, 2), nyg - 1) - 2);
        gu[h] = c + nxp * (min(r, nyg) - 1);
        gv[h] = c + nxp * (min(r, ny) - 1);
        so[h] = sy * PX + x;
    }
    auto fetch = [&](int r, int b) {
        const int k = wrapn(r, nzp) - 2;
        const float *Q = a.q + (long)nxp * a.nym * k, *U = a.uf + (long)nxp * nyg * k, *V = a.vf + (long)nxp * ny * k,
                    *Wp = a.wf + (long)nxp * nyg * k;
        float *d = st + b * (TL::NA * NP);
#pragma unroll
        for (int h = 0; h < NH; h++) {
            if (!on[h]) continue;
            if (warp < 3) {
#pragma unroll
                for (int q = 0; q < 9; q++) copy_async<VEC * 4>(d + q * NP + so[h], Q + q * a.n + gq[h]);
                copy_async<VEC * 4>(d + 9 * NP + so[h], U + gu[h]);
                copy_async<VEC * 4>(d + 10 * NP + so[h], V + gv[h]);
                copy_async<VEC * 4>(d + 11 * NP + so[h], Wp + gu[h]);
            } else {
#pragma unroll
                for (int q = 0; q < 9; q++) copy_async<8>(d + q * NP + so[h], Q + q * a.n + gq[h]);
                copy_async<8>(d + 9 * NP + so[h], U + gu[h]);
                copy_async<8>(d + 10 * NP + so[h], V + gv[h]);
                copy_async<8>(d + 11 * NP + so[h], Wp + gu[h]);
            }
        }
        copy_commit();
    };
    // rows j-1, j, j+1 in the tile; those of the canonical arrays reflected at rows 2 and nyg-1
    const int t1 = (ty + 1) * PX + 2 * l, ta = t1 - PX, tc = t1 + PX;
    const int q1 = t1, qa = j == 2 ? tc : ta, qc = j == nyg - 1 ? ta : tc;
    const int iA = min(c0 + 2 * l + 1, nxp - 1) + 2, iB = iA + 1 > nxp + 1 ? 2 : iA + 1;  // the lane's columns, 1-based
    const int jg = min(j, nyg - 1);
    SGeo g;
    g.rx = f2(a.rc.dx[iA], a.rc.dx[iB]);
    g.rx0 = f2(a.rc.dxg[iA], a.rc.dxg[iB]);
    g.rx1 = f2(a.rc.dxg[iA + 1], a.rc.dxg[iB + 1]);
    g.ry = a.rc.dy[jg];
    g.ry0 = a.rc.dyg[jg];
    g.ry1 = a.rc.dyg[jg + 1];
    const bool wrow = j == 2 || j == nyg - 1;
    const int fe = j == 2 ? 0 : nxp;  // its one-sided row
    float2 h0[NQ], h1[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) h0[q] = h1[q] = sp(0.f);
    Strain s = {};
    float2 fw = sp(0.f);
    float2 lmd = sp(0.f), lmo = sp(0.f), mmd = sp(0.f), mmo = sp(0.f);
#pragma unroll
    for (int d = 0; d < D32_NB - 1; d++) fetch(kb - 1 + d, d);
    float dzg = 0.f, dzw = 0.f;
    for (int r = kb - 1, b = 0; r <= ke + 1; r++, b = b + 1 == D32_NB ? 0 : b + 1) {
        copy_wait<D32_NB - 2>();
        __syncthreads();  // plane r is in; the buffer of r-1 is no longer read
        const int bn = b == 0 ? D32_NB - 1 : b - 1;
        if (r + D32_NB - 1 <= ke + 1) fetch(r + D32_NB - 1, bn);
        else copy_commit();
        const float dzg0 = dzg, dzw0 = dzw;  // of plane r; the next plane's on their way
        dzg = a.rc.dzg[min(r + 1, ke + 1)];
        dzw = a.rc.dz[min(r + 1, ke)];
        if (!rowok) continue;
        const float *T = st + b * (TL::NA * NP);
        // 4 |Sf| Sf_ij and hat(u_i) at plane r-1, from plane r (the first two
        // planes complete none: weight 0 below)
        float2 m[6], f[3], fe0 = sp(0.f), fe1 = sp(0.f), fe2 = sp(0.f);
        if (wrow) {
            const int k1 = wrapn(max(r - 1, 1), nzp) - 2, k0 = wrapn(max(r - 2, 1), nzp) - 2, cm = iA - 3;
            const long e1 = fe + 2L * nxp * k1, e0 = fe + 2L * nxp * k0;
            fe0 = f2(a.ue[e1 + iA - 2] + a.ue[e1 + cm], a.ue[e1 + iB - 2] + a.ue[e1 + iA - 2]);
            fe1 = f2(a.ve[e1 + iA - 2], a.ve[e1 + iB - 2]);
            fe2 = f2(a.we[e1 + iA - 2] + a.we[e0 + iA - 2], a.we[e1 + iB - 2] + a.we[e0 + iB - 2]);
        }
        {
            const float *U = T + 9 * NP, *V = T + 10 * NP, *Wp = T + 11 * NP;
            const Quad ua = quad(U + ta), u = quad(U + t1), uc = quad(U + tc);
            const Quad va = quad(V + ta), v = quad(V + t1), w = quad(Wp + t1);
            const float2 wa = f2(Wp[ta + 1], Wp[ta + 2]), wc = f2(Wp[tc + 1], Wp[tc + 2]);
            strain_z(s, u.c(), u.p, v.c(), va.c(), dzg0);
            const float2 t13 = add2(s.p13, s.du), t23 = add2(s.p23, s.dv);
            const float2 S = s_mag(s.d0, s.d1, s.d2, s.t12, t13, t23), c4 = mul2(S, sp(SC_M)), ch = mul2(S, sp(0.125f * SC_M));
            m[0] = mul2(c4, s.d0);
            m[1] = mul2(c4, s.d1);
            m[2] = mul2(c4, s.d2);
            m[3] = mul2(ch, s.t12);
            m[4] = mul2(ch, t13);
            m[5] = mul2(ch, t23);
            f[0] = wrow ? fe0 : add2(s.u0, s.um);
            f[1] = wrow ? fe1 : add2(s.v1, s.va);
            f[2] = wrow ? fe2 : fw;
            fw = add2(w.c(), s.w0);
            strain_plane(s, g, ua, u, uc, va, v, wa, w, wc, dzw0);
        }
        // a quantity's x and z filters from its y-filtered plane r; returns plane r-1's
        auto filt = [&](int q, float2 P, float2 Q) {
            return wz(h0[q], h1[q], wx(P, Q));
        };
        float2 L[6];
        {
            Quad cu[3][3];
#pragma unroll
            for (int e = 0; e < 3; e++) {
                cu[e][0] = quad(T + e * NP + qa);
                cu[e][1] = quad(T + e * NP + q1);
                cu[e][2] = quad(T + e * NP + qc);
            }
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const int x = pa_of(q), y = pb_of(q);
                L[q] = filt(q, wf(mul2(cu[x][0].p, cu[y][0].p), mul2(cu[x][1].p, cu[y][1].p), mul2(cu[x][2].p, cu[y][2].p)),
                            wf(mul2(cu[x][0].q, cu[y][0].q), mul2(cu[x][1].q, cu[y][1].q), mul2(cu[x][2].q, cu[y][2].q)));
            }
        }
        float2 fl[3];
#pragma unroll
        for (int e = 0; e < 3; e++) {
            fl[e] = mul2(f[e], sp(-SC_A));
            f[e] = mul2(f[e], sp(SC_B));
        }
#pragma unroll
        for (int q = 0; q < 6; q++) L[q] = fma2(fl[pa_of(q)], f[pb_of(q)], L[q]);
        const float wk = r <= kb ? 0.f : (r - 1 == 2 ? 2.f : 1.f);  // plane 2 stands for its duplicate too
#pragma unroll
        for (int q = 6; q < NQ; q++) {
            const float *C = T + (S_Q + q - 6) * NP;
            const Quad x0 = quad(C + qa), x1 = quad(C + q1), x2 = quad(C + qc);
            const float2 H = filt(q, wf(x0.p, x1.p, x2.p), wf(x0.q, x1.q, x2.q));
            const float2 M = sub2(m[q - 6], H), Mw = mul2(M, sp(wk));
            if (q < 9) {
                lmd = fma2(L[q - 6], Mw, lmd);
                mmd = fma2(M, Mw, mmd);
            } else {
                lmo = fma2(L[q - 6], Mw, lmo);
                mmo = fma2(M, Mw, mmo);
            }
        }
    }
    // the mixed components count twice; column 2 stands for its duplicate too
    const float2 lm = fma2(sp(2.f), lmo, lmd), mm = fma2(sp(2.f), mmo, mmd);
    const float wb = iB == 2 ? 2.f : 1.f;
    float ah = 0.f, al = 0.f, bh = 0.f, bl = 0.f;
    if (own) {
        two_sum(lm.x, wb * lm.y, ah, al);
        two_sum(mm.x, wb * mm.y, bh, bl);
    }
#pragma unroll
    for (int o = LS / 2; o > 0; o >>= 1) {
        const float a1 = __shfl_down_sync(0xffffffffu, ah, o, LS), a2 = __shfl_down_sync(0xffffffffu, al, o, LS);
        const float b1 = __shfl_down_sync(0xffffffffu, bh, o, LS), b2 = __shfl_down_sync(0xffffffffu, bl, o, LS);
        ff_add2(ah, al, a1, a2);
        ff_add2(bh, bl, b1, b2);
    }
    if (l == 0 && rowok) {
        // float-float times the scale, the products' rounding recovered
        const float x = ah * SC_P, y = bh * SC_P;
        a.part[(long)(j - 2) * (a.ntx * a.nkc) + blockIdx.x * a.nkc + blockIdx.z] =
            make_float4(x, fmaf(ah, SC_P, -x) + al * SC_P, y, fmaf(bh, SC_P, -y) + bl * SC_P);
    }
}

template <int LS>
int lm_blocks_per_sm(int nxp) {
    int per = 1;
    if (nxp % 4 == 0) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_dsm32_lm<LS, 4>, D32_T, LTile<LS>::bytes);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_dsm32_lm<LS, 2>, D32_T, LTile<LS>::bytes);
    return std::max(per, 1);
}

template <int LS>
void d32_run(cf_ctx *ctx, const D32 &a) {
    constexpr int R = D32_T / LS;
    // (the last block row: the one-sided rows)
    k_dsm32_q<LS><<<dim3(a.ntx, cdiv(ctx->nyg, R) + 1, a.nkc), D32_T, 0, ctx->st>>>(a);
    count_launch(ctx, "k_dsm32_q");
    const dim3 grd(a.ntx, cdiv(ctx->nym, R), a.nkc);
    if (ctx->nxp % 4 == 0) k_dsm32_lm<LS, 4><<<grd, D32_T, LTile<LS>::bytes, ctx->st>>>(a);
    else k_dsm32_lm<LS, 2><<<grd, D32_T, LTile<LS>::bytes, ctx->st>>>(a);
    count_launch(ctx, "k_dsm32_lm");
}

}  // namespace

// shared-memory opt-in (called at context creation)
int dsm32_setup() {
#define CF_D32_ATTR(LS)                                                                                            \
    cudaFuncSetAttribute(k_dsm32_lm<LS, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LTile<LS>::bytes);  \
    cudaFuncSetAttribute(k_dsm32_lm<LS, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LTile<LS>::bytes);
    CF_D32_ATTR(32) CF_D32_ATTR(16) CF_D32_ATTR(8)
#undef CF_D32_ATTR
    return 0;
}

// z-chunk length (of the filter kernel's blocks; the first kernel's time is
// within 3 % over a factor of two around it)
int dsm32_plan(int nxp, int nym, int nzp, int sms) {
    const int ls = tile_lanes(nxp);
    const int per = ls == 32 ? lm_blocks_per_sm<32>(nxp) : (ls == 16 ? lm_blocks_per_sm<16>(nxp) : lm_blocks_per_sm<8>(nxp));
    return chunk_len((long)cdiv(nxp, 2 * ls) * cdiv(nym, D32_T / ls), per, sms, nzp);
}

int dsm32_slots(int nxp, int nzp, int kc) { return cdiv(nxp, 2 * tile_lanes(nxp)) * cdiv(nzp, kc); }

// |S| into the canonical scratch, the plane partials into dsm_part
int launch_dsm32(cf_ctx *ctx, int b, int *nchunk) {
    D32 a;
    a.U = make_fld<float>(ctx->U[b], ctx->nx, ctx->nyg);
    a.V = make_fld<float>(ctx->V[b], ctx->nxg, ctx->ny);
    a.W = make_fld<float>(ctx->W[b], ctx->nxg, ctx->nyg);
    a.rc = rcp_of<float>(ctx);
    a.n = (long)ctx->nCan;
    a.q = (float *)ctx->dsm_q;
    const long row = (long)ctx->nxp * ctx->nzp;  // elements per row of all planes
    a.uf = a.q + S_F * a.n;
    a.vf = a.uf + row * ctx->nyg;
    a.wf = a.vf + row * ctx->nyg;
    a.ue = a.wf + row * ctx->nyg;
    a.ve = a.ue + 2 * row;
    a.we = a.ve + 2 * row;
    a.part = (float4 *)ctx->dsm_part;
    a.ny = ctx->ny; a.nz = ctx->nz; a.nyg = ctx->nyg;
    a.nxp = ctx->nxp; a.nym = ctx->nym; a.nzp = ctx->nzp;
    const int ls = tile_lanes(ctx->nxp);
    a.ntx = cdiv(ctx->nxp, 2 * ls);
    a.kc_len = ctx->dsm_kc;
    a.nkc = cdiv(ctx->nzp, ctx->dsm_kc);
    *nchunk = a.ntx * a.nkc;
    if ((size_t)*nchunk > ctx->dsm_part_nch) return cf_fail(ctx, CF_ERR_INVALID, "plane-partial slots");
    if (ls == 32) d32_run<32>(ctx, a);
    else if (ls == 16) d32_run<16>(ctx, a);
    else d32_run<8>(ctx, a);
    CF_CUDA(cudaGetLastError());
    return 0;
}
