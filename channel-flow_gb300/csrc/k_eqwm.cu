// k_eqwm.cu -- equilibrium wall model (Larsson), wallmodel.f90:591-685 and
// eqwm.f90:20-223, FP64.
//
// W at the matching row is moved to the U location with the 3-point Lagrange
// interpolations of interpolation.f90:114-252; their stencil choice depends
// only on indices, so the host precomputes (jj, w0, w1, w2) per output index
// with the reference's formulas.  The ODE of a wall point is solved by Picard
// iteration on tau_w (<= 101 passes, tol 1e-7; k_eq_solve below).
#include "cf_internal.cuh"

// temp_1 = interpolate_z_2nd of W(:, jw, :) at both walls: (nxg, 2, nzg)
template <typename T>
__global__ void k_eq_zinterp_t(Fld<T> W, int jref, int nxg, int nyg, int nzg, const int *zst, const double *zw,
                               double *t1) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int k = blockIdx.y + 1;
    int w = blockIdx.z;
    if (i > nxg) return;
    int jw = w == 0 ? jref : nyg - jref + 1;
    int jj = zst[k];
    const double *c = zw + 3 * k;
    t1[(i - 1) + (long)nxg * (w + 2L * (k - 1))] =
        c[0] * (double)W(i, jw, jj - 1) + c[1] * (double)W(i, jw, jj) + c[2] * (double)W(i, jw, jj + 1);
}

struct EqParams {
    int ncv, jref, nx, nxg, nyg, nzg;
    double nu, h_wm, tau_mean;
};

// |u| at the matching row of wall point t = (i, wall, k) (wallmodel.f90:
// 597-612): U there and W moved to the U location by interpolate_x_2nd of
// temp_1; returns u_les and, through Uv / wv, the two components.
struct WallPt {
    int i, w, k, jj;
    long toff;
};
__device__ __forceinline__ WallPt wall_point(long t, const EqParams &ep) {
    WallPt p;
    p.i = (int)(t % ep.nx) + 1;
    const long r = t / ep.nx;
    p.w = (int)(r % 2);
    p.k = (int)(r / 2) + 1;
    p.jj = p.w == 0 ? ep.jref : ep.nyg - ep.jref + 1;
    p.toff = (long)(p.i - 1) + (long)ep.nx * (p.w + 2L * (p.k - 1));
    return p;
}
__device__ __forceinline__ double wall_ules(const WallPt &p, const EqParams &ep, const Fld<double> &Ud, const float *Uf32,
                                            int use_f32, int sy, int sz, const double *t1, const int *xst,
                                            const double *xw, double *Uv_out, double *wv_out) {
    const int xj = xst[p.i];
    const double *c = xw + 3 * p.i;
    const double *row = t1 + (long)ep.nxg * (p.w + 2L * (p.k - 1)) - 1;
    const double wv = c[0] * row[xj - 1] + c[1] * row[xj] + c[2] * row[xj + 1];
    const long uoff = (long)(p.i - 1) + (long)sy * (p.jj - 1) + (long)sz * (p.k - 1);
    const double Uv = use_f32 ? (double)Uf32[uoff] : Ud.p[uoff];
    *Uv_out = Uv;
    *wv_out = wv;
    return sqrt(Uv * Uv + wv * wv);
}

// u_les of every wall point (the input of the learned wall stress)
__global__ void k_wm_ules(const Fld<double> Ud, const float *Uf32, int use_f32, int sy, int sz, const double *t1,
                          const int *xst, const double *xw, EqParams ep, double *ules) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)ep.nx * ep.nzg * 2) return;
    const WallPt p = wall_point(t, ep);
    double Uv, wv;
    ules[p.toff] = wall_ules(p, ep, Ud, Uf32, use_f32, sy, sz, t1, xst, xw, &Uv, &wv);
}

// Learned-stress state of the wall model: the network's stress and envelope
// flag per point, the call counter and checking period, the checked eqwm
// stress.  mode 0: eqwm everywhere (the reference).
struct WmState {
    const double *tau_nn;
    const int *inside;
    const int *calls;
    int check_every;
    int mode;
    double *tau_eq;
};

// ---------------------------------------------------------------------------
// solve_u_eqwm (eqwm.f90:90-223) for every wall point.
//
// The ODE's tridiagonal system (eqwm.f90:152-205) says that the flux
// mu (u_{q+1} - u_q) / (y_cv(q+1) - y_cv(q)) is the same through every face
// between the wall and the top cell, whose velocity is given, so the stress
// of a pass is that of resistances in series,
//   tau = u_les / sum_q g_q / mu_q,
// g_0 = y_cv(1) - y_fa(1) with mu = nu and g_q = y_cv(q+1) - y_cv(q) with the
// mixing-length viscosity of face q+1.  The sum is kept as a quotient
// (N, D) <- (N mu + g D, D mu) with mu in units of nu: three operations a
// cell and one division a pass, every term positive.  P lanes share a point's
// cells and add their sums by shuffles: the FP64 pipe of each of an SM's
// sub-partitions issues one warp instruction per 64 clocks whether or not
// others have work, so that a wall with few points is spread over all of
// them (66 x 66 x 2 points of 100 cells: 270 warps for 608 sub-partitions).
//
// exp(-y cd) of a pass is the last pass's value (kept per thread in shared
// memory) times exp(-y dcd) as its Taylor polynomial where |y dcd| <= 2e-2
// (degree 7; 4 up to 1e-3, 2 up to 1e-6: truncation below 1e-17 relative),
// from a table otherwise (exp_neg).
//
// Split path: the Picard passes in FP32 (at most 50, until the change is below
// 1e-5 of tau), which also give the slope of the fixed-point map, G'(tau) =
// (1/2r) sum g c y D (D + 2 x E) / mu^2; then one FP64 pass and the Newton
// step t0 + (t1 - t0)/(1 - G'), whose error is that of the slope, about 1e-5
// of a correction of 1e-6; then the reference's FP64 passes to its criterion,
// which the first of them meets.  (Two passes and Aitken's extrapolation
// instead needed a third FP64 pass, and a pass took a continuant recurrence
// with seven operations a cell: 567 us per call against 340 at Re_tau 2000,
// 258 x 258 x 2 points of 30 cells, 295 with the table of exponentials;
// all-FP64 4.62 ms against 2.32 and 2.16.)
// ---------------------------------------------------------------------------
constexpr int EQ_T = 128;                 // threads per block

// exp(-x), x >= 0, by table (Tang's method): exp(-n/32) at the nearest n/32
// times the Taylor polynomial of the rest, |r| <= 1/64 (degree 6: truncation
// 5e-17).  About 9 FP64 instructions, the library's function 16.  Past x = 40
// the value is below half an ulp of the 1 it is taken from: 0.
__device__ __forceinline__ double exp_neg(double x, const double2 *__restrict__ tab) {
    const float xf = (float)x;
    const double2 t = __ldg(&tab[min((int)fmaf(xf, 32.f, 0.5f), EQ_EXPN)]);  // (n/32, exp(-n/32))
    const double r = t.x - x;
    double p = fma(r, 1.0 / 720.0, 1.0 / 120.0);
    p = fma(r, p, 1.0 / 24.0);
    p = fma(r, p, 1.0 / 6.0);
    p = fma(r, p, 0.5);
    p = fma(r, p, 1.0);
    const double e = fma(t.y * r, p, t.y);
    return xf > 40.f ? 0.0 : e;
}
constexpr size_t EQ_SMEM = 100 * 1024;    // shared memory of a block at most
__host__ __device__ __forceinline__ int eq_grid_doubles(int ncv) { return 2 * ncv + (ncv + 1); }

template <int P, bool MIXED>
__global__ void __launch_bounds__(EQ_T) k_eq_solve(const Fld<double> Ud, const float *Uf32, int sy, int sz,
                                                   const double *t1, const int *xst, const double *xw,
                                                   const double *grid, const double2 *etab, EqParams ep,
                                                   const void *nut, int keep_ex,
                                                   double *tau0, double *alpha_x, double *alpha_zt, int *counters,
                                                   WmState wm) {
    extern __shared__ double sg[];
    const int ncv = ep.ncv, nt = ncv - 1;  // terms with a mixing-length viscosity
    // y and g of term m = 0 .. nt-1 (face m + 2), FP32 copies after them, then the kept exponentials
    double *y64 = sg, *g64 = sg + ncv;
    float *y32 = (float *)(sg + 2 * ncv), *g32 = y32 + ncv;
    double *Ex = sg + eq_grid_doubles(ncv) + threadIdx.x;
    for (int m = threadIdx.x; m < nt; m += EQ_T) {
        y64[m] = grid[ncv + m + 2];
        g64[m] = grid[m + 2] - grid[m + 1];
        y32[m] = (float)y64[m];
        g32[m] = (float)g64[m];
    }
    __syncthreads();
    const double g0 = grid[1] - grid[ncv + 1], ymax = y64[nt - 1];
    const int part = threadIdx.x % P;
    const long npts = (long)ep.nx * ep.nzg * 2;
    long t = ((long)blockIdx.x * EQ_T + threadIdx.x) / P;
    const bool act = t < npts;
    if (!act) t = npts - 1;  // whole warps stay: the lanes of a point add by shuffles
    const WallPt pt = wall_point(t, ep);
    const int i = pt.i, w = pt.w, k = pt.k;
    const int nxg = ep.nxg, nyg = ep.nyg;
    double Uv, wv;
    const double u_les = wall_ules(pt, ep, Ud, Uf32, MIXED, sy, sz, t1, xst, xw, &Uv, &wv);
    const long toff = pt.toff;
    const bool served = wm.mode == 1 && wm.inside[toff] != 0;
    const bool check = wm.mode == 1 && wm.check_every > 0 && (*wm.calls % wm.check_every) == 0;
    double tau = tau0[toff];
    const bool solve = act && (!served || check);
    if (__any_sync(0xffffffffu, solve)) {
        // solve_u_eqwm(u_les, nu, 1.0, yg(jref), ncv, stretch, tau, iter, tau_in)
        const double nu = ep.nu, rnu = 1.0 / nu, kn = 0.41 * rnu, cA = rnu / 17.0;  // kappa / nu, 1 / (nu A+)
        const int max_iter = 100;
        const double tol = 0.0000001 * (nu * u_les / ep.h_wm);  // 1e-7 of the laminar stress
        const double nuu = nu * u_les;
        auto psum = [](auto v) {
#pragma unroll
            for (int o = 1; o < P; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            return v;
        };
        int iter = 0;
        bool mixed_ok = false;  // the FP32 passes gave the FP64 ones their start
        float slope = 0.f;
        if constexpr (MIXED) {
            const float nuu32 = (float)nuu, g00 = (float)g0, kn32 = (float)kn, cA32 = (float)cA;
            float tq = (float)tau;
            int it = 0;
            bool run = solve;
            // lanes whose point has converged idle until their warp's others have
            while (__any_sync(0xffffffffu, run)) {
                const float ut = sqrtf(tq), c = kn32 * ut, cd = ut * cA32;
                float r = 0.f, sl = 0.f;
                for (int m = part; m < nt; m += P) {
                    const float y = y32[m], x = y * cd, E = __expf(-x), D = 1.f - E, cyD = c * y * D;
                    const float q = 1.f / fmaf(cyD, D, 1.f), gq = g32[m] * q;
                    r += gq;
                    sl = fmaf(gq * q, cyD * fmaf(2.f * x, E, D), sl);
                }
                r = g00 + psum(r);
                sl = psum(sl);
                const float tn = nuu32 / r;
                if (run) {
                    const float tp = tq;
                    tq = tn;
                    slope = 0.5f * sl / r;
                    if (fabsf(tq - tp) < 1e-5f * fabsf(tq)) run = false;
                    else if (++it >= 50) run = false;
                }
            }
            if (isfinite(tq) && tq > 0.f) {
                tau = (double)tq;
                iter = it;
                mixed_ok = true;
            }
        }
        // one FP64 Picard pass of solve_u_eqwm (eqwm.f90:121-205)
        double cd_last = -1.0;  // no exponentials kept yet
        auto pass64 = [&](double tau) -> double {
            const double ut = sqrt(tau), c = kn * ut, cd = ut * cA;
            const double dcd = cd - cd_last, xmax = fabs(dcd) * ymax;
            // the polynomial of the warp's largest step (3: exp)
            int lev = (cd_last >= 0.0 && xmax <= 2e-2) ? (xmax <= 1e-6 ? 0 : (xmax <= 1e-3 ? 1 : 2)) : 3;
            lev = keep_ex ? __reduce_max_sync(0xffffffffu, lev) : 3;
            cd_last = cd;
            double N = 0.0, Dn = 1.0;
            auto sweep = [&](auto &&ex) {
                int s = 0;
                for (int m = part; m < nt; m += P, s++) {
                    const double y = y64[m], E = ex(y, s), D = 1.0 - E;
                    if (keep_ex) Ex[s * EQ_T] = E;
                    const double mu = fma(c * y, D * D, 1.0);
                    N = fma(g64[m], Dn, N * mu);
                    Dn *= mu;
                    if ((s & 7) == 7) {  // powers of two out (exact), well before the range ends
                        const int e = ((__double2hiint(Dn) >> 20) & 0x7ff) - 1023;
                        if (e > 128 && e < 1024) {
                            const double sc = __hiloint2double((1023 - e) << 20, 0);  // 2^-e
                            N *= sc;
                            Dn *= sc;
                        }
                    }
                }
            };
            if (lev == 3) {
                sweep([&](double y, int) { return exp_neg(y * cd, etab); });
            } else if (lev == 2) {
                sweep([&](double y, int s) {
                    const double x = y * -dcd;
                    double p = fma(x, 1.0 / 5040.0, 1.0 / 720.0);
                    p = fma(x, p, 1.0 / 120.0);
                    p = fma(x, p, 1.0 / 24.0);
                    p = fma(x, p, 1.0 / 6.0);
                    p = fma(x, p, 0.5);
                    p = fma(x, p, 1.0);
                    const double e = Ex[s * EQ_T];
                    return fma(e * x, p, e);
                });
            } else if (lev == 1) {
                sweep([&](double y, int s) {
                    const double x = y * -dcd;
                    double p = fma(x, 1.0 / 24.0, 1.0 / 6.0);
                    p = fma(x, p, 0.5);
                    p = fma(x, p, 1.0);
                    const double e = Ex[s * EQ_T];
                    return fma(e * x, p, e);
                });
            } else {
                sweep([&](double y, int s) {
                    const double x = y * -dcd, p = fma(x, 0.5, 1.0), e = Ex[s * EQ_T];
                    return fma(e * x, p, e);
                });
            }
            return nuu / (g0 + psum(N / Dn));
        };
        bool run = solve;
        if constexpr (MIXED) {
            if (__any_sync(0xffffffffu, run && mixed_ok)) {
                const double t0 = tau, tn = pass64(t0);
                if (run && mixed_ok) {
                    if (fabs(tn - t0) < tol) {
                        tau = tn;
                        run = false;
                    } else {
                        iter = iter + 1;
                        const double ta = t0 + (tn - t0) / (1.0 - (double)slope);
                        tau = (slope < 0.9f && isfinite(ta) && ta > 0.0) ? ta : tn;
                    }
                }
            }
        }
        while (__any_sync(0xffffffffu, run)) {
            const double tn = pass64(tau);
            if (run) {
                if (fabs(tn - tau) < tol) run = false;
                else if (++iter > max_iter) run = false;
                tau = tn;
            }
        }
        // wallmodel.f90:620-640
        if (solve) {
            if (isnan(tau)) {
                if (part == 0) atomicAdd(&counters[0], 1);
                tau = ep.tau_mean;
            }
            if (iter == 100) {
                tau = ep.tau_mean;
                if (part == 0) atomicAdd(&counters[1], 1);
            }
            if (check && part == 0) wm.tau_eq[toff] = tau;
        }
    }
    if (!act || part != 0) return;
    if (served) tau = wm.tau_nn[toff];
    tau0[toff] = tau;
    const int ja = w == 0 ? 1 : nyg, jb = w == 0 ? 2 : nyg - 1;
    const long cs = (long)nxg * nyg;
    auto NT = [&](int ii, int j) -> double {
        const long o = (long)(ii - 1) + (long)nxg * (j - 1) + cs * (k - 1);
        return MIXED ? (double)((const float *)nut)[o] : ((const double *)nut)[o];
    };
    const double nu_t_ik = 0.25 * ((NT(i, ja) + NT(i + 1, ja)) + (NT(i, jb) + NT(i + 1, jb)));
    const double f = tau / (u_les * (ep.nu + nu_t_ik));
    alpha_x[toff] = f * Uv;
    alpha_zt[toff] = f * wv;
}

// lanes per point: the count that minimises (warps on the busiest
// sub-partition) x (45 + 16 per cell of a lane) FP64 instructions of a pass
static int eq_parts(long npts, int ncv) {
    int best = 1;
    double best_cost = 1e300;
    for (int p = 1; p <= 8; p *= 2) {
        const double cost = (double)cdiv(cdiv(npts * p, 32), 4 * 152) * (45.0 + 16.0 * cdiv(ncv - 1, p));
        if (cost < best_cost) {
            best_cost = cost;
            best = p;
        }
    }
    return best;
}

template <int P, bool MIXED>
static void eq_launch(cf_ctx *ctx, const Fld<double> &Ud, const EqParams &ep, int b, const WmState &wm) {
    const long npts = (long)ep.nx * ep.nzg * 2;
    const size_t base = (size_t)eq_grid_doubles(ep.ncv) * sizeof(double),
                 ex = (size_t)cdiv(ep.ncv - 1, P) * EQ_T * sizeof(double);
    const int keep = base + ex <= EQ_SMEM;
    k_eq_solve<P, MIXED><<<cdiv(npts * P, EQ_T), EQ_T, base + (keep ? ex : 0), ctx->st>>>(
        Ud, (const float *)ctx->U[b], ep.nx, ep.nx * ep.nyg, ctx->wtemp1, ctx->eq_xst, ctx->eq_xw, ctx->eq_grid, ctx->eq_exp,
        ep, ctx->nut, keep, ctx->tau0, ctx->alpha_x, ctx->alpha_zt, (int *)ctx->d_red, wm);
}

template <bool MIXED>
static void eq_launch_parts(cf_ctx *ctx, const Fld<double> &Ud, const EqParams &ep, int b, const WmState &wm) {
    switch (eq_parts((long)ep.nx * ep.nzg * 2, ep.ncv)) {
    case 1: eq_launch<1, MIXED>(ctx, Ud, ep, b, wm); break;
    case 2: eq_launch<2, MIXED>(ctx, Ud, ep, b, wm); break;
    case 4: eq_launch<4, MIXED>(ctx, Ud, ep, b, wm); break;
    default: eq_launch<8, MIXED>(ctx, Ud, ep, b, wm);
    }
}

// shared-memory opt-in (called at context creation)
int eqwm_setup() {
#define CF_EQ_ATTR(P)                                                                                           \
    cudaFuncSetAttribute(k_eq_solve<P, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EQ_SMEM); \
    cudaFuncSetAttribute(k_eq_solve<P, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EQ_SMEM);
    CF_EQ_ATTR(1) CF_EQ_ATTR(2) CF_EQ_ATTR(4) CF_EQ_ATTR(8)
#undef CF_EQ_ATTR
    return 0;
}

// The error record of checked calls: max and mean |tau_nn/tau_eq - 1| over
// the points the network served, their count and the fallback count; every
// call advances the call counter.  One block.
__global__ void __launch_bounds__(1024) k_wm_audit(long npts, const double *tau_nn, const int *inside,
                                                  const double *tau_eq, int *calls, int check_every, double *log) {
    __shared__ double sm[3][32];
    const bool check = check_every > 0 && (*calls % check_every) == 0;
    if (check) {
        double mx = 0.0, sum = 0.0, cnt = 0.0;
        for (long t = threadIdx.x; t < npts; t += blockDim.x) {
            if (!inside[t]) continue;
            const double e = fabs(tau_nn[t] / tau_eq[t] - 1.0);
            mx = fmax(mx, e);
            sum += e;
            cnt += 1.0;
        }
        for (int o = 16; o > 0; o >>= 1) {
            mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
            sum += __shfl_down_sync(0xffffffffu, sum, o);
            cnt += __shfl_down_sync(0xffffffffu, cnt, o);
        }
        if ((threadIdx.x & 31) == 0) {
            sm[0][threadIdx.x >> 5] = mx;
            sm[1][threadIdx.x >> 5] = sum;
            sm[2][threadIdx.x >> 5] = cnt;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int q = 1; q < (int)(blockDim.x >> 5); q++) {
                mx = fmax(mx, sm[0][q]);
                sum += sm[1][q];
                cnt += sm[2][q];
            }
            log[0] = (double)(*calls + 1);
            log[1] = mx;
            log[2] = cnt > 0 ? sum / cnt : 0.0;
            log[3] = cnt;
            log[4] = (double)npts - cnt;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) *calls = *calls + 1;
}

// alpha_z: 4-point average of alpha_z_temp and its copies (wallmodel.f90:656-664)
__global__ void k_eq_alphaz(const double *azt, double *az, int nx, int nxg, int nz, int nzg) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int k = blockIdx.y + 1;
    int w = blockIdx.z;
    if (i > nxg) return;
    // value of alpha_z(i,w,k) after the three copy statements
    int ii = i, kk = k;
    if (kk == nz) kk = 2;
    if (ii == nxg) ii = 3;
    else if (ii == nxg - 1) ii = 2;
    auto T = [&](int a, int c) { return azt[(a - 1) + (long)nx * (w + 2L * (c - 1))]; };
    double v = 0.25 * (T(ii, kk) + T(ii + 1, kk) + T(ii, kk + 1) + T(ii + 1, kk + 1));
    az[(i - 1) + (long)nxg * (w + 2L * (k - 1))] = v;
}

template <typename T>
int launch_eqwm(cf_ctx *ctx, int b) {
    if (int rc = launch_nut_wall_rows<T>(ctx)) return rc;  // the rows k_eq_solve reads
    int nx = ctx->nx, nxg = ctx->nxg, nyg = ctx->nyg, nz = ctx->nz, nzg = ctx->nzg;
    Fld<T> W = make_fld<T>(ctx->W[b], ctx->nxg, ctx->nyg);
    k_eq_zinterp_t<T><<<dim3(cdiv(nxg, 128), nzg, 2), 128, 0, ctx->st>>>(W, ctx->prm.jref_eqwm, nxg, nyg, nzg,
                                                                         ctx->eq_zst, ctx->eq_zw, ctx->wtemp1);
    count_launch(ctx, "k_eq_zinterp_t");
    EqParams ep;
    ep.ncv = ctx->prm.eqwm_ncv;
    ep.jref = ctx->prm.jref_eqwm;
    ep.nx = nx; ep.nxg = nxg; ep.nyg = nyg; ep.nzg = nzg;
    ep.nu = ctx->prm.nu;
    ep.h_wm = ctx->hyg[ep.jref];
    ep.tau_mean = ctx->hs.tau_mean_eqwm;
    CF_CUDA(cudaMemsetAsync(ctx->d_red, 0, 2 * sizeof(int), ctx->st));
    long npts = (long)nx * nzg * 2;
    Fld<double> Ud = make_fld<double>(ctx->U[b], nx, nyg);
    WmState wm = {};
    if (ctx->wmlp) {
        // the learned stress of every point, then the solve where it does not serve
        k_wm_ules<<<cdiv(npts, 256), 256, 0, ctx->st>>>(Ud, (const float *)ctx->U[b], sizeof(T) == 4, nx, nx * nyg,
                                                        ctx->wtemp1, ctx->eq_xst, ctx->eq_xw, ep, ctx->wm_u);
        count_launch(ctx, "k_wm_ules");
        if (int rc = wall_mlp_infer(ctx, (int)npts, ep.h_wm, ep.nu)) return rc;
        wm.tau_nn = ctx->wm_tau;
        wm.inside = ctx->wm_inside;
        wm.calls = ctx->wm_calls;
        wm.check_every = ctx->wm_check_every;
        wm.mode = 1;
        wm.tau_eq = ctx->wm_tau_eq;
    }
    eq_launch_parts<sizeof(T) == 4>(ctx, Ud, ep, b, wm);
    count_launch(ctx, "k_eq_solve");
    if (ctx->wmlp) {
        k_wm_audit<<<1, 1024, 0, ctx->st>>>(npts, ctx->wm_tau, ctx->wm_inside, ctx->wm_tau_eq, ctx->wm_calls,
                                            ctx->wm_check_every, ctx->wm_log);
        count_launch(ctx, "k_wm_audit");
    }
    k_eq_alphaz<<<dim3(cdiv(nxg, 128), nz, 2), 128, 0, ctx->st>>>(ctx->alpha_zt, ctx->alpha_z, nx, nxg, nz, nzg);
    count_launch(ctx, "k_eq_alphaz");
    CF_CUDA(cudaGetLastError());
    return 0;
}

template int launch_eqwm<double>(cf_ctx *, int);
template int launch_eqwm<float>(cf_ctx *, int);

// The matching-plane velocity |u| of every wall point for state buffer b --
// the input the wall model hands to the eqwm solve (wallmodel.f90:597-621) --
// into ules (device, nx * 2 * nzg values, wall-point order (i, wall, k)).
template <typename T>
int launch_wm_inputs(cf_ctx *ctx, int b, double *ules) {
    int nx = ctx->nx, nxg = ctx->nxg, nyg = ctx->nyg, nzg = ctx->nzg;
    Fld<T> W = make_fld<T>(ctx->W[b], ctx->nxg, ctx->nyg);
    k_eq_zinterp_t<T><<<dim3(cdiv(nxg, 128), nzg, 2), 128, 0, ctx->st>>>(W, ctx->prm.jref_eqwm, nxg, nyg, nzg,
                                                                         ctx->eq_zst, ctx->eq_zw, ctx->wtemp1);
    EqParams ep = {};
    ep.ncv = ctx->prm.eqwm_ncv;
    ep.jref = ctx->prm.jref_eqwm;
    ep.nx = nx; ep.nxg = nxg; ep.nyg = nyg; ep.nzg = nzg;
    ep.nu = ctx->prm.nu;
    ep.h_wm = ctx->hyg[ep.jref];
    const long npts = (long)nx * nzg * 2;
    Fld<double> Ud = make_fld<double>(ctx->U[b], nx, nyg);
    k_wm_ules<<<cdiv(npts, 256), 256, 0, ctx->st>>>(Ud, (const float *)ctx->U[b], sizeof(T) == 4, nx, nx * nyg,
                                                    ctx->wtemp1, ctx->eq_xst, ctx->eq_xw, ep, ules);
    CF_CUDA(cudaGetLastError());
    return 0;
}

template int launch_wm_inputs<double>(cf_ctx *, int, double *);
template int launch_wm_inputs<float>(cf_ctx *, int, double *);
