"""FP64 kernels against the CPU oracle at the sizes where their tilings,
chunks and tails end: rows around the tridiagonal replay's chunk of 8, mode
counts off and on a multiple of 32, transform lengths with and without a
compile-time plan."""
import numpy as np
import pytest

from conftest import assert_close, channel_case

pytestmark = pytest.mark.gpu


def pair(case, **extra):
    from oracle import Oracle
    import channelflow as cf
    o = Oracle(case["x"], case["y"], case["z"], case["prm"])
    o.set_fields(case["U"], case["V"], case["W"])
    kw = dict(case["prm"])
    kw.update(extra)
    ch = cf.Channel(case["x"], case["y"], case["z"], precision=0, **kw)
    ch.upload(case["U"], case["V"], case["W"])
    return o, ch


@pytest.mark.parametrize("dims", [(6, 5, 6), (12, 9, 10), (18, 10, 14), (32, 11, 22), (34, 18, 18), (20, 130, 8)])
def test_projection_edges(dims):
    """One projection of a field that is far from divergence-free: U, V, W
    within the per-routine 1e-12 of the oracle, P (a Poisson solution of
    condition number ~(rows)^2, so 1e-16 times at most 2e4) within 1e-11."""
    case = channel_case(*dims)
    o, ch = pair(case)
    for d in (o, ch):
        d.apply_boundary_conditions()
    ch.set_scalars(dt=case["dt"], rk_step=1)
    o.set_scalar("dt", case["dt"])
    o.set_scalar("rk_step", 1)
    for d in (o, ch):
        d.compute_projection_step()
        d.apply_boundary_conditions()
    g, f = ch.download(), o.fields()
    for n in ("U", "V", "W"):
        assert_close(g[n], f[n], 1e-12, n)
    assert_close(g["P"], f["P"], 1e-11, "P")
    ch.close()
    o.close()


# every transform length with a compile-time plan (even, factors 2, 3, 5, 16 to
# 512), and two outside that range
LENGTHS = sorted(a * b * c for a in (2, 4, 8, 16, 32, 64, 128, 256, 512) for b in (1, 3, 9, 27, 81, 243)
                 for c in (1, 5, 25, 125) if 16 <= a * b * c <= 512) + [12, 540]


@pytest.mark.parametrize("nx,nz", list(zip(LENGTHS, reversed(LENGTHS))))
def test_projection_lengths(nx, nz):
    """Transforms of every length in x and in z, in both precisions, with the
    last block of lines partly full: the FP64 projection within the
    per-routine 1e-12 of the oracle's (P within 1e-11, as above), the split
    path's (FP32 transforms) within the 1e-5 (P 1e-3) it is held to elsewhere."""
    import channelflow as cf
    case = channel_case(nx + 2, 7, nz + 2)
    o, ch = pair(case)
    sp = cf.Channel(case["x"], case["y"], case["z"], precision=cf.PREC_SPLIT, **case["prm"])
    sp.upload(case["U"], case["V"], case["W"])
    o.set_scalar("dt", case["dt"])
    o.set_scalar("rk_step", 1)
    for d in (ch, sp):
        d.set_scalars(dt=case["dt"], rk_step=1)
    for d in (o, ch, sp):
        d.apply_boundary_conditions()
        d.compute_projection_step()
        d.apply_boundary_conditions()
    f, g, h = o.fields(), ch.download(), sp.download()
    for n in ("U", "V", "W"):
        assert_close(g[n], f[n], 1e-12, n)
        assert_close(h[n], g[n], 1e-5, n)
    assert_close(g["P"], f["P"], 1e-11, "P")
    assert_close(h["P"], g["P"], 1e-3, "P")
    ch.close()
    sp.close()
    o.close()


@pytest.mark.parametrize("dims,wall,kw", [((6, 5, 6), 0, {}), ((18, 6, 8), 0, {}), ((22, 9, 34), 0, {"dirichlet": 1}),
                                          ((34, 17, 12), 0, {}), ((50, 7, 18), 0, {}), ((66, 12, 20), 0, {}),
                                          ((18, 17, 18), 3, {}), ((34, 8, 22), 3, {}), ((50, 13, 10), 3, {})])
def test_dsm_segments_and_chunks(dims, wall, kw):
    """The FP64 dynamic Smagorinsky pass with one and several row segments of
    16 and 32 lanes, full and ragged, rows packed in pairs (odd and even row
    counts), chunks of one plane and more; with the wall model after an eqwm
    boundary update, whose wall ghosts are not periodic at the seams.  nu_t
    and the plane coefficients within the per-routine 1e-12."""
    if wall:
        case = channel_case(*dims, stretch=0.0, wall=3, retau=2000.0, profile="plug", jref=2, ncv=30)
    else:
        case = channel_case(*dims)
    if "dirichlet" in kw:
        case["prm"]["Dirichlet_nu_t"] = kw["dirichlet"]
    o, ch = pair(case)
    for d in (o, ch):
        d.apply_boundary_conditions()
        d.compute_eddy_viscosity()
        if wall:
            d.compute_wall_model()
            d.apply_boundary_conditions()
            d.compute_eddy_viscosity()
    assert_close(ch.download()["nu_t"], o.fields()["nu_t"], 1e-12, "nu_t")
    assert_close(ch.avg_nu_t()[1:-1], o.array("avg_nu_t").ravel()[1:-1], 1e-12, "avg_nu_t")
    ch.close()
    o.close()


@pytest.mark.parametrize("dims,les,wall,vary,kw", [((6, 5, 6), 0, 0, True, {}), ((18, 9, 10), 2, 0, False, {}),
                                                   ((34, 16, 8), 3, 0, True, {}),
                                                   ((22, 17, 66), 2, 0, False, dict(Rossby_plus=2.0)),
                                                   ((50, 33, 14), 2, 0, False, {}), ((66, 10, 12), 2, 3, False, {}),
                                                   ((98, 23, 6), 0, 0, True, dict(Rossby_plus=2.0)),
                                                   ((18, 10, 130), 3, 0, True, {})])
def test_rhs_segments_rows_and_chunks(dims, les, wall, vary, kw):
    """The FP64 fused right-hand side through one whole step: segments of 16
    and 32 lanes, full and ragged, one and several row tiles with full and
    partial last tiles, one and several chunks, with rotation, with and
    without eddy viscosity and wall model.  vary: x and z spacings that
    change from cell to cell, where the reference's upper- and lower-face
    formulas differ (not with the dynamic model, whose plane sums the library
    takes with the duplicate column as a copy, which it is on uniform x and z
    only).  U, V, W after the step within the per-routine 1e-12."""
    nx, ny, nz = dims
    case = channel_case(*dims, les=les, wall=wall, stretch=0.0 if wall else 1.5, retau=2000.0 if wall else 180.0,
                        profile="plug" if wall else "laminar", jref=2, ncv=30)
    if vary:
        for c, n in (("x", nx), ("z", nz)):
            d = np.diff(case[c])
            d *= 1.0 + 0.2 * np.cos(2 * np.pi * np.arange(n - 1) / (n - 2))  # periodic over the n - 2 cells
            case[c] = np.concatenate([[0.0], np.cumsum(d)])
    case["prm"].update(kw)
    o, ch = pair(case)
    for d in (o, ch):
        d.init_mass_flow()
        d.apply_boundary_conditions()
    o.compute_dt()
    o.time_step_rk3()
    ch.time_step_rk3(1)
    g, f = ch.download(), o.fields()
    for n in ("U", "V", "W"):
        assert_close(g[n], f[n], 1e-12, n)
    ch.close()
    o.close()


def eqwm_stress(u_les, h, nu, ncv, stretch, tau):
    """The wall stress of solve_u_eqwm (eqwm.f90:20-223) in extended precision:
    the same Picard passes to the same criterion, each from the resistances of
    the faces in series, which is what the tridiagonal system solves."""
    L = np.longdouble
    fa = np.concatenate([[0.0], np.cumsum(np.cumprod(np.r_[1.0, np.full(ncv - 1, stretch)]))])
    cv = (fa[1:] + fa[:-1]) / 2
    fa, cv = (fa / cv[-1] * h).astype(L), (cv / cv[-1] * h).astype(L)
    u_les, nu, tau = u_les.astype(L), L(nu), tau.astype(L)
    tol, run = L("1e-7") * nu * u_les / L(h), np.full(tau.shape, True)
    for _ in range(101):
        ut = np.sqrt(tau)
        r = (cv[0] - fa[0]) / nu + np.zeros_like(tau)
        for q in range(1, ncv):
            y = fa[q]
            r += (cv[q] - cv[q - 1]) / (nu + L("0.41") * ut * y * (1 - np.exp(-y * ut / nu / 17)) ** 2)
        new = u_les / r
        tau, run = np.where(run, new, tau), run & ~(np.abs(new - tau) < tol)
        if not run.any():
            break
    return tau.astype(float)


@pytest.mark.parametrize("dims,ncv,stretch", [((18, 9, 18), 30, 1.10), ((18, 9, 18), 100, 1.10), ((18, 9, 18), 3, 1.10),
                                              ((18, 9, 18), 2000, 1.001), ((50, 9, 50), 45, 1.10),
                                              ((66, 9, 82), 30, 1.10), ((130, 9, 130), 30, 1.10)])
def test_eqwm_lanes_per_point(dims, ncv, stretch):
    """The FP64 equilibrium wall model with one to eight lanes per wall point
    (the count falls with the number of points), few and many ODE cells, with
    and without room for the kept exponentials; a first call from the mean
    stress and a second one from the first's result.  Both iterate the same
    map to the same criterion, so that they stop at the same pass and agree to
    rounding: 1e-12, counters equal.  With 2000 cells the oracle's Thomas sweep
    is itself 1e-12 to 1e-11 from the exact solution of its system (its
    rounding grows as the square of the cells), so that the stress is held to
    the same passes in extended precision and alpha_x to the oracle's
    alpha_x / stress."""
    case = channel_case(*dims, stretch=0.0, wall=3, retau=2000.0, profile="plug", jref=3, ncv=ncv)
    case["prm"]["eqwm_stretch"] = stretch
    from channelflow.wallmlp import wall_model_inputs
    o, ch = pair(case)
    for d in (o, ch):
        d.apply_boundary_conditions()
        d.compute_eddy_viscosity()
    for _ in range(2):
        if ncv > 1000:
            u_les, h, nu = (v.cpu().numpy() if hasattr(v, "cpu") else v for v in wall_model_inputs(ch))
            tau_in = ch.download_wall()["tau_eqwm_initial"]
            want = eqwm_stress(u_les.reshape(tau_in.shape, order="F"), h, nu, ncv, stretch, tau_in)
        o.compute_wall_model()
        ch.compute_wall_model()
        w = ch.download_wall()
        if ncv > 1000:
            tau, t0 = w["tau_eqwm_initial"], o.array("tau_eqwm_initial")
            assert_close(tau, want, 1e-12, "tau_eqwm_initial")
            assert_close(w["alpha_x"] / tau, o.array("alpha_x") / t0, 1e-12, "alpha_x / tau")
        else:
            for n in ("alpha_x", "alpha_z", "tau_eqwm_initial"):
                assert_close(w[n], o.array(n), 1e-12, n)
        assert ch.eqwm_counters() == (int(o.scalar("n_nan_eqwm")), int(o.scalar("n_iter_eqwm")))
    ch.close()
    o.close()
