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
