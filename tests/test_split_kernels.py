"""Split-path kernels at the sizes where their tilings, chunks and tails end,
against the FP64 path on the same inputs."""
import numpy as np
import pytest

from conftest import channel_case, rel_err

pytestmark = pytest.mark.gpu


def run_pair(case, calls, **extra):
    """The same calls on an FP64 and a split-path channel; both channels."""
    import channelflow as cf
    out = []
    for prec in (cf.PREC_FP64, cf.PREC_SPLIT):
        kw = dict(case["prm"])
        kw.update(extra)
        ch = cf.Channel(case["x"], case["y"], case["z"], precision=prec, **kw)
        ch.upload(case["U"], case["V"], case["W"])
        calls(ch)
        out.append(ch)
    return out


@pytest.mark.parametrize("dims,wall,dirichlet", [((6, 5, 6), 0, 0), ((18, 6, 8), 0, 0), ((20, 9, 34), 0, 1),
                                                 ((34, 17, 12), 0, 0), ((50, 7, 18), 0, 0), ((66, 12, 20), 0, 0),
                                                 ((98, 14, 10), 0, 0), ((130, 10, 8), 0, 1), ((102, 13, 38), 0, 0),
                                                 ((18, 17, 18), 3, 0), ((34, 8, 22), 3, 0), ((130, 11, 10), 3, 0)])
def test_dsm_segments_and_chunks(dims, wall, dirichlet):
    """The FP32 dynamic Smagorinsky pass with segments of 16, 32 and 64
    columns, full and ragged, several rows to a warp, chunks of one plane and
    more, ghosts unfilled at the first call; with the wall model after an eqwm
    boundary update.  The velocities (up to 1.5) are rounded to FP32 and the
    strain rates are differences of neighbours of order 0.1: relative errors of
    1e-6 per difference; C(j) and nu_t are held to the 2e-4 the split path's
    eddy viscosity is held to elsewhere."""
    if wall:
        case = channel_case(*dims, stretch=0.0, wall=3, retau=2000.0, profile="plug", jref=2, ncv=30)
    else:
        case = channel_case(*dims)
    case["prm"]["Dirichlet_nu_t"] = dirichlet

    def calls(ch):
        ch.apply_boundary_conditions()
        ch.compute_eddy_viscosity()
        if wall:
            ch.compute_wall_model()
            ch.apply_boundary_conditions()
            ch.compute_eddy_viscosity()

    a, b = run_pair(case, calls)
    assert rel_err(b.avg_nu_t()[1:-1], a.avg_nu_t()[1:-1]) <= 2e-4
    assert rel_err(b.download()["nu_t"], a.download()["nu_t"]) <= 2e-4
    a.close()
    b.close()


@pytest.mark.parametrize("dims,les,wall,vary,kw", [((6, 5, 6), 0, 0, False, {}), ((18, 6, 8), 2, 0, False, {}),
                                                   ((20, 9, 34), 0, 0, True, dict(Rossby_plus=2.0)),
                                                   ((34, 17, 12), 3, 0, True, {}), ((50, 12, 18), 2, 3, False, {}),
                                                   ((66, 7, 20), 2, 0, False, dict(Dirichlet_nu_t=1)),
                                                   ((98, 14, 10), 0, 0, True, {}), ((130, 10, 8), 3, 0, True, dict(Rossby_plus=2.0)),
                                                   ((18, 21, 74), 2, 0, False, {})])
def test_rhs_tiles_and_chunks(dims, les, wall, vary, kw):
    """The FP32 right-hand side with the update through one whole step: tiles
    of 64 x 4, 32 x 8 and 16 x 16 cells, full and ragged, chunks of one plane
    and more, nu_t from |S| and from its field, rotation, x and z spacings
    that change from cell to cell (vary).  A right-hand side is a sum of about
    20 terms of at most U^2/dx, each rounded to FP32: 1.2e-6 of the largest,
    so that dt times it is 6e-7 U off at CFL 0.5, three times a step, against
    fluctuations of V and W of a tenth of U: 2e-5."""
    nx, ny, nz = dims
    case = channel_case(*dims, les=les, wall=wall, stretch=0.0 if wall else 1.5, retau=2000.0 if wall else 180.0,
                        profile="plug" if wall else "laminar", jref=2, ncv=30)
    if vary:
        for c, n in (("x", nx), ("z", nz)):
            d = np.diff(case[c])
            d *= 1.0 + 0.2 * np.cos(2 * np.pi * np.arange(n - 1) / (n - 2))  # periodic over the n - 2 cells
            case[c] = np.concatenate([[0.0], np.cumsum(d)])

    def calls(ch):
        ch.init_mass_flow()
        ch.apply_boundary_conditions()
        ch.set_fixed_dt(case["dt"])
        ch.time_step_rk3(1)

    a, b = run_pair(case, calls, **kw)
    f, g = a.download(), b.download()
    for n in ("U", "V", "W"):
        assert rel_err(g[n], f[n]) <= 2e-5, n
    a.close()
    b.close()


@pytest.mark.parametrize("dims,rule", [((6, 5, 6), 0), ((18, 6, 8), 1), ((20, 9, 34), 2), ((34, 17, 12), 0), ((50, 7, 18), 1),
                                       ((66, 12, 20), 0), ((98, 14, 10), 2), ((130, 10, 8), 0), ((102, 13, 38), 1)])
def test_amd_tiles_and_chunks(dims, rule):
    """The FP32 anisotropic minimum dissipation pass with tiles of 64 x 4,
    32 x 8 and 16 x 16 cells, full and ragged, chunks of one plane and more,
    the duplicate and ghost images and the three wall rules.  Velocities of up
    to 1.5 rounded to FP32 and differences of order 0.1 as in the dynamic
    model's test: nu_t and its plane means within 2e-4."""
    case = channel_case(*dims, les=3)
    case["prm"]["Dirichlet_nu_t"] = rule

    def calls(ch):
        ch.apply_boundary_conditions()
        ch.compute_eddy_viscosity()

    a, b = run_pair(case, calls)
    assert rel_err(b.download()["nu_t"], a.download()["nu_t"]) <= 2e-4
    assert rel_err(b.avg_nu_t()[1:-1], a.avg_nu_t()[1:-1]) <= 2e-4
    a.close()
    b.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_nut_of_steps_after_uploads(prec):
    """nu_t downloaded after each step of a state uploaded without its ghosts
    filled, and after a step of each of several uploads: bit for bit that of a
    channel that is stepped once from the upload on and downloaded once."""
    import channelflow as cf
    case = channel_case(18, 9, 18, mass=0)

    def make(scale):
        ch = cf.Channel(case["x"], case["y"], case["z"], precision=prec, **case["prm"])
        ch.upload(scale * case["U"], scale * case["V"], scale * case["W"])
        ch.set_fixed_dt(case["dt"])
        return ch

    ch = make(1.0)
    for n in range(1, 5):
        ch.time_step_rk3(1)
        got = ch.download()["nu_t"]
        ref = make(1.0)
        ref.time_step_rk3(n)
        assert np.array_equal(got, ref.download()["nu_t"]), n
        ref.close()
    for n in range(6):
        scale = 1.0 + 0.1 * n
        ch.upload(scale * case["U"], scale * case["V"], scale * case["W"])
        ch.time_step_rk3(1)
        got = ch.download()["nu_t"]
        ref = make(scale)
        ref.time_step_rk3(1)
        assert np.array_equal(got, ref.download()["nu_t"]), scale
        ref.close()
    ch.close()
