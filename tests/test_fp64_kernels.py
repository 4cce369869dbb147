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
