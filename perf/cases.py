"""Performance cases of the channel solver: what its users run, through the public entry points.

A case advances seeded turbulent channels by a few RK3 steps and fetches the
fields, as a simulation does between two outputs (nmonitor / nsave of the
input_parameters file).  Three kinds:

  step      Channel.time_step_rk3 -- the device-resident fast path
  mirror    compute_dt + compute_time_step_rk3_mirror -- the call sequence of
            the Fortran drop-in, one subroutine at a time
  ensemble  Ensemble.step over independent channels of several grids

Fields of the FP64 path are returned as they arrive in the pinned host
buffers; fields of the split path (FP32 state) are handed on as FP32 device
tensors, the precision they carry, as a post-processing program keeps them.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "channel-flow_gb300"))

NONE, DSM, AMD = 0, 2, 3  # LES_model
EQWM = 3                  # iwall_model


def _case(name, kind, precision, nx, ny, nz, steps, retau, **kw):
    """nx, ny, nz are numbers of cells; the options not given take the values
    a plain channel simulation uses."""
    c = dict(name=name, kind=kind, precision=precision, nx=nx, ny=ny, nz=nz, steps=steps, retau=float(retau),
             les=DSM, wall=0, jref=3, ncv=30, stretch=1.5, mass=1, rossby=0.0, dirichlet=0, members="")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest grid the tests and the smoke run use: latency of a step's launches
        _case("tiny_dsm_fp64", "step", "fp64", 16, 16, 16, 5, 180),
        # Re_tau 180 in a small box, the production precision: a debugging or teaching run
        _case("re180_dsm_split", "step", "split", 64, 64, 64, 10, 180),
        # a ragged grid (radix 3 and 5 transforms, odd row count), rotating channel at a fixed
        # pressure gradient with the Dirichlet rule of nu_t
        _case("ragged_dsm_split", "step", "split", 100, 75, 90, 10, 395, mass=0, rossby=0.5, dirichlet=1),
        # the headline workload: wall-resolved LES at Re_tau 550
        _case("re550_dsm_split", "step", "split", 192, 128, 192, 10, 550),
        # the same in the default precision, the parity path with the reference
        _case("re550_dsm_fp64", "step", "fp64", 192, 128, 192, 2, 550),
        # the headline grid with the anisotropic minimum dissipation model
        _case("re550_amd_split", "step", "split", 192, 128, 192, 10, 550, les=AMD),
        # a ragged AMD run in the default precision
        _case("ragged_amd_fp64", "step", "fp64", 120, 81, 96, 4, 395, les=AMD),
        # wall-modelled LES at Re_tau 2000
        _case("re2000_eqwm_split", "step", "split", 256, 96, 256, 6, 2000, wall=EQWM, jref=6, stretch=0.0),
        # a coarse wall-modelled run in the default precision with the reference's 100 ODE cells
        _case("re1000_eqwm_fp64", "step", "fp64", 64, 48, 64, 4, 1000, wall=EQWM, jref=4, stretch=0.0, ncv=100),
        # the largest production grid: wall-modelled LES at Re_tau 5200
        _case("re5200_eqwm_split", "step", "split", 512, 128, 512, 6, 5200, wall=EQWM, jref=8, stretch=0.0),
        # the Fortran drop-in: the reference's call sequence, one subroutine per call
        _case("mirror_dsm_fp64", "mirror", "fp64", 64, 48, 64, 4, 180),
        # a parameter study: independent channels advanced together
        _case("ensemble_split", "ensemble", "split", 0, 0, 0, 4, 395,
              members="64x64x64,64x64x64,64x64x64,96x64x96,96x64x96,96x64x96,128x96x128,128x96x128"),
    ]


# even lengths of the periodic directions that factor into 2, 3 and 5
LENGTHS = sorted(n for n in {2 ** a * 3 ** b * 5 ** c for a in range(1, 10) for b in range(6) for c in range(4)}
                 if 16 <= n <= 512)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(LENGTHS, key=lambda n: abs(math.log(n / want)))


def draw(rng):
    kind = rng.choice(["step"] * 8 + ["mirror", "ensemble"])
    precision = rng.choice(["split", "split", "fp64"])
    # cell-steps of a pass: at most a tenth of the largest listed case in FP64 (its step costs up
    # to thirty times the split one's per cell), at most half of it in the split path
    budget = 1.0e7 if precision == "fp64" else 1.0e8
    if kind == "ensemble":
        steps = rng.randint(2, 4)
        n = rng.randint(3, 10)
        members = ",".join("%dx%dx%d" % (_length(rng, 32, 96), _log_int(rng, 24, 96), _length(rng, 32, 96))
                           for _ in range(n))
        if precision == "fp64":
            members = ",".join(members.split(",")[:4])
        return _unnamed(kind, precision, 0, 0, 0, steps, rng.uniform(150, 700), les=rng.choice([DSM, DSM, AMD]),
                        members=members)
    steps = rng.randint(2, 8)
    les = rng.choice([DSM, DSM, DSM, AMD, NONE])
    wall = rng.choice([0, 0, EQWM])
    for _ in range(1000):
        nx, ny, nz = _length(rng, 16, 512), _log_int(rng, 12, 160), _length(rng, 16, 512)
        if nx * ny * nz * steps <= budget:
            break
    else:
        nx, ny, nz = 64, 49, 64
    if wall:
        return _unnamed(kind, precision, nx, ny, nz, steps, rng.uniform(500, 6000), les=les, wall=wall,
                        jref=rng.randint(2, max(2, min(8, ny // 3))), ncv=rng.choice([20, 30, 45, 100]), stretch=0.0)
    return _unnamed(kind, precision, nx, ny, nz, steps, rng.uniform(150, 700), les=les,
                    mass=rng.choice([1, 1, 0]), rossby=rng.choice([0.0, 0.0, 0.5]), dirichlet=rng.choice([0, 0, 1]),
                    stretch=rng.choice([1.5, 1.5, 1.2, 0.0]))


def _unnamed(*args, **kw):
    c = _case("", *args, **kw)
    del c["name"]
    return c


def _channels(case):
    """The single channels of a case: (cells, seed offset) of each."""
    if case["kind"] != "ensemble":
        return [(case["nx"], case["ny"], case["nz"])]
    return [tuple(int(v) for v in m.split("x")) for m in case["members"].split(",")]


def _params(case):
    nu = 2.0 / (case["retau"] / 0.09) ** (1.0 / 0.88)  # Dean's correlation, unit bulk velocity and half-height
    return dict(nu=nu, CFL=0.5, dPdx=(case["retau"] * nu) ** 2, Rossby_plus=case["rossby"], x_mass_cte=case["mass"],
                LES_model=case["les"], iwall_model=case["wall"], Dirichlet_nu_t=case["dirichlet"],
                jref_eqwm=case["jref"], eqwm_ncv=case["ncv"])


def _faces(cells, stretch):
    """Face coordinates x, y, z of a 2 pi x 2 x pi channel: cells + 2, cells + 1
    and cells + 2 faces, as the input_parameters file counts them."""
    nxp, nym, nzp = cells
    x = np.arange(nxp + 2, dtype=np.float64) * (2 * math.pi / nxp)
    z = np.arange(nzp + 2, dtype=np.float64) * (math.pi / nzp)
    y = 2.0 * np.arange(nym + 1, dtype=np.float64) / nym - 1.0
    if stretch > 0:
        y = np.tanh(stretch * y) / math.tanh(stretch)
    return x, (y - y[0]) * (2.0 / (y[-1] - y[0])), z


def _centres(f):
    m = 0.5 * (f[:-1] + f[1:])
    return np.concatenate([[2 * f[0] - m[0]], m, [2 * f[-1] - m[-1]]])


def _wrap(n, n_per):
    """0-based canonical position (0..n_per-1) of each of n stored entries
    (the first one is the periodic image below the first canonical entry)."""
    return torch.arange(-1, n - 1) % n_per


def _fields(cells, stretch, seed, dev):
    """A turbulent-looking channel: a 1/7 power-law mean profile of unit bulk
    velocity plus broadband fluctuations of about a tenth of it that vanish at
    the walls, the discrete curl of a random vector potential and therefore
    divergence-free on the staggered grid.  U, V, W on the unique cells with V
    on all faces, [z][y][x], FP64."""
    nxp, nym, nzp = cells
    x, y, z = _faces(cells, stretch)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)
    yg = t(_centres(y))[1:-1]
    yf = t(y)
    dx, dz = x[1] - x[0], z[1] - z[0]
    kx = torch.arange(nxp // 2 + 1, device=dev, dtype=torch.float64)
    kz = torch.fft.fftfreq(nzp, 1.0 / nzp, device=dev, dtype=torch.float64) * 2.0
    k2 = kz[:, None] ** 2 + kx[None, :] ** 2
    spec = (1.0 + k2 / 16.0) ** (-17.0 / 12.0 - 0.25)
    spec = torch.where(k2 > (0.66 * min(nxp, 2 * nzp) / 2) ** 2, torch.zeros_like(spec), spec)
    spec[0, 0] = 0.0

    def potential(rows, shape):
        a = torch.randn((nzp, rows, nxp), generator=gen, device=dev, dtype=torch.float64)
        for _ in range(6):  # correlated over a few rows in y
            b = a.clone()
            b[:, 1:] += 0.5 * a[:, :-1]
            b[:, :-1] += 0.5 * a[:, 1:]
            a = 0.5 * b
        h = torch.fft.rfftn(a, dim=(0, 2)) * spec[:, None, :]
        a = torch.fft.irfftn(h, s=(nzp, nxp), dim=(0, 2))
        return a * shape[None, :, None]

    wf, wc = yf * (2.0 - yf), yg * (2.0 - yg)
    Ax, Ay, Az = potential(nym + 1, wf ** 2), potential(nym, wc ** 2), potential(nym + 1, wf ** 2)
    dy = (yf[1:] - yf[:-1])[None, :, None]
    # a face array's entry is the upper face of its cell: the difference over a cell is F - roll(F, 1)
    dn = lambda a, d: torch.roll(a, 1, d)
    U = (Az[:, 1:] - Az[:, :-1]) / dy - (Ay - dn(Ay, 0)) / dz
    V = (Ax - dn(Ax, 0)) / dz - (Az - dn(Az, 2)) / dx
    W = (Ay - dn(Ay, 2)) / dx - (Ax[:, 1:] - Ax[:, :-1]) / dy
    scale = 0.1 / torch.sqrt((U * U).mean() + 1e-300)
    U, V, W = U * scale, V * scale, W * scale
    V[:, 0] = 0.0
    V[:, -1] = 0.0
    eta = torch.clamp(1.0 - (1.0 - yg).abs(), 0.0, 1.0)
    U += (8.0 / 7.0) * eta[None, :, None] ** (1.0 / 7.0)
    return U, V, W


def _stored(U, V, W):
    """The arrays the solver takes, [z][y][x] with the ghost layers and
    periodic duplicates of a no-slip channel (the wall model refills its own
    ghosts): x fastest, which is the Fortran array (nx, ny+1, nz+1)."""
    nzp, nym, nxp = U.shape
    ix, ixc = _wrap(nxp + 2, nxp).to(U.device), _wrap(nxp + 3, nxp).to(U.device)
    iz, izc = _wrap(nzp + 2, nzp).to(U.device), _wrap(nzp + 3, nzp).to(U.device)
    u = U[izc][:, :, ix]
    u = torch.cat([-u[:, :1], u, -u[:, -1:]], 1)
    v = V[izc][:, :, ixc]
    w = W[iz][:, :, ixc]
    w = torch.cat([-w[:, :1], w, -w[:, -1:]], 1)
    return u, v, w


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _outputs(case):
    """Names of the fields a pass returns: the velocities, the eddy viscosity
    and, in FP64, the pressure (in FP32 the pseudo-pressure of one substep is
    mostly rounding: it carries the O(dt) cancellation of div u)."""
    names = ["U", "V", "W"]
    if case["les"] != NONE:
        names.append("nu_t")
    if case["precision"] == "fp64":
        names.append("P")
    return names


def prepare(case, seed):
    import channelflow as cf
    dev = torch.device("cuda")
    prec = cf.PREC_FP64 if case["precision"] == "fp64" else cf.PREC_SPLIT
    chans, bufs = [], []
    for m, cells in enumerate(_channels(case)):
        x, y, z = _faces(cells, case["stretch"])
        ch = cf.Channel(x, y, z, precision=prec, **_params(case))
        host = [_pinned(a.shape).copy_(a) for a in _stored(*_fields(cells, case["stretch"], seed * 64 + m, dev))]
        ch.upload(*(h.numpy().T for h in host))
        ch.init_mass_flow()
        ch.apply_boundary_conditions()
        buf = dict(zip("UVW", host))
        for n in _outputs(case)[3:]:
            buf[n] = _pinned(tuple(reversed(ch.shapes[n])))
        chans.append(ch)
        bufs.append(buf)
    # members solve their own pressure systems inside their branches, the mode the autotuner
    # keeps for ensembles of this kind
    ens = cf.Ensemble(chans, batched_tri=False) if case["kind"] == "ensemble" else None
    return dict(case=dict(case), chans=chans, bufs=bufs, ens=ens)


def run(state):
    case, n = state["case"], state["case"]["steps"]
    if case["kind"] == "ensemble":
        state["ens"].step(n)
    elif case["kind"] == "mirror":
        ch = state["chans"][0]
        for _ in range(n):
            ch.compute_dt()
            ch.compute_time_step_rk3_mirror()
    else:
        state["chans"][0].time_step_rk3(n)
    out = []
    for ch, buf in zip(state["chans"], state["bufs"]):
        ch.download_into(**{k: b.numpy().T for k, b in buf.items()})
        if case["precision"] == "fp64":
            out.append(dict(buf))
        else:
            out.append({k: b.to("cuda").float() for k, b in buf.items()})
    return out


def work(case):
    """One read or write of a field per pass that the data dependencies of a
    step force -- per substep: velocities in and one field out for the eddy
    viscosity (plane averages of all of it precede the right-hand side),
    velocities, nu_t, old state and F1 in and the new state out for the
    right-hand side, divergence to spectrum, the y solves, back to the
    pressure, and the projection; per step the mass flow and the dt rule --
    plus the fields fetched at the end.  FP64: 8 B everywhere; split: 4 B, old
    state and spectrum 8 B.  Operations: those of the formulas per cell."""
    nbytes = flops = 0.0
    fp64 = case["precision"] == "fp64"
    for nxp, nym, nzp in _channels(case):
        cells = nxp * nym * nzp
        es, wide = (8, 8) if fp64 else (4, 8)
        les = 4 * 3 * es if case["les"] != NONE else 0
        rhs = 3 * (3 + 1) * es + 9 * wide + 6 * es + 6 * es + 3 * wide
        poisson = 3 * (3 * es + wide + 2 * wide + wide + es)
        proj = 3 * 7 * es
        nbytes += cells * (case["steps"] * (les + rhs + poisson + proj + 2 * es + 3 * es) + 8.0 * len(_outputs(case)))
        ops = {DSM: 450, AMD: 330, NONE: 0}[case["les"]]
        fft = 2 * 2.5 * (math.log2(nxp) + math.log2(nzp))
        flops += cells * case["steps"] * 3.0 * (ops + 190 + fft + 20 + 15)
        if case["wall"]:  # eqwm: a few passes of an ODE solve per wall point
            flops += case["steps"] * 2 * nxp * nzp * 3 * case["ncv"] * 30
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    """The first pass in 64 bits by plain torch operations on the same
    inputs."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    out = []
    for m, cells in enumerate(_channels(case)):
        s = _Step64(case, cells, *_fields(cells, case["stretch"], seed * 64 + m, dev))
        for _ in range(case["steps"]):
            s.step()
        got = dict(U=s.U, V=s.V, W=s.W, nu_t=s.nut, P=s.P)
        out.append({n: got[n] for n in _outputs(case)})
    return out


class _Step64:
    """The RK3 step on stored arrays [z][y][x] (ghosts and duplicates
    included), written from the scheme: staggered second-order differences,
    modified-wavenumber pressure solve, RK3 with the (8/15, 1/4, 5/12, 1/4, 0,
    3/4) weights, constant mass flow."""

    def __init__(self, case, cells, U, V, W):
        self.dev = U.device
        self.case, p = case, _params(case)
        self.nu, self.les, self.wall = p["nu"], p["LES_model"], p["iwall_model"]
        self.dirichlet, self.dPdx, self.Om = p["Dirichlet_nu_t"], p["dPdx"], p["Rossby_plus"] * math.sqrt(p["dPdx"]) / 2
        self.tau_mean, self.mass = p["dPdx"], p["x_mass_cte"]
        self.jref, self.ncv, self.cfl = p["jref_eqwm"], p["eqwm_ncv"], p["CFL"]
        self.nxp, self.nym, self.nzp = cells
        self.hx, self.hy, self.hz = _faces(cells, case["stretch"])
        self.hxg, self.hyg, self.hzg = (_centres(a) for a in (self.hx, self.hy, self.hz))
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=self.dev)
        self.x, self.xg = t(self.hx), t(self.hxg)
        self.y, self.yg = t(self.hy)[:, None], t(self.hyg)[:, None]
        self.z, self.zg = t(self.hz)[:, None, None], t(self.hzg)[:, None, None]
        w0 = (self.yg[1:] - self.y) / (self.yg[1:] - self.yg[:-1])  # weight of the row below a face
        self.w0, self.w1 = w0, 1.0 - w0
        nx, nz = self.nxp + 2, self.nzp + 2
        idx = lambda n, m: _wrap(n, m).to(self.dev)
        self.ix, self.ixc = idx(nx, self.nxp), idx(nx + 1, self.nxp)
        self.iz, self.izc = idx(nz, self.nzp), idx(nz + 1, self.nzp)
        self.U, self.V, self.W = _stored(U, V, W)
        # wall model: stress per wall point [z][wall][x] and the wall-normal gradients it gives
        self.tau = torch.full((nz + 1, 2, nx), self.tau_mean, dtype=torch.float64, device=self.dev)
        self.ax = torch.zeros((nz + 1, 2, nx), dtype=torch.float64, device=self.dev)
        self.az = torch.zeros((nz, 2, nx + 1), dtype=torch.float64, device=self.dev)
        self.nut = torch.zeros((nz + 1, self.nym + 2, nx + 1), dtype=torch.float64, device=self.dev)
        self.P = torch.zeros_like(self.nut)
        self.Q0 = self.flow()
        self.bc()
        self.poisson_setup()

    # canonical cells of a stored array shifted by (a, b, c) in x, y, z
    def c(self, F, a=0, b=0, c=0, rows=None):
        n = self.nym if rows is None else rows
        return F[1 + c:1 + c + self.nzp, 1 + b:1 + b + n, 1 + a:1 + a + self.nxp]

    def dx(self, a=0):   # x(i+a) - x(i+a-1)
        return self.x[1 + a:1 + a + self.nxp] - self.x[a:a + self.nxp]

    def dxg(self, a=0):
        return self.xg[1 + a:1 + a + self.nxp] - self.xg[a:a + self.nxp]

    def dy(self, b=0, rows=None):
        n = self.nym if rows is None else rows
        return self.y[1 + b:1 + b + n] - self.y[b:b + n]

    def dyg(self, b=0, rows=None):
        n = self.nym if rows is None else rows
        return self.yg[1 + b:1 + b + n] - self.yg[b:b + n]

    def dz(self, c=0):
        return self.z[1 + c:1 + c + self.nzp] - self.z[c:c + self.nzp]

    def dzg(self, c=0):
        return self.zg[1 + c:1 + c + self.nzp] - self.zg[c:c + self.nzp]

    def bc(self):
        """Periodic images from the canonical entries, then the walls."""
        U, V, W = self.c(self.U), self.V[1:1 + self.nzp, :, 1:1 + self.nxp], self.c(self.W)
        U, V, W = U[self.izc][:, :, self.ix], V[self.izc][:, :, self.ixc].clone(), W[self.iz][:, :, self.ixc]
        V[:, 0] = 0.0
        V[:, -1] = 0.0
        if self.wall:
            d0, d1 = self.hyg[1] - self.hyg[0], self.hyg[-1] - self.hyg[-2]
            ends = lambda F, al: (F[:, :1] - d0 * al[:, :1], F[:, -1:] - d1 * al[:, 1:])
            (u0, u1), (w0, w1) = ends(U, self.ax), ends(W, self.az)
        else:
            u0, u1, w0, w1 = -U[:, :1], -U[:, -1:], -W[:, :1], -W[:, -1:]
        self.U, self.V, self.W = torch.cat([u0, U, u1], 1), V, torch.cat([w0, W, w1], 1)

    def flow(self):
        """Mean of U by the trapezoid rule between the first and last centres;
        the planes counted are the canonical ones and the first again."""
        u = self.c(self.U)
        h = self.dyg(1, self.nym - 1)
        s = ((u[:, 1:] + u[:, :-1]) * 0.5 * h).sum((1, 2))
        return float((s.sum() + s[0]) / (h.sum() * self.nxp * (self.nzp + 1)))

    def dt_rule(self):
        # spacing over |velocity| at its largest, over all interior points; then the viscous limit and the cap
        U, V, W = self.U[1:-1, 1:-1, 1:], self.V[1:-1, 1:, 1:-1], self.W[1:, 1:-1, 1:-1]
        lu = (self.dxg(1)[0] / U.abs().min()).item()
        dyc = (self.yg[2:] - self.yg[1:-1]).reshape(-1)
        lv = (dyc / V.abs().amin((0, 2))).max().item()
        lw = (self.dzg(1).reshape(-1)[0] / W.abs().min()).item()
        lim = [(np.diff(g).min()) ** 2 / self.nu for g in (self.hxg, self.hyg, self.hzg)]
        return min(self.cfl * min(lu, lv, lw), self.cfl * min(lim), 5e-3)

    # ---- eddy viscosity
    def strain(self, U, V, W):
        """S_ij at the centres (the mixed components as means of the four
        edges) and |S| = sqrt(2 S_ij S_ij)."""
        c = self.c
        s = [(c(U) - c(U, -1)) / self.dx(), (c(V) - c(V, 0, -1)) / self.dy(), (c(W) - c(W, 0, 0, -1)) / self.dz()]
        e4 = e5 = e6 = 0.0
        for a in (0, 1):
            for b in (0, 1):
                e4 = e4 + (c(U, a - 1, b) - c(U, a - 1, b - 1)) / self.dyg(b) + \
                    (c(V, a, b - 1) - c(V, a - 1, b - 1)) / self.dxg(a)
                e5 = e5 + (c(U, a - 1, 0, b) - c(U, a - 1, 0, b - 1)) / self.dzg(b) + \
                    (c(W, a, 0, b - 1) - c(W, a - 1, 0, b - 1)) / self.dxg(a)
                e6 = e6 + (c(V, 0, a - 1, b) - c(V, 0, a - 1, b - 1)) / self.dzg(b) + \
                    (c(W, 0, a, b - 1) - c(W, 0, a - 1, b - 1)) / self.dyg(a)
        s += [e4 / 8, e5 / 8, e6 / 8]
        return s, torch.sqrt(2 * (s[0] ** 2 + s[1] ** 2 + s[2] ** 2) + 4 * (s[3] ** 2 + s[4] ** 2 + s[5] ** 2))

    @staticmethod
    def fy(q):
        """Simpson filter in y, one-sided in the end rows."""
        r = torch.empty_like(q)
        r[:, 1:-1] = (q[:, :-2] + 4 * q[:, 1:-1] + q[:, 2:]) / 6
        r[:, 0] = (2 * q[:, 0] + q[:, 1]) / 3
        r[:, -1] = (q[:, -2] + 2 * q[:, -1]) / 3
        return r

    def filt(self, q):
        """Test filter of a periodic quantity on the canonical cells."""
        q = self.fy(q)
        for d in (0, 2):
            q = (torch.roll(q, 1, d) + 4 * q + torch.roll(q, -1, d)) / 6
        return q

    def filt_stored(self, F, iz, ix):
        """Test filter of a stored velocity (its own ghosts), periodic images
        of the result filled in."""
        g = self.fy(F)
        g = (g[:, :, :-2] + 4 * g[:, :, 1:-1] + g[:, :, 2:]) / 6
        g = (g[:-2] + 4 * g[1:-1] + g[2:]) / 6
        return g[:self.nzp, :, :self.nxp][iz][:, :, ix]

    def eddy(self):
        if self.les == NONE:
            return
        nut = self.dsm() if self.les == DSM else self.amd()
        nut = torch.where(nut > 0, nut, torch.zeros_like(nut))[self.izc][:, :, self.ixc]
        s = -1.0 if self.dirichlet else 1.0
        self.nut = torch.cat([s * nut[:, :1], nut, s * nut[:, -1:]], 1)

    def dsm(self):
        c, U, V, W = self.c, self.U, self.V, self.W
        vel = [(c(U, -1) + c(U)) / 2, (c(V, 0, -1) + c(V)) / 2, (c(W, 0, 0, -1) + c(W)) / 2]
        pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
        hat = [self.filt(v) for v in vel]
        s, S = self.strain(U, V, W)
        sf, Sf = self.strain(self.filt_stored(U, self.izc, self.ix), self.filt_stored(V, self.izc, self.ixc),
                             self.filt_stored(W, self.iz, self.ixc))
        lm = mm = 0.0
        for q, (a, b) in enumerate(pairs):
            L = self.filt(vel[a] * vel[b]) - hat[a] * hat[b]
            M = 4 * Sf * sf[q] - self.filt(S * s[q])
            wq = 1.0 if q < 3 else 2.0
            lm = lm + wq * L * M
            mm = mm + wq * M * M
        # the plane sums count the first canonical column and plane twice
        both = torch.stack([lm, mm])
        both = both.sum(3) + both[..., 0]
        both = both.sum(1) + both[:, 0]
        return -0.5 * (both[0] / both[1])[:, None] * S

    def amd(self):
        """Minus 0.3 times the production over the gradient norm, the gradients
        taken where the staggered differences live and averaged to centres."""
        c = self.c
        F = {"u": self.U, "v": self.V, "w": self.W}

        def d(f, ax, a=0, b=0, cc=0):
            o = [[1, 0, 0], [0, 1, 0], [0, 0, 1]][ax]
            return c(F[f], a, b, cc) - c(F[f], a - o[0], b - o[1], cc - o[2])

        sp = [self.dxg, self.dyg, self.dzg]

        def mean4(f, ax, g):
            """Mean over the two faces of component f and the two sides in
            direction ax of g(difference, side)."""
            own = {"u": 0, "v": 1, "w": 2}[f]
            tot = 0.0
            for face in (-1, 0):
                for side in (0, 1):
                    o = [0, 0, 0]
                    o[own], o[ax] = face, side
                    tot = tot + g(d(f, ax, *o), side)
            return tot / 4

        def cross(f, g, ax):
            """Mean over the two sides in direction ax of the product of the
            two components' face-averaged differences."""
            fo, go = {"u": 0, "v": 1, "w": 2}[f], {"u": 0, "v": 1, "w": 2}[g]
            tot = 0.0
            for side in (0, 1):
                m = []
                for h, own in ((f, fo), (g, go)):
                    v = 0.0
                    for face in (-1, 0):
                        o = [0, 0, 0]
                        o[own], o[ax] = face, side
                        v = v + d(h, ax, *o)
                    m.append(v / 2)
                tot = tot + m[0] * m[1]
            return tot / 2

        s, _ = self.strain(self.U, self.V, self.W)
        dd = {("u", 0): (d("u", 0), self.dx()), ("v", 1): (d("v", 1), self.dy()), ("w", 2): (d("w", 2), self.dz())}
        num = den = 0.0
        mean = {}
        for q, f in enumerate("uvw"):
            for ax in range(3):
                if (f, ax) in dd:
                    e, h = dd[f, ax]
                    num, den = num + e ** 2 * s[q], den + (e / h) ** 2
                    mean[f, ax] = e
                else:
                    num = num + mean4(f, ax, lambda e, side: e ** 2) * s[q]
                    den = den + mean4(f, ax, lambda e, side: (e / sp[ax](side)) ** 2)
                    mean[f, ax] = mean4(f, ax, lambda e, side: e)
        for (f, g), q in ((("u", "v"), 3), (("u", "w"), 4), (("v", "w"), 5)):
            for ax in range(3):
                prod = cross(f, g, ax) if ax not in ("uvw".index(f), "uvw".index(g)) else mean[f, ax] * mean[g, ax]
                num = num + 2 * prod * s[q]
        return torch.where(den > 0, -0.3 * num / den, torch.zeros_like(num))

    # ---- wall model
    @staticmethod
    def lagrange(y, yi, strict):
        """Second-order interpolation stencils of the points yi on y: first
        index and three weights of each, the search that of the solver."""
        n, st, w = len(y), [], []
        for q, p in enumerate(yi):
            above = [m for m in range(2, n) if (y[m] > p if strict else y[m] >= p)]
            if above:
                j = above[0] - 1
            else:
                j = n - 2 if q == len(yi) - 1 else st[-1] + 1
            a, b, c = y[j - 1], y[j], y[j + 1]
            st.append(j - 1)
            w.append(((p - b) * (p - c) / ((a - b) * (a - c)), (p - a) * (p - c) / ((b - a) * (b - c)),
                      (p - a) * (p - b) / ((c - a) * (c - b))))
        return st, w

    def wall_model(self):
        if not self.wall:
            return
        st, w = self.lagrange(self.hz, self.hzg, True)
        sx, wx = self.lagrange(self.hxg, self.hx, False)
        t = lambda a: torch.as_tensor(np.array(a), device=self.dev)
        zs, zw, xs, xw = t(st), t(w), t(sx), t(wx)
        j0, j1 = self.jref - 1, self.nym + 2 - self.jref
        Wj = torch.stack([self.W[:, j0], self.W[:, j1]], 1)                      # [nz][wall][nxg]
        Wz = sum(zw[:, m, None, None] * Wj[zs + m] for m in range(3))            # [nzg][wall][nxg]
        Wx = sum(xw[:, m] * Wz[:, :, xs + m] for m in range(3))                  # [nzg][wall][nx]
        Uj = torch.stack([self.U[:, j0], self.U[:, j1]], 1)
        ul = torch.sqrt(Uj * Uj + Wx * Wx)
        self.tau = self.eqwm(ul, self.tau)
        n = self.nut
        nw = torch.stack([n[:, 0] + n[:, 1], n[:, -1] + n[:, -2]], 1) / 2
        nw = self.nu + (nw[:, :, :-1] + nw[:, :, 1:]) / 2
        self.ax = self.tau * Uj / ul / nw
        az = self.tau * Wx / ul / nw
        m = (az[:-1, :, :-1] + az[:-1, :, 1:] + az[1:, :, :-1] + az[1:, :, 1:]) / 4  # [nz][wall][nx-1]
        full = torch.zeros_like(self.az)
        full[:-1, :, :-2] = m[:-1]
        full[:, :, -1], full[:, :, -2] = full[:, :, 2], full[:, :, 1]
        full[-1] = full[1]
        self.az = full

    def eqwm(self, ul, tau):
        """Wall stress of the equilibrium boundary layer: mixing-length
        viscosity with van Driest damping, fixed-point iteration until the
        change is below 1e-7 of the laminar stress (101 passes at most)."""
        ncv, h = self.ncv, self.hyg[self.jref - 1]
        inc = 1.10 ** np.arange(ncv)
        fa = np.concatenate([[0.0], np.cumsum(inc)])
        cv = 0.5 * (fa[1:] + fa[:-1])
        fa, cv = fa / cv.max() * h, cv / cv.max() * h
        shape, ul, tau = ul.shape, ul.reshape(-1), tau.reshape(-1).clone()
        left = torch.arange(ul.numel(), device=self.dev)
        f = torch.as_tensor(fa[1:], device=self.dev)[:, None]
        g = np.concatenate([[cv[0] - fa[0]], np.diff(cv)])
        for it in range(101):
            u, old = ul[left], tau[left]
            ut = torch.sqrt(old)
            D = 1 - torch.exp(-f * ut / self.nu / 17.0)
            mu = torch.cat([torch.full_like(ut, self.nu)[None], self.nu + 0.41 * f * ut * D * D])
            # the flux is the same through every face below the top centre: a chain of resistances
            r = sum(torch.as_tensor(g[q]) / mu[q] for q in range(ncv))
            new = u / r
            tau[left] = new
            left = left[~((new - old).abs() / (self.nu * u / h) < 1e-7)]
            if not left.numel():
                break
        bad = torch.isnan(tau)
        tau[bad] = self.tau_mean
        return tau.reshape(shape)

    # ---- right-hand sides
    def rhs(self):
        U, V, W, n, nu = self.U, self.V, self.W, self.nut, self.nu
        c, m = self.c, self.nym - 1  # V lives on the nym - 1 inner faces
        # canonical entry of a face is the upper face of its cell: fluxes are formed at the centres or
        # edges on both sides and differenced
        wy = lambda F, a, b, cc, rows=None: (self.w0[1 + b:1 + b + (rows or self.nym)] * c(F, a, b, cc, rows) +
                                             self.w1[1 + b:1 + b + (rows or self.nym)] * c(F, a, b + 1, cc, rows))
        # u: x flux at centres i+1, i; y flux at edges j, j-1; z flux at edges k, k-1
        fx = lambda a: 2 * (nu + c(n, a)) * (c(U, a) - c(U, a - 1)) / self.dx(a) - ((c(U, a - 1) + c(U, a)) / 2) ** 2
        # (the viscous cross term of the lower edges divides by the spacing below the face)
        def fuy(b):
            nue = nu + (wy(n, 0, b, 0) + wy(n, 1, b, 0)) / 2
            g = (c(U, 0, b + 1) - c(U, 0, b)) / self.dyg(b + 1) + (c(V, 1, b) - c(V, 0, b)) / self.dx(1 + b)
            return nue * g - wy(U, 0, b, 0) * (c(V, 0, b) + c(V, 1, b)) / 2

        def fuz(k):
            nue = nu + (c(n, 0, 0, k) + c(n, 0, 0, k + 1) + c(n, 1, 0, k) + c(n, 1, 0, k + 1)) / 4
            g = (c(U, 0, 0, k + 1) - c(U, 0, 0, k)) / self.dzg(k + 1) + (c(W, 1, 0, k) - c(W, 0, 0, k)) / self.dx(1 + k)
            return nue * g - (c(U, 0, 0, k) + c(U, 0, 0, k + 1)) / 2 * (c(W, 0, 0, k) + c(W, 1, 0, k)) / 2

        ru = (fx(1) - fx(0)) / self.dxg(1) + (fuy(0) - fuy(-1)) / self.dy() + (fuz(0) - fuz(-1)) / self.dz() + self.dPdx

        # v
        def fvx(a):
            nue = nu + (wy(n, a, 0, 0, m) + wy(n, a + 1, 0, 0, m)) / 2
            g = (c(V, a + 1, 0, 0, m) - c(V, a, 0, 0, m)) / self.dxg(1 + a) + \
                (c(U, a, 1, 0, m) - c(U, a, 0, 0, m)) / self.dyg(1, m)
            return nue * g - wy(U, a, 0, 0, m) * (c(V, a, 0, 0, m) + c(V, a + 1, 0, 0, m)) / 2

        fvy = lambda b: 2 * (nu + c(n, 0, b, 0, m)) * (c(V, 0, b, 0, m) - c(V, 0, b - 1, 0, m)) / self.dy(b, m) - \
            ((c(V, 0, b - 1, 0, m) + c(V, 0, b, 0, m)) / 2) ** 2

        def fvz(k):
            nue = nu + (wy(n, 0, 0, k, m) + wy(n, 0, 0, k + 1, m)) / 2
            g = (c(V, 0, 0, k + 1, m) - c(V, 0, 0, k, m)) / self.dzg(k + 1) + \
                (c(W, 0, 1, k, m) - c(W, 0, 0, k, m)) / self.dyg(1, m)
            return nue * g - wy(W, 0, 0, k, m) * (c(V, 0, 0, k, m) + c(V, 0, 0, k + 1, m)) / 2

        rv = (fvx(0) - fvx(-1)) / self.dx() + (fvy(1) - fvy(0)) / self.dyg(1, m) + (fvz(0) - fvz(-1)) / self.dz()

        # w
        def fwx(a):
            nue = nu + (c(n, a) + c(n, a, 0, 1) + c(n, a + 1) + c(n, a + 1, 0, 1)) / 4
            g = (c(W, a + 1) - c(W, a)) / self.dxg(1 + a) + (c(U, a, 0, 1) - c(U, a)) / self.dzg(1)
            return nue * g - (c(U, a) + c(U, a, 0, 1)) / 2 * (c(W, a) + c(W, a + 1)) / 2

        def fwy(b):
            nue = nu + (wy(n, 0, b, 0) + wy(n, 0, b, 1)) / 2
            g = (c(W, 0, b + 1) - c(W, 0, b)) / self.dyg(b + 1) + (c(V, 0, b, 1) - c(V, 0, b)) / self.dzg(1)
            return nue * g - wy(W, 0, b, 0) * (c(V, 0, b) + c(V, 0, b, 1)) / 2

        fwz = lambda k: 2 * (nu + c(n, 0, 0, k)) * (c(W, 0, 0, k) - c(W, 0, 0, k - 1)) / self.dz(k) - \
            ((c(W, 0, 0, k - 1) + c(W, 0, 0, k)) / 2) ** 2
        rw = (fwx(0) - fwx(-1)) / self.dx() + (fwy(0) - fwy(-1)) / self.dy() + (fwz(1) - fwz(0)) / self.dzg(1)
        if abs(self.Om) > 1e-6:
            ru = ru + 2 * self.Om * (c(V, 0, -1) + c(V) + c(V, 1, -1) + c(V, 1)) / 4
            t = lambda b: (c(U, -1, b, 0, m) + c(U, 0, b, 0, m)) / 2
            rv = rv - 2 * self.Om * (self.w0[1:1 + m] * t(0) + self.w1[1:1 + m] * t(1))
        return ru, rv, rw

    # ---- pressure
    def poisson_setup(self):
        n, d = self.nym, self.dev
        y, yg = self.hy, self.hyg
        q = np.arange(n)
        up = 1 / (y[q + 1] - y[q]) / (yg[q + 2] - yg[q + 1])
        lo = 1 / (y[q + 1] - y[q]) / (yg[q + 1] - yg[q])
        up[-1], lo[0] = 0.0, 0.0
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=d)
        dxm, dzm = np.diff(self.hxg).min(), np.diff(self.hzg).min()
        kx = t(2 * (np.cos(2 * math.pi * np.arange(self.nxp // 2 + 1) / self.nxp) - 1) / dxm ** 2)
        kz = t(2 * (np.cos(2 * math.pi * np.arange(self.nzp) / self.nzp) - 1) / dzm ** 2)
        kk = kz[:, None] + kx[None, :]
        self.up, self.lo = up, lo
        diag = [(-(up[r] + lo[r]) + kk) for r in range(n)]
        diag[0] = diag[0].clone()
        diag[0][0, 0] *= 1.5  # the mean mode's matrix is singular: its first diagonal is changed
        # Thomas factors of every mode
        self.rd = [1 / diag[0]]
        for r in range(1, n):
            self.rd.append(1 / (diag[r] - lo[r] * up[r - 1] * self.rd[-1]))

    def project(self, store, dt):
        c = self.c
        div = (c(self.U) - c(self.U, -1)) / self.dx() + (c(self.V) - c(self.V, 0, -1)) / self.dy() + \
            (c(self.W) - c(self.W, 0, 0, -1)) / self.dz()
        b = torch.fft.rfftn(div, dim=(0, 2))
        n = self.nym
        g = [b[:, 0] * self.rd[0]]
        for r in range(1, n):
            g.append((b[:, r] - self.lo[r] * g[-1]) * self.rd[r])
        for r in range(n - 2, -1, -1):
            g[r] = g[r] - self.up[r] * self.rd[r] * g[r + 1]
        phi = torch.fft.irfftn(torch.stack(g, 1), s=(self.nzp, self.nxp), dim=(0, 2))
        full = phi[self.izc][:, :, self.ixc]
        if store:
            P = phi / (dt * 8 / 15)
            first = lambda m: torch.cat([torch.zeros(1, dtype=torch.long), torch.arange(m),
                                         torch.zeros(2, dtype=torch.long)]).to(self.dev)
            P = P[first(self.nzp)][:, :, first(self.nxp)]
            self.P = torch.cat([P[:, :1], P, P[:, -1:]], 1)
        sl = slice(1, 1 + self.nxp)
        p0 = full[1:1 + self.nzp, :, sl]
        c(self.U).sub_((full[1:1 + self.nzp, :, 2:2 + self.nxp] - p0) / self.dxg(1))
        c(self.V, 0, 0, 0, n - 1).sub_((p0[:, 1:] - p0[:, :-1]) / self.dyg(1, n - 1))
        c(self.W).sub_((full[2:2 + self.nzp, :, sl] - p0) / self.dzg(1))

    def step(self):
        dt = self.dt_rule()
        old = [self.c(self.U).clone(), self.c(self.V, 0, 0, 0, self.nym - 1).clone(), self.c(self.W).clone()]
        F1 = None
        for s in (1, 2, 3):
            self.eddy()
            if s == 1:
                self.wall_model()
            F = self.rhs()
            if s == 1:
                inc, F1 = [8 / 15 * f for f in F], F
            else:
                a, b = ((1 / 4, 5 / 12), (1 / 4, 3 / 4))[s - 2]
                inc = [a * f1 + b * f for f1, f in zip(F1, F)]
            for o, dst, i in zip(old, (self.c(self.U), self.c(self.V, 0, 0, 0, self.nym - 1), self.c(self.W)), inc):
                dst.copy_(o + dt * i)
            self.bc()
            self.project(s == 1, dt)
            self.bc()
        if self.mass == 1:
            corr = self.Q0 - self.flow()
            self.c(self.U).add_(corr)
            self.dPdx = corr / dt
            self.bc()
