"""What the performance of this package is measured on: time steps, ensembles and single operators.

A case is one use of the library through its Python binding (``lsbflow_b200.lib``):

* ``step``  -- a resident run (``Solver``) advanced by ``steps`` calls of timestep() and its velocity
               copied to the caller's device arrays, as a driver does between its own output steps;
               with ``exchange`` the caller hands its velocity in before each pass as well, as a
               program does that keeps u, v, w itself (assimilation, forcing of its own);
* ``batch`` -- ``members`` runs of one grid with their own Re, dipole and noise, advanced together
               (``Batch``), as a parameter study does;
* ``helm``  -- the Helmholtz solve on device arrays that the caller owns (``solve_helmholtz_noalloc``);
* ``nlterm``-- the nonlinear term on host arrays (``Solver.nlterm``), as a host time loop calls the
               subroutine of that name.

Runs are handed over after their start-up steps, with seeded divergence-free noise as the
initial field, and go on from where the last pass left them, or from the caller's velocity with
``exchange``.  The sigma model and the mixed form are stepped by exchange: left to themselves
they carry the last bit of one step into the eighth digit of the next.  Sizes are (nx, ny, nz): x and y
periodic, nz + 1 Chebyshev points in z.
"""
import functools
import math

import numpy as np
import torch

from lsbflow_b200 import hostsetup, lib
from lsbflow_b200.config import LsbConfig, ensemble_configs, workload

SGS = {"none": None, "static": 0, "dynamic": 1, "sigma": 2, "interscale": 3, "tns": 4}
START_UP = 3        # steps before a run is steady: Euler, BDF2, then BDF3
AMPLITUDE = 5e-3    # rms of the initial noise over the free-stream velocity


def listed():
    def case(name, kind, nx, ny, nz, flow="les", sgs="none", dealias=1, precision="fp64", steps=1, members=1,
             exchange=False):
        return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, flow=flow, sgs=sgs, dealias=dealias,
                    precision=precision, steps=steps, members=members, exchange=exchange)

    return [
        # the smallest grid that is run in earnest, one step at a time: launches and latency
        case("dns64", "step", 64, 16, 64, flow="dns"),
        # linear stability: a thin, tall grid without products on a finer grid, several steps a call
        case("os128", "step", 128, 4, 96, flow="os", dealias=0, steps=10),
        # the reference's shipped set-up: x length 224, spectral filter, wall suction, adaptive dt
        # (checked every 5 steps), an x transform that is no power of two times three
        case("shipped224", "step", 224, 24, 32, flow="suction", dealias=2, steps=5),
        # one sigma-model run of an ensemble's grid, alone on the GPU
        case("sigma128", "step", 128, 32, 64, sgs="sigma", exchange=True),
        # an ensemble of such runs advanced together
        case("ensemble128", "batch", 128, 32, 64, sgs="sigma", members=8, exchange=True),
        # a tall LES of a serving mix
        case("interscale128", "step", 128, 32, 96, sgs="interscale"),
        # an LES on lengths off the powers of two (padded 288 x 72)
        case("static192", "step", 192, 48, 80, sgs="static"),
        # the LES that the package's benchmark steps, in both of its precisions
        case("dynamic256", "step", 256, 64, 128, sgs="dynamic"),
        case("mixed256", "step", 256, 64, 128, sgs="dynamic", precision="mixed", exchange=True),
        # twice that streamwise resolution: the largest run
        case("dynamic512", "step", 512, 64, 128, sgs="dynamic"),
        # a caller that owns its device memory: one Helmholtz solve
        case("helm256", "helm", 256, 64, 128),
        # a host time loop that calls the nonlinear term as a subroutine
        case("nlterm128", "nlterm", 128, 32, 64, flow="dns"),
    ]


def draw(rng):
    """One more case: mostly single runs, their sizes spread evenly over the logarithm."""
    kind = rng.choices(["step", "batch", "helm", "nlterm"], [10, 2, 2, 1])[0]
    form = rng.choices(["plain", "sigma", "mixed"], [7, 1, 2])[0] if kind in ("step", "batch") else "plain"
    if form == "plain":     # lengths with the prime factors 2, 3, 5, 7
        xs = [48, 64, 80, 96, 112, 128, 144, 160, 192, 224, 240, 256, 288, 320, 384, 448, 512]
        ys = [4, 6, 8, 10, 12, 16, 20, 24, 28, 32, 36, 40, 48, 56, 60, 64, 80, 96]
    else:                   # the lengths of the package's ensembles and mixed runs
        xs, ys = [64, 128, 256], [8, 16, 32, 64]

    def near(values, lo, hi):
        x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min(values, key=lambda v: abs(math.log(v / x)))

    members = rng.randint(2, 8) if kind == "batch" else 1
    most = 512 * 64 * 129 // 2 // members
    while True:
        nx, ny = near(xs, 48, 512), near(ys, 4, 96)
        # runs with fewer points in z than this don't resolve the layer under the ceiling's dipole
        nz = round(math.exp(rng.uniform(math.log(17 if kind == "helm" else 33), math.log(129)))) - 1
        if 64 * 16 * 17 <= nx * ny * (nz + 1) <= most and (kind != "nlterm" or nx * ny * nz < 1 << 20):
            break
    if form == "sigma" or kind == "helm":
        flow = "les"
    elif kind == "nlterm":
        flow = "dns"
    elif form == "mixed":
        flow = rng.choice(["les", "dns"])
    else:
        flow = rng.choices(["les", "dns", "os", "suction"], [6, 2, 1, 1])[0]
    sgs = "none"
    if form == "sigma":
        sgs = "sigma"
    elif flow == "les" and kind == "step":
        sgs = rng.choice(["none", "static", "dynamic", "interscale", "tns"])
    elif flow == "les" and kind == "batch":
        sgs = "dynamic"
    exchange = form != "plain" or (kind == "step" and flow in ("les", "dns") and rng.random() < 0.2)
    if kind not in ("step", "batch"):
        exchange, steps = False, 1
    elif flow == "suction":
        steps = 5
    else:
        steps = 1 if exchange or nx * ny * nz >= 1 << 19 else rng.choice([1, 1, 2, 5])
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, flow=flow, sgs=sgs, dealias={"os": 0, "suction": 2}.get(flow, 1),
                precision="mixed" if form == "mixed" else "fp64", steps=steps, members=members, exchange=exchange)


# ------------------------------------------------------------------ inputs
def config(case) -> LsbConfig:
    size = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], precision=1 if case["precision"] == "mixed" else 0,
                dealiasflag=case["dealias"])
    model = SGS[case["sgs"]]
    size.update(sgsflag=0 if model is None else 1, sgsmodel=model or 0)
    if case["flow"] == "suction":   # run/input.dat: Spalart's suction profile, dt from the CFL number
        return LsbConfig(bctype=1, forcing=1, dtadapt=1, **size)
    if case["kind"] == "nlterm":    # the term itself: no forcing added to it
        return workload("dns64", forcing=0, **size)
    return workload({"les": "les256", "dns": "dns64", "os": "os128"}[case["flow"]], **size)


@functools.lru_cache(maxsize=16)
def setup_of(key):
    return hostsetup.make_setup(config(dict(key)))


def setup(case):
    return setup_of(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "members", "exchange"))))


def noise(st, seed):
    """(3, nzp, ny, nx) spectral velocity on the GPU: the curl of a random vector potential on the
    lower two thirds of the modes, zero on both walls, of rms AMPLITUDE u0 over the grid."""
    c, g, dev = st.cfg, st.grid, "cuda"
    f64 = dict(dtype=torch.float64, device=dev)
    gen = torch.Generator(device=dev).manual_seed(seed)
    kx = torch.arange(c.nx // 2, device=dev)
    ky = torch.from_numpy(np.fft.fftfreq(c.ny, 1.0 / c.ny).astype(np.int64)).to(dev)
    keep = ((kx <= c.nx // 3)[None, :] & (ky.abs() <= c.ny // 3)[:, None]).to(torch.float64)
    z = torch.tensor(g.zpts, **f64)
    xi = (z - z[-1]) / (z[0] - z[-1])
    psi = torch.randn((3, c.nzp, c.ny, c.nx // 2, 2), generator=gen, **f64)
    psi *= ((xi * (1.0 - xi)) ** 2)[:, None, None, None] * keep[..., None]
    psi = torch.view_as_complex(psi)
    # real fields: the kx = 0 modes of ky and -ky are conjugate
    zero = psi[..., 0]
    psi[..., 0] = 0.5 * (zero + zero[..., (-ky) % c.ny].conj())
    ix = 1j * torch.tensor(g.wavx[0::2], **f64)
    iy = 1j * torch.tensor(g.wavy, **f64)[:, None]
    d = torch.tensor(st.d, **f64).to(torch.complex128)
    ddz = lambda f: (d @ f.reshape(c.nzp, -1)).reshape(f.shape)  # noqa: E731
    u = torch.stack([iy * psi[2] - ddz(psi[1]), ddz(psi[0]) - ix * psi[2], ix * psi[1] - iy * psi[0]])
    u[:, 0] = u[:, -1] = 0.0
    power = 2.0 * u.abs().square().sum() - u[..., 0].abs().square().sum()
    u *= AMPLITUDE * c.u0 / torch.sqrt(power / (3.0 * c.nzp))
    return torch.view_as_real(u).reshape(3, c.nzp, c.ny, c.nx).contiguous()


class Run:
    """A run with its start-up steps behind it, and the caller's arrays for its velocity."""

    def __init__(self, st, seed, exchange):
        self.solver = lib.Solver(st)
        u = noise(st, seed)
        self.given = u if exchange else None
        self.solver.upload(*u.cpu().numpy(), dt=st.dt)
        for _ in range(START_UP):
            self.give()
            self.solver.step(1)
        self.solver.synchronize()
        self.out = torch.empty_like(u)

    def give(self):
        if self.given is not None:
            self.solver.upload_device(*(f.data_ptr() for f in self.given))

    def velocity(self):
        self.solver.download_device(*(f.data_ptr() for f in self.out))
        return self.out


class Ensemble:
    """Runs advanced together; closed before its members."""

    def __init__(self, runs):
        self.runs = runs
        self.batch = lib.Batch([r.solver for r in runs])

    def __del__(self):
        self.batch.close()


def helm_inputs(case, seed):
    """The right-hand side and shift of an implicit diffusion step."""
    st = setup(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (st.cfg.nzp, st.cfg.ny, st.cfg.nx)
    return st, torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda"), 11.0 / (6.0 * st.cfg.xnu * st.dt)


def prepare(case, seed):
    st = setup(case)
    if case["kind"] == "helm":
        st, rhs, shift = helm_inputs(case, seed)
        mats = [torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
                for a in (st.lam, st.E, st.Ei, st.grid.wavx, st.grid.wavy)]
        return dict(case, rhs=rhs, out=torch.empty_like(rhs), mats=mats, shift=shift)
    if case["kind"] == "nlterm":
        return dict(case, solver=lib.Solver(st), u=noise(st, seed).cpu().numpy())
    if case["kind"] == "batch":
        cfg = config(case)
        keep = ("xnu", "x0", "xlen", "ylen", "zlen", "bc3_amp", "bc3_xc", "bc3_s")
        drawn = ensemble_configs(case["members"], seed)
        runs = [Run(hostsetup.make_setup(cfg.replace(**{k: getattr(m, k) for k in keep})), seed + 100 * i, case["exchange"])
                for i, m in enumerate(drawn)]
        return dict(case, ensemble=Ensemble(runs))
    return dict(case, run=Run(st, seed, case["exchange"]))


def run(state):
    kind = state["kind"]
    if kind == "step":
        r = state["run"]
        r.give()
        r.solver.step(state["steps"])
        return r.velocity()
    if kind == "batch":
        e = state["ensemble"]
        for r in e.runs:
            r.give()
        e.batch.step(state["steps"])
        return [r.velocity() for r in e.runs]
    if kind == "helm":
        lib.solve_helmholtz_noalloc(state["nx"], state["ny"], state["nz"], state["rhs"].data_ptr(),
                                    state["out"].data_ptr(), *(m.data_ptr() for m in state["mats"]), state["shift"],
                                    torch.cuda.current_stream().cuda_stream)
        return state["out"]
    return state["solver"].nlterm(state["u"])


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    nx, ny, nzp = case["nx"], case["ny"], case["nz"] + 1
    nzm, points = nzp - 2, nx * ny * nzp
    solve = 2.0 * (nzm * nzm + nzp * nzm) * nx * ny          # E^-1 and E over all columns
    if case["kind"] == "helm":
        return {"bytes": 8.0 * (2 * points + 2 * nzm * nzm), "flops": solve}
    deriv = 2.0 * nzp * points
    fine = 2.25 if case["dealias"] == 1 else 1.0
    fft = 2.5 * math.log2(nx * ny * fine) * points * fine    # one real transform of a (padded) field
    nonlinear = 6 * deriv + 18 * fft + 40 * points * fine
    if case["kind"] == "nlterm":
        return {"bytes": 8.0 * 6 * points, "flops": nonlinear}
    # a step reads u, u^{n-1}, u^{n-2}, N^{n-1}, N^{n-2} (3 fields each), p, p^{n-1} and writes u, N, p
    flops = nonlinear + 4 * solve + 2 * deriv + 60 * points
    if case["sgs"] not in ("none", "tns"):
        flops += (12 + 6) * 2.5 * math.log2(nx * ny) * points + 200 * points
    n = case["steps"] * case["members"]
    return {"bytes": 8.0 * 24 * points * n, "flops": flops * n}


# ------------------------------------------------------------------ the single operators in plain float64
def exact(case, seed):
    if case["kind"] == "helm":
        st, rhs, shift = helm_inputs(case, seed)
        lam, e, ei = (torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda") for a in (st.lam, st.E, st.Ei))
        k2 = torch.tensor(st.grid.wavy[:, None] ** 2 + st.grid.wavx[None, :] ** 2, device="cuda").reshape(-1)
        t = ei @ rhs[1:-1].reshape(st.cfg.nz - 1, -1) / (lam[:, None] - k2 - shift)
        out = torch.zeros_like(rhs)
        out[1:-1] = (e @ t).reshape(rhs[1:-1].shape)
        return out
    if case["kind"] == "nlterm":
        return exact_nlterm(setup(case), noise(setup(case), seed).cpu().numpy())
    return None


def exact_nlterm(st, u):
    """-(u . grad u + div(u u)) / 2 for u + ubar, products by the 3/2 rule, numpy's transforms."""
    c = st.cfg
    nx, ny, nxl, nyl, h = c.nx, c.ny, st.nx_lg, st.ny_lg, c.ny // 2
    f = u[..., 0::2] + 1j * u[..., 1::2]
    ix, iy = 1j * st.grid.wavx[0::2], 1j * st.grid.wavy[:, None]
    ddz = lambda a: np.tensordot(st.dz1, a, 1)  # noqa: E731

    def physical(a):
        p = np.zeros(a.shape[:-2] + (nyl, nxl // 2 + 1), dtype=complex)
        p[..., :h, : nx // 2] = a[..., :h, :]
        p[..., nyl - h:, : nx // 2] = a[..., h:, :]
        return np.fft.irfft2(p, s=(nyl, nxl)) * (nxl * nyl)

    def spectral(p):
        a = np.fft.rfft2(p)[..., : nx // 2] / (nxl * nyl)
        a = np.concatenate([a[..., :h, :], a[..., nyl - h:, :]], axis=-2)
        zero = np.fft.ifft(a[..., 0], axis=-1)           # kx = 0 of a real field on the ny grid
        a[..., 0] = np.fft.fft(zero.real, axis=-1)
        return a

    q = [physical(f[l]) for l in range(3)]
    q[0] = q[0] + st.ubar[:, None, None]
    out = []
    for l in range(3):
        grad = [physical(ix * f[l]), physical(iy * f[l]), physical(ddz(f[l]))]
        if l == 0:
            grad[2] = grad[2] + st.ubarp[:, None, None]
        uu = [spectral(q[l] * q[m]) for m in range(3)]
        n = spectral(sum(q[m] * grad[m] for m in range(3))) + ix * uu[0] + iy * uu[1] + ddz(uu[2])
        out.append(-0.5 * n)
    n = np.stack(out)
    return np.stack([n.real, n.imag], axis=-1).reshape(u.shape)
