"""The z contractions at the sizes where their kernels change: every remainder of the matrix
size over a tile of 16 rows, the smallest and the largest, on column counts that take the
kernels for small grids (a part of a CTA, one and several CTAs of 8, 16 and 32 columns) and
the ones for large grids.

The bound is elementwise: a length-n dot product in floating point is off by at most
n eps sum |a||b|, so the solve E (E^-1 r / den) is off by at most (2 n + 8) eps
|E| (|E^-1| |r| / |den|) on each side of the comparison (8 for the lift, the scale and the
boundary terms, which enter |r| and the result by their absolute values).
"""
import numpy as np
import pytest

from lsbflow_b200 import hostsetup as hs
from lsbflow_b200.config import workload
from oracle import lsb_oracle as O

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def setup(nx, ny, nz):
    return hs.make_setup(workload("dns64", nx=nx, ny=ny, nz=nz, dealiasflag=0))


def solve_bound(st, rhs, bc, dtnui):
    c = st.cfg
    w2 = O.wav2(st)
    hb, ht = np.abs(st.hbot)[:, None, None], np.abs(st.htop)[:, None, None]
    fac = (w2 + abs(dtnui))[None]
    mag = np.abs(rhs) + (np.abs(st.d2hbot)[:, None, None] + fac * hb) * np.abs(bc[-1]) \
        + (np.abs(st.d2htop)[:, None, None] + fac * ht) * np.abs(bc[0])
    den = np.abs(st.lam[:, None, None] - (w2 + dtnui)[None])
    y = np.tensordot(np.abs(st.Ei), mag[1:-1], 1) / den
    out = np.zeros_like(rhs)
    out[1:-1] = np.tensordot(np.abs(st.E), y, 1)
    out += hb * np.abs(bc[-1]) + ht * np.abs(bc[0])
    return (2 * c.nz + 8) * EPS * out


COLS = [(4, 2), (20, 3), (64, 8), (128, 16), (96, 50), (256, 32)]  # 8 .. 8192 columns
NZ = [4, 16, 17, 18, 32, 33, 48, 63, 64, 65, 80, 81, 96, 97, 112, 127, 128, 129, 130, 142]


@pytest.mark.parametrize("nz", NZ)
def test_helmholtz_every_tile_count(nz):
    from lsbflow_b200 import lib
    for nx, ny in (COLS if nz in (17, 64, 96, 97) else COLS[2:4]):
        st = setup(nx, ny, nz)
        s = lib.Solver(st)
        rng = np.random.default_rng(nz + nx)
        rhs = rng.standard_normal((nz + 1, ny, nx))
        bc = np.zeros_like(rhs)
        bc[0], bc[-1] = rng.standard_normal((2, ny, nx))
        for dtnui in (1.0 / (st.cfg.xnu * st.dt), 0.25):
            got = s.solve_nhom_helmholtz(rhs, bc, dtnui)
            err = np.abs(got - O.solve_nhom_helmholtz(st, rhs.copy(), bc, dtnui))
            assert np.all(err <= 2 * solve_bound(st, rhs, bc, dtnui)), (nx, ny, dtnui)
            got = s.solve_helmholtz(rhs, dtnui)
            assert np.all(got[0] == 0.0) and np.all(got[-1] == 0.0)
            err = np.abs(got - O.solve_helmholtz(st, rhs.copy(), dtnui))
            assert np.all(err <= 2 * solve_bound(st, rhs, 0 * bc, dtnui)), (nx, ny, dtnui)
        s.close()


@pytest.mark.parametrize("nz", NZ)
def test_derivatives_every_tile_count(nz):
    from lsbflow_b200 import lib
    for nx, ny in (COLS if nz in (17, 64, 96, 97) else COLS[2:4]):
        st = setup(nx, ny, nz)
        s = lib.Solver(st)
        u = np.random.default_rng(nz + nx).standard_normal((nz + 1, ny, nx))
        for got, m in ((s.dfdz(u), st.dz1), (s.d2fdz2(u), st.dz2)):
            bound = (nz + 1) * EPS * np.tensordot(np.abs(m), np.abs(u), 1)
            assert np.all(np.abs(got - np.tensordot(m, u, 1)) <= 2 * bound), (nx, ny)
        s.close()


@pytest.mark.parametrize("nz", [16, 32, 48, 64, 80, 97, 128])
def test_steps_of_small_grids_equal_the_large_kernels_bit_for_bit(nz):
    # a tuned width takes the kernels for large grids: every epilogue of a step (plain,
    # divergence, Poisson right-hand side, pressure, solves) against the ones for small grids
    from lsbflow_b200 import ic, lib
    for nx, ny, over in ((64, 8, dict(dealiasflag=1)), (32, 16, dict(dealiasflag=0)), (48, 6, dict(dealiasflag=1))):
        st = hs.make_setup(workload("dns64", nx=nx, ny=ny, nz=nz, **over))
        u, v, w = ic.seeded_noise(st, 3, 1e-2)
        outs = []
        for warps in (0, 4, 7):
            s = lib.Solver(st)
            s.set_schedule({"gemm_warps": warps})
            s.upload(u, v, w, dt=st.dt)
            s.step(5)
            outs.append(s.download())
            s.close()
        for k in ("uf", "vf", "wf", "pf", "nlnif"):
            assert np.array_equal(outs[0][k], outs[1][k]) and np.array_equal(outs[0][k], outs[2][k]), (nx, ny, k)


@pytest.mark.parametrize("nz", [3, 17, 64, 97, 128])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "8-byte aligned"])
def test_noalloc_solve_on_any_alignment(nz, shift):
    import torch
    from lsbflow_b200 import lib
    for nx, ny in ((6, 3), (64, 8), (160, 40)):
        st = setup(nx, ny, nz) if nz > 3 else hs.make_setup(workload("dns64", nx=nx, ny=ny, nz=nz, dealiasflag=0))
        rng = np.random.default_rng(nz + nx)
        rhs = rng.standard_normal((nz + 1, ny, nx))
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()  # noqa: E731
        n = rhs.size
        src = torch.zeros(n + 2, dtype=torch.float64, device="cuda")
        dst = torch.full((n + 2,), float("nan"), dtype=torch.float64, device="cuda")
        src[shift:shift + n] = put(rhs).reshape(-1)
        mats = [put(a) for a in (st.lam, st.E, st.Ei, st.grid.wavx, st.grid.wavy)]
        lib.solve_helmholtz_noalloc(nx, ny, nz, src[shift:].data_ptr(), dst[shift:].data_ptr(),
                                    *(m.data_ptr() for m in mats), 7.5, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got = dst[shift:shift + n].cpu().numpy().reshape(rhs.shape)
        err = np.abs(got - O.solve_helmholtz(st, rhs.copy(), 7.5))
        assert np.all(err <= 2 * solve_bound(st, rhs, 0 * rhs, 7.5)), (nx, ny)
        assert bool(dst[shift + n:].isnan().all()) and bool(dst[:shift].isnan().all())
