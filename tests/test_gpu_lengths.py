"""Transforms and product rows at every kind of length: register counts 1 .. 9, 12 and 15 per
lane, lane groups of 1 .. 32, rows that do not fill a warp's last groups, and lengths without a
register plan, on the padded and the unpadded grid, against the oracle.

The tolerance is the one of the single-operator parity tests: an FFT of N points is off by about
eps log2(N) relative (4e-15 at these lengths), a product row runs two of them around pointwise
products, and the 1e-12 leaves two decimal digits for the derivative's weighting of the highest
modes.
"""
import numpy as np
import pytest

from lsbflow_b200 import hostsetup as hs
from lsbflow_b200.config import workload
from oracle import lsb_oracle as O

pytestmark = pytest.mark.gpu

TOL_OP = 1e-12

# (nx, ny): half and padded half lengths nx/2, 3 nx/4 and spanwise ny, 3 ny/2
GRIDS = [(20, 4), (24, 6), (28, 10), (36, 12), (40, 14), (48, 18), (56, 20), (60, 28), (64, 30), (72, 36), (80, 40),
         (96, 48), (112, 56), (120, 60), (128, 14), (144, 80), (160, 6), (192, 96), (224, 8), (240, 16),
         (256, 6), (288, 4), (320, 10), (384, 24), (448, 4), (512, 20)]


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b)


@pytest.mark.parametrize("nx,ny", GRIDS)
def test_transforms(nx, ny):
    from lsbflow_b200 import lib
    st = hs.make_setup(workload("dns64", nx=nx, ny=ny, nz=4, dealiasflag=0))
    s = lib.Solver(st)
    rng = np.random.default_rng(nx + ny)
    a = np.zeros((5, ny, nx + 2))
    a[..., :nx] = rng.standard_normal((5, ny, nx))
    assert rel(s.horfft(a, None, -1), O.horfft_fwd(a, nx, ny)) < TOL_OP
    f = rng.standard_normal((5, ny, nx))
    assert rel(s.horfft(None, f, 1), O.horfft_inv(f, nx, ny)) < TOL_OP
    s.close()


@pytest.mark.parametrize("over", [dict(dealiasflag=1, dealias_layout="correct"),
                                  dict(dealiasflag=1, dealias_layout="ref"), dict(dealiasflag=0, forcing=1)],
                         ids=["padded", "padded-ref", "fringe"])
@pytest.mark.parametrize("nx,ny", GRIDS)
def test_product_rows(nx, ny, over):
    from lsbflow_b200 import lib
    st = hs.make_setup(workload("dns64", nx=nx, ny=ny, nz=6, **{"forcing": 0, **over}))
    s = lib.Solver(st)
    rng = np.random.default_rng(nx * ny)
    u = [rng.standard_normal((7, ny, nx)) for _ in range(3)]
    O.norm(u, ny)
    got, ref = s.nlterm(np.array(u)), O.nlterm_skewsym(st, u)
    for l in range(3):
        assert rel(got[l], ref[l]) < TOL_OP, l
    s.close()


def test_product_rows_of_384_modes_over_several_rows_per_warp():
    # 144 x 13 rows on 148 blocks of 7 warps: every warp stages its next row, some have one, some two
    from lsbflow_b200 import lib
    st = hs.make_setup(workload("dns64", nx=512, ny=96, nz=12, dealiasflag=1, forcing=0))
    s = lib.Solver(st)
    rng = np.random.default_rng(0)
    u = [rng.standard_normal((13, 96, 512)) for _ in range(3)]
    O.norm(u, 96)
    got, ref = s.nlterm(np.array(u)), O.nlterm_skewsym(st, u)
    for l in range(3):
        assert rel(got[l], ref[l]) < TOL_OP, l
    s.close()


@pytest.mark.parametrize("layout", ["correct", "ref"])
@pytest.mark.parametrize("ny", [4, 6, 8, 12, 14, 16, 18, 20, 24, 30, 42, 32, 36, 48, 64, 72, 80, 96, 112, 128])
def test_forcing_accumulates_over_every_spanwise_split(ny, layout):
    # the fringe forcing of padded runs is added to N by the forward spanwise pass
    from lsbflow_b200 import lib
    st = hs.make_setup(workload("dns64", nx=64, ny=ny, nz=5, dealiasflag=1, dealias_layout=layout, forcing=1))
    s = lib.Solver(st)
    rng = np.random.default_rng(ny)
    u = [rng.standard_normal((6, ny, 64)) for _ in range(3)]
    O.norm(u, ny)
    got, ref = s.nlterm(np.array(u)), O.nlterm_skewsym(st, u)
    for l in range(3):
        assert rel(got[l], ref[l]) < TOL_OP, l
    s.close()


def test_mixed_form_takes_the_lengths_it_took():
    # the register counts that only FP64 has do not open the mixed form to new lengths
    from lsbflow_b200 import lib
    for nx, ny in ((144, 8), (224, 8), (64, 36), (320, 8)):
        with pytest.raises(lib.LsbError, match="mixed precision"):
            lib.Solver(hs.make_setup(workload("dns64", nx=nx, ny=ny, nz=8, dealiasflag=0, precision=1)))
