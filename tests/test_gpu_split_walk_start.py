"""Where a block of the split path's update starts its walk up z must not show
in the result, in the fast build either.  A state that repeats along z every
five planes is stepped on a periodic grid: a plane is the first of a block's
walk in one period and in the middle of one in the next, and all copies of it
must stay equal bit for bit.  The spacing is 3/64, so that positions and cell
widths are exact (the same numbers in every period) while products with a width
round.  Odd Ntot_x loads per thread, even Ntot_x by TMA."""
import numpy as np
import pytest

from bonzo_b200._lib import Context

pytestmark = pytest.mark.gpu

H, PERIOD = 3. / 64, 5


@pytest.mark.parametrize("exact", [False, True], ids=["fast", "exact"])
@pytest.mark.parametrize("kw", [dict(rsolver="hlld", limiter="vl"), dict(rsolver="hll", limiter="mc")],
                         ids=["hlld", "hll"])
@pytest.mark.parametrize("nx,ny,nz", [(7, 9, 40), (8, 9, 40), (33, 20, 40), (34, 20, 40), (65, 33, 70), (33, 200, 45)])
def test_result_does_not_depend_on_the_walks_start(nx, ny, nz, kw, exact):
    c = Context(Nx=nx, Ny=ny, Nz=nz, dims=3, lmax=(nx * H, ny * H, nz * H), gam=5. / 3, cour=0.3, path="split",
                exact_fp=exact, **kw)
    rng = np.random.default_rng(nx + nz)
    prim, bfld = np.zeros((9,) + c.shape), np.zeros((3,) + c.shape)
    a = np.s_[3:3 + nz, 3:3 + ny, 3:3 + nx]
    rep = lambda x: np.tile(x, (nz // PERIOD, 1, 1))
    shp = (PERIOD, ny, nx)
    prim[0][a] = rep(np.exp(0.2 * rng.standard_normal(shp)))
    for v in (1, 2, 3):
        prim[v][a] = rep(0.3 * rng.standard_normal(shp))
    prim[4][a] = rep(np.exp(0.2 * rng.standard_normal(shp)))
    prim[5][a] = rep(rng.random(shp))
    for q, b in enumerate((0.5, -0.4, 0.3)):  # uniform: divergence free
        bfld[q] = b
    c.set_state(prim, bfld)
    c.init()
    for _ in range(2):
        c.step(0.002)
    P, _, B = c.get_state()
    for x in (P[(slice(None),) + a], B[(slice(None),) + a]):
        assert np.array_equal(x[:, PERIOD:], x[:, :-PERIOD]), np.argwhere(x[:, PERIOD:] != x[:, :-PERIOD])[:5]
