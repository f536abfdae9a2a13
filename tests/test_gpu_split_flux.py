"""The split path's flux kernels at the sizes where their walks can go wrong:
rows that end just before, at and just after a warp's segment of cells, columns
cut by the walk length, grids of a few cells, one plane or one row, for donor
cells, PLM and characteristic slopes.  The exact build must reproduce the
oracle bit for bit (it takes the reference's arithmetic), so no tolerance."""
import numpy as np
import pytest

from bonzo_b200 import problems as P
from helpers import device_ctx, oracle_sim

pytestmark = pytest.mark.gpu

SIZES = [(4, 4, 4), (5, 7, 4), (28, 5, 4), (29, 4, 6), (30, 6, 5), (31, 5, 5), (32, 4, 4), (33, 5, 4), (59, 4, 5),
         (60, 5, 4), (61, 4, 4), (4, 40, 5), (5, 4, 41), (6, 33, 1), (64, 4, 1), (27, 70, 1), (200, 1, 1), (25, 1, 1)]
# columns whose walks share blocks: one walk a column and several, a block of one
# walk of many columns, lanes of a warp in two walks
SIZES += [(30, 600, 1), (3, 900, 1), (125, 33, 1), (126, 130, 1), (400, 300, 1), (40, 41, 42)]


def _state(n, reconstr, hydro, seed):
    dims = 1 + (n[1] > 1) + (n[2] > 1)
    gc = P.make_grid(*n, dims=dims, bc=((0, 0), (1, 1), (2, 2)), reconstr=reconstr)
    rng = np.random.default_rng(seed)
    prim = np.zeros((9,) + gc.shape)
    bfld = np.zeros((3,) + gc.shape)
    a = gc.active
    shp = prim[0][a].shape
    prim[0][a] = np.exp(0.3 * rng.standard_normal(shp))
    for v in (1, 2, 3):
        prim[v][a] = 0.4 * rng.standard_normal(shp)
    prim[4][a] = np.exp(0.3 * rng.standard_normal(shp))
    prim[5][a] = rng.random(shp)
    if not hydro:  # uniform field: divergence free on any grid
        for c, b in enumerate((0.6, -0.4, 0.3)):
            bfld[c] = b
    opts = dict(Nx=n[0], Ny=n[1], Nz=n[2], dims=dims, bc=((0, 0), (1, 1), (2, 2)), gam=5. / 3, cour=0.3,
                reconstr=reconstr)
    return prim, bfld, opts


@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("kw", [dict(reconstr="const"), dict(), dict(charact_proj=1, limiter="mc"),
                                dict(hydro=True, rsolver="hllc", limiter="mm")],
                         ids=["donor", "plm", "charact", "hydro"])
def test_split_flux_walks_bitwise_vs_oracle(n, kw):
    kw = dict(kw)
    prim, bfld, opts = _state(n, kw.pop("reconstr", "linear"), kw.get("hydro", False), sum(n))
    o = oracle_sim(opts, **kw)
    d = device_ctx(opts, exact_fp=True, path="split", **kw)
    nv = 6 if kw.get("hydro") else 9  # the hydro oracle holds no field
    o.set_state(prim[:nv], bfld)
    d.set_state(prim, bfld)
    o.init()
    d.init()
    for _ in range(2):
        dt = o.new_dt()
        assert d.new_dt() == dt
        o.step(dt)
        d.step(dt)
    (Po, Uo, Bo), (Pd, Ud, Bd) = o.get_state(), d.get_state()
    assert np.array_equal(Pd[:nv], Po) and np.array_equal(Ud[:nv], Uo)
    assert not Bd.any() if nv == 6 else np.array_equal(Bd, Bo)
