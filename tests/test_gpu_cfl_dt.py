"""The one-launch CFL time step (bcdt::k_cfl_dt) over grids of one block, of a
few and of more blocks than one pass, asked for again and again: the maximum and
the count of finished blocks must be back at zero each time.  Bitwise the
oracle's dt in the exact build."""
import numpy as np
import pytest

from bonzo_b200 import problems as P
from helpers import device_ctx, oracle_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(5, 1, 1), (255, 1, 1), (257, 1, 1), (16, 16, 1), (33, 31, 1), (700, 650, 1), (9, 8, 7),
                               (70, 61, 83)])
def test_cfl_dt_bitwise_vs_oracle(n):
    dims = 1 + (n[1] > 1) + (n[2] > 1)
    gc = P.make_grid(*n, dims=dims, bc=0)
    rng = np.random.default_rng(sum(n))
    prim, bfld = np.zeros((9,) + gc.shape), np.zeros((3,) + gc.shape)
    a = gc.active
    opts = dict(Nx=n[0], Ny=n[1], Nz=n[2], dims=dims, bc=((0, 0),) * 3, gam=5. / 3, cour=0.3)
    o, d = oracle_sim(opts), device_ctx(opts, exact_fp=True, path="split")
    for c, b in enumerate((0.5, 0.3, 0.2)):
        bfld[c] = b
    for _ in range(3):
        prim[0][a] = np.exp(0.4 * rng.standard_normal(prim[0][a].shape))
        for v in (1, 2, 3):
            prim[v][a] = rng.standard_normal(prim[0][a].shape)
        prim[4][a] = np.exp(0.4 * rng.standard_normal(prim[0][a].shape))
        for s in (o, d):
            s.set_state(prim, bfld)
            s.init()
        assert d.new_dt() == o.new_dt()
        assert d.new_dt() == o.new_dt()


def test_host_stepping_stops_at_tmax():
    """advance clips the last step to tmax: the record's dt is then the host's."""
    gc = P.make_grid(33, 31, 1, dims=2, bc=0)
    prim, bfld = P.otvortex(gc)
    opts = dict(Nx=33, Ny=31, Nz=1, dims=2, bc=((0, 0),) * 3, gam=5. / 3, cour=0.3)
    for path in ("fused", "split", "plain"):
        o, d = oracle_sim(opts), device_ctx(opts, exact_fp=True, path=path)
        for s in (o, d):
            s.set_state(prim, bfld)
            s.init()
        tmax = 2.5 * o.new_dt()
        o.advance(tmax)
        assert d.advance(tmax) == (o.time, o.nstep)
        for x, y in zip(d.get_state(), o.get_state()):
            assert np.array_equal(x, y)
