"""The strip walks of large 2D batches and grids (bnz_walk2d.cuh) and the tile
shapes of small single grids.

Both build from the same expressions as the tile kernels, so in the exact build
the states must be equal bit for bit: a batch that walks against the same batch
on the tile variant 9, a single grid against the split path, which shares no
kernel with either.  The fast build's walks round like its tiles too (they fix
by hand what the compiler would contract another way), so there as well a batch
that walks must equal one on tiles.  Sizes put the strips' edges everywhere: one
column or row more and less than a strip holds, grids of a few cells, both sides
of the size where a batch or a grid starts to walk.  (The walks against the
oracle over 100 steps: test_gpu_parity_scale.py.)"""
import numpy as np
import pytest

from bonzo_b200 import problems as P
from bonzo_b200._lib import BNZ_ERR_UNSUPPORTED, WALK_VARIANT, Batch, BnzError, Context

pytestmark = pytest.mark.gpu

SMALL = [(4, 4), (5, 40), (33, 6), (29, 9), (30, 8), (31, 7), (60, 17), (61, 16), (59, 33), (90, 91), (121, 25)]
LARGE = [(640, 640), (641, 600), (600, 641), (512, 640)]  # 1.5 M zones: the batch walks


def _state(n, bc, seed):
    gc = P.make_grid(n[0], n[1], 1, dims=2, bc=bc)
    rng = np.random.default_rng(seed)
    prim, bfld = np.zeros((9,) + gc.shape), np.zeros((3,) + gc.shape)
    a = gc.active
    shp = prim[0][a].shape
    prim[0][a] = np.exp(0.2 * rng.standard_normal(shp))
    for v in (1, 2, 3):
        prim[v][a] = 0.3 * rng.standard_normal(shp)
    prim[4][a] = np.exp(0.2 * rng.standard_normal(shp))
    prim[5][a] = rng.random(shp)
    for c, b in enumerate((0.5, -0.4, 0.3)):  # uniform: divergence free
        bfld[c] = b
    return prim, bfld


BCS = [((0, 0), (0, 0), (0, 0)), ((1, 1), (2, 2), (0, 0)), ((2, 2), (0, 0), (0, 0)), ((0, 0), (1, 1), (0, 0))]


@pytest.mark.parametrize("bc,kw", [(BCS[0], {}), (BCS[1], dict(limiter="mc")), (BCS[2], dict(rsolver="hll")),
                                   (BCS[3], dict(rsolver="hllt", limiter="mm")),
                                   (BCS[1], dict(grav=(0.1, -0.4, 0.0)))])
def test_walking_batch_bitwise_vs_tiles(bc, kw):
    grids = [dict(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=bc) for n in SMALL + LARGE]
    walk = Batch(grids, exact_fp=True, cour=0.3, **kw)
    tile = Batch(grids, exact_fp=True, cour=0.3, **kw)
    walk.set_variant(WALK_VARIANT)
    tile.set_variant(9)
    for q, n in enumerate(SMALL + LARGE):
        s = _state(n, bc, q)
        for b in (walk, tile):
            b[q].set_state(*s)
            b[q].init()
    for b in (walk, tile):
        b.advance(1e30, 3)
    for q in range(len(grids)):
        assert walk[q].time() == tile[q].time()
        for x, y in zip(walk[q].get_state(), tile[q].get_state()):
            assert np.array_equal(x, y), (q, grids[q])


def test_walking_batch_stops_at_tmax():
    """An instance at tmax is carried over unchanged while the others step."""
    bc = BCS[0]
    grids = [dict(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=bc) for n in SMALL + LARGE]
    walk, tile = Batch(grids, exact_fp=True, cour=0.3), Batch(grids, exact_fp=True, cour=0.3)
    walk.set_variant(WALK_VARIANT)
    tile.set_variant(9)
    for q, n in enumerate(SMALL + LARGE):
        s = _state(n, bc, q)
        for b in (walk, tile):
            b[q].set_state(*s)
            b[q].init()
    for b in (walk, tile):
        b.advance(2e-3, 6)  # coarse grids arrive in one step, the large ones step on
    steps = [walk[q].time()[1] for q in range(len(grids))]
    assert min(steps) < max(steps)
    for q in range(len(grids)):
        assert walk[q].time() == tile[q].time()
        for x, y in zip(walk[q].get_state(), tile[q].get_state()):
            assert np.array_equal(x, y), q


def test_variant_numbers_mean_one_kernel_each():
    """A large batch starts on the walks; any tile variant can still be chosen
    and is what runs, and a small batch can be made to walk."""
    bc = BCS[0]
    big = Batch([dict(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=bc) for n in LARGE], cour=0.3)
    for q, n in enumerate(LARGE):
        big[q].set_state(*_state(n, bc, q))
        big[q].init()
    assert big.variant == WALK_VARIANT
    assert all(big.time_variant(v) > 0 for v in (8, WALK_VARIANT)) and big.variant == WALK_VARIANT
    big.set_variant(8)
    assert big.variant == 8
    small = [dict(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=BCS[1]) for n in SMALL]
    out = []
    for v in (None, 8, 9, WALK_VARIANT):
        b = Batch(small, exact_fp=True, cour=0.3)
        assert b.variant == 8 and b.walk_variant == WALK_VARIANT
        if v is not None:
            b.set_variant(v)
            assert b.variant == v
        for q, n in enumerate(SMALL):
            b[q].set_state(*_state(n, BCS[1], q))
            b[q].init()
        b.advance(1e30, 3)
        out.append([c.get_state() for c in b.instances])
    for o in out[1:]:
        for s, s0 in zip(o, out[0]):
            assert all(np.array_equal(x, y) for x, y in zip(s, s0))
    for grids, kw in ((small, dict(charact_proj=1)), ([dict(Nx=8, Ny=8, Nz=8, dims=3, bc=bc)], {})):
        b = Batch(grids, cour=0.3, **kw)
        assert b.walk_variant is None
        with pytest.raises(BnzError) as e:
            b.set_variant(WALK_VARIANT)
        assert e.value.code == BNZ_ERR_UNSUPPORTED
    with pytest.raises(BnzError):
        big.set_variant(WALK_VARIANT + 1)


@pytest.mark.parametrize("n", [(4, 5), (13, 14), (14, 29), (64, 64), (201, 150), (256, 256), (270, 250), (499, 500),
                               (500, 500), (501, 500), (640, 397)])
@pytest.mark.parametrize("bc", BCS[:2])
def test_single_grid_shapes_bitwise_vs_split(n, bc):
    """14 x 14 tiles, 32 x 8 tiles and (from 250 000 cells) walks of one grid."""
    s = _state(n, bc, n[0])
    out = []
    for path in ("fused", "split"):
        c = Context(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=bc, exact_fp=True, cour=0.3, path=path)
        c.set_state(*s)
        c.init()
        for _ in range(2):
            c.step(0.2 / max(n) / 4)
        out.append(c.get_state())
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("bc", BCS)
@pytest.mark.parametrize("kw", [dict(), dict(limiter="mc"), dict(limiter="mm", grav=(0.1, -0.4, 0.2)),
                                dict(rsolver="hll", limiter="mc"), dict(rsolver="hllt"),
                                dict(rsolver="hllt", limiter="mm", grav=(0.1, -0.4, 0.2))],
                         ids=lambda k: "-".join(str(v) for v in k.values()) or "default")
def test_fast_walks_round_like_tiles(bc, kw):
    sizes = SMALL + [(200, 151), (256, 256)]
    grids = [dict(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=bc) for n in sizes]
    out = []
    for v in (WALK_VARIANT, 8, 9):
        b = Batch(grids, cour=0.3, **kw)
        b.set_variant(v)
        for q, n in enumerate(sizes):
            b[q].set_state(*_state(n, bc, q))
            b[q].init()
        b.advance(1e30, 5)
        out.append([c.get_state() + (np.array(c.time()),) for c in b.instances])
    for o in out[1:]:
        for n, s, s0 in zip(sizes, o, out[0]):
            assert all(np.array_equal(x, y) for x, y in zip(s, s0)), n


@pytest.mark.parametrize("kw", [dict(grav=(0.1, -0.3, 0.0), drive_f0=0.8, drive_tau=0.05, drive_nmod=2, drive_seed=3),
                                dict(drive_f0=0.5, drive_tau=0.1, drive_nmod=1, drive_seed=7, rsolver="hll")])
def test_driven_walking_grid_bitwise_vs_split(kw):
    n, bc = (520, 490), BCS[0]
    out = []
    for path in ("fused", "split"):
        c = Context(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=bc, exact_fp=True, cour=0.3, path=path, **kw)
        assert c.variant == (WALK_VARIANT if path == "fused" else -1)
        c.set_state(*_state(n, bc, 2))
        c.init()
        c.advance(1e30, max_steps=3)
        out.append(c.get_state())
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [(40, 40, 40), (41, 23, 37), (64, 30, 17), (97, 65, 50)])
def test_short_update_walks_bitwise_vs_plain(n):
    """3D grids of few columns: the update and EMF kernels walk fewer planes a block."""
    bc = ((0, 0), (1, 1), (2, 2))
    gc = P.make_grid(*n, dims=3, bc=bc)
    prim, bfld = P.blast(gc, b_mag=0.4, b_angle=0.6, center=(0.45, 0.55, 0.5), radius=0.2, p_ratio=40.)
    out = []
    for path in ("plain", "split"):
        c = Context(Nx=n[0], Ny=n[1], Nz=n[2], dims=3, bc=bc, exact_fp=True, cour=0.3, path=path)
        c.set_state(prim, bfld)
        c.init()
        c.advance(1e30, max_steps=3)
        out.append(c.get_state())
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def _pinned(b):
    import torch
    host = []
    for c in b.instances:
        P_ = torch.empty((9,) + c.shape, dtype=torch.float64, pin_memory=True).numpy()
        B_ = torch.empty((3,) + c.shape, dtype=torch.float64, pin_memory=True).numpy()
        c.get_state_into(P_, None, B_)
        host.append((P_, B_))
    return [h[0] for h in host], [h[1] for h in host]


@pytest.mark.parametrize("nchunks", [1, 2, 5, 0])
def test_walking_batch_host_stepping(nchunks):
    """Host stepping of a walking batch, as one group (walks) and in groups
    (tiles), then walks on the device again: bitwise the batch on tiles."""
    bc = BCS[1]
    grids = [dict(Nx=n[0], Ny=n[1], Nz=1, dims=2, bc=bc) for n in SMALL + LARGE]
    walk, tile = Batch(grids, exact_fp=True, cour=0.3), Batch(grids, exact_fp=True, cour=0.3)
    walk.set_variant(WALK_VARIANT)
    tile.set_variant(9)
    for q, n in enumerate(SMALL + LARGE):
        s = _state(n, bc, q)
        for b in (walk, tile):
            b[q].set_state(*s)
            b[q].init()
    P_, B_ = _pinned(walk)
    walk.step_host(P_, B_, 1e30, 3, nchunks)
    walk.advance(1e30, 2)
    tile.advance(1e30, 3)
    for q in range(len(grids)):
        x = tile[q].get_state()
        assert np.array_equal(P_[q], x[0]) and np.array_equal(B_[q], x[2]), q
    tile.advance(1e30, 2)
    assert walk.variant == WALK_VARIANT
    for q in range(len(grids)):
        assert walk[q].time() == tile[q].time()
        for x, y in zip(walk[q].get_state(), tile[q].get_state()):
            assert np.array_equal(x, y), q


def test_walking_batch_host_stepping_is_not_slower_in_groups():
    """The groups of a host-stepped batch are small: they must not take strips
    cut for a launch of the whole batch (2.5 times the time of tiles)."""
    import time
    bc = BCS[0]
    grids = [dict(Nx=320, Ny=320, Nz=1, dims=2, bc=bc)] * 32
    ms = []
    for v in (WALK_VARIANT, 8):
        b = Batch(grids, cour=0.3)
        assert b.variant == WALK_VARIANT
        b.set_variant(v)
        for q in range(len(grids)):
            b[q].set_state(*_state((320, 320), bc, 0))
            b[q].init()
        P_, B_ = _pinned(b)
        b.step_host(P_, B_, 1e30, 10)
        best = 1e9
        for _ in range(3):
            t = time.perf_counter()
            b.step_host(P_, B_, 1e30, 10)
            best = min(best, time.perf_counter() - t)
        ms.append(best)
    assert ms[0] < 1.3 * ms[1], ms


@pytest.mark.parametrize("grids,kw,variant", [
    ([(640, 640)] * 4, {}, WALK_VARIANT), ([(640, 640)] * 4, dict(rsolver="hll"), WALK_VARIANT),
    ([(640, 640)] * 4, dict(rsolver="hllt"), 8),          # its walks cost more than its tiles
    ([(640, 640)] * 4, dict(charact_proj=1), 8),
    ([(640, 640)] * 3, {}, 8),                            # too few zones
    ([(25, 15000)] * 5, {}, WALK_VARIANT),                # one strip of 25 columns
    ([(40, 9500)] * 4, {}, 8), ([(64, 6000)] * 4, dict(rsolver="hll"), 8)])  # half empty strips
def test_batch_starts_on_the_faster_kernels(grids, kw, variant):
    b = Batch([dict(Nx=n[0], Ny=n[1], Nz=1, dims=2) for n in grids], cour=0.3, **kw)
    assert b.variant == variant


@pytest.mark.parametrize("n,kw,variant", [
    ((64, 64), {}, 9), ((224, 224), {}, 9), ((256, 256), {}, 0), ((384, 384), {}, 9), ((499, 500), {}, 9),
    ((500, 500), {}, WALK_VARIANT), ((500, 500), dict(rsolver="hllt"), 9), ((500, 500), dict(charact_proj=1), 9),
    ((640, 640), dict(rsolver="hllt"), WALK_VARIANT), ((4000, 60), {}, 0), ((60, 4000), {}, 9),
    ((31, 10000), {}, 9), ((80000, 4), {}, WALK_VARIANT), ((80000, 4), dict(charact_proj=1), 0)])
def test_single_grid_takes_the_faster_kernels(n, kw, variant):
    assert Context(Nx=n[0], Ny=n[1], Nz=1, dims=2, path="fused", **kw).variant == variant
    assert Context(Nx=n[0], Ny=n[1], Nz=1, dims=2, path="split", **kw).variant == -1
