"""The forms of the 3-D dendrite step against one another, bit for bit: FP32 8^3 blocks on the
double-buffered tiles (grids of more than 2960 tiles, tiles = 1) and on the general tiles from a list
(the same grids, tiles = 0), FP64 and 4^3 blocks from a list, and a part of a periodic domain too
small for a list.  dba_info.grid_ctas tells the forms apart."""
import numpy as np
import pytest

import dba_b200
from cases import DENDRITE_REF, dendrite_cfg

pytestmark = pytest.mark.gpu

PRM = dict(DENDRITE_REF, Delta=1.15, delta=0.2, metric_p=1e-3, metric_T=1e-5)
BIG = (256, 192, 128)                            # 8 x 24 x 16 tiles


def _seeds(shape, seed, n=3, r=9.0):
    """A few tanh seeds, one on a corner, in undercooled melt; (nz, ny, nx)."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    z, y, x = np.mgrid[0:nz, 0:ny, 0:nx].astype(np.float32)
    p = np.zeros((nz, ny, nx), np.float32)
    for c in [(0, 0, 0)] + [tuple(rng.random(3) * (nx, ny, nz)) for _ in range(n - 1)]:
        d = np.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2)
        p = np.maximum(p, 0.5 * (1.0 - np.tanh((d - r) / 2.0)))
    return [p.astype(np.float64), np.full(p.shape, -1.15)]


def _same(a, b, copies=(1, 1, 1)):
    for f in ("p", "T"):
        u = a.field_f32(f) if a.cfg.precision else a.field(f)
        v = b.field_f32(f) if b.cfg.precision else b.field(f)
        assert np.isfinite(u).all()
        assert np.array_equal(np.tile(u, copies), v), f
    B = a.cfg.block
    for w in (0, 1, 2, 3):
        u = a.flags(w).reshape(a.cfg.nz // B, a.cfg.ny // B, -1)
        assert np.array_equal(np.tile(u, copies).ravel(), b.flags(w)), w


def _sim(shape, B, precision, ic, bc=0, prm=PRM, **kw):
    return dba_b200.Simulation(dendrite_cfg(prm, *shape, B, precision=precision, bc=bc, **kw)).init(ic)


@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("shape", [BIG, (232, 232, 120)])
def test_double_buffered_tiles_equal_listed_tiles(bc, shape):
    ic = _seeds(shape, 5)
    a, b = (_sim(shape, 8, 1, ic, bc, tiles=t) for t in (1, 0))
    assert a.info.grid_ctas != b.info.grid_ctas
    act = []
    for steps, mode in ((1, 1), (1, 1), (1, 1), (5, 1), (60, 1), (3, 0), (1, 1), (30, 1)):
        a.step(steps, mode)
        b.step(steps, mode)
        _same(a, b)
        act.append((a.flags(0).mean(), a.flags(2).mean()))
    assert min(v[0] for v in act) < 0.2 and 0.0 < min(v[1] for v in act) < 0.5
    a.sync()
    b.sync()


@pytest.mark.parametrize("B,precision,tiles", [(8, 1, 1), (8, 1, 0), (4, 1, 1), (4, 0, 1), (8, 0, 1)])
def test_listed_equal_unlisted(B, precision, tiles):
    """2 x 2 x 2 copies of a periodic domain (a list) and the domain (none)."""
    shape = (128, 96, 64)
    ic = _seeds(shape, 7)
    a = _sim(shape, B, precision, ic, tiles=tiles)
    b = _sim(tuple(2 * n for n in shape), B, precision, [np.tile(f, (2, 2, 2)) for f in ic], tiles=tiles)
    for steps, mode in ((1, 1), (2, 1), (50, 1), (2, 0), (1, 1), (20, 1)):
        a.step(steps, mode)
        b.step(steps, mode)
        _same(a, b, (2, 2, 2))
    a.sync()
    b.sync()


@pytest.mark.parametrize("B,precision,tiles", [(8, 1, 1), (8, 1, 0), (4, 0, 1)])
def test_lists_without_an_entry(B, precision, tiles):
    """Thresholds that no cell passes: after the first step nothing is active and every list is empty;
    regular and DBA steps that follow match the domain without a list."""
    prm = dict(PRM, metric_p=0.6, metric_T=1e30)
    shape = (128, 96, 64)
    ic = _seeds(shape, 9)
    a = _sim(shape, B, precision, ic, prm=prm, tiles=tiles)
    b = _sim(tuple(2 * n for n in shape), B, precision, [np.tile(f, (2, 2, 2)) for f in ic], prm=prm, tiles=tiles)
    for s in (a, b):
        s.step(1, 1)
    c0 = b.cell_updates()
    for steps, mode in ((1, 1), (7, 1), (48, 1)):
        for s in (a, b):
            s.step(steps, mode)
    assert b.cell_updates() == c0
    for steps, mode in ((5, 0), (1, 1), (6, 1), (3, 0)):
        for s in (a, b):
            s.step(steps, mode)
        _same(a, b, (2, 2, 2))
    a.sync()
    b.sync()


@pytest.mark.parametrize("tiles", [1, 0])
def test_large_grids_report_non_finite_values(tiles):
    ic = _seeds(BIG, 11)
    ic[1][5, 6, 7] = np.nan                      # in the corner seed: an active block
    s = _sim(BIG, 8, 1, ic, tiles=tiles)
    s.step(2, 1)
    with pytest.raises(dba_b200.DBAError) as e:
        s.sync()
    assert e.value.code == 5
