"""The dendrite tile kernels and the two Model B kernels where their tiles end: grids that
are multiples of the block edge only, one tile or several, the smallest grids, partial
activity.  FP64 must equal the CPU restatement bit for bit, flags at every step; FP32 stays
within the tolerances of test_gpu_parity.py (2e-5 for the dendrite's fields, relative L2 1e-4
for Model B: rounding of a few 1e-7 per step over the steps taken here)."""
import numpy as np
import pytest

import dba_b200
from cases import DENDRITE_REF, MODELB_REF, dendrite_cfg, modelb_cfg
from oracle_lib import OracleDendrite, OracleModelB

pytestmark = pytest.mark.gpu

DEN = dict(DENDRITE_REF, Delta=1.15, delta=0.2, metric_p=1e-3, metric_T=1e-5)


def _seed(nx, ny, nz, r):
    """A solid corner piece and its warm layer, off the tile centres."""
    z, y, x = np.mgrid[0:nz, 0:ny, 0:nx].astype(np.float64)
    d = np.sqrt((x - 0.3 * nx) ** 2 + (y - 0.6 * ny) ** 2 + (z - 0.4 * nz) ** 2) - r
    return 0.5 * (1 - np.tanh(d / 2)), -1.15 + 0.5 * (1 - np.tanh(d / 3))


@pytest.mark.parametrize("nx,ny,nz,B,mode,bc,precision", [
    (36, 20, 12, 4, 1, 0, 0), (36, 20, 12, 4, 1, 1, 0), (40, 24, 16, 8, 1, 0, 0), (72, 24, 8, 8, 1, 1, 0),
    (4, 4, 4, 4, 1, 0, 0), (8, 8, 8, 8, 1, 1, 0), (68, 12, 20, 4, 0, 1, 0), (40, 16, 24, 8, 0, 0, 0),
    (36, 20, 12, 4, 1, 1, 1), (68, 12, 20, 4, 0, 0, 1), (40, 24, 16, 8, 1, 1, 1), (200, 128, 144, 4, 1, 0, 0),
    (136, 144, 168, 8, 1, 1, 0),                         # the last two work from a tile list
    (36, 20, 1, 4, 1, 1, 0), (36, 20, 1, 4, 0, 0, 0), (40, 24, 1, 8, 1, 0, 0), (48, 80, 1, 16, 1, 1, 0),
    (96, 32, 1, 32, 1, 0, 0), (4, 4, 1, 4, 1, 1, 0), (40, 24, 1, 8, 1, 1, 1), (48, 80, 1, 16, 0, 1, 1),
    (1000, 256, 1, 8, 1, 1, 0), (1000, 260, 1, 4, 1, 0, 0)])   # these two have more tiles than a DBA step takes by tile
def test_dendrite_tile_edges(nx, ny, nz, B, mode, bc, precision):
    p, T = _seed(nx, ny, nz, 3.0 if nx < 100 else 12.0)
    o = OracleDendrite(nx, ny, nz, B, DEN, bc=bc)
    o.set_fields(p, T)
    s = dba_b200.Simulation(dendrite_cfg(DEN, nx, ny, nz, B, precision=precision, bc=bc)).init([p, T])
    for t in range(1, 31 if nx < 100 else 9):
        o.step(1, mode)
        s.step(1, mode)
        if precision:
            continue
        d = o.get()
        assert np.array_equal(s.field("p"), d["p"]), t
        assert np.array_equal(s.field("T"), d["T"]), t
        if mode:
            for w, k in enumerate(("wake_p", "next_p", "wake_T", "next_T")):
                assert np.array_equal(s.flags(w), d[k]), (k, t)
    d = o.get()
    assert np.max(np.abs(s.field("p") - d["p"])) <= 2e-5 and np.max(np.abs(s.field("T") - d["T"])) <= 2e-5
    s.sync()


@pytest.mark.parametrize("nx,ny,nz,bc", [(200, 256, 256, 0), (136, 256, 256, 1), (256, 256, 128, 1)])
def test_dendrite3_fp32_tiles_past_the_grid(nx, ny, nz, bc):
    """FP32 8^3 blocks on grids that work from a tile list: the double-buffered tiles, whose last
    tile of a row may reach past the grid, equal the general tile kernel bit for bit."""
    p, T = _seed(nx, ny, nz, 20.0)
    a, b = (dba_b200.Simulation(dendrite_cfg(DEN, nx, ny, nz, 8, precision=1, bc=bc, tiles=t)).init([p, T]) for t in (1, 0))
    for n, mode in ((1, 1), (1, 1), (30, 1), (3, 0), (40, 1)):
        for s in (a, b):
            s.step(n, mode)
        for q in ("p", "T"):
            assert np.array_equal(a.field(q), b.field(q)), (q, n)
        for w in range(4):
            assert np.array_equal(a.flags(w), b.flags(w)), (w, n)
    a.sync()
    b.sync()


@pytest.mark.parametrize("nx,ny,nz,B,mode,conserved,precision", [
    (36, 20, 12, 4, 1, 1, 0), (40, 24, 16, 8, 1, 1, 0), (4, 4, 4, 4, 1, 1, 0), (8, 8, 8, 8, 1, 0, 0),
    (36, 12, 20, 4, 0, 0, 0), (24, 16, 40, 8, 0, 0, 0), (36, 20, 1, 4, 1, 1, 0), (40, 24, 1, 8, 1, 1, 0),
    (48, 80, 1, 16, 1, 1, 0), (96, 32, 1, 32, 1, 1, 0), (4, 4, 1, 4, 1, 0, 0), (36, 20, 12, 4, 1, 1, 1),
    (40, 24, 16, 8, 1, 0, 1), (40, 16, 24, 8, 0, 0, 1)])
def test_modelb_tile_edges(nx, ny, nz, B, mode, conserved, precision):
    prm = dict(MODELB_REF, metric_eps=1e-3, rx=3)      # rx = 3: the division that no product replaces
    rng = np.random.default_rng(7)
    f = [v + 0.02 * (rng.random((nz, ny, nx)) - 0.5) for v in (0.2, 0.2, 0.1)]
    for a, v in zip(f, (0.2, 0.2, 0.1)):
        a[:, :, (nx // 2 // B) * B + 1:] = v           # the far part starts uniform, hence asleep
    o = OracleModelB(nx, ny, nz, B, prm, conserved=conserved)
    o.set_fields(*f)
    s = dba_b200.Simulation(modelb_cfg(prm, nx, ny, nz, B, precision=precision, conserved=conserved)).init(f)
    for t in range(1, 21):
        o.step(1, mode)
        s.step(1, mode)
        if precision:
            continue
        for q in ("x", "y", "z"):
            assert np.array_equal(s.field(q), o.field(q)), (q, t)
        if mode:
            w, nxt = o.flags()
            assert np.array_equal(s.flags(0), w) and np.array_equal(s.flags(1), nxt), t
    for q in ("x", "y", "z"):
        a, b = s.field(q), o.field(q)
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), q
    s.sync()
