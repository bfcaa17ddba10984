"""FP64 2-D Model B on tiles of 16 rows (4^2 and 8^2 blocks, more than 1776 tiles of 8 rows) against the
CPU restatement, bit for bit: just past the size from which it takes them, with a last row and
column of tiles past the grid, partly active, plain and conserved, DBA and regular; and the
largest grid that does not take them."""
import numpy as np
import pytest

import dba_b200
from cases import MODELB_REF, modelb_cfg
from oracle_lib import OracleModelB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,B,mode,conserved", [
    (1000, 456, 8, 1, 1), (1004, 460, 4, 1, 0), (1004, 468, 4, 1, 1), (1000, 456, 8, 0, 0), (1024, 448, 8, 1, 0),
    (32, 14216, 8, 1, 0), (1024, 444, 4, 1, 1)])
def test_tall_tiles(nx, ny, B, mode, conserved):
    prm = dict(MODELB_REF, metric_eps=1e-3)
    rng = np.random.default_rng(11)
    f = [v + 0.02 * (rng.random((1, ny, nx)) - 0.5) for v in (0.2, 0.2, 0.1)]
    for a, v in zip(f, (0.2, 0.2, 0.1)):
        a[:, ny // 3:, (nx // 3 // B) * B + 1:] = v    # this part starts uniform, hence asleep
    o = OracleModelB(nx, ny, 1, B, prm, conserved=conserved)
    o.set_fields(*f)
    s = dba_b200.Simulation(modelb_cfg(prm, nx, ny, 1, B, conserved=conserved)).init(f)
    for n in (1, 1, 5):
        o.step(n, mode)
        s.step(n, mode)
        for q in ("x", "y", "z"):
            assert np.array_equal(s.field(q), o.field(q)), (q, n)
        if mode:
            w, nxt = o.flags()
            assert np.array_equal(s.flags(0), w) and np.array_equal(s.flags(1), nxt), n
            assert nx == 32 or 0.0 < s.flags(0).mean() < 1.0      # (a column of tiles: each has an active neighbour)
    s.sync()
