"""FP32 2-D Model B on 32x32-cell tiles where the last tiles reach past the grid, and 32^2 blocks:
bit for bit the one-block kernel, with partly active grids whose noisy disc crosses the wrap."""
import pytest

import dba_b200
from cases import MODELB_REF, modelb_cfg
from test_gpu_modelb_tiles import _same, patch_ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,B,conserved,form", [
    (264, 264, 8, 1, 1), (72, 936, 8, 0, 2), (272, 304, 16, 1, 1), (1032, 64, 8, 0, 1), (64, 1048, 8, 1, 1), (400, 176, 16, 0, 2),
    (96, 64, 32, 1, 1), (64, 96, 32, 0, 1), (1000, 760, 8, 1, 1)])
def test_ragged_tiles_bitexact_vs_block_kernel(nx, ny, B, conserved, form):
    prm = dict(MODELB_REF, metric_eps=3e-4, k_0=0.3)
    ic = patch_ic(nx, ny, cx=8, cy=ny - 10, radius=22)
    t, k = (dba_b200.Simulation(modelb_cfg(prm, nx, ny, 1, B, precision=1, conserved=conserved, tiles=m)).init(ic)
            for m in (form, 0))
    act = []
    for n, mode in ((1, 1), (1, 1), (1, 1), (9, 1), (20, 1), (2, 0), (40, 1)):
        t.step(n, mode)
        k.step(n, mode)
        _same(t, k)
        act.append(t.flags(0).mean())
    assert B == 32 or min(act) < 1.0      # (6 blocks of 32^2 are all awake around the disc)
    t.sync()
    k.sync()
