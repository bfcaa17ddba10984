"""bench.py's count of kernel launches per step follows the engine's choice of form."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def _w(model, nx, ny, nz, precision, mode=1, conserved=0):
    return dict(model=model, nx=nx, ny=ny, nz=nz, precision=precision, mode=mode, conserved=conserved)


@pytest.mark.parametrize("w,grid_ctas,count", [
    (_w("kh", 2048, 2048, 1, 1), 444, 3), (_w("kh", 2048, 2048, 1, 1, mode=0), 444, 2), (_w("kh", 512, 512, 1, 1), 444, 2),
    (_w("kh", 2048, 2048, 1, 0), 296, 2), (_w("kh", 2048, 2048, 1, 1, conserved=1), 444, 4),
    (_w("kh", 2048, 2048, 1, 1, mode=0, conserved=1), 444, 2),
    (_w("dendrite", 512, 512, 1, 0), 740, 1), (_w("dendrite", 256, 256, 256, 0), 444, 2),     # listed: 8192 tiles
    (_w("dendrite", 128, 128, 128, 0), 444, 1), (_w("dendrite", 256, 128, 128, 1), 740, 1),   # 1024, 2048 tiles
    (_w("dendrite", 512, 512, 512, 1), 444, 2), (_w("dendrite", 256, 192, 128, 1), 444, 2),   # double-buffered tiles
    (_w("modelb", 2048, 2048, 1, 1, conserved=1), 592, 1), (_w("modelb", 256, 256, 256, 0), 592, 2),
    (_w("modelb", 768, 768, 1, 0, conserved=1), 592, 4), (_w("modelb", 768, 768, 1, 0, mode=0, conserved=1), 592, 2)])
def test_launches_of_a_step(w, grid_ctas, count):
    assert len(bench.step_launches(w, grid_ctas)) == count
