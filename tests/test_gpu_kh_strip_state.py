"""A state saved by FP32 KH strips holds the stale values of the blocks that fell asleep in its last
step, computed with the step's own constants: a context that loads it and goes on with another
time step matches the tile kernel's run (a quarter of the domain, too small for strips) that
does the same, bit for bit."""
import numpy as np
import pytest

from test_gpu_kh_strips import _flow

import dba_b200

pytestmark = pytest.mark.gpu


def _sim(n, copies, B, ic=None, **more):
    h = 1.0 / n
    kw = dict(dt=0.1 * h, kh_gamma=1.4, metric_eps=60.0)   # blocks with gradients fall asleep
    kw.update(more)
    c = dba_b200.config("kh", nx=n * copies, ny=n * copies, nz=1, block=B, precision=1, dx=h, dy=h, dz=h, **kw)
    s = dba_b200.Simulation(c)
    return s.init([np.tile(f, (copies, copies)) for f in ic]) if ic is not None else s


@pytest.mark.parametrize("how", ["blob", "file"])
@pytest.mark.parametrize("B,cfl,change", [(16, 0.0, dict(dt=0.03 / 512)), (8, 0.4, dict(cfl=0.2)), (8, 0.0, dict(kh_gamma=1.6)),
                                          (16, 0.4, {})])
def test_resume_with_other_constants(tmp_path, B, cfl, change, how):
    n = 512
    ic = _flow(n, 3)
    out = []
    for copies in (1, 2):
        a = _sim(n, copies, B, ic, cfl=cfl)
        before = a.flags(0)
        a.step(1, 1)           # every block active, hence strips; then the quiet ones fall asleep
        after = a.flags(0)
        assert (before == 1).all() and 0 < after.mean() < 1
        b = _sim(n, copies, B, **dict(dict(cfl=cfl), **change))
        if how == "file":
            a.checkpoint(tmp_path / f"{copies}.bin")
            b.restore(tmp_path / f"{copies}.bin")
        else:
            blob = np.empty(a.state_size(), np.uint8)
            a.save_state(blob)
            b.load_state(blob)
        for steps in (1, 1, 30):
            b.step(steps, 1)
        out.append([b.field_f32(f)[0] for f in ("Mass", "Momx", "Momy", "Energy")] + [b.flags(0).reshape(n * copies // B, -1)])
        b.sync()
    for u, v in zip(*out):
        assert np.array_equal(np.tile(u, (2, 2)), v)
