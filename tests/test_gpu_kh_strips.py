"""FP32 KH strips (grids of 2^20 cells and more) against the tile kernel (smaller grids): a 1024^2
periodic domain made of 2 x 2 copies of a 512^2 one evolves as four copies of it, bit for bit --
fields and flags, fixed and CFL time step, with a quiet region (partly active grids: strips,
tiles and the persisted values between them), blocks falling asleep, and in regular mode."""
import numpy as np
import pytest

import dba_b200

pytestmark = pytest.mark.gpu


def _flow(n, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:n, 0:n] / n
    d = np.hypot(x - 0.3, y - 0.6)
    env = np.clip((d - 0.12) / 0.05, 0.0, 1.0)           # quiet inside a disc
    vx, vy, rho = 0.0 * x, 0.0 * x, 1.0 + 0.0 * x
    for _ in range(8):
        k, m, p, a = rng.integers(1, 6), rng.integers(1, 6), rng.random(), rng.random()
        w = np.cos(2 * np.pi * (k * x + m * y + p))
        vx, vy, rho = vx + 0.1 * m * w * env, vy - 0.1 * k * w * env, rho + 0.03 * a * w * env
    return [rho, 2.5 + 0.0 * x, vx, vy]


def _sim(n, copies, B, cfl, eps, ic):
    h = 1.0 / n
    c = dba_b200.config("kh", nx=n * copies, ny=n * copies, nz=1, block=B, precision=1, dx=h, dy=h, dz=h, dt=0.1 * h,
                        kh_gamma=1.4, metric_eps=eps, cfl=cfl)
    return dba_b200.Simulation(c).init([np.tile(f, (copies, copies)) for f in ic])


@pytest.mark.parametrize("B,cfl,eps", [(16, 0.4, 1e-3), (8, 0.0, 1e-3), (8, 0.4, 8.0), (16, 0.0, 16.0), (16, 0.4, 0.0)])
def test_strips_equal_tiles(B, cfl, eps):
    n = 512
    ic = _flow(n, 3)
    a, b = _sim(n, 1, B, cfl, eps, ic), _sim(n, 2, B, cfl, eps, ic)
    nb = n // B
    act = []
    for steps, mode in ((1, 1), (1, 1), (7, 1), (40, 1), (3, 0), (1, 1), (30, 1)):
        for s in (a, b):
            s.step(steps, mode)
        for f in ("Mass", "Momx", "Momy", "Energy"):
            u, v = a.field_f32(f)[0], b.field_f32(f)[0]
            assert np.array_equal(np.tile(u, (2, 2)), v), (f, steps, mode)
        for w in (0, 1):
            assert np.array_equal(np.tile(a.flags(w).reshape(nb, nb), (2, 2)).ravel(), b.flags(w)), (w, steps, mode)
        act.append(b.flags(0).mean())
    if cfl:
        assert a.observables()["time"] == b.observables()["time"]
    assert min(act) < 1.0 or eps == 0.0
    a.sync()
    b.sync()


@pytest.mark.parametrize("eps", [1e-3, 16.0])
def test_strips_resume_from_a_saved_state(eps):
    """A context that loads a state in the middle of a run goes on bit for bit like the one that
    saved it: what strips leave to the next step is in the state."""
    ic = _flow(512, 5)
    a, b = _sim(512, 2, 16, 0.4, eps, ic), _sim(512, 2, 16, 0.4, eps, ic)
    a.step(25, 1)
    blob = np.empty(a.state_size(), np.uint8)
    a.save_state(blob)
    b.step(4, 1)
    b.load_state(blob)
    for steps in (1, 1, 20):
        for s in (a, b):
            s.step(steps, 1)
        for f in ("Mass", "Momx", "Momy", "Energy"):
            assert np.array_equal(a.field_f32(f), b.field_f32(f)), (f, steps)
        assert np.array_equal(a.flags(0), b.flags(0)) and np.array_equal(a.flags(1), b.flags(1)), steps
    a.sync()
    b.sync()
