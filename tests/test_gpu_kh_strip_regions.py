"""FP32 KH strips beside tiles, at the shapes and activities where they can go wrong: units of 32 rows
with a short last one, grids of unequal edges and narrower than a strip, many steps in which some
tiles go by strips and some by tiles while blocks fall asleep and wake.  Against the four stage
kernels (tiles = 0; every KH formula of both goes through the same rounded helpers), or, for the
CFL step that those do not have, against a part of the domain too small for strips; bit for bit."""
import numpy as np
import pytest

import dba_b200

pytestmark = pytest.mark.gpu


def _flow(nx, ny, quiet, seed=3):
    """Random modes outside a disc of share `quiet`."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:ny, 0:nx]
    r = np.sqrt(quiet * nx * ny / np.pi)
    env = np.clip((np.hypot(x - 0.4 * nx, y - 0.55 * ny) - r) / 4.0, 0.0, 1.0) if quiet else np.ones((ny, nx))
    vx, vy, rho = 0.0 * env, 0.0 * env, 1.0 + 0.0 * env
    for _ in range(6):
        k, m, p, a = rng.integers(1, 6), rng.integers(1, 6), rng.random(), rng.random()
        w = np.cos(2 * np.pi * (k * x / nx + m * y / ny + p))
        vx, vy, rho = vx + 0.1 * m * w * env, vy - 0.1 * k * w * env, rho + 0.03 * a * w * env
    return [rho, 2.5 + 0.0 * rho, vx, vy]


def _sim(nx, ny, B, ic, copies=(1, 1), **more):
    h = 1.0 / 512
    kw = dict(precision=1, dx=h, dy=h, dz=h, dt=0.1 * h, kh_gamma=1.4, metric_eps=1e-3)
    kw.update(more)
    s = dba_b200.Simulation(dba_b200.config("kh", nx=nx * copies[1], ny=ny * copies[0], nz=1, block=B, **kw))
    return s.init([np.tile(f, copies) for f in ic])


def _full(s, B):
    """Share of the tiles whose blocks and all blocks around them are active in the next step."""
    nby, nbx = s.cfg.ny // B, s.cfg.nx // B
    a = s.flags(0).reshape(nby, nbx) != 0
    f = a.copy()
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            f &= np.roll(a, (dy, dx), (0, 1))
    t = 16 // B
    return f.reshape(nby // t, t, nbx // t, t).all(axis=(1, 3)).mean()


def _same(a, b, copies=(1, 1)):
    for f in ("Mass", "Momx", "Momy", "Energy"):
        u = a.field_f32(f)[0]
        assert np.isfinite(u).all()
        assert np.array_equal(np.tile(u, copies), b.field_f32(f)[0]), f
    for w in (0, 1):
        u = a.flags(w).reshape(a.cfg.ny // a.cfg.block, -1)
        assert np.array_equal(np.tile(u, copies).ravel(), b.flags(w)), w


@pytest.mark.parametrize("B,eps", [(16, 1e-3), (8, 12.0)])
def test_strips_of_32_rows_with_a_short_last_unit(B, eps):
    """2048 x 2064: 2240 units of 32 rows and a row of 16; a fifth of the domain quiet."""
    nx, ny, copies = 1024, 688, (3, 2)
    ic = _flow(nx, ny, 0.2)
    a, b = _sim(nx, ny, B, ic, cfl=0.4, metric_eps=eps), _sim(nx, ny, B, ic, copies, cfl=0.4, metric_eps=eps)
    mixed = 0
    for k in range(24):
        a.step(1, 1)
        b.step(1, 1)
        mixed += 0.62 < _full(b, B) < 1.0       # strips on, beside tiles
        if k in (0, 1, 2, 12):
            _same(a, b, copies)
    assert mixed >= 16
    for steps, mode in ((48, 1), (2, 0), (1, 1), (30, 1)):
        a.step(steps, mode)
        b.step(steps, mode)
        _same(a, b, copies)
    assert a.observables()["time"] == b.observables()["time"]
    a.sync()
    b.sync()


@pytest.mark.parametrize("nx,ny,B,quiet", [(48, 21856, 16, 0.04), (48, 21856, 8, 0.3), (1216, 880, 8, 0.08), (4096, 272, 16, 0.5),
                                            (1040, 1024, 16, 0.05)])
def test_strips_equal_stage_kernels(nx, ny, B, quiet):
    ic = _flow(nx, ny, quiet)
    a, b = _sim(nx, ny, B, ic, tiles=0), _sim(nx, ny, B, ic)
    for steps, mode in ((1, 1), (1, 1), (1, 1), (20, 1), (3, 0), (1, 1), (25, 1)):
        a.step(steps, mode)
        b.step(steps, mode)
        _same(a, b)
    a.sync()
    b.sync()


def test_conserved_context_regular_then_dba():
    """Regular steps of a conserved context go by strips, its DBA steps by tiles with block sums."""
    ic = _flow(1024, 1024, 0.1)
    a, b = (_sim(1024, 1024, 16, ic, tiles=t, conserved=1) for t in (0, 1))
    for steps, mode in ((2, 0), (6, 1), (1, 0), (1, 1), (12, 1), (2, 0)):
        a.step(steps, mode)
        b.step(steps, mode)
        _same(a, b)
    a.sync()
    b.sync()


@pytest.mark.parametrize("mode", [0, 1])
def test_strips_report_non_finite_values(mode):
    ic = _flow(1024, 1024, 0.0)
    ic[0][700, 333] = np.nan
    s = _sim(1024, 1024, 16, ic, metric_eps=0.0)
    s.step(2, mode)
    with pytest.raises(dba_b200.DBAError) as e:
        s.sync()
    assert e.value.code == 5
