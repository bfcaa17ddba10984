"""The launches that bench.py counts for a step are the kernels that run in it."""
import pytest
import torch

import bench
import dba_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,size,precision,block,mode,conserved", [
    ("kh", (1024, 1024, 1), 1, 16, 1, 0), ("kh", (1024, 1024, 1), 1, 16, 0, 0), ("kh", (256, 256, 1), 0, 8, 1, 1),
    ("dendrite", (256, 192, 128), 1, 8, 1, 0), ("dendrite", (64, 64, 64), 1, 8, 1, 0), ("dendrite", (128, 128, 256), 0, 4, 1, 0),
    ("dendrite", (256, 256, 1), 0, 8, 1, 0), ("modelb", (64, 64, 64), 0, 4, 1, 1), ("modelb", (256, 256, 1), 1, 16, 1, 1)])
def test_counted_launches_run(model, size, precision, block, mode, conserved):
    nx, ny, nz = size
    sim = dba_b200.Simulation(dba_b200.config(model, nx=nx, ny=ny, nz=nz, block=block, precision=precision,
                                              conserved=conserved)).init()
    sim.step(1, mode)
    sim.sync()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        sim.step(3, mode)
        sim.sync()
    n = sum(e.count for e in prof.key_averages() if "Memcpy" not in e.key and "Memset" not in e.key and e.self_device_time_total > 0)
    if n == 0:
        pytest.skip("the profiler records no kernels here")
    w = dict(model=model, nx=nx, ny=ny, nz=nz, precision=precision, mode=mode, conserved=conserved)
    assert n == 3 * len(bench.step_launches(w, sim.info.grid_ctas))
