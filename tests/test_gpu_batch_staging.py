"""Staging of the batch kernel: every block edge, type and thread count, in an arena whose
capacity is no multiple of a 16-byte piece, with a partly filled last group."""
import numpy as np
import pytest

import dba_b200
from cases import DENDRITE_REF, dendrite_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("precision,B,bc", [(1, 4, 0), (1, 16, 1), (1, 8, 0), (0, 4, 1), (0, 8, 0), (0, 16, 1)])
def test_batch_staging_equals_single_simulation(precision, B, bc, threads):
    """Both evaluate the same rounded point formulas: the same bits, after direct launches and graphs."""
    b = dba_b200.Batch(precision=precision, block=B, max_slots=4, block_capacity=4096, cell_capacity=(1 << 14) + 5,
                       threads=threads)
    b.add(dendrite_cfg(dict(DENDRITE_REF, Delta=0.6), 32, 48, 1, B, precision=precision, bc=1 - bc))
    k = dendrite_cfg(DENDRITE_REF, 48, 80, 1, B, precision=precision, bc=bc)
    s = b.add(k)
    sim = dba_b200.Simulation(k).init()
    for n in (1, 60):
        b.step(n)
        sim.step(n, 1)
        assert np.array_equal(b.field(s, "p"), sim.field("p")), n
        assert np.array_equal(b.field(s, "T"), sim.field("T")), n
    b.sync()
    sim.sync()
