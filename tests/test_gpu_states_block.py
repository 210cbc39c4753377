"""Ion states that lie in one block go over in one copy, others array by array: the same results, odd counts
included, and nothing beside the arrays is written."""
import numpy as np
import pytest

import multiq_workbench_gb300 as mq
from multiq_workbench_gb300.channel import ION_FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [mq.PREC_MIXED, mq.PREC_F64])
@pytest.mark.parametrize("n", [1, 33, 20001])
def test_block_and_separate_arrays_agree(coarse, prec, n):
    ph = mq.Physics(legacy_force=True, pressure_pa=0.133322, temp_k=300.0, dt=1e-7, t_max=200 * 1e-7, launch=mq.LAUNCH_GAUSSIAN,
                    sigma_mm=0.1)
    jobs = [mq.Job(mq.Species(499.0, 1.0, 2.95 * 499.0 ** (2 / 3)), mq.RfAc(100.0, 500e3, 0.5, 100e3), n, 3)]
    with mq.Engine(coarse, prec) as e:
        e.set_dc([0.0, 5.0, -5.0, 0.0])
        block = e.inject(jobs, ph).copy()
        guard = 64
        room = {k: np.full(n + 2 * guard, 7, dt) for k, dt in ION_FIELDS}
        apart = mq.IonStates(**{k: room[k][guard:guard + n] for k, _ in ION_FIELDS})
        for k, _ in ION_FIELDS:
            getattr(apart, k)[:] = getattr(block, k)
        for s in (block, apart):
            e.run_ions(jobs, ph, s, max_more=101)
    for k, _ in ION_FIELDS:
        assert np.array_equal(getattr(block, k).view(np.uint8), getattr(apart, k).view(np.uint8)), k
        assert (room[k][:guard] == 7).all() and (room[k][-guard:] == 7).all(), k
    assert (block.steps > 0).all()
