"""Ion states in one block of which a part is page-locked (a host program may register the arrays that it
reads itself): they lie one after the other like any block's, but no single copy may span the two kinds of
memory. The results are those of states in separate arrays."""
import numpy as np
import pytest

import multiq_workbench_gb300 as mq
from multiq_workbench_gb300.channel import ION_FIELDS, _ION_BYTES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first, last", [(0, 6), (8, 9), (9, 14)])
def test_block_registered_in_part(coarse, first, last):
    torch = pytest.importorskip("torch")
    ph = mq.Physics(legacy_force=True, pressure_pa=0.133322, temp_k=300.0, dt=1e-7, t_max=200 * 1e-7, launch=mq.LAUNCH_GAUSSIAN,
                    sigma_mm=0.1)
    n = 1 << 16   # every array begins on a page
    jobs = [mq.Job(mq.Species(499.0, 1.0, 2.95 * 499.0 ** (2 / 3)), mq.RfAc(100.0, 500e3, 0.5, 100e3), n, 3)]
    page = 1 << 16
    room = np.zeros(n * _ION_BYTES + page, np.uint8)
    at = -room.ctypes.data % page
    st = mq.IonStates._in_block(room[at:at + n * _ION_BYTES], n)
    names = [k for k, _ in ION_FIELDS]
    begin = getattr(st, names[first]).ctypes.data
    size = sum(getattr(st, k).nbytes for k in names[first:last])
    rt = torch.cuda.cudart()
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        e.set_dc([0.0, 5.0, -5.0, 0.0])
        ref = e.inject(jobs, ph)
        for k in names:
            getattr(st, k)[:] = getattr(ref, k)
        e.run_ions(jobs, ph, ref, max_more=101)
        assert int(rt.cudaHostRegister(begin, size, 0)) == 0
        try:
            e.run_ions(jobs, ph, st, max_more=101)
        finally:
            assert int(rt.cudaHostUnregister(begin)) == 0
    for k in names:
        assert np.array_equal(getattr(st, k).view(np.uint8), getattr(ref, k).view(np.uint8)), k
    assert (st.steps > 0).all()
