"""The mixed engine's one-lane kernel in every form a tuning can give it: lists longer than the lane groups hold, cut
into launches that queue the ions again at every position of a four-step window, with both record widths, the L1
prefetch, the cell sort, as a graph and as single launches. Bit for bit what the lane groups make of the same
ions in short lists."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent))
from test_gpu_parity import FIELDS, _mq, _variants  # noqa: E402

pytestmark = pytest.mark.gpu

DC = [0.0, 5.0, -5.0, 0.0]
N = 31000   # more than the 29,184 that lane groups hold with nearest-node fields on 152 SMs
SHAPES = [dict(wide_records=w, prefetch=p, sort_cells=s, chunk=c, use_graph=g, blocks_per_sm=b)
          for w in (True, False)
          for p, s, c, g, b in ((False, False, 37, True, 3), (True, False, 701, True, 1), (True, True, 301, False, 2), (False, True, 149, True, 3))]


@pytest.mark.parametrize("name", ["corrected_disc", "half_kick_gauss", "legacy_all", "legacy_coll_trilinear", "thermal_nearest"])
def test_every_form_equals_the_groups(coarse, name):
    mq = _mq()
    ph = _variants()[name]
    sp = mq.Species(499.0 * 5, 5.0, 0.0) if name.startswith("legacy") else mq.Species(499.0, 1.0, 2.95 * 499.0 ** (2 / 3))
    jobs = [mq.Job(sp, mq.RfAc(100.0, 500e3, 0.5, 100e3), N, 9)]
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        e.set_dc(DC)
        st = e.inject(jobs, ph)
        st.steps[:] = np.arange(N) % 13

        def run(i0, i1):
            s = mq.IonStates.empty(i1 - i0)
            for f in FIELDS:
                getattr(s, f)[:] = getattr(st, f)[i0:i1]
            e.run_ions(jobs, ph, s, max_more=1000)
            return s
        parts = [run(i, min(i + 8000, N)) for i in range(0, N, 8000)]
        want = {f: np.concatenate([getattr(p, f) for p in parts]) for f in FIELDS}
        for shape in SHAPES:
            e.set_tuning(**shape)
            got = run(0, N)
            for f in FIELDS:
                assert np.array_equal(want[f].view(np.uint8), getattr(got, f).view(np.uint8)), (name, shape, f)
