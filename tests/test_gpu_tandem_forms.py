"""The mixed tandem's two step kernels, for tracks that stay in the cube and for tracks that come and go: which of them
takes a chunk is read off all tracks, so the same tracks run alone, beside others that lie in ports, and in parts
that are too short for the choice take one or the other. Their states are the same, bit for bit, whichever steps them, on their way into the ports too."""
import numpy as np
import pytest

import multiq_workbench_gb300 as mq
from multiq_workbench_gb300.tandem import TRACK_FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mouth", [False, True])
def test_both_forms_step_alike(tandem_small, mouth):
    n, more = 384 * 152 + 3001, 4000   # shorter advances have one form only
    alone = tandem_small(n=n, seed=11, mouth_start=mouth, precision=mq.PREC_MIXED)
    beside = tandem_small(n=n + more, seed=12, precision=mq.PREC_MIXED)
    if mouth:   # some in the cube's middle, on their way to the mouths
        alone.tracks.z[::2] -= 0.012
    part = tandem_small(n=5000, seed=13, precision=mq.PREC_MIXED)
    for k, _ in TRACK_FIELDS:
        getattr(beside.tracks, k)[:n] = getattr(alone.tracks, k)
        getattr(part.tracks, k)[:] = getattr(alone.tracks, k)[:5000]
    beside.tracks.region[n:] = 5
    for a in "xy":
        getattr(beside.tracks, a)[n:] = beside.axis
    beside.tracks.z[n:] = 5e-3
    for steps in (1, 255, 300, 444):
        sa, sb = alone.advance(steps), beside.advance(steps)
        assert sa.steps_cube > 0 and sb.track_steps > sa.track_steps
        part.advance(steps)
        for k, _ in TRACK_FIELDS:
            a, b, c = getattr(alone.tracks, k), getattr(beside.tracks, k)[:n], getattr(part.tracks, k)
            assert np.array_equal(a.view(np.uint8), np.ascontiguousarray(b).view(np.uint8)), (k, steps)
            assert np.array_equal(a[:c.size].view(np.uint8), c.view(np.uint8)), (k, steps)
    if mouth:
        assert sa.steps_port + sa.steps_idle > 0
    for m in (alone, beside, part):
        m.close()
