"""Where the mixed tandem kernel sends a track, against the oracle: tracks at rest all over the cube, its
walls, mouths, ports and what lies outside, one step. The kernel's positions are FP32 in millimetres when
it asks the cube's geometry (an error of 5e-6 mm at 40 mm) and surfaces take up about 1 mm^2 per mm^3, so of
20,000 random tracks 0.2 are expected close enough to one to go the other way; 3 are allowed."""
import numpy as np
import pytest

import multiq_workbench_gb300 as mq
from oracle import mqtandem as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("region", [0, 10, 5])
def test_mixed_routing_is_the_oracles(tandem_small, region):
    n = 20000
    m = tandem_small(n=n, seed=3, precision=mq.PREC_MIXED)
    d = O.desc_from(m.desc)
    ref = O.inject(d, 3, True, n)
    rng = np.random.default_rng(region)
    if region in (0, 10):
        hi = [m.cube.lo_mm[a] + m.cube_h * (m.cube.dims[a] - 1) for a in range(3)]
        lo = list(m.cube.lo_mm)
        scale = 1e-3
    else:
        f = m.desc.port[region - 1]
        lo = [-0.3 * f.h] * 3
        hi = [(f.dims[a] - 0.7) * f.h for a in range(3)]
        scale = 1.0
    cnt = np.zeros((9, O.NC), np.uint32)
    for t in (m.tracks, ref):
        t.region[:] = region
        t.last[:] = np.arange(n) % 10 - 1
    for a, k in enumerate("xyz"):
        x = (lo[a] + (hi[a] - lo[a]) * rng.random(n)) * scale
        for t in (m.tracks, ref):
            getattr(t, k)[:] = x
            getattr(t, "v" + k)[:] = 0.0
    m.advance(1)
    O.advance(d, ref, 0, 1, counts=cnt)
    off = int((m.tracks.region != ref.region).sum())
    assert off <= 3 and int(np.abs(m.counts_array().astype(np.int64) - cnt).sum()) <= 3 * off
    assert len(np.unique(ref.region)) >= (3 if region in (0, 10) else 2)
    m.close()
