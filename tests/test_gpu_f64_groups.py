"""The FP64 step kernel's lane groups against the CPU oracle, bit for bit, at the sizes where their
choice and their queue can go wrong: one ion, an odd few, one below and above the largest call that 16-lane
groups take alone (8 ions per SM; 152 SMs), and a call that starts in 4-lane groups, refills them
and hands its last ions over. Each for thermal and for legacy collisions, trilinear and
nearest-node fields, with ions that are already finished, that are about to time out or past it, that
stand on the box faces or planes, and velocities of negative zero; in two parts, the first of which
ends in the middle of most flights."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent))
from test_gpu_parity import _assert_bitequal, _jobs, _mq, _variants  # noqa: E402

pytestmark = pytest.mark.gpu

DC = [0.0, 5.0, -5.0, 0.0]


@pytest.mark.parametrize("n", [1, 33, 1215, 1217, 13001])
@pytest.mark.parametrize("name", ["half_kick_gauss", "legacy_all", "thermal_nearest", "legacy_coll_trilinear"])
def test_groups_equal_oracle(coarse, name, n):
    mq = _mq()
    from oracle import mqref as R
    ph = _variants()[name]
    jobs = _jobs((n + 2) // 3, legacy_species=name.startswith("legacy"))
    ions = mq.inject(coarse, jobs, ph)
    for k, _ in mq.channel.ION_FIELDS:
        setattr(ions, k, np.ascontiguousarray(getattr(ions, k)[:n]))
    if n > 1:
        lim = 1e-3 * 0.4 * (coarse.nx - 1)
        ions.status[3::7] = 2
        ions.steps[5::11] = ph.max_steps() - 1
        ions.steps[6::11] = ph.max_steps() + 3
        ions.x[8::13] = 0.0
        ions.x[9::13] = lim
        ions.y[10::13] = 0.4e-3 * 7
        ions.z[11::13] = 0.5e-3
        ions.vx[4::9] = -0.0
        ions.vy[4::9] = -0.0
    g = coarse.geom
    G = R.Grid3(coarse.nx, coarse.ny, coarse.nz, coarse.h, coarse.rf, coarse.ac, coarse.dc_field(DC))
    b = R.batch(ph, jobs[0].drive.v_rf, jobs[0].drive.f_rf, g.axis(), g.layers())
    ref = R.State.from_arrays(ions)
    with mq.Engine(coarse, mq.PREC_F64) as e:
        e.set_dc(DC)
        st = e.run_ions(jobs, ph, ions, max_more=61)
        assert st.ion_steps == R.run(G, b, jobs, ref, max_more=61)
        _assert_bitequal(ions, ref, f"{name} n={n}: first 61 steps")
        st = e.run_ions(jobs, ph, ions)
        assert st.ion_steps == R.run(G, b, jobs, ref)
    _assert_bitequal(ions, ref, f"{name} n={n}: to completion")
    assert (ions.status != 0).all()


@pytest.mark.parametrize("mouth", [True, False])
@pytest.mark.parametrize("n", [1, 17, 1216, 1217, 5003])
def test_tandem_groups_equal_oracle(tandem_small, n, mouth):
    """The FP64 tandem kernel at the sizes where its lane groups change width or refill, tracks of every
    region side by side (a first advance spreads them; some are then set lost), in two advances."""
    from oracle import mqtandem as O
    m = tandem_small(n=n, seed=77, mouth_start=mouth)
    d = O.desc_from(m.desc)
    ref = O.inject(d, 77, mouth, n)
    cnt = np.zeros((9, O.NC), np.uint32)
    for s0, k in ((0, 2999), (2999, 1)):
        m.advance(k)
        O.advance(d, ref, s0, k, counts=cnt)
        if n > 1:
            m.tracks.region[3::17] = 11
            ref.region[3::17] = 11
    for k, _ in O.TRACK_FIELDS:
        a, b = getattr(m.tracks, k), getattr(ref, k)
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), k
    assert np.array_equal(m.counts_array(), cnt)
    m.close()
