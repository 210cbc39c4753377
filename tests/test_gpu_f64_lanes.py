"""Collisions on most steps on the FP64 engine, legacy ones and those of a dense gas, where long lists go one ion to a
lane: against the CPU oracle, bit for bit, one ion above and below the line (72 live ions per SM and wave of 128 per SM with
legacy collisions, 90 and 80 with the two densities here; 152 SMs), with a second wave, with so many finished ions in the list that the groups take it, and across launches
that change from one kernel to the other."""
import dataclasses
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent))
from test_gpu_parity import _assert_bitequal, _jobs, _mq, _variants  # noqa: E402

pytestmark = pytest.mark.gpu

DC = [0.0, 5.0, -5.0, 0.0]
LINE = 72 * 152


@pytest.mark.parametrize("name, pressure, n, dead", [(p, None, n, d) for p in ("legacy_all", "legacy_coll_trilinear") for n, d in (
    (LINE, 0), (LINE + 1, 0), (LINE + 9, 3), (19457, 2), (2 * LINE + 1, 0))] + [
    (p, pr, n, d) for p, pr, line in (("half_kick_gauss", 5.0, 90), ("half_kick_gauss", 30.0, 80), ("thermal_nearest", 5.0, 90)) for n, d in (
        (line * 152, 0), (line * 152 + 153, 0), (line * 152 + 161, 3), (2 * 152 * (line + 1), 0))])
def test_lanes_equal_oracle(coarse, name, pressure, n, dead):
    mq = _mq()
    from oracle import mqref as R
    ph = _variants()[name]
    if pressure:
        ph = dataclasses.replace(ph, pressure_pa=pressure)
    jobs = _jobs((n + 2) // 3, legacy_species=name.startswith("legacy"))
    ions = mq.inject(coarse, jobs, ph)
    for k, _ in mq.channel.ION_FIELDS:
        setattr(ions, k, np.ascontiguousarray(getattr(ions, k)[:n]))
    lim = 1e-3 * 0.4 * (coarse.nx - 1)
    if dead:
        ions.status[::dead] = 2
    ions.steps[5::11] = ph.max_steps() - 1
    ions.steps[6::11] = ph.max_steps() + 3
    ions.x[8::13] = 0.0
    ions.x[9::13] = lim
    ions.y[10::13] = 0.4e-3 * 7
    ions.z[11::13] = 0.5e-3
    ions.vx[4::9] = -0.0
    ions.leg[7::17] = 1
    ions.leg[8::17] = -5
    g = coarse.geom
    G = R.Grid3(coarse.nx, coarse.ny, coarse.nz, coarse.h, coarse.rf, coarse.ac, coarse.dc_field(DC))
    b = R.batch(ph, jobs[0].drive.v_rf, jobs[0].drive.f_rf, g.axis(), g.layers())
    ref = R.State.from_arrays(ions)
    with mq.Engine(coarse, mq.PREC_F64) as e:
        e.set_dc(DC)
        for more in (61, None):
            st = e.run_ions(jobs, ph, ions, **({} if more is None else {"max_more": more}))
            assert st.ion_steps == R.run(G, b, jobs, ref, **({} if more is None else {"max_more": more}))
            _assert_bitequal(ions, ref, f"{name} n={n}: {more}")
    assert (ions.status != 0).all()


def test_allocation_free_entry_takes_the_same_way(coarse):
    """The same call on device memory of the caller's, whose launches follow the same rule without a hand-over list."""
    from test_zz_no_alloc import _device_call
    mq = _mq()
    ph = _variants()["legacy_all"]
    jobs = _jobs(LINE // 3 + 1, legacy_species=True)
    with mq.Engine(coarse, mq.PREC_F64) as e:
        e.set_dc(DC)
        ions = e.inject(jobs, ph)
        got, steps = _device_call(mq, coarse, DC, ph, jobs, ions, 0xFFFFFFFF)
        assert e.run_ions(jobs, ph, ions).ion_steps == steps
    _assert_bitequal(got, ions, "allocation-free")
