"""The mixed engine's launch shape: what a caller sets is what runs, and an engine that was given no blocks
per SM keeps choosing them itself whatever else is set. Results do not depend on it."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent))
from test_gpu_parity import FIELDS, _mq, _variants  # noqa: E402

pytestmark = pytest.mark.gpu

DC = [0.0, 5.0, -5.0, 0.0]
LONG = 2048 * 152 + 1   # ions above which the engine's own choice for wide records is four


def _jobs(n, k=1):
    mq = _mq()
    return [mq.Job(mq.Species(499.0, 1.0, 2.95 * 499.0 ** (2 / 3)), mq.RfAc(100.0, 500e3, 0.5, 100e3), n, 5 + s) for s in range(k)]


@pytest.mark.parametrize("name, narrow", [("half_kick_gauss", 2), ("legacy_coll_trilinear", 3)])
def test_given_blocks_run_and_the_engines_choice_stays(coarse, name, narrow):
    mq = _mq()
    ph = _variants()[name]
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        def runs(*ions):
            return [e.blocks_per_sm(n, ph) for n in ions]
        assert runs(1000, 60000, LONG) == [0, 3, 4]
        e.set_tuning(chunk=301, use_graph=False)
        assert e.tuning()["blocks_per_sm"] == 3 and runs(LONG) == [4]
        e.set_tuning(wide_records=False)          # what fits of the narrow kernel
        assert runs(256 * 152, 60000, LONG) == [2, narrow, narrow]
        for wide, most in ((False, narrow), (True, 3)):
            for b in (1, 2, 3):
                e.set_tuning(blocks_per_sm=b, wide_records=wide)
                assert e.tuning()["blocks_per_sm"] == b
                e.set_tuning(chunk=400)
                assert runs(60000, LONG) == [min(b, most)] * 2, (wide, b)
        assert e.blocks_per_sm(60000, _variants()["legacy_all"]) > 3   # nearest-node fields: as many as fit
        for b in (0, 4, 9, -1):
            with pytest.raises(mq.MqError):
                e.set_tuning(blocks_per_sm=b)
    with mq.Engine(coarse, mq.PREC_F64) as e, pytest.raises(mq.MqError):
        e.blocks_per_sm(1000)


@pytest.mark.parametrize("name", ["half_kick_gauss", "legacy_coll_trilinear"])
def test_any_shape_gives_the_same_ions(coarse, name):
    mq = _mq()
    ph = _variants()[name]
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        want, _ = e.run_batch_ions(_jobs(LONG), DC, ph)
        rate = {}
        for wide in (True, False):
            for b in (1, 2, 3):
                e.set_tuning(blocks_per_sm=b, wide_records=wide)
                got, _ = e.run_batch_ions(_jobs(LONG), DC, ph)
                rate[wide, b] = e.last_stats.step_kernel_ms
                for f in FIELDS:
                    assert np.array_equal(getattr(want, f).view(np.uint8), getattr(got, f).view(np.uint8)), (wide, b, f)
    # one block of 128 lanes per SM has half the ions in flight that two have, and does show it
    assert rate[True, 1] > 1.15 * rate[True, 2] and rate[False, 1] > 1.15 * rate[False, 2], rate


@pytest.mark.parametrize("n, sample", [(64, 64), (3000, 3000), (48000, 3000)])
def test_autotune_on_few_ions_leaves_what_it_cannot_time(coarse, n, sample):
    """A sample that runs in the lane groups alone says nothing about the other kernel's shape, be it the whole batch
    or the beginning of a long one."""
    mq = _mq()
    ph = _variants()["half_kick_gauss"]
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        e.set_tuning(chunk=12345)
        before = e.tuning()
        t, rate = e.autotune(_jobs(n, 4), DC, ph, sample_per_job=sample)
        assert rate > 0 and {**t, "wide_records": before["wide_records"]} == before
        e.set_tuning(wide_records=True)
        assert e.blocks_per_sm(LONG) == 4


def test_autotune_keeps_no_shape_that_is_slower(built):
    """60,000 ions on the 0.1 mm channel: the L1 prefetch costs a tenth, narrow records more."""
    mq = _mq()
    f = mq.Fields.build(mq.Geom.with_spacing(0.1), bases=[0, 1, 3, 4], cache=False, device=0)
    ph = _variants()["half_kick_gauss"]
    got = []
    for _ in range(4):
        with mq.Engine(f, mq.PREC_MIXED) as e:
            t, _ = e.autotune(_jobs(15000, 4), DC, ph, sample_per_job=15000)
            got.append((t["wide_records"], t["prefetch"]))
    assert got == [(True, False)] * 4, got


def test_the_last_ions_are_handed_over_wherever_they_are(built):
    """58,368 lanes: the queue's last ions of 60,000 fill warps that took nothing else and never come to it again. They go
    on in lane groups like any others: 3,000 steps take little more than with 50,000 ions (kernel times 7.8 and 5.8 ms;
    10.4 where these warps kept them), and give the same states as in short lists."""
    mq = _mq()
    f = mq.Fields.build(mq.Geom.with_spacing(0.1), bases=[0, 1, 3, 4], cache=False, device=0)
    ph = mq.Physics.legacy(0.133322)
    ph.legacy_fields = False
    ph.t_max = 3000 * ph.dt
    with mq.Engine(f, mq.PREC_MIXED) as e:
        ms = {}
        for n in (50000, 60000):
            jobs = [mq.Job(mq.Species(499.0 * 5, 5.0, 0.0), mq.RfAc(100.0, 500e3, 0.5, 100e3), k, 5) for k in (n - 10000, 10000)]
            t = []
            for _ in range(4):
                whole, jid = e.run_batch_ions(jobs, DC, ph)
                t.append(e.last_stats.step_kernel_ms)
            ms[n] = min(t)
            part, _ = e.run_batch_ions(jobs[1:], DC, ph)
            for fld in FIELDS[:-1]:
                assert np.array_equal(getattr(whole, fld)[jid == 1].view(np.uint8), getattr(part, fld).view(np.uint8)), (n, fld)
        assert ms[60000] < 1.55 * ms[50000], ms
