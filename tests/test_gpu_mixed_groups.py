"""The mixed engine's lane groups: an ion's final state does not depend on which kernel stepped it. A batch
larger than the groups hold (19,456 or, with nearest-node fields, 29,184 ions on 152 SMs) starts in the
one-lane kernel, is spread over its warps unevenly, and hands its last ions to the groups in the
middle of their flights; the same jobs run alone, odd sizes down to one ion, go through the groups
from their first step. Bit for bit the same for every physics, both node record widths, and launches of
37 steps, which re-queue ions at every position of a 16-step block and cut the groups' legs."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent))
from test_gpu_parity import FIELDS, _mq, _variants  # noqa: E402

pytestmark = pytest.mark.gpu

DC = [0.0, 5.0, -5.0, 0.0]
SIZES = (1, 7, 33, 1217, 4865, 23878)   # 30,001 together; the 23,878 alone are also above 19,456


def _jobs(legacy_species):
    mq = _mq()
    out = []
    for k, n in enumerate(SIZES):
        mz = 493.0 + 2 * k
        sp = mq.Species(mz * 5, 5.0, 0.0) if legacy_species else mq.Species(mz, 1.0, 2.95 * mz ** (2 / 3))
        out.append(mq.Job(sp, mq.RfAc(100.0, 500e3, 0.5 if k else 0.0, 100e3 + 1e3 * k), n, 77 + k))
    return out


@pytest.mark.parametrize("wide", [True, False], ids=["wide", "narrow"])
@pytest.mark.parametrize("name", ["corrected_disc", "half_kick_gauss", "legacy_all", "legacy_coll_trilinear", "thermal_nearest",
                                  "no_gas_rf_random"])
def test_groups_equal_one_lane_kernel(coarse, name, wide):
    mq = _mq()
    ph = _variants()[name]
    jobs = _jobs(name.startswith("legacy"))
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        e.set_tuning(wide_records=wide)
        whole, jid = e.run_batch_ions(jobs, DC, ph)
        steps = e.last_stats.ion_steps
        assert steps == int(whole.steps.astype(np.int64).sum())
        assert (whole.status != 0).all()
        alone = [e.run_batch_ions([j], DC, ph)[0] for j in jobs]
        e.set_tuning(chunk=37)
        cut, _ = e.run_batch_ions(jobs[:5], DC, ph)
    for k in range(len(jobs)):
        m = jid == k
        for f in FIELDS[:-1]:
            a, b = getattr(whole, f)[m], getattr(alone[k], f)
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), f"{name}: job {k}, {f}"
    m = jid < 5
    for f in FIELDS:
        assert np.array_equal(getattr(whole, f)[m].view(np.uint8), getattr(cut, f).view(np.uint8)), f"{name}: 37-step launches, {f}"


def test_two_engines_at_once(coarse):
    """Blocks of one batch that start only after others have ended (another engine's kernels hold their SMs):
    no ion is left behind when the last ones are handed over."""
    from concurrent.futures import ThreadPoolExecutor
    mq = _mq()
    ph = _variants()["half_kick_gauss"]
    jobs = [mq.Job(mq.Species(499.0, 1.0, 2.95 * 499.0 ** (2 / 3)), mq.RfAc(100.0, 500e3, 0.5, 100e3), n, 5) for n in (23878, 31000)]
    engines = [mq.Engine(coarse, mq.PREC_MIXED) for _ in jobs]
    try:
        alone = [e.run_batch_ions([j], DC, ph)[0] for e, j in zip(engines, jobs)]
        with ThreadPoolExecutor(2) as pool:
            for _ in range(4):
                both = [f.result()[0] for f in [pool.submit(e.run_batch_ions, [j], DC, ph) for e, j in zip(engines, jobs)]]
                for a, b in zip(alone, both):
                    assert (b.status != 0).all()
                    for f in FIELDS:
                        assert np.array_equal(getattr(a, f).view(np.uint8), getattr(b, f).view(np.uint8)), f
    finally:
        for e in engines:
            e.close()


@pytest.mark.parametrize("wide", [True, False], ids=["wide", "narrow"])
def test_states_at_the_edges_equal_one_lane_kernel(coarse, wide):
    """States a caller can hand in: outside the box, on its faces, at and past the step cap, at every
    residue of the step count; 24,000 of them through the one-lane kernel, and in parts through the groups."""
    mq = _mq()
    ph = _variants()["half_kick_gauss"]
    jobs = [mq.Job(mq.Species(499.0, 1.0, 2.95 * 499.0 ** (2 / 3)), mq.RfAc(100.0, 500e3, 0.5, 100e3), 24000, 9)]
    rng = np.random.default_rng(3)
    cap = int(round(ph.t_max / ph.dt))
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        e.set_dc(DC)
        e.set_tuning(wide_records=wide)
        st = e.inject(jobs, ph)
        h = coarse.h
        for f, n in (("x", coarse.nx), ("y", coarse.ny), ("z", coarse.nz)):
            v = getattr(st, f)
            pick = rng.random(v.size)
            v[:] = np.where(pick < 0.05, h * (n - 1) * rng.choice([-0.01, 0.0, 0.999, 1.0, 1.02], v.size),
                            np.where(pick < 0.1, h * rng.integers(0, n, v.size), v))
        st.steps[:] = rng.integers(0, 64, st.steps.size)
        late = rng.random(st.steps.size) < 0.05
        st.steps[late] = cap + rng.integers(-3, 3, int(late.sum()))

        def run(i0, i1):
            s = mq.IonStates.empty(i1 - i0)
            for f in FIELDS:
                getattr(s, f)[:] = getattr(st, f)[i0:i1]
            e.run_ions(jobs, ph, s, max_more=301)
            return s
        whole = run(0, 24000)
        parts = [run(i, i + 6000) for i in range(0, 24000, 6000)]
    for f in FIELDS:
        b = np.concatenate([getattr(p, f) for p in parts])
        assert np.array_equal(getattr(whole, f).view(np.uint8), b.view(np.uint8)), f


@pytest.mark.parametrize("name", ["corrected_disc", "legacy_coll_trilinear", "no_gas_rf_random"])
def test_long_lists_equal_their_parts(coarse, name):
    """Lists above 2,048 ions per SM run the one-lane kernel at four blocks per SM, shorter ones at three."""
    mq = _mq()
    ph = _variants()[name]
    sp = mq.Species(499.0 * 5, 5.0, 0.0) if name.startswith("legacy") else mq.Species(499.0, 1.0, 2.95 * 499.0 ** (2 / 3))
    jobs = [mq.Job(sp, mq.RfAc(100.0, 500e3, 0.5, 100e3 + 1e3 * k), 110000, 5 + k) for k in range(3)]
    with mq.Engine(coarse, mq.PREC_MIXED) as e:
        e.set_tuning(chunk=301)
        whole, jid = e.run_batch_ions(jobs, DC, ph)
        for k, j in enumerate(jobs):
            part, _ = e.run_batch_ions([j], DC, ph)
            for f in FIELDS[:-1]:
                assert np.array_equal(getattr(whole, f)[jid == k].view(np.uint8), getattr(part, f).view(np.uint8)), f
