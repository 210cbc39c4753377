"""Workloads for the bounds-checked build that are long enough to leave the lane groups: more ions than these
hold (so that the one-lane kernel runs, refills, queues ions again and hands its last ones over), more
FP64 ions and tracks than 16-lane groups take alone, both record widths, the L1 prefetch and the cell sort,
states that are NaN, outside the box or on its faces in all of these, and device field solves. Run with MQ_LIB
pointing at libmqgb_check.so (tests/test_gpu_check_long.py does); prints one JSON line with the records."""
import dataclasses
import json
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
sys.path.insert(0, str(Path(__file__).resolve().parent))

import multiq_workbench_gb300 as mq  # noqa: E402
from check_workloads import status  # noqa: E402

DC = [0.0, 5.0, -5.0, 0.0]


def edges(ions, f):
    n = len(ions)
    lim = np.array([(f.nx - 1) * f.h, (f.ny - 1) * f.h, (f.nz - 1) * f.h])
    ions.x[::11] = lim[0]
    ions.y[1::11] = 0.0
    ions.z[2::11] = lim[2] + 1e-3
    ions.x[3::97] = np.nan
    ions.vz[4::97] = np.nan
    ions.y[5::97] = np.inf
    ions.vx[6::97] = -np.inf
    ions.steps[:] = np.arange(n) % 23
    return ions


def main():
    out = {}
    status(reset=1)
    # field solves of two geometries, the second with rows that are no multiple of a warp
    f = mq.Fields.build(mq.Geom.with_spacing(0.4), bases=[0, 1, 2, 3, 4, 5], cache=False, device=0)
    mq.Fields.build(mq.Geom(h_mm=0.5, n_xy=33), cache=False, device=0)
    out["solve"] = status(reset=1)

    base = dict(pressure_pa=0.133322, temp_k=300.0, dt=1e-7, t_max=400e-7)
    variants = [
        mq.Physics(**base, legacy_force=True, launch=mq.LAUNCH_GAUSSIAN, sigma_mm=0.1),
        mq.Physics(True, True, False, True, True, 0.133322, 300.0, 1e-7, 400e-7, 0.0, mq.LAUNCH_LEGACY),
        mq.Physics(True, True, True, True, True, 0.133322, 300.0, 1e-7, 400e-7, 0.0, mq.LAUNCH_LEGACY),
        mq.Physics(**base, legacy_fields=True, legacy_force=True, launch=mq.LAUNCH_GAUSSIAN),
    ]
    jobs = [mq.Job(mq.Species(mz, 1.0, 2.95 * mz ** (2 / 3)), mq.RfAc(100.0, 500e3, 0.5, 100e3 + 1e3 * k), 11000, 30 + k)
            for k, mz in enumerate((493.0, 499.0, 505.0))]
    with mq.Engine(f, mq.PREC_MIXED) as e:
        for wide in (True, False):
            for prefetch, sort, chunk in ((False, False, 20000), (True, False, 53), (False, True, 53)):
                e.set_tuning(wide_records=wide, prefetch=prefetch, sort_cells=sort, chunk=chunk)
                for ph in variants:
                    e.set_dc(DC)
                    e.run_ions(jobs, ph, edges(e.inject(jobs, ph), f))
            e.set_tuning(sort_cells=False)
            e.run_batch([mq.Job(jobs[0].sp, jobs[0].drive, 2048 * 152 + 1, 3)], DC, variants[0])
        out["loads"] = int(e.last_stats.cell_loads)
    with mq.Engine(f, mq.PREC_F64) as e:
        # with legacy collisions and in the dense gas one ion to a lane, else in groups
        short = [mq.Job(j.sp, j.drive, 5000, j.seed) for j in jobs]
        for ph in variants + [dataclasses.replace(variants[0], pressure_pa=5.0)]:
            e.set_dc(DC)
            e.run_ions(short, ph, edges(e.inject(short, ph), f))
    out["channel"] = status(reset=1)

    s14 = mq.Fields.build(mq.Geom.s14(h_mm=0.4, n_xy=40), cache=False)
    for prec in (0, 1):
        m = mq.TandemModel(n=9000, seed=486, mouth_start=True, channel=s14, cube_h=2.0, precision=prec)
        for _ in range(2):
            m.advance(700)
        m.tracks.x[::50] = np.nan
        m.advance(100)
        m.close()
    out["tandem"] = status(reset=1)
    print(json.dumps(out))


if __name__ == "__main__":
    main()
