"""Device set-up against the host's, bit for bit, where its splits end: rows that are no multiple of a
warp, one level only, a coarsest level too large for shared memory, more planes than a grid axis has
blocks, values at the ends of the range; and every channel basis formed on the device."""
import ctypes as C

import numpy as np
import pytest

import multiq_workbench_gb300 as mq
from multiq_workbench_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _both(dims, mask, fixed, outer, tol):
    out = []
    for device in (None, 0):
        phi = np.zeros(mask.size)
        st = N.mq_solve_stats()
        if device is None:
            rc = N.lib().mq_laplace_solve(*dims, mask.ctypes.data, fixed.ctypes.data, outer, tol, 0, phi.ctypes.data, C.byref(st))
        else:
            rc = N.lib().mq_laplace_solve_device(*dims, mask.ctypes.data, fixed.ctypes.data, outer, tol, device, phi.ctypes.data,
                                                 C.byref(st))
        out.append((rc, st.iterations, st.converged, st.final_residual, phi.view(np.uint64)))
    return out


@pytest.mark.parametrize("dims, scale", [((3, 3, 3), 1.0), ((4, 5, 6), 1.0), ((5, 6, 7), -3.0), ((33, 34, 35), 1.0), ((65, 31, 18), 7.0),
                                         ((32, 16, 64), 1e-150), ((97, 12, 9), 1e-306), ((40, 20, 21), 1e140), ((4, 40, 40), 1.0),
                                         ((3, 3, 65600), 1.0)])
def test_any_size_bitwise(built, dims, scale):
    rng = np.random.default_rng(dims[0] * 1000 + dims[2])
    n = dims[0] * dims[1] * dims[2]
    mask = (rng.random(n) < 0.04).astype(np.uint8)
    fixed = np.where(mask, scale * rng.uniform(-1, 1, n), 0.0)
    fixed[(mask != 0) & (rng.random(n) < 0.1)] = -0.0
    host, dev = _both(dims, mask, fixed, 0.25 * scale, 1e-8)
    assert host[:4] == dev[:4] and np.array_equal(host[4], dev[4])


@pytest.mark.parametrize("kw", [dict(h_mm=0.5, n_xy=33), dict(h_mm=0.4, n_xy=41, tilt_mode=1, ac_mode=1),
                                dict(h_mm=0.4, n_xy=40, tilt_mode=2, q2_flare_bug=0, grow=0.5)])
def test_channel_bases_formed_on_the_device(built, kw):
    g = mq.Geom().native()
    for k, v in kw.items():
        setattr(g, k, v)
    d = (C.c_int32 * 3)()
    assert N.lib().mq_geom_dims(C.byref(g), d) == 0
    n = d[0] * d[1] * d[2]
    for basis in range(6):
        got = []
        for device in (-1, 0):
            e4, phi, st = np.zeros(4 * n, np.float32), np.zeros(n), N.mq_solve_stats()
            rc = N.lib().mq_channel_basis_ex(C.byref(g), basis, 1e-7, 0, device, e4.ctypes.data, phi.ctypes.data, C.byref(st))
            got.append((rc, st.iterations, e4.view(np.uint32), phi.view(np.uint64)))
        assert got[0][:2] == got[1][:2]
        assert np.array_equal(got[0][2], got[1][2]) and np.array_equal(got[0][3], got[1][3])
