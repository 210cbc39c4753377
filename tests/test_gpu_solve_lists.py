"""The device solver without lists of free nodes, as it runs on grids of 2^32 nodes and more (the lists hold 32-bit
numbers), on small grids: the same potential, bit for bit, as with them and as the host's."""
import ctypes as C

import numpy as np
import pytest

from multiq_workbench_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 5, 6), (33, 34, 35), (65, 31, 18), (97, 12, 9), (4, 40, 40), (3, 3, 65600), (80, 81, 60)])
def test_without_lists_bitwise(built, dims):
    L = N.lib()
    f = L.mq_laplace_solve_device_lists
    f.restype = C.c_int32
    f.argtypes = [C.c_int32] * 3 + [C.c_void_p] * 2 + [C.c_double] * 2 + [C.c_int32] * 2 + [C.c_void_p] * 2
    rng = np.random.default_rng(dims[0] * 1000 + dims[2])
    n = dims[0] * dims[1] * dims[2]
    mask = (rng.random(n) < 0.04).astype(np.uint8)
    fixed = np.where(mask, rng.uniform(-1, 1, n), 0.0)
    fixed[(mask != 0) & (rng.random(n) < 0.1)] = -0.0
    got = []
    for lists in (0, 1, None):
        phi, st = np.zeros(n), N.mq_solve_stats()
        if lists is None:
            rc = L.mq_laplace_solve(*dims, mask.ctypes.data, fixed.ctypes.data, 0.25, 1e-8, 0, phi.ctypes.data, C.byref(st))
        else:
            rc = f(*dims, mask.ctypes.data, fixed.ctypes.data, 0.25, 1e-8, 0, lists, phi.ctypes.data, C.byref(st))
        got.append((rc, st.iterations, st.converged, st.final_residual, phi.view(np.uint64)))
    for g in got[:2]:
        assert g[:4] == got[2][:4] and np.array_equal(g[4], got[2][4])
