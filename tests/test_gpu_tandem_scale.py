"""The FP64 tandem's electrode test does not depend on the cube's size: its FP32 filter leaves to the exact
test whatever lies as close to a surface as FP32 is off by, which grows with the lengths. The cube as it
is and 65,536 times as large; tracks at rest by the walls of posts, posts' tops and the wall planes, at distances
from 3e-8 to 1e-6 of a pitch, and half way between posts, one step; and the oracle's result bit for bit. Also
with clearance holes so wide that the two posts beside such a point both count."""
import numpy as np
import pytest

import multiq_workbench_gb300 as mq  # noqa: F401
from oracle import mqtandem as O

pytestmark = pytest.mark.gpu

LENGTHS = ("d", "pitch", "height", "t_pcb", "gap", "stem_r", "clear_r", "l_ext", "ap_r", "rod_clear_extra", "cap_gap", "cap_r")


@pytest.mark.parametrize("scale, wider", [(1, 0.0), (65536, 0.0), (1, 1.2)])
@pytest.mark.parametrize("n", [900, 9000])   # 16 lanes a track, and 4
def test_surfaces_of_a_cube_of_any_size(tandem_small, n, scale, wider):
    m = tandem_small(n=n, seed=5)
    g = m.desc.cube
    g.rod_clear_extra += wider
    g.clear_r += wider
    for k in LENGTHS:
        setattr(g, k, getattr(g, k) * scale)
    m.desc.cube_h_mm *= scale
    for a in range(3):
        m.desc.cube_lo_mm[a] *= scale
    rng = np.random.default_rng(n)
    c0 = g.t_pcb + g.gap + g.d / 2
    size = 2 * c0 + (g.n - 1) * g.pitch
    off = g.pitch * 10.0 ** rng.uniform(-7.5, -6, n) * rng.choice([-1.0, 1.0], n)
    top = g.t_pcb + g.gap + g.height
    what = rng.integers(0, 4, n)   # a post's side, its top, the wall plane, between two posts
    r = np.where(what == 0, g.d / 2 + off, g.d * rng.uniform(0, 0.45, n))
    r = np.where(what == 2, g.pitch * rng.uniform(0.4, 0.6, n), r)
    u = np.where(what == 0, rng.uniform(g.t_pcb + g.gap, top, n), np.where(what == 1, top + off, g.t_pcb + off))
    u = np.where((what == 3) & (rng.random(n) < 0.5), rng.uniform(0, 1.1 * top, n), u)
    phi = rng.uniform(0, 2 * np.pi, n)
    pb = c0 + g.pitch * rng.integers(2, g.n - 2, n) + r * np.cos(phi)
    pc = c0 + g.pitch * rng.integers(2, g.n - 2, n) + r * np.sin(phi)
    mid = what == 3   # some of them half way along both axes, as on a port's axis
    pb[mid] = c0 + g.pitch * (rng.integers(1, g.n - 2, n) + 0.5)[mid] + off[mid]
    both = mid & (rng.random(n) < 0.4)
    pc[both] = c0 + g.pitch * (rng.integers(1, g.n - 2, n) + 0.5)[both] + np.roll(off, 1)[both]
    face = rng.integers(0, 6, n)
    face[both & (rng.random(n) < 0.5)] = 3
    p = np.zeros((3, n))
    pa = np.where(face % 2 == 0, u, size - u)
    for a in range(3):
        own = face // 2 == a
        p[a][own] = pa[own]
        p[(a + 1) % 3][own] = pb[own]
        p[(a + 2) % 3][own] = pc[own]
    d = O.desc_from(m.desc)
    ref = O.inject(d, 5, True, n)
    for t in (m.tracks, ref):
        t.region[:] = 0
        t.last[:] = -1
        for a, k in enumerate("xyz"):
            getattr(t, k)[:] = p[a] * 1e-3
            getattr(t, "v" + k)[:] = 0.0
    cnt = np.zeros((9, O.NC), np.uint32)
    m.advance(1)
    O.advance(d, ref, 0, 1, counts=cnt)
    assert 0.1 < float((ref.region == 11).mean()) < 0.9
    for k, _ in O.TRACK_FIELDS:
        a, b = getattr(m.tracks, k), getattr(ref, k)
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), (k, int((a != b).sum()))
    assert np.array_equal(m.counts_array(), cnt)
    m.close()
