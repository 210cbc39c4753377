"""The byte counts behind bench.py's rooflines, against counts made by hand."""
from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("steps, chunks", [(0, 0), (1, 1), (256, 1), (1000, 4), (65536, 256), (65537, 257), (200000, 782)])
def test_tandem_state_is_counted_once_per_step_launch(steps, chunks):
    import bench
    launches = 2 + 2 * chunks + -(-steps // 65536)   # load, store; bucket and step kernel; one drive table per 65,536 steps
    st = SimpleNamespace(launches=launches, cell_fills_cube=3, cell_fills_port=5)
    assert bench.tandem_moved(st, 7, steps) == 3 * 256 + 5 * 192 + 7 * bench.TRACK_STATE_BYTES * chunks


@pytest.mark.parametrize("wide, nearest, fill", [(True, False, 384), (False, False, 192), (True, True, 48), (False, True, 48)])
def test_a_fill_counts_what_it_cannot_do_without(wide, nearest, fill):
    import bench
    st = SimpleNamespace(cell_loads=11, ions_queued=2)
    assert bench.stepping_bytes(st, wide, nearest) == 11 * fill + 2 * bench.ION_STATE_BYTES
