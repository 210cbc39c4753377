"""No gather, queue, hand-over or node-list index out of range in the kernels that only long calls reach
(tests/check_workloads_long.py on the bounds-checked build)."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


def test_long_calls_stay_in_range(built):
    from multiq_workbench_gb300 import build as B
    env = dict(os.environ, MQ_LIB=str(B.build(check=True)))
    r = subprocess.run([sys.executable, str(HERE / "check_workloads_long.py")], env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    rec = json.loads(r.stdout.strip().splitlines()[-1])
    for part in ("solve", "channel", "tandem"):
        assert rec[part]["enabled"] == 1 and rec[part]["hits"] == 0, (part, rec[part])
    assert rec["loads"] > 0
