"""Specialised kernels with one and with two consumer groups forced on every sweep (QSV_JIT_GROUPS13, read once per
process): exact and coarse structures give the interpreter's and the oracle's values. Left alone, the count follows a
sweep's multiply-adds and its warp-shuffle ops."""
import os
import subprocess
import sys

import pytest

from test_gpu_jit import _SWITCH_SCRIPT

pytestmark = pytest.mark.gpu


@pytest.mark.timeout(900)
@pytest.mark.parametrize("groups", ["1", "2"])
def test_forced_group_counts_exact(groups, tmp_path):
    script = tmp_path / "groups.py"
    script.write_text(_SWITCH_SCRIPT)
    r = subprocess.run([sys.executable, str(script), os.path.dirname(os.path.abspath(__file__))],
                       env={**os.environ, "QSV_JIT_GROUPS13": groups}, capture_output=True, text=True, timeout=800)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
