"""A fill of the tensor-memory kernel that never comes: its waits run out, the
kernel ends soon after, reports it in its status, writes nothing that it summed
from what was not there, and the next call is right again.  In the index-checked
build, which can leave out a fill; a child process (tests/_lost_fill_run.py)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lost_fill(cuda):
    lib = os.path.join(ROOT, "beampower_b200", "lib", "libbeampower_b200_checked.so")
    assert os.path.exists(lib), "build it with: python -m beampower_b200.build --checked"
    env = dict(os.environ, BEAMPOWER_B200_LIBRARY=lib)
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "_lost_fill_run.py")],
                       env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "LOST FILL OK" in r.stdout
