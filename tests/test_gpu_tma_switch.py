"""WQL3D_TMA, read once per process: unset or empty, a separable Cartesian block
runs the point kernel (one launch a stage); a value names how the interior tile
fills its planes, so the block runs the tile beside the shell (two launches)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.abspath(__file__))

RUNNER = r"""
import sys
sys.path.insert(0, sys.argv[1])
from cases import small_case
from waveqlab3d_q_gpu_b200.domain import Domain
g = Domain(small_case(n=(31, 23, 25)), nsteps_hint=4)
before = g.kernel_launches()
g.stage(1)
print("LAUNCHES", g.kernel_launches() - before)
g.close()
"""


@pytest.mark.parametrize("value,launches", [(None, 1), ("", 1), ("0", 2)])
def test_launches_of_a_stage(wql3d_lib, value, launches):
    env = dict(os.environ)
    env.pop("WQL3D_TMA", None)
    if value is not None:
        env["WQL3D_TMA"] = value
    env["PYTHONPATH"] = os.path.dirname(ROOT) + os.pathsep + env.get("PYTHONPATH", "")
    r = subprocess.run([sys.executable, "-c", RUNNER, ROOT], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    assert f"LAUNCHES {launches}" in r.stdout, r.stdout
