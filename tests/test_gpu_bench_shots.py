"""bench.py's batched-shot line names what its autotuner chose: two shots that
both run the point kernels report CTAs per SM (3 to 8) as the launch shape, and
no z-chunk, which no kernel of theirs has."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_shape_of_the_shots_line(wql3d_lib):
    r = subprocess.run([sys.executable, "bench.py", "--workload", "shots", "--nshots", "2", "--steps", "4", "--warmup",
                        "3", "--no-cpu"], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    b = line["batched"]
    assert "zchunk" not in b
    assert set(b["tuning_ms_per_step"]) == {"3", "4", "5", "6", "7", "8"} and str(b["launch_shape"]) in b["tuning_ms_per_step"]
    assert "CTAs per SM" in b["what"]
