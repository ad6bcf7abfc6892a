"""WQL3D_SHELL_OVERLAP=0 keeps a stage on one stream.  A stage of a two-block
domain is captured from the domain's stream and the captured graph's edges are
read: with the side stream the second block's kernels branch off (a node with
two successors), without it every node has one successor.  The switch is read
once per process, so each setting runs in a subprocess."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.abspath(__file__))

RUNNER = r"""
import ctypes as C
import sys
sys.path.insert(0, sys.argv[2])
from cases import two_block_case
from waveqlab3d_q_gpu_b200.domain import Domain
p = two_block_case(mesh=sys.argv[1])
g = Domain(p, nsteps_hint=4)
g.run(2)
g.synchronize()
cu = C.CDLL("libcuda.so.1")
def ck(rc):
    assert rc == 0, rc
s, graph, n = C.c_void_p(g.stream_handle()), C.c_void_p(), C.c_size_t(0)
ck(cu.cuStreamBeginCapture_v2(s, 1))          # thread-local capture mode
g.stage(1)
ck(cu.cuStreamEndCapture(s, C.byref(graph)))
ck(cu.cuGraphGetEdges(graph, None, None, C.byref(n)))
a, b = (C.c_void_p * n.value)(), (C.c_void_p * n.value)()
ck(cu.cuGraphGetEdges(graph, a, b, C.byref(n)))
print("SUCCESSORS", max(list(a).count(x) for x in a))
ck(cu.cuGraphDestroy(graph))
"""


@pytest.mark.parametrize("mesh", ["cartesian", "curvilinear"])
@pytest.mark.parametrize("overlap,successors", [(1, 2), (0, 1)])
def test_second_block_follows_the_overlap_switch(wql3d_lib, mesh, overlap, successors):
    env = dict(os.environ)
    env["WQL3D_SHELL_OVERLAP"] = str(overlap)
    env["PYTHONPATH"] = os.path.dirname(ROOT) + os.pathsep + env.get("PYTHONPATH", "")
    r = subprocess.run([sys.executable, "-c", RUNNER, mesh, ROOT], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    assert f"SUCCESSORS {successors}" in r.stdout, r.stdout
