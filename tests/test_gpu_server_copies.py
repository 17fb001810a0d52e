"""A server's uploads take the same way whether or not a renderer exists beside it: in a process
that holds nothing but a server, a large scene is copied by the helper threads of a set of
page-locked slots, which go with the server."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import os, sys
sys.path.insert(0, sys.argv[1])
from __graft_entry__ import load_package
rg = load_package()

def helpers():
    return sum(open("/proc/self/task/%s/comm" % t).read().strip() == "rg_copy" for t in os.listdir("/proc/self/task"))

server = rg.RenderServer()
scene = rg.Scene.builtin(4, 1, [400000, 8])  # 14 MB of positions, as much of normals
for _ in range(2):
    job = server.submit(scene, 16, 16, 1)
    server.wait(job)
during = helpers()
server.close()
print(during, helpers())
"""


def test_a_server_alone_uses_the_helpers():
    if len(os.sched_getaffinity(0)) < 4:
        pytest.skip("copies are direct on few cores")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", PROGRAM, root], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    during, after = map(int, out.stdout.split())
    assert during > 0
    assert after == 0
