"""A scene's batch memory is the driver's again when the scene is destroyed, also
what an earlier load of the scene held, and a cleared scene that is loaded again
takes no more.  In a process of its own: the device's pool and its free memory
belong to the whole process."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import numpy as np, torch
from heavyrt_gb300 import SceneRT, workload as wl
free = lambda: torch.cuda.mem_get_info()[0]
meshes = [wl.soup(k, 100000, off=0.01) for k in range(8)]
small = [wl.soup(9, 1000)]
load = lambda s, m: s.add_geoms_batched([v for v, _ in m], [i for _, i in m])
torch.zeros(1).cuda()
s = SceneRT(); load(s, small); s.close()
s = SceneRT()
load(s, meshes)
first = free()
s.ClearGeom(); load(s, meshes); s.ClearGeom(); load(s, small)
again = free()
s.close()
print(first - again, free() - again)
"""


def test_batch_memory_is_given_back(native):
    out = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, check=True, capture_output=True, text=True).stdout
    grown, back = (int(x) for x in out.split())
    held = 800000 * (5 * 4 + 2 * 36 + 64 + 48 + 12 + 48)  # codes, order, runs; nodes, pairs, triangles, indices, vertices
    assert grown <= held // 8
    assert back >= held * 3 // 4
