"""The count of living meshes whose last one gives the scratch back, with meshes in reference cycles that the
collector finds while another mesh is being counted.  In a process of its own: the fault this guards against is a
thread that waits for itself."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import contextlib, gc, sys, threading
sys.path[:0] = [{root!r}, {pkg!r}]
import torch
from xkgpu import device as D

trims = []
D.L.call = lambda name, keep: trims.append((name, keep))
torch.cuda.device = lambda index: contextlib.nullcontext()

class Mesh:
    device = torch.device("cuda", 3)
    def __init__(self):
        self.me = self
        D._count_mesh(self)

gc.collect()
gc.set_threshold(3)
def work():
    for _ in range(20000):
        Mesh()
threads = [threading.Thread(target=work) for _ in range(3)]
kept = Mesh()
for t in threads:
    t.start()
work()
for t in threads:
    t.join()
gc.collect()
assert not trims, len(trims)  # one mesh was alive throughout
del kept
gc.collect()
assert trims == [("xk_scratch_trim", 0)], trims
print("counted")
"""


def test_meshes_in_cycles_are_counted():
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(ROOT), pkg=str(ROOT / "xkep-cae_gb300"))],
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "counted" in r.stdout, r.stderr[-3000:]
