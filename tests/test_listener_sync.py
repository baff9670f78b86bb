"""The receiver ACA is enqueued like the other parts of a call: the host does not wait for it by itself."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import os, sys
import numpy as np, torch
from torch.profiler import ProfilerActivity, profile
from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM
R = meshes.relief(0.6, 0.6, 0.05, 16, 3, 14, 0, meshes.smooth_heightmap(16, 5))
Ls = meshes.semicircle(5.0, 37)
for listener in ("dense", "aca"):
    bem = DiffBEM(32, 2.0, [1000.0], 1, 1e-4, 1e-4, 1e-6, precision="mixed", listener=listener)
    bem.silent = True
    bem.set_krylov("gmres")
    bem.set_mesh(R.Ps, R.Es)
    bem.pvals(1000.0, Ls)
    waits = 0
    for _ in range(4):  # a profile can stay empty, the first one does
        if waits == 0:
            with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
                bem.pvals(1000.0, Ls)
                torch.cuda.synchronize()
            waits = sum(e.name == "cudaStreamSynchronize" for e in p.events())
    print("waits", listener, waits, bem.stats()["iterations"])
sys.stdout.flush()
os._exit(0)
"""


@pytest.mark.gpu
def test_receiver_aca_adds_no_wait(gpu_lib):
    """As many stream synchronisations in a call with the receivers by ACA as with the exact ones. A process
    of its own: the profiler stays attached to it."""
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    rows = [ln.split() for ln in r.stdout.splitlines() if ln.startswith("waits ")]
    assert len(rows) == 2, r.stdout + r.stderr
    dense, aca = (int(x[2]) for x in rows)
    assert rows[0][3] == rows[1][3] and dense > 0
    assert aca == dense
