"""The FP64 transposed matvec's sums stay in one order whatever kernel forms them, so that an adjoint BiCGSTAB
solve ends on the same iterate."""
import os

import numpy as np
import pytest

from acoustic_reliefs_gb300.acoustics3d import DiffBEM

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "fp64_adjoint.npz")


@pytest.mark.gpu
@pytest.mark.parametrize("i", range(5))
def test_adjoint_iterates(gpu_lib, i):
    """Gradients of 768 to 1280 triangles at 2.5 to 4 kHz in leaves of up to 16, 32, 47, 100 and 200, solved to
    1e-3 in 63 to 247 BiCGSTAB iterations both ways: to rounding (1e-9) those that the FP32 layout's passes gave in
    FP64 (csrc/matvec.cu, before csrc/matvec64.cu took their place). Another order of the near field's sums
    ends up to 7e-4 away."""
    g = np.load(GOLDEN)
    leaf, f, factor = g[f"par{i}"]
    bem = DiffBEM(int(leaf), factor, [f], 1, 1e-5, 1e-5, 1e-3, (0.0, 50.0, 1.0), 10, 4, precision="fp64")
    bem.silent = True
    bem.set_krylov("bicgstab")
    bem.precompute(g[f"Ps{i}"], g[f"Es{i}"], g[f"diff{i}"])
    c, grad = bem.gradient(g[f"x{i}"])
    want = g[f"g{i}"]
    assert abs(c - g[f"c{i}"]) < 1e-9
    assert np.linalg.norm(grad - want) < 1e-9 * np.linalg.norm(want)
