"""The FP64 assembly's pivots on symmetric geometries, where many candidates are equal but for rounding."""
import os

import numpy as np
import pytest

from acoustic_reliefs_gb300.acoustics3d import DiffBEM

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "fp64_pivots.npz")


@pytest.mark.gpu
@pytest.mark.parametrize("i", range(5))
def test_pivots_of_equal_candidates(gpu_lib, i):
    """Spheres of 80 to 1280 panels in leaves of 1 to 32: the ranks and, to rounding (1e-9; other pivots are
    3e-6 to 1.6e-2 away), the surface solutions that the assembly by one warp per block gave
    (csrc/assemble.cu's kernel in FP64, before csrc/aca_f64.cu took its place)."""
    g = np.load(GOLDEN)
    leaf, f, aca = g[f"par{i}"]
    bem = DiffBEM(int(leaf), 2.0, [f], 1, aca, aca, 1e-6, precision="fp64", incident=("plane", (0.3, -1.0, 0.2)))
    bem.silent = True
    bem.set_krylov("gmres")
    bem.set_mesh(g[f"Ps{i}"], g[f"Es{i}"])
    x, want = bem.surface_vals(f), g[f"x{i}"]
    assert np.array_equal(bem.ranks(), g[f"rank{i}"])
    assert np.linalg.norm(x - want) < 1e-9 * np.linalg.norm(want)


@pytest.mark.gpu
@pytest.mark.parametrize("i", range(5))
def test_gmres_solution_keeps_its_bits(gpu_lib, i):
    """The same solutions by GMRES in FP64, bit for bit: the back substitution rounds as in its former shape
    whatever the compiler makes of the present one."""
    g = np.load(GOLDEN)
    leaf, f, aca = g[f"par{i}"]
    bem = DiffBEM(int(leaf), 2.0, [f], 1, aca, aca, 1e-6, precision="fp64", incident=("plane", (0.3, -1.0, 0.2)))
    bem.silent = True
    bem.set_krylov("gmres")
    bem.set_mesh(g[f"Ps{i}"], g[f"Es{i}"])
    assert np.array_equal(bem.surface_vals(f), g[f"x{i}"])
