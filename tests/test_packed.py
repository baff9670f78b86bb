"""The packed double-float arithmetic of the assembly and the ACA groups built on it."""
import ctypes

import numpy as np
import pytest

from acoustic_reliefs_gb300 import _lib as L
from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", [0, 1, 2])
def test_packed_arithmetic_is_the_scalar_bits(gpu_lib, op):
    bad = ctypes.c_longlong(-1)
    assert L.lib().ac3d_packed_selftest(op, ctypes.byref(bad)) == L.OK
    assert bad.value == 0


@pytest.mark.parametrize("leaf,nx", [(8, 13), (32, 33), (61, 31), (128, 26), (256, 30)])
def test_aca_groups_match_oracle(oracle_lib, gpu_lib, leaf, nx):
    """Admissible blocks of odd sides in each of the groups (sides up to 64, 128, 256 and above; with
    larger leaves only the larger ones) against the oracle: its stored ranks, but for a block where
    two pivot candidates agree to the entries' 1e-13 (on the box's regular faces), and its pressures
    to the ACA tolerance."""
    R = meshes.relief(0.6, 0.6, 0.05, nx, 3, nx - 2, 0, meshes.smooth_heightmap(16, 5))
    Ls = meshes.semicircle(5.0, 37)
    f, d = 1500.0, np.array([0.0, -1.0, 0.0])
    bem = DiffBEM(leaf, 2.0, [f], 1, 1e-4, 1e-4, 1e-9, precision="mixed", incident=("plane", d))
    bem.silent = True
    bem.set_krylov("gmres")
    bem.set_mesh(R.Ps, R.Es)
    y = bem.pvals(f, Ls)
    m = oracle_lib.Mesh(R.Ps, R.Es, leaf, 2.0)
    k = oracle_lib.wavenumber(f)
    H = oracle_lib.HMat(m, k, 1e-4)
    differ = np.sum(bem.ranks() != H.stored_ranks())
    assert differ <= 1 + len(H.ranks) // 1000
    yo, _, _ = oracle_lib.solve_pressures(m, k, d, 1, Ls, 1e-4, 1e-4, 1e-9, listener="dense")
    assert np.linalg.norm(y - yo) / np.linalg.norm(yo) < 1e-4
