"""The FP64 assembly's ACA kernels against the oracle."""
import numpy as np
import pytest

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,nx,L,listener", [(32, 33, 17, "aca"), (64, 25, 300, "aca"), (61, 31, 2, "aca"),
                                                (128, 26, 37, "dense"), (256, 30, 37, "dense")])
def test_fp64_aca_matches_oracle(oracle_lib, gpu_lib, leaf, nx, L, listener):
    """Admissible blocks of odd sides below and above 64, and the receivers' block: the
    oracle's stored ranks, but for a block where two pivot candidates agree to rounding (on the box's
    regular faces), and its pressures to ten times the ACA tolerance."""
    R = meshes.relief(0.6, 0.6, 0.05, nx, 3, nx - 2, 0, meshes.smooth_heightmap(16, 5))
    Ls = meshes.semicircle(5.0, L)
    f, d = 1500.0, np.array([0.0, -1.0, 0.0])
    bem = DiffBEM(leaf, 2.0, [f], 1, 1e-6, 1e-6, 1e-9, precision="fp64", incident=("plane", d), listener=listener)
    bem.silent = True
    bem.set_krylov("gmres")
    bem.set_mesh(R.Ps, R.Es)
    y = bem.pvals(f, Ls)
    m = oracle_lib.Mesh(R.Ps, R.Es, leaf, 2.0)
    k = oracle_lib.wavenumber(f)
    H = oracle_lib.HMat(m, k, 1e-6)
    assert np.sum(bem.ranks() != H.stored_ranks()) <= 1 + len(H.ranks) // 1000
    yo, _, _ = oracle_lib.solve_pressures(m, k, d, 1, Ls, 1e-6, 1e-6, 1e-9, listener=listener)
    assert np.linalg.norm(y - yo) / np.linalg.norm(yo) < 1e-5
