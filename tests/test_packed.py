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


@pytest.mark.parametrize("nx,L", [(4, 17), (5, 2), (9, 3), (9, 181), (23, 700), (40, 37)])
def test_receiver_aca_matches_oracle(oracle_lib, gpu_lib, nx, L):
    """The receiver ACA by one CTA (128 panels) and over the GPU (ranges of columns and rows that do
    not divide evenly, fewer receivers than CTAs): the oracle's receiver ACA product."""
    R = meshes.relief(0.6, 0.6, 0.05, nx, 2, nx, 0, meshes.smooth_heightmap(16, 5))
    Ls = meshes.semicircle(5.0, L) + np.random.default_rng(L).uniform(-0.2, 0.2, size=(L, 3))
    f, d = 1200.0, np.array([0.2, -1.0, 0.1]) / np.linalg.norm([0.2, -1.0, 0.1])
    bem = DiffBEM(32, 2.0, [f], 1, 1e-6, 1e-5, 1e-9, precision="mixed", incident=("plane", d), listener="aca")
    bem.silent = True
    bem.set_krylov("gmres")
    bem.set_mesh(R.Ps, R.Es)
    y = bem.pvals(f, Ls)
    m = oracle_lib.Mesh(R.Ps, R.Es, 32, 2.0)
    yo, _, _ = oracle_lib.solve_pressures(m, oracle_lib.wavenumber(f), d, 1, Ls, 1e-6, 1e-5, 1e-9, listener="aca")
    assert np.linalg.norm(y - yo) / np.linalg.norm(yo) < 1e-4
