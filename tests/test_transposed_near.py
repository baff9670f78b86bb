"""The near field of the transposed matvec: read from its transposed copy, and in place where the device has
no room for the copy."""
import ctypes

import numpy as np
import pytest

from acoustic_reliefs_gb300 import _lib as L
from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("leaf,factor", [(7, 1.5), (32, 2.0), (61, 2.0), (100, 1.5), (256, 2.0), (50, 1e6)])
def test_copy_and_in_place_agree(gpu_lib, precision, leaf, factor):
    """The same sums in the same order from either: no bit of A^T x differs."""
    R = meshes.relief(0.6, 0.6, 0.05, 14, 3, 12, 0, meshes.smooth_heightmap(16, 5))
    bem = DiffBEM(leaf, factor, [1500.0], 1, 1e-5, 1e-5, 1e-6, precision=precision)
    bem.silent = True
    bem.set_mesh(R.Ps, R.Es)
    bem.pvals(1500.0, meshes.semicircle(5.0, 9))
    bad = ctypes.c_longlong(-1)
    L.check(bem._h, L.lib().ac3d_transposed_selftest(bem._h, ctypes.byref(bad)))
    assert bad.value == 0


@pytest.mark.parametrize("precision,size", [("mixed", 8), ("fp64", 16)])
def test_hmat_bytes_count_the_copy(gpu_lib, precision, size):
    """An adjoint call's H-matrix holds the copy: its near entries (but the forward layout's padding, less
    than a column per row) once more."""
    R = meshes.relief(0.3, 0.3, 0.05, 10, 2, 10, 0, meshes.smooth_heightmap(16, 2))
    bem = DiffBEM(32, 2.0, [1000.0], 1, 1e-4, 1e-4, 1e-6, (0.0, 100.0, 0.0), 50, 15, precision=precision)
    bem.silent = True
    bem.precompute(R.Ps, R.Es, R.diff_pts)
    x = np.zeros(len(R.diff_pts))
    bem.value(x)
    forward = bem.stats()["hmat_bytes"]
    bem.gradient(x)
    st = bem.stats()
    assert st["hmat_bytes"] - forward >= size * (st["near_entries"] - st["n_elements"])
