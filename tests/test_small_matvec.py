"""The mixed-precision matvec where several CTAs share a leaf (few leaves), and where none do."""
import numpy as np
import pytest

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,nx,method", [(256, 5, "gmres"), (250, 9, "bicgstab"), (120, 14, "gmres"),
                                            (64, 25, "bicgstab"), (37, 31, "gmres"), (20, 12, "bicgstab"),
                                            (5, 12, "gmres"), (9, 40, "bicgstab")])
def test_shared_leaves_match_oracle(oracle_lib, gpu_lib, leaf, nx, method):
    """Leaves of 2 to 256 elements, from a handful of them to more than four per SM, columns that do not
    divide into the parts: pressures within 1e-4 of the oracle's (FP32 storage, an ACA tolerance of
    1e-5), as the mixed precision's other tests."""
    R = meshes.relief(0.6, 0.6, 0.05, nx, 3, nx - 2, 0, meshes.smooth_heightmap(16, 5))
    Ls = meshes.semicircle(5.0, 37)
    f, d = 1500.0, np.array([0.0, -1.0, 0.0])
    bem = DiffBEM(leaf, 2.0, [f], 1, 1e-5, 1e-5, 1e-9, precision="mixed", incident=("plane", d))
    bem.silent = True
    bem.set_krylov(method)
    bem.set_mesh(R.Ps, R.Es)
    m = oracle_lib.Mesh(R.Ps, R.Es, leaf, 2.0)
    yo, _, _ = oracle_lib.solve_pressures(m, oracle_lib.wavenumber(f), d, 1, Ls, 1e-5, 1e-5, 1e-9, listener="dense")
    y = bem.pvals(f, Ls)
    assert np.linalg.norm(y - yo) / np.linalg.norm(yo) < 1e-4


@pytest.mark.parametrize("leaf,factor", [(7, 1.5), (40, 1.5), (100, 1.5), (200, 1.5), (16, 1e6)])
def test_shared_leaves_transposed_matches_oracle(oracle_lib, gpu_lib, leaf, factor):
    """The adjoint solve on the same kinds of leaf: the coefficient's derivative against the oracle's
    to 1e-3, as the mixed precision's other gradient tests."""
    R = meshes.relief(0.3, 0.3, 0.05, 10, 2, 10, 0, meshes.smooth_heightmap(16, 2))
    kw = dict(cluster_size=leaf, radius_factor=factor, freq_bands=[2000.0], n_freqs=1, approx_ACA_tol=1e-6,
              Q_ACA_tol=1e-6, solver_tol=1e-9, src_pt=(0.0, 100.0, 0.0), listener_radius=50, listener_ds=15)
    gpu = DiffBEM(**kw, precision="mixed", listener="dense")
    gpu.silent = True
    orc = oracle_lib.OracleDiffBEM(**kw)
    gpu.precompute(R.Ps, R.Es, R.diff_pts)
    orc.precompute(R.Ps, R.Es, R.diff_pts)
    x = np.random.default_rng(leaf).uniform(0, 0.02, size=len(R.diff_pts))
    cg, gg = gpu.gradient(x)
    co, go = orc.gradient(x)
    assert abs(cg - co) < 1e-3
    assert np.linalg.norm(gg - go) / np.linalg.norm(go) < 1e-3
