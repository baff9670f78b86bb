"""The FP64 matvec on leaves of odd sizes, few and many leaves, and both directions."""
import numpy as np
import pytest

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,nx,factor", [(32, 33, 2.0), (64, 25, 2.0), (85, 21, 2.0), (129, 9, 2.0),
                                            (256, 30, 2.0), (256, 5, 2.0), (32, 20, 1e6)])
def test_fp64_matvec_matches_oracle(oracle_lib, gpu_lib, leaf, nx, factor):
    """A column per lane, per 2, 4 and 8 lanes; rows that do not divide the CTA; leaves over 1 to 8 CTAs;
    no low-rank part (factor 1e6): pressures against the oracle's H-matrix solves at the same tolerances. The
    blocks agree to the ACA tolerance of 1e-8 and the solves to 1e-10."""
    R = meshes.relief(0.6, 0.6, 0.05, nx, 3, nx - 2, 0, meshes.smooth_heightmap(16, 5))
    Ls = meshes.semicircle(5.0, 37)
    f, d = 1500.0, np.array([0.0, -1.0, 0.0])
    bem = DiffBEM(leaf, factor, [f], 1, 1e-8, 1e-8, 1e-10, precision="fp64", incident=("plane", d))
    bem.silent = True
    bem.set_mesh(R.Ps, R.Es)
    m = oracle_lib.Mesh(R.Ps, R.Es, leaf, factor)
    k = oracle_lib.wavenumber(f)
    yo, _, _ = oracle_lib.solve_pressures(m, k, d, 1, Ls, 1e-8, 1e-8, 1e-10, listener="dense")
    for method in ("gmres", "bicgstab"):
        bem.set_krylov(method)
        y = bem.pvals(f, Ls)
        assert np.linalg.norm(y - yo) / np.linalg.norm(yo) < 1e-6


@pytest.mark.parametrize("leaf", [7, 40, 100, 200])
def test_fp64_transposed_matvec_matches_oracle(oracle_lib, gpu_lib, leaf):
    """The adjoint solve (segments and near copy of the transpose) at the same kinds of leaf: the
    coefficient's derivative against the oracle's, both at an ACA tolerance of 1e-8."""
    R = meshes.relief(0.3, 0.3, 0.05, 10, 2, 10, 0, meshes.smooth_heightmap(16, 2))
    kw = dict(cluster_size=leaf, radius_factor=1.5, freq_bands=[2000.0], n_freqs=1, approx_ACA_tol=1e-8,
              Q_ACA_tol=1e-8, solver_tol=1e-10, src_pt=(0.0, 100.0, 0.0), listener_radius=50, listener_ds=15)
    gpu = DiffBEM(**kw, precision="fp64", listener="dense")
    gpu.silent = True
    orc = oracle_lib.OracleDiffBEM(**kw)
    gpu.precompute(R.Ps, R.Es, R.diff_pts)
    orc.precompute(R.Ps, R.Es, R.diff_pts)
    x = np.random.default_rng(leaf).uniform(0, 0.02, size=len(R.diff_pts))
    cg, gg = gpu.gradient(x)
    co, go = orc.gradient(x)
    assert abs(cg - co) < 1e-6
    assert np.linalg.norm(gg - go) / np.linalg.norm(go) < 1e-4
