"""Block solves where the gather pass's tiles, rings and chunks differ: leaves of 2 to 64 elements (one and
two rows per lane), 4, 8 and 16 right-hand sides, no low-rank blocks, both directions, the leaf limit."""
import numpy as np
import pytest

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import AC3DError, DiffBEM
from tests import cases

pytestmark = pytest.mark.gpu


def _dirs(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d[:, 1] = -np.abs(d[:, 1]) - 0.5
    return d / np.linalg.norm(d, axis=1, keepdims=True)


@pytest.mark.parametrize("leaf,nx,factor,nrhs,method", [
    (5, 12, 2.0, 2, "gmres"), (9, 10, 2.0, 16, "bicgstab"), (20, 20, 2.0, 5, "bicgstab"), (37, 22, 2.0, 16, "gmres"),
    (37, 13, 2.0, 3, "bicgstab"), (64, 25, 2.0, 5, "gmres"), (64, 16, 2.0, 16, "bicgstab"), (64, 33, 2.0, 8, "gmres"),
    (50, 12, 1e6, 16, "gmres"), (61, 11, 1e6, 5, "bicgstab"), (32, 6, 1e6, 2, "gmres")])
def test_block_solve_matches_single_solves(gpu_lib, leaf, nx, factor, nrhs, method):
    """Every column within 1e-6 of the single solve of its direction on the same H-matrix, both to a relative
    residual of 1e-9, as the block solves' other tests."""
    R = meshes.relief(0.6, 0.6, 0.05, nx, 3, nx - 2, 0, meshes.smooth_heightmap(16, 5))
    Ls, dirs, f = meshes.semicircle(5.0, 37), _dirs(nrhs, leaf), 1500.0
    bem = DiffBEM(leaf, factor, [f], 1, 1e-5, 1e-5, 1e-9, precision="mixed")
    bem.silent = True
    bem.set_krylov(method)
    bem.set_mesh(R.Ps, R.Es)
    P = bem.pvals_multi(f, dirs, Ls)
    assert bem.stats()["rel_residual"] <= 1e-9
    for i, d in enumerate(dirs):
        bem.set_incident("plane", d)
        assert cases.rel_l2(P[i], bem.pvals(f, Ls)) < 1e-6, i


@pytest.mark.parametrize("leaf,factor,nd", [(7, 1.5, 2), (20, 2.0, 5), (40, 1.5, 9), (64, 2.0, 5), (64, 1e6, 3)])
def test_transposed_block_solve_matches_single_solves(gpu_lib, leaf, factor, nd):
    """The multi-direction gradient's adjoint block solves: the mean of the single directions' gradients
    within 1e-4, as its other tests (solves to 1e-8)."""
    R = meshes.relief(0.3, 0.3, 0.05, 10, 2, 10, 0, meshes.smooth_heightmap(16, 2))
    x, dirs, f = np.random.default_rng(leaf).uniform(0, 0.02, size=len(R.diff_pts)), _dirs(nd, leaf), 2000.0

    def bem(d):
        b = DiffBEM(leaf, factor, [f], 1, 1e-6, 1e-6, 1e-8, precision="mixed", incident=("plane", d))
        b.silent = True
        b.set_krylov("gmres")
        b.set_listeners(meshes.semicircle(10.0, 91))
        b.precompute(R.Ps, R.Es, R.diff_pts)
        return b

    loss, g, _ = bem(dirs[0]).gradient_multi(x, [f], dirs)
    singles = [bem(d).gradient(x) for d in dirs]
    assert abs(loss - (1 - np.mean([c for c, _ in singles]))) < 1e-6
    gref = -np.mean([s for _, s in singles], axis=0)
    assert np.linalg.norm(g - gref) / np.linalg.norm(gref) < 1e-4


@pytest.mark.parametrize("method", ["gmres", "bicgstab"])
def test_more_leaves_than_supported_are_refused(gpu_lib, method):
    """33852 leaves of one triangle (the passes' reduction has room for 32768): refused before a launch."""
    R = meshes.relief(0.6, 0.6, 0.05, 91, 1, 91, 0, meshes.smooth_heightmap(16, 5))
    bem = DiffBEM(1, 0.2, [500.0], 1, 1e-3, 1e-3, 1e-6, precision="mixed")
    bem.silent = True
    bem.set_krylov(method)
    bem.set_mesh(R.Ps, R.Es)
    with pytest.raises(AC3DError, match="32768 leaf clusters"):
        bem.pvals_multi(500.0, _dirs(2, 1), meshes.semicircle(5.0, 9))
