"""The ACA pool's first size: where the terms fit, the assembly runs once; where they do not, it runs
again with a larger pool and ends on the same bits."""
import numpy as np
import pytest

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM
from tests import cases

pytestmark = pytest.mark.gpu


def _calls(c, freqs, leaf=32, tol=1e-4):
    bem = DiffBEM(leaf, 2.0, [freqs[0]], 1, tol, tol, 1e-6, precision="mixed", incident=("plane", c["vec"]))
    bem.silent = True
    bem.set_krylov("gmres")
    bem.set_mesh(c["Ps"], c["Es"])
    out = []
    for f in freqs:
        y = bem.pvals(f, c["Ls"])
        launches = bem.stats()["kernel_launches"]
        assert launches > 0
        out.append((y, bem.ranks(), launches))
    return out


def _relief(nx):
    R = meshes.relief(0.6, 0.6, 0.05, nx, 3, nx - 2, 0, meshes.smooth_heightmap(16, 5))
    return dict(Ps=R.Ps, Es=R.Es, vec=np.array([0.0, -1.0, 0.0]), Ls=meshes.semicircle(5.0, 37))


@pytest.mark.parametrize("nx,f", [(0, 4500.0), (8, 2000.0), (20, 2000.0), (33, 6000.0)])
def test_terms_that_fit_are_assembled_once(gpu_lib, nx, f):
    """14.6 to 15.2 places of terms per row and column, and the first pool has 16 (nx 0: the 5280-triangle
    relief): a first call launches what a later one launches, whatever places the blocks leave unused."""
    (y0, r0, n0), (y1, r1, n1) = _calls(_relief(nx) if nx else cases.relief_small(), [f, f])
    assert np.array_equal(r0, r1) and np.array_equal(y0, y1)
    assert n0 == n1


def test_overflow_ends_on_the_same_bits(gpu_lib):
    """A tight tolerance (24 places of terms per row and column): the first call's pool is too small, the
    second's is that of the first."""
    (y0, r0, n0), (y1, r1, n1) = _calls(_relief(33), [3000.0, 3000.0], leaf=64, tol=1e-6)
    assert n0 > n1
    assert np.array_equal(r0, r1) and np.array_equal(y0, y1)
