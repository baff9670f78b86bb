"""What a context says about its last H-matrix after another mesh has been set: the H-matrix keeps its
own mesh, so its ranks and timings are those of the mesh it was assembled on."""
import numpy as np
import pytest

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import AC3DError, DiffBEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,other", [(8, 20), (20, 8)])
def test_another_mesh_leaves_the_last_hmatrix_alone(gpu_lib, nx, other):
    A, B = (meshes.relief(0.6, 0.6, 0.05, n, 3, n, 0, meshes.smooth_heightmap(16, 5)) for n in (nx, other))
    Ls = meshes.semicircle(5.0, 9)
    bem = DiffBEM(32, 2.0, [1000.0], 1, 1e-4, 1e-4, 1e-6, precision="mixed")
    bem.silent = True
    bem.set_mesh(A.Ps, A.Es)
    y = bem.pvals(1000.0, Ls)
    _, nbytes = bem.matvec_timing(2)
    _, nbytes_block = bem.block_matvec_timing(8, 2)
    bem.set_mesh(B.Ps, B.Es)
    with pytest.raises(AC3DError, match="admissible blocks"):
        bem.ranks()
    assert bem.matvec_timing(2)[1] == nbytes
    assert bem.matvec_timing(2, transposed=True)[1] == nbytes
    assert bem.block_matvec_timing(8, 2)[1] == nbytes_block
    with pytest.raises(AC3DError, match="admissible blocks"):
        bem.ranks()
    bem.set_mesh(A.Ps, A.Es)  # its block count again: the last H-matrix's ranks
    r = bem.ranks()
    assert r.min() >= 0 and 0 < r.max() < 32
    assert np.array_equal(bem.pvals(1000.0, Ls), y)
    assert np.array_equal(bem.ranks(), r)
