"""The receiver ACA with more than a million receivers, where a bit per row takes most of the shared memory:
calls that had been taken before the entries' items were kept there as well."""
import numpy as np
import pytest

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import AC3DError, DiffBEM

pytestmark = pytest.mark.gpu


def _bem(Ps, Es, listener):
    bem = DiffBEM(32, 2.0, [300.0], 1, 1e-6, 1e-6, 1e-9, precision="mixed", incident=("plane", (0.0, -1.0, 0.0)),
                  listener=listener)
    bem.silent = True
    bem.set_mesh(Ps, Es)
    return bem


# by one CTA; over the GPU with half of the entries at a time; with all of them
@pytest.mark.parametrize("case,L", [("sphere80", 1612000), ("relief164", 1585000), ("relief1120", 1250000)])
def test_receiver_aca_of_many_receivers(gpu_lib, case, L):
    """Against the exact receiver product on the same solution: the ACA tolerance is 1e-6, ten times that in
    the relative L2 norm."""
    if case == "sphere80":
        Ps, Es = meshes.icosphere(1, 0.2)
    else:
        R = meshes.relief(0.6, 0.6, 0.05, *((6, 1, 5) if case == "relief164" else (14, 3, 14)), 0,
                          meshes.smooth_heightmap(16, 5))
        Ps, Es = R.Ps, R.Es
    Ls = meshes.semicircle(5.0, L)
    y, yd = (_bem(Ps, Es, m).pvals(300.0, Ls) for m in ("aca", "dense"))
    assert np.linalg.norm(y - yd) / np.linalg.norm(yd) < 1e-5


def test_too_many_receivers_are_refused(gpu_lib):
    Ps, Es = meshes.icosphere(1, 0.2)
    with pytest.raises(AC3DError, match="receiver ACA too large"):
        _bem(Ps, Es, "aca").pvals(300.0, meshes.semicircle(5.0, 1640000))
