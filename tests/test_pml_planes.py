"""x/y-CPML items with two planes at a time (yee.cuh e_pmlx, h_pmlx) against the
general kernels, one plane at a time (AEFDTD_ALL_BOUNDARY): chunks and CPML that
end on either plane of a pair, grids of a few planes, odd rows."""
import numpy as np
import pytest

from aether_b200 import _abi as A
from aether_b200 import configs as CF
from aether_b200 import fdtd

pytestmark = pytest.mark.gpu
NM = 1e-9


@pytest.mark.parametrize("precision", [A.FP64, A.FP32])
@pytest.mark.parametrize("n,pml", [((70, 58, 51), 7), ((41, 39, 23), 4), ((96, 40, 18), 3), ((33, 70, 37), 8)])
def test_planes_in_pairs_equal_the_general_kernels(n, pml, precision, monkeypatch):
    scene = CF.random_spheres_scene(n_total=n, pml=pml, n_dielectric=8, n_lorentz=2, r_range=(10 * NM, 20 * NM),
                                    nsteps=60, nl=3, precision=precision, seed=2)
    monkeypatch.setenv("AEFDTD_RESIDENT", "0")
    got = []
    for general in (False, True):
        if general:
            monkeypatch.setenv("AEFDTD_ALL_BOUNDARY", "1")
        with fdtd.build_simulation(scene) as s:
            s.step(60)
            got.append(s.fields())
    assert np.abs(got[1]).max() > 0
    if precision == A.FP64:
        assert np.array_equal(got[0], got[1])
    else:   # contraction may differ per kernel: about one rounding (6e-8) per value and step
        assert np.linalg.norm(got[0] - got[1]) <= 1e-5 * np.linalg.norm(got[1])
