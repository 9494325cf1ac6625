"""Resident steps of the grids that need the long runs: E and H share one
exchange array, z-CPML psi has slots for the CPML planes alone, and the pole
update is staged through shared memory. Against the split kernels as in
test_resident.py: FP64 bit-identical, FP32 within rounding. Scenes: near the
capacity with and without poles, odd sizes, CPML that ends within a run, and
more poles than a staged trip carries (also in the short runs)."""
import numpy as np
import pytest

from aether_b200 import _abi as A
from aether_b200 import configs as CF
from test_resident import run

pytestmark = pytest.mark.gpu
NM = 1e-9


def sphere(nx, ny, nz, pml, r, material=None):
    def build(precision):
        sc = CF.sphere_scene(nx=nx, ny=ny, nz_total=nz, pml=pml, radius=r * NM, nsteps=200, nl=5, sensor_gap=4,
                             precision=precision)
        if material is not None:
            sc.materials[1] = material()
        return sc
    return build


def seven_poles():
    return A.material_desc(1.1, drude=[(1.3e16, 1.1e14)], debye=[(0.3, 2e-15)], lorentz=[(0.2, 3.0e15, 1.0e14)],
                           critpoint=[(0.9, 4.0e15, -0.8, 1.1e15), (1.3, 5.6e15, -0.5, 1.9e15),
                                      (0.1, 5.0e15, -0.3, 0.9e15), (0.2, 6.6e15, -0.1, 1.2e15)])


def slab(nx, ny, nz, pml):
    return lambda precision: CF.slab_scene(nx=nx, ny=ny, nz_total=nz, pml=pml, nl=5, nsteps=200, sensor_gap=4,
                                           precision=precision)


FP64 = {"slab": slab(64, 64, 128, 16), "slab_odd": slab(61, 59, 131, 11), "sphere": sphere(50, 44, 150, 9, 15),
        "sphere_odd": sphere(55, 53, 121, 13, 13), "seven_poles": sphere(51, 47, 150, 9, 10, seven_poles),
        "seven_poles_short": sphere(24, 20, 90, 9, 20, seven_poles)}
FP32 = {"slab": slab(64, 64, 250, 8), "sphere": sphere(64, 61, 150, 9, 20), "sphere_long": sphere(60, 60, 200, 16, 20),
        "seven_poles": sphere(63, 57, 151, 9, 15, seven_poles)}


@pytest.mark.parametrize("name", sorted(FP64))
def test_fp64_bit_identical_to_the_split_kernels(name):
    chunks = (64, 37, 1, 30)
    scene = FP64[name](precision=A.FP64)
    a, b = run(scene, True, chunks), run(scene, False, chunks)
    assert a["launches"] < b["launches"] / 8
    assert np.abs(b["fields"]).max() > 0
    assert np.array_equal(a["fields"], b["fields"])
    assert np.array_equal(a["sums"], b["sums"])
    for key in ("dft", "flux"):
        for x, y in zip(a[key], b[key]):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("name", sorted(FP32))
def test_fp32_agrees_with_the_split_kernels(name):
    # 130 steps: about one rounding (6e-8) per value and step, below 1e-5 of the norm
    chunks = (64, 66)
    scene = FP32[name](precision=A.FP32)
    a, b = run(scene, True, chunks), run(scene, False, chunks)
    assert a["launches"] < b["launches"] / 8
    assert np.linalg.norm(a["fields"] - b["fields"]) <= 1e-5 * np.linalg.norm(b["fields"])
    for x, y in zip(a["flux"], b["flux"]):
        assert np.linalg.norm(x - y) <= 1e-4 * np.linalg.norm(y)
