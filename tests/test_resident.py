"""Resident time steps (resident.cuh): a grid that fits the SMs' shared memory
is advanced by one cooperative launch per chunk of steps. FP64 fields, plane
sums and sensor samples are bit-identical to the split half-step kernels
(AEFDTD_RESIDENT=0), which the other tests hold to the reference; FP32 agrees
within rounding. Scenes: one block and many, rows and planes that do not
divide, one-column grids, blocks that hold both CPML ends of an axis, CPML on
six faces with an oscillator, poles in the CPML, flux planes of every
orientation with their wrapped neighbours, uneven chunks of steps."""
import os

import numpy as np
import pytest

from aether_b200 import _abi as A
from aether_b200 import configs as CF
from aether_b200 import fdtd
import scenes

pytestmark = pytest.mark.gpu

WAIT_CYCLES, WITHHOLD = 7, 8   # AEFDTD_TEST_RESIDENT_WAIT_CYCLES, AEFDTD_TEST_RESIDENT_WITHHOLD
NM = 1e-9


def substrate_of_poles(precision):
    """A dispersive substrate that reaches through the lower CPML."""
    sc = CF.sphere_scene(nx=30, ny=26, nz_total=110, pml=10, radius=14 * NM, nsteps=200, nl=5, sensor_gap=4,
                         precision=precision)
    sc.materials[2] = CF.lorentz_model()
    return sc


SCENES = {
    **{k: v for k, v in scenes.ALL.items() if k != "custom_many_materials"},
    "cell": lambda precision: CF.sphere_scene(nx=45, ny=37, nz_total=101, pml=11, radius=22 * NM, nl=9, nsteps=200,
                                              sensor_gap=4, precision=precision),
    "wide_rows": lambda precision: CF.slab_scene(nx=160, ny=9, nz_total=90, pml=8, slab=8, nl=5, nsteps=200,
                                                 sensor_gap=4, precision=precision),
    "poles_in_cpml": substrate_of_poles,
    "box": lambda precision: CF.random_spheres_scene(n_total=(70, 58, 50), pml=7, n_dielectric=20, n_lorentz=5,
                                                     r_range=(10 * NM, 30 * NM), nsteps=120, nl=3,
                                                     precision=precision, seed=3),
    "flat_box": lambda precision: CF.random_spheres_scene(n_total=(34, 33, 19), pml=3, n_dielectric=6, n_lorentz=2,
                                                          r_range=(10 * NM, 20 * NM), nsteps=120, nl=3,
                                                          precision=precision, seed=4),
}


def run(scene, resident, chunks):
    saved = os.environ.get("AEFDTD_RESIDENT")
    os.environ["AEFDTD_RESIDENT"] = "1" if resident else "0"
    try:
        with fdtd.build_simulation(scene) as s:
            box = None
            if scene.grid.mode == A.MODE_CUSTOM:
                g = scene.grid
                box = s.add_box_sensor((1, g.nx - 1, 0, g.ny, 0, g.nz - 1), 3, 500 * NM, 700 * NM)
            n0 = s.launch_count()
            for n in chunks:
                s.step(n)
            out = {"launches": s.launch_count() - n0, "fields": s.fields(),
                   "flux": [s.sensor_flux(i) for i in range(len(s.sensor_nl))],
                   "dft": [s.sensor_dft(i) for i in range(len(s.sensor_nl))]}
            if box is not None:
                out["flux"].append(s.box_flux(box))
            if scene.grid.mode == A.MODE_NORMAL:
                out["sums"] = s.plane_sums()
            return out
    finally:
        if saved is None:
            del os.environ["AEFDTD_RESIDENT"]
        else:
            os.environ["AEFDTD_RESIDENT"] = saved


@pytest.mark.parametrize("name", sorted(SCENES))
def test_fp64_bit_identical_to_the_split_kernels(name):
    chunks = (64, 37, 1, 70)
    scene = SCENES[name](precision=A.FP64)
    a, b = run(scene, True, chunks), run(scene, False, chunks)
    assert a["launches"] < b["launches"] / 8
    assert np.abs(b["fields"]).max() > 0
    assert np.array_equal(a["fields"], b["fields"])
    if "sums" in a:
        assert np.array_equal(a["sums"], b["sums"])
    for x, y in zip(a["dft"], b["dft"]):
        assert np.array_equal(x, y)
    for x, y in zip(a["flux"], b["flux"]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("name", ["gold_sphere", "cell", "poles_in_cpml", "box", "thin_column"])
def test_fp32_agrees_with_the_split_kernels(name):
    # 130 steps of single-precision updates; contraction may differ per kernel,
    # about one rounding (6e-8) per value and step adds up to below 1e-5 of the norm
    chunks = (64, 66)
    scene = SCENES[name](precision=A.FP32)
    a, b = run(scene, True, chunks), run(scene, False, chunks)
    assert np.linalg.norm(a["fields"] - b["fields"]) <= 1e-5 * np.linalg.norm(b["fields"])
    for x, y in zip(a["flux"], b["flux"]):
        assert np.linalg.norm(x - y) <= 1e-4 * np.linalg.norm(y)


def test_split_segments_from_graphs_match_direct_launches(monkeypatch):
    """The split path's captured segments, on a scene that now runs resident."""
    monkeypatch.setenv("AEFDTD_RESIDENT", "0")
    scene = scenes.gold_sphere()
    with fdtd.build_simulation(scene) as s:
        s.step(200)
        want = s.fields()
    monkeypatch.setenv("AEFDTD_NO_GRAPHS", "1")
    with fdtd.build_simulation(scene) as s:
        s.step(200)
        assert np.array_equal(s.fields(), want)


def test_restored_fields_and_resets_between_launches():
    """The state is in the public arrays between calls: a field written there
    is stepped, a reset clears it, and a second run repeats the first."""
    scene = SCENES["cell"](precision=A.FP64)
    rng = np.random.default_rng(5)
    nx, ny, nz = scene.total_dims()
    start = rng.standard_normal((6, nz, ny, nx))
    got = []
    for resident in (True, False):
        os.environ["AEFDTD_RESIDENT"] = "1" if resident else "0"
        try:
            with fdtd.build_simulation(scene) as s:
                s.step(20)
                s.reset()
                for c in range(6):
                    s.set_field(c, start[c])
                s.step(50)
                got.append(s.fields())
        finally:
            del os.environ["AEFDTD_RESIDENT"]
    assert np.array_equal(got[0], got[1])


def test_wait_runs_out_then_handle_recovers():
    scene = SCENES["cell"](precision=A.FP64)
    want = run(scene, True, (40,))["fields"]
    with fdtd.build_simulation(scene) as s:
        lib = s._lib
        assert lib.aefdtd_test_hook(s._h, WAIT_CYCLES, 1 << 20) == 0
        assert lib.aefdtd_test_hook(s._h, WITHHOLD, 1) == 0
        s.step(8)
        with pytest.raises(fdtd.AefdtdError) as e:
            s.synchronize()
        assert e.value.status == 3   # AEFDTD_TIMEOUT
        assert lib.aefdtd_test_hook(s._h, WAIT_CYCLES, 1 << 31) == 0
        assert lib.aefdtd_test_hook(s._h, WITHHOLD, 0) == 0
        s.reset()
        s.step(40)
        s.synchronize()
        assert np.array_equal(s.fields(), want)
