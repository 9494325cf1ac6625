"""The split half-step kernels (AEFDTD_RESIDENT=0, what every larger grid runs
on) and the resident steps (the default of the small scenes), each held to the
reference's golden fixtures and through calls cut into pieces and results read
mid-run; the split path's captured segments against direct launches and its
concurrent groups against serial ones. Launch counts show which path ran."""
import os

import numpy as np
import pytest

import scenes
from aether_b200 import _abi as A
from aether_b200 import fdtd
from test_gpu_parity import GOLDEN, GOLDEN_DIR, RTOL_FLUX, RTOL_PLANE, RTOL_SPECTRA, rel, sha
from test_resident import SCENES, run

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["split", "resident"])
def path(request, monkeypatch):
    monkeypatch.setenv("AEFDTD_RESIDENT", "1" if request.param == "resident" else "0")
    return request.param


def took(path, launches, steps):
    """A split step is at least an E and an H launch; a resident chunk of 64
    steps a handful."""
    assert (launches >= 2 * steps) == (path == "split"), (path, launches, steps)


@pytest.mark.parametrize("name", GOLDEN)
def test_fp64_bit_identical_to_reference_golden(name, path):
    g = np.load(os.path.join(GOLDEN_DIR, f"{name}.npz"))
    scene = scenes.ALL[name]()
    r = fdtd.run(scene)
    took(path, r["launches"], scene.nsteps)
    assert sha(r["fields"]) == list(g["field_sha256"])
    if "plane_sums" in g:
        assert rel(r["plane_sums"], g["plane_sums"]) < RTOL_PLANE
        assert rel(r["spectra"], g["spectra"]) < RTOL_SPECTRA
    for i, f in enumerate(r["flux"]):
        assert rel(f, g[f"flux{i}"]) < RTOL_FLUX


def test_fp64_step_in_pieces_equals_one_call(path):
    with fdtd.build_simulation(scenes.gold_sphere()) as s1, fdtd.build_simulation(scenes.gold_sphere()) as s2:
        s1.step(90)
        took(path, s1.launch_count(), 90)
        for n in (1, 10, 33, 46):
            s2.step(n)
        assert np.array_equal(s1.fields(), s2.fields())
        assert np.array_equal(s1.plane_sums(), s2.plane_sums())
        for i in range(2):
            assert np.array_equal(s1.sensor_flux(i), s2.sensor_flux(i))


@pytest.mark.parametrize("precision", [A.FP64, A.FP32])
def test_reading_sensors_mid_run_then_continuing(precision, path):
    """Pending and partial DFT blocks drained by a read after 150 of 330 steps:
    the fields unchanged, the flux up to the regrouping of the block sums."""
    scene = scenes.gold_sphere(precision=precision, nsteps=330)
    with fdtd.build_simulation(scene) as s1, fdtd.build_simulation(scene) as s2:
        s1.step(330)
        took(path, s1.launch_count(), 330)
        s2.step(150)
        mid = [s2.sensor_flux(i) for i in range(2)]
        s2.step(180)
        assert np.array_equal(s1.fields(), s2.fields())
        for i in range(2):
            assert rel(s2.sensor_flux(i), s1.sensor_flux(i)) < (RTOL_FLUX if precision == A.FP64 else 1e-6)
            assert np.all(np.isfinite(mid[i]))


@pytest.mark.parametrize("precision", [A.FP64, A.FP32])
def test_graph_replay_matches_direct_launches(precision, monkeypatch):
    """Whole 64-step segments replayed from CUDA graphs against the same steps
    launched one by one: fields, sums, flux and the launches of both."""
    monkeypatch.setenv("AEFDTD_RESIDENT", "0")
    scene = scenes.gold_sphere(precision=precision, nsteps=200)
    a = fdtd.run(scene)
    monkeypatch.setenv("AEFDTD_NO_GRAPHS", "1")
    b = fdtd.run(scene)
    took("split", a["launches"], 200)
    assert np.array_equal(a["fields"], b["fields"])
    assert np.array_equal(a["plane_sums"], b["plane_sums"])
    for fa, fb in zip(a["flux"], b["flux"]):
        assert np.array_equal(fa, fb)
    assert a["launches"] == b["launches"]


@pytest.mark.parametrize("name", ["gold_sphere", "custom_box"])
def test_concurrent_groups_match_serial_groups(name, monkeypatch):
    monkeypatch.setenv("AEFDTD_RESIDENT", "0")
    scene = getattr(scenes, name)(nsteps=90)
    a = fdtd.run(scene)
    monkeypatch.setenv("AEFDTD_SERIAL_GROUPS", "1")
    b = fdtd.run(scene)
    took("split", a["launches"], 90)
    assert np.array_equal(a["fields"], b["fields"])
    for fa, fb in zip(a["flux"], b["flux"]):
        assert np.array_equal(fa, fb)


@pytest.mark.parametrize("name,precision", [(n, A.FP32) for n in ("gold_sphere", "cell", "poles_in_cpml", "box",
                                                                  "thin_column")] + [("cell", A.FP64)])
def test_scenes_of_the_resident_tests_run_resident(name, precision):
    """The scenes that test_resident.py compares between the paths without a
    look at the launches."""
    scene = SCENES[name](precision=precision)
    chunks = (64, 66) if precision == A.FP32 else (20, 50)
    assert run(scene, True, chunks)["launches"] < run(scene, False, chunks)["launches"] / 8
