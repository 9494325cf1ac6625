"""Resident time steps (resident.cuh) beside the normal run: a wait that runs
out and how it is reported, several threads with a simulation each, DFT blocks
(so segments) of a few steps, a device that refuses the plan, and fields with
infinities, and other work on the device at the same time."""
import threading

import numpy as np
import pytest

from aether_b200 import _abi as A
from aether_b200 import fdtd
from test_resident import SCENES, WAIT_CYCLES, WITHHOLD, run
from test_resident_long import FP32 as FP32_LONG, FP64 as FP64_LONG

pytestmark = pytest.mark.gpu
TIMEOUT = 3   # AEFDTD_TIMEOUT


def withhold(s, on):
    """Launches whose first block never sends H; waits end after 2^20 cycles."""
    assert s._lib.aefdtd_test_hook(s._h, WAIT_CYCLES, 1 << 20 if on else 1 << 31) == 0
    assert s._lib.aefdtd_test_hook(s._h, WITHHOLD, int(on)) == 0


REFUSE = 9    # AEFDTD_TEST_RESIDENT_REFUSE
READS = {"fields": lambda s: s.fields(), "sums": lambda s: s.plane_sums(), "spectra": lambda s: s.normal_spectra(),
         "flux": lambda s: s.sensor_flux(1), "dft": lambda s: s.sensor_dft(0), "synchronize": lambda s: s.synchronize()}


@pytest.mark.parametrize("read", sorted(READS))
def test_a_wait_that_runs_out_is_reported_by_the_call_that_reads(read):
    """No call hands out what an aborted launch left, whichever comes first;
    steps and reads are refused until the reset, which mends the handle."""
    scene = SCENES["cell"](precision=A.FP64)
    want = run(scene, True, (40,))["fields"]
    with fdtd.build_simulation(scene) as s:
        withhold(s, True)
        s.step(8)
        with pytest.raises(fdtd.AefdtdError) as e:
            READS[read](s)
        assert e.value.status == TIMEOUT
        withhold(s, False)
        for call in (lambda s: s.step(1), READS["fields"], READS["flux"]):
            with pytest.raises(fdtd.AefdtdError) as e:
                call(s)
            assert e.value.status == TIMEOUT
        s.reset()
        s.step(40)
        assert np.array_equal(s.fields(), want)


def test_a_reset_leaves_no_report_of_the_run_before():
    scene = SCENES["cell"](precision=A.FP64)
    want = run(scene, True, (40,))["fields"]
    with fdtd.build_simulation(scene) as s:
        withhold(s, True)
        s.step(8)
        s.reset()   # without a synchronising call before
        withhold(s, False)
        s.step(40)
        s.synchronize()
        assert np.array_equal(s.fields(), want)


def test_threads_with_plans_of_different_sizes():
    """One owning thread per handle: launches of simulations whose plans take
    the same kernel with different amounts of shared memory do not disturb
    each other."""
    names = ["gold_sphere", "slab_tm", "slab_te", "debye_lorentz_sphere"]
    want = {n: run(SCENES[n](precision=A.FP64), True, (64,) * 6)["fields"] for n in names}
    got, start = {}, threading.Barrier(len(names))

    def work(name):
        try:
            with fdtd.build_simulation(SCENES[name](precision=A.FP64)) as s:
                start.wait(60)
                for _ in range(6):
                    for _ in range(16):   # short calls: many launches
                        s.step(4)
                got[name] = s.fields()
        except Exception as e:   # kept for the assertion below
            got[name] = e

    threads = [threading.Thread(target=work, args=(n,)) for n in names]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for n in names:
        assert isinstance(got[n], np.ndarray), got[n]
        assert np.array_equal(got[n], want[n])


@pytest.mark.parametrize("sensors", [True, False])
@pytest.mark.parametrize("block", [1, 2, 3, 5])
def test_segments_of_a_few_steps(block, sensors):
    """A launch carries at most a segment (dft_block steps), however few."""
    scene = SCENES["cell"](precision=A.FP64)
    scene.grid.dft_block = block
    if not sensors:
        scene.sensors = []
    a, b = run(scene, True, (1, 17, 4)), run(scene, False, (1, 17, 4))
    for key in ("fields", "sums"):
        assert np.array_equal(a[key], b[key])
    for x, y in zip(a["dft"] + a["flux"], b["dft"] + b["flux"]):
        assert np.array_equal(x, y)
    assert len(a["flux"]) == len(scene.sensors)


def runs_resident(scene, chunks):
    """Whether the run issues fewer launches than the split kernels do."""
    counts = [run(scene, resident, chunks)["launches"] for resident in (True, False)]
    assert counts[0] <= counts[1]
    return counts[0] < counts[1]


def test_few_steps_per_launch_run_on_the_split_kernels():
    """A launch of few steps does not pay for loading and storing the state:
    short DFT blocks and, in FP64, single steps of the larger grids take the
    split kernels, which give the same bits."""
    scene = FP64_LONG["slab"](precision=A.FP64)
    assert runs_resident(scene, (64,)) and runs_resident(scene, (2,))
    assert not runs_resident(scene, (1,) * 4)
    assert runs_resident(SCENES["gold_sphere"](precision=A.FP64), (1,) * 4)
    for block in (1, 4, 7, 8):
        scene.grid.dft_block = block
        assert runs_resident(scene, (64,)) == (block >= 8), block
    scene.sensors = []
    for block in (3, 4):
        scene.grid.dft_block = block
        assert runs_resident(scene, (64,)) == (block >= 4), block


@pytest.mark.parametrize("name,precision", [("slab", A.FP64), ("sphere_odd", A.FP64), ("slab", A.FP32)])
def test_single_steps_among_longer_calls(name, precision):
    """However a run is cut into calls: the same fields and sums, bit for bit,
    and the flux up to the regrouping of its block sums."""
    scene = {A.FP64: FP64_LONG, A.FP32: FP32_LONG}[precision][name](precision=precision)
    a, b = run(scene, True, (100,)), run(scene, True, (1, 60, 1, 1, 2, 34, 1))
    assert np.abs(a["fields"]).max() > 0
    for key in ("fields", "sums"):
        assert np.array_equal(a[key], b[key])
    for x, y in zip(a["flux"], b["flux"]):
        assert np.linalg.norm(x - y) <= (1e-10 if precision == A.FP64 else 1e-6) * np.linalg.norm(x)


@pytest.mark.parametrize("name", ["gold_sphere", "box"])
@pytest.mark.parametrize("where", [1, 2, 3])
def test_a_refused_plan_falls_back_to_the_split_kernels(where, name):
    """No memory for the plan, blocks that do not fit at once, a refused launch
    (also after resident steps): the run goes on as if there were no resident
    path, and takes it again when the refusal and the plan are gone."""
    scene = SCENES[name](precision=A.FP64)
    want = run(scene, False, (40, 30, 30))
    with fdtd.build_simulation(scene) as s:
        assert s._lib.aefdtd_test_hook(s._h, REFUSE, where) == 0
        s.step(40)
        n = s.launch_count()
        assert n >= 3 * 40   # launches: E, H and their sensors or boundaries each step
        assert s._lib.aefdtd_test_hook(s._h, REFUSE, 0) == 0
        s.step(30)
        assert s.launch_count() < n + 60
        assert s._lib.aefdtd_test_hook(s._h, REFUSE, where) == 0
        s.step(30)
        assert np.array_equal(s.fields(), want["fields"])
        for i in range(len(s.sensor_nl)):
            if i < len(scene.sensors):
                assert np.array_equal(s.sensor_flux(i), want["flux"][i])
        if "sums" in want:
            assert np.array_equal(s.plane_sums(), want["sums"])


@pytest.mark.parametrize("precision", [A.FP64, A.FP32])
@pytest.mark.parametrize("name", ["slab_tm", "gold_sphere", "poles_in_cpml", "thin_column", "custom_box"])
def test_infinities_and_nans_spread_as_in_the_split_kernels(name, precision, monkeypatch):
    """Infinite and NaN values in and beside the CPML, at the faces of blocks
    and in the interior: the same cells are finite, infinite and NaN after
    three steps (the shortest run that sees both updates of both)."""
    scene = SCENES[name](precision=precision)
    nx, ny, nz = scene.total_dims()
    rng = np.random.default_rng(8)
    start = rng.standard_normal((6, nz, ny, nx))
    for c in range(6):
        for v in (np.inf, -np.inf, np.nan):
            for k in rng.integers(0, nz, 3):
                start[c, k, rng.integers(0, ny), rng.integers(0, nx)] = v
        start[c, 0, 0, 0] = start[c, nz - 1, ny - 1, nx - 1] = np.inf
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("AEFDTD_RESIDENT", resident)
        with fdtd.build_simulation(scene) as s:
            for c in range(6):
                s.set_field(c, start[c])
            s.step(3)
            got.append((s.fields(), s.launch_count()))
    (a, na), (b, nb) = got
    assert na < nb
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.isnan(b).any()
    assert np.array_equal(np.isinf(a), np.isinf(b)) and np.isinf(b).any()
    if precision == A.FP64:
        assert np.array_equal(a, b, equal_nan=True)


def test_two_simulations_that_fill_the_device():
    """Both launches want every SM: they take turns, and no wait runs out."""
    scenes = [FP64_LONG[n](precision=A.FP64) for n in ("slab", "sphere")]
    want = [run(sc, True, (256,) * 4)["fields"] for sc in scenes]
    got, start = [None, None], threading.Barrier(2)

    def work(k):
        with fdtd.build_simulation(scenes[k]) as s:
            start.wait(60)
            for _ in range(4):
                s.step(256)
            got[k] = s.fields()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_a_launch_beside_a_long_kernel_of_another_stream():
    """A kernel of 2.4e9 cycles holds a part of one SM for longer than a wait's
    bound of 2^31: the blocks start together all the same."""
    import torch
    scene = FP64_LONG["slab"](precision=A.FP64)
    want = run(scene, True, (64, 64))["fields"]
    with fdtd.build_simulation(scene) as s:
        s.step(64)
        s.synchronize()
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(int(2.4e9))
        s.step(64)
        assert np.array_equal(s.fields(), want)
        stream.synchronize()


def test_a_batch_member_gives_back_its_plan(monkeypatch):
    """Subsets are sized by what their members hold on the device; a member
    that ran resident before, and runs so again after, holds no plan in it."""
    scene = SCENES["cell"](precision=A.FP32)
    scene.sensors = []
    held, got = [], []
    for resident in ("1", "0"):
        monkeypatch.setenv("AEFDTD_RESIDENT", resident)
        with fdtd.build_simulation(scene) as s:
            s.step(64)
            with fdtd.Batch() as b:
                b.add(s, 64)
                held.append(s.dims().device_bytes)
                b.run(64)
                b.remove(s)
            n = s.launch_count()
            s.step(64)
            assert (s.launch_count() - n < 64) == (resident == "1")
            got.append(s.fields())
    assert held[0] == held[1]
    assert np.linalg.norm(got[0] - got[1]) <= 1e-5 * np.linalg.norm(got[1])
