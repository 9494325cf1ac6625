"""Resident time steps (resident.cuh) beside the normal run: a wait that runs
out and how it is reported, several threads with a simulation each, and DFT
blocks (so segments) of a few steps."""
import threading

import numpy as np
import pytest

from aether_b200 import _abi as A
from aether_b200 import fdtd
from test_resident import SCENES, WAIT_CYCLES, WITHHOLD, run

pytestmark = pytest.mark.gpu
TIMEOUT = 3   # AEFDTD_TIMEOUT


def withhold(s, on):
    """Launches whose first block never sends H; waits end after 2^20 cycles."""
    assert s._lib.aefdtd_test_hook(s._h, WAIT_CYCLES, 1 << 20 if on else 1 << 31) == 0
    assert s._lib.aefdtd_test_hook(s._h, WITHHOLD, int(on)) == 0


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
