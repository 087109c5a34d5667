"""Which way seis2d_run_steps takes: one persistent launch or graph replay.  By rule (no mode set) runs of 16
steps or more are persistent once a session has made 512 of them, on grids that fit on the chip and
need at most two rows of split cells per thread; a gather of more than 1024 receivers is
replayed.  The way is read off the launch counter, the results are those of single steps."""
import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu


def context(size, npml, scheme, up, steps, receivers, src_type=capi2d.EXPLOSIVE):
    nx, nz = size
    top = npml if scheme == 3 and up else 0
    return models2d.layered_context(nx, nz, npml, 5.0, 0.0005, steps,
                                    [(0, 2200.0, 1200.0, 1900.0), (nz // 3, 3000.0, 1700.0, 2200.0)], f0=60.0,
                                    src=(nx // 2, max(nz // 2, top + 1)), src_type=src_type, receivers=receivers,
                                    flag_type=scheme, up=up)


def session(c, samples):
    gpu = seis2d.GPUSimData()
    seis2d.initializeGpuSimulation(gpu, c)
    if samples:
        seis2d.gatherBegin(gpu, 0, 1, samples)
    return gpu


def launches(gpu, first, count, c):
    before = gpu.kernelLaunches
    seis2d.runGpuSimulationSteps(gpu, first, count, c)
    return gpu.kernelLaunches - before


PERSISTENT = 2   # the run's configuration and one launch


def replayed(count):
    return 2 * count + (count + 63) // 64 + 1


def results(gpu, c, samples, stored):
    vx, vz, taken = seis2d.gatherFetch(gpu, samples)
    assert taken == samples
    return [vx[: c.num_rcv], vz[: c.num_rcv]] + [seis2d.copyField(gpu, n) for n in capi2d.FIELDS[:stored]]


# The sizes of test_gpu_resident2d.py, and three that no tiling of a 148-SM device takes.
FIT = [((9, 9), 0), ((10, 13), 0), ((2000, 9), 0), ((11, 900), 1), ((331, 330), 9), ((460, 460), 20), ((465, 465), 20),
       ((60, 110), 8), ((330, 205), 14)]
TOO_LARGE = [((470, 470), 20), ((514, 401), 20), ((900, 900), 20)]


@pytest.mark.parametrize("scheme,up", [(1, False), (2, False), (3, True)])
def test_sizes_of_persistent_runs(scheme, up, solver2d_lib, cuda_device):
    for fits, sizes in ((True, FIT), (False, TOO_LARGE)):
        for size, npml in sizes:
            if scheme == 3 and npml < 4:
                continue
            c = context(size, npml, scheme, up, 100, [(size[0] // 2, size[1] // 2)])
            gpu = session(c, 0)
            seis2d.setRunMode(gpu, capi2d.RUN_PERSISTENT)
            for first, count in ((0, 1), (1, 20)):
                assert launches(gpu, first, count, c) == (PERSISTENT if fits else replayed(count)), (size, count)
            seis2d.synchronize(gpu)
            seis2d.releaseGpuSimulation(gpu)


@pytest.mark.parametrize("scheme,up,size,npml", [(3, True, (120, 100), 12), (2, False, (128, 96), 12), (1, False, (200, 90), 0)])
def test_choice_by_rule_within_one_session(scheme, up, size, npml, solver2d_lib, cuda_device):
    # The run that comes to 512 long steps is the first persistent one; short runs are replayed
    # before and after it.  A gather is open throughout.
    runs = [(100, False), (15, False), (300, False), (10, False), (111, False), (15, False), (16, True), (70, True),
            (15, False), (1, False), (33, True)]
    assert sum(n for n, _ in runs[:6] if n >= 16) == 511
    steps = sum(n for n, _ in runs)
    top = npml if up else 4
    c = context(size, npml, scheme, up, steps, [(x, top + 5) for x in range(4, size[0] - 4, 7)])
    gpu = session(c, steps)
    done = 0
    for count, persistent in runs:
        assert launches(gpu, done, count, c) == (PERSISTENT if persistent else replayed(count)), (done, count)
        done += count
    stored = 15 if scheme == 2 else 10
    got = results(gpu, c, steps, stored)
    seis2d.releaseGpuSimulation(gpu)
    single = session(c, steps)
    for n in range(steps):
        seis2d.runGpuSimulationStep(single, n, c, -1)
    want = results(single, c, steps, stored)
    seis2d.releaseGpuSimulation(single)
    assert np.abs(want[1]).max() > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_grids_of_three_rows_are_replayed_by_rule(solver2d_lib, cuda_device):
    for scheme, persistent in ((1, False), (2, True)):
        c = context((460, 460), 20, scheme, False, 600, [(230, 230)])
        gpu = session(c, 0)
        assert launches(gpu, 0, 520, c) == (PERSISTENT if persistent else replayed(520))
        seis2d.synchronize(gpu)
        seis2d.releaseGpuSimulation(gpu)


@pytest.mark.parametrize("count,persistent", [(1024, True), (1025, False)])
def test_receivers_of_a_persistent_gather(count, persistent, solver2d_lib, cuda_device):
    # 1024 receivers of one tile fill its list; one more and the run is replayed, in either mode.
    size, lead, steps = (120, 100), 512, 40
    receivers = [(20 + n % 4, 30 + n // 4 % 3) for n in range(count)]
    c = context(size, 12, 1, False, lead + steps, receivers)
    got = []
    for way in ("mode", "rule", "single"):
        gpu = session(c, 0)
        if way != "rule":
            seis2d.setRunMode(gpu, capi2d.RUN_PERSISTENT if way == "mode" else capi2d.RUN_GRAPH)
        assert launches(gpu, 0, lead, c) == (replayed(lead) if way == "single" else PERSISTENT)
        seis2d.gatherBegin(gpu, lead, 1, steps)
        if way == "single":
            for n in range(lead, lead + steps):
                seis2d.runGpuSimulationStep(gpu, n, c, -1)
        else:
            assert launches(gpu, lead, steps, c) == (PERSISTENT if persistent else replayed(steps))
        got.append(results(gpu, c, steps, 10))
        seis2d.releaseGpuSimulation(gpu)
    assert np.abs(got[0][1]).max() > 0
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)
