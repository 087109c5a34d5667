"""2-D runs by rule where several sessions share the device: a persistent run takes all of its SMs, so a
run beside another session's is replayed.  The way is read off the launch counter."""
import threading

import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu

RUN, PERSISTENT, REPLAYED = 32, 2, 2 * 32 + 2


def context():
    return models2d.small_shot2d(steps=2000).context


def session(c, steps=512):
    gpu = seis2d.GPUSimData()
    seis2d.initializeGpuSimulation(gpu, c)
    if steps:
        seis2d.runGpuSimulationSteps(gpu, 0, steps, c)
        seis2d.synchronize(gpu)
    return gpu


def launches(gpu, c, first=512):
    before = gpu.kernelLaunches
    seis2d.runGpuSimulationSteps(gpu, first, RUN, c)
    return gpu.kernelLaunches - before


def test_a_run_beside_another_sessions_is_replayed(solver2d_lib, cuda_device):
    c = context()
    a, b = session(c), session(c)
    assert launches(a, c) == PERSISTENT           # b's run is over
    seis2d.synchronize(a)
    for way in (capi2d.RUN_GRAPH, capi2d.RUN_PERSISTENT):
        seis2d.setRunMode(b, way)
        seis2d.runGpuSimulationSteps(b, 0, 20000, c)          # some tens of ms
        assert launches(a, c) == REPLAYED
        assert launches(a, c) == REPLAYED
        seis2d.synchronize(b)
        assert launches(a, c) == PERSISTENT       # its own earlier runs do not count
        seis2d.synchronize(a)
    seis2d.runGpuSimulationSteps(b, 0, 20000, c)
    seis2d.setRunMode(a, capi2d.RUN_PERSISTENT)
    assert launches(a, c) == PERSISTENT           # the caller's choice holds
    seis2d.releaseGpuSimulation(b)
    seis2d.synchronize(a)
    seis2d.releaseGpuSimulation(a)
    a = session(c)
    assert launches(a, c) == PERSISTENT           # a released session is not looked at
    seis2d.synchronize(a)
    seis2d.releaseGpuSimulation(a)


def test_sessions_on_threads(solver2d_lib, cuda_device):
    # Whatever way each run takes, every session has the bits of a session alone.
    c = context()
    alone = session(c, 0)
    for n in range(30):
        seis2d.runGpuSimulationSteps(alone, n * RUN, RUN, c)
    want = [seis2d.copyField(alone, n) for n in capi2d.FIELDS[:10]]
    seis2d.releaseGpuSimulation(alone)
    assert np.abs(want[2]).max() > 0
    got, errors = {}, []

    def work(k):
        try:
            gpu = session(c, 0)
            for n in range(30):
                seis2d.runGpuSimulationSteps(gpu, n * RUN, RUN, c)
                if n % (k + 2) == 0:
                    seis2d.synchronize(gpu)
            got[k] = [seis2d.copyField(gpu, n) for n in capi2d.FIELDS[:10]]
            seis2d.releaseGpuSimulation(gpu)
        except Exception as e:   # pytest reports it from the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k in range(4):
        for a, b in zip(got[k], want):
            assert np.array_equal(a, b)
