"""A context may refuse the cooperative launch of a 2-D persistent run (it has fewer SMs than the device).
The steps are then replayed, by rule and in the persistent mode, with the same results; nothing
is left of the refusal.  The refusal is the library's test hook, which answers in the launch's place."""
import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu

RUNS = [32] * 17 + [5, 40]   # past the 512 steps after which long runs are persistent by rule


@pytest.mark.parametrize("scheme,up", [(3, True), (2, False)])
@pytest.mark.parametrize("mode", [None, capi2d.RUN_PERSISTENT])
def test_refused_launch_is_replayed(scheme, up, mode, solver2d_lib, cuda_device):
    steps = sum(RUNS)
    c = models2d.small_shot2d(scheme, up, steps=steps).context
    results = []
    for refused in (True, False):
        gpu = seis2d.GPUSimData()
        seis2d.initializeGpuSimulation(gpu, c)
        chosen = mode if refused else capi2d.RUN_GRAPH
        if chosen is not None:
            seis2d.setRunMode(gpu, chosen)
        seis2d._check(solver2d_lib.seis2d_debug_refuse_persistent(seis2d._session(gpu), int(refused)))
        seis2d.gatherBegin(gpu, 0, 1, steps)
        done = 0
        for count in RUNS:
            before = gpu.kernelLaunches
            seis2d.runGpuSimulationSteps(gpu, done, count, c)
            assert gpu.kernelLaunches - before == 2 * count + 2      # one replay and its configuration
            done += count
        seis2d.synchronize(gpu)
        vx, vz, taken = seis2d.gatherFetch(gpu, steps)
        assert taken == steps
        results.append([vx, vz] + [seis2d.copyField(gpu, n) for n in capi2d.FIELDS[:10]])
        seis2d.releaseGpuSimulation(gpu)
    assert np.abs(results[1][1]).max() > 0
    for a, b in zip(*results):
        assert np.array_equal(a, b)
