"""A 2-D gather keeps the receivers it began with: replaced by fewer or by more, the session's receivers
change neither its traces nor the size of what is fetched."""
import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import models2d, seis2d

pytestmark = pytest.mark.gpu

STEPS = 60


@pytest.mark.parametrize("later", [None, 1, 90])
def test_gather_after_a_change_of_receivers(later, solver2d_lib, cuda_device):
    c = models2d.small_shot2d(steps=STEPS).context
    gpu = seis2d.GPUSimData()
    seis2d.initializeGpuSimulation(gpu, c)
    seis2d.gatherBegin(gpu, 0, 1, STEPS)
    seis2d.runGpuSimulationSteps(gpu, 0, STEPS // 2, c)
    if later is not None:
        seis2d.updateGpuReceivers(gpu, np.arange(later) + 30 * c.NX)
    seis2d.runGpuSimulationSteps(gpu, STEPS // 2, STEPS - STEPS // 2, c)
    vx, vz, taken = seis2d.gatherFetch(gpu, STEPS)
    assert taken == STEPS and vx.shape == vz.shape == (max(c.num_rcv, later or 0), STEPS)
    seis2d.releaseGpuSimulation(gpu)
    plain = seis2d.GPUSimData()
    seis2d.initializeGpuSimulation(plain, c)
    seis2d.gatherBegin(plain, 0, 1, STEPS)
    seis2d.runGpuSimulationSteps(plain, 0, STEPS, c)
    wx, wz, _ = seis2d.gatherFetch(plain, STEPS)
    seis2d.releaseGpuSimulation(plain)
    assert np.abs(wz).max() > 0
    assert np.array_equal(vx[: c.num_rcv], wx) and np.array_equal(vz[: c.num_rcv], wz)
