"""Stepping a 2-D session on its own stream while the same thread captures other work into a CUDA graph
(torch's default, the strictest capture mode): the call in which the library goes over to
persistent runs, at 512 long steps, must leave the capture alone, as replayed steps do."""
import numpy as np
import pytest
import torch

from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu

RUN, RUNS, BEFORE = 32, 20, 15   # the 16th run crosses the line


def test_stepping_during_another_capture(solver2d_lib, cuda_device):
    c = models2d.small_shot2d(steps=RUN * RUNS).context
    results = []
    x = torch.arange(1000, dtype=torch.float32, device="cuda")
    for capture in (True, False):
        gpu = seis2d.GPUSimData()
        seis2d.initializeGpuSimulation(gpu, c)
        for n in range(BEFORE):
            seis2d.runGpuSimulationSteps(gpu, n * RUN, RUN, c)
        seis2d.synchronize(gpu)
        before = gpu.kernelLaunches
        if capture:
            graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                y = x * 2.0
                for n in range(BEFORE, RUNS):
                    seis2d.runGpuSimulationSteps(gpu, n * RUN, RUN, c)
                y = y + 1.0
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, 2.0 * x + 1.0)
        else:
            for n in range(BEFORE, RUNS):
                seis2d.runGpuSimulationSteps(gpu, n * RUN, RUN, c)
        assert gpu.kernelLaunches - before == 2 * (RUNS - BEFORE)     # persistent from the 16th run on
        results.append([seis2d.copyField(gpu, n) for n in capi2d.FIELDS[:10]])
        seis2d.releaseGpuSimulation(gpu)
    assert np.abs(results[0][2]).max() > 0
    for a, b in zip(*results):
        assert np.array_equal(a, b)
