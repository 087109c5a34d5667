"""A 2-D persistent run that gave up is reported by the next synchronising call, whatever was enqueued
in between.  The wait is made to run out as in test_gpu_bounded_waits.py: one block sends nothing in
its first exchange and every wait is bounded by 0.1 ms."""
import pytest
import torch

from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu

SHORT_WAIT = 200_000   # SM cycles


def session(c, stream=None):
    gpu = seis2d.GPUSimData()
    seis2d.initializeGpuSimulation(gpu, c)
    seis2d.setRunMode(gpu, capi2d.RUN_PERSISTENT)
    if stream is not None:
        seis2d._check(capi2d.load().seis2d_set_stream(seis2d._session(gpu), stream.cuda_stream))
    seis2d.runGpuSimulationSteps(gpu, 0, 3, c)
    seis2d.synchronize(gpu)
    return gpu


def withhold(gpu, block):
    seis2d._check(capi2d.load().seis2d_debug_barrier_wait(seis2d._session(gpu), SHORT_WAIT if block >= 0 else 0, block))


@pytest.mark.parametrize("later", [capi2d.RUN_PERSISTENT, capi2d.RUN_GRAPH])
def test_a_later_run_does_not_hide_the_failure(later, solver2d_lib, cuda_device):
    c = models2d.small_shot2d(steps=40).context
    gpu = session(c)
    withhold(gpu, 0)
    seis2d.runGpuSimulationSteps(gpu, 3, 5, c)
    withhold(gpu, -1)
    seis2d.setRunMode(gpu, later)
    seis2d.runGpuSimulationSteps(gpu, 8, 5, c)
    with pytest.raises(RuntimeError, match="gave up"):
        seis2d.synchronize(gpu)
    # Reported once; runs after the report are runs like any other.
    seis2d.synchronize(gpu)
    seis2d.setRunMode(gpu, capi2d.RUN_PERSISTENT)
    before = seis2d.copyField(gpu, "vz_1")
    seis2d.runGpuSimulationSteps(gpu, 13, 5, c)
    seis2d.synchronize(gpu)
    assert (seis2d.copyField(gpu, "vz_1") != before).any()
    seis2d.releaseGpuSimulation(gpu)


def test_every_replay_of_a_captured_run_is_reported(solver2d_lib, cuda_device):
    c = models2d.small_shot2d(steps=40).context
    stream = torch.cuda.Stream()
    gpu = session(c, stream)
    withhold(gpu, 0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        seis2d.runGpuSimulationSteps(gpu, 3, 5, c)
    for _ in range(2):
        with torch.cuda.stream(stream):
            graph.replay()
            graph.replay()
        with pytest.raises(RuntimeError, match="gave up"):
            seis2d.synchronize(gpu)
    del graph
    seis2d.releaseGpuSimulation(gpu)
