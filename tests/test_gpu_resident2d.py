"""The 2-D persistent run at the edges of its tiles and of its range: the same bits as single
steps, whose traces are held against the CPU FP32 oracle with the bound of
test_gpu_parity2d.py (1e-4 relative L2; the same scheme in another rounding)."""
import numpy as np
import pytest
import torch

import oracle
from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu

ORACLE32_TOL = 1e-4
STEPS = 90


def shot(size, npml, scheme, up, src_type):
    nx, nz = size
    top = npml if scheme == 3 and up else 0
    rows = range(max(4, top), nz - 4, max(1, nz // 12))
    receivers = [(x, z) for z in rows for x in range(4, nx - 4, max(1, nx // 12))]
    return models2d.layered_context(nx, nz, npml, 5.0, 0.0005, STEPS,
                                    [(0, 2200.0, 1200.0, 1900.0), (nz // 3, 3000.0, 1700.0, 2200.0)],
                                    f0=60.0, src=(nx // 2, max(nz // 2, top + 1)), src_type=src_type, src_angle=30.0,
                                    receivers=receivers, flag_type=scheme, up=up)


def session(c):
    gpu = seis2d.GPUSimData()
    seis2d.initializeGpuSimulation(gpu, c)
    seis2d.gatherBegin(gpu, 0, 1, STEPS)
    return gpu


def results(gpu, c, stored):
    vx, vz, taken = seis2d.gatherFetch(gpu, STEPS)
    assert taken == STEPS
    return [vx[: c.num_rcv], vz[: c.num_rcv]] + [seis2d.copyField(gpu, n) for n in capi2d.FIELDS[:stored]]


# One row per thread down to two tiles of a few cells and to strips of tiles one wide; two and
# three rows; the last size that fits and one that does not (replayed).  The air rows are swept
# over a tile's height, so that the images cross the border between two tiles at every offset.
SIZES = [((9, 9), 0), ((10, 13), 0), ((2000, 9), 0), ((11, 900), 1), ((331, 330), 9), ((460, 460), 20), ((470, 470), 20)]
CASES = [(size, npml, 1, False, capi2d.ROTATED_FORCE) for size, npml in SIZES] + \
        [(size, npml, 2, False, capi2d.SHEAR) for size, npml in SIZES] + \
        [(size, npml, 3, True, capi2d.EXPLOSIVE) for size, npml in SIZES if npml >= 4] + \
        [((60, 110), npml, 3, True, capi2d.EXPLOSIVE) for npml in range(8, 16)] + \
        [((330, 205), npml, 3, True, capi2d.SHEAR) for npml in (14, 15, 16, 18, 19, 20)]


@pytest.mark.parametrize("size,npml,scheme,up,src_type", CASES)
def test_persistent_run_equals_single_steps(size, npml, scheme, up, src_type, solver2d_lib, cuda_device):
    c = shot(size, npml, scheme, up, src_type)
    stored = 15 if scheme == 2 else 10
    gpu = session(c)
    seis2d.setRunMode(gpu, capi2d.RUN_PERSISTENT)
    for first, count in ((0, 1), (1, 2), (3, 37), (40, 50)):
        seis2d.runGpuSimulationSteps(gpu, first, count, c)
    got = results(gpu, c, stored)
    steps = session(c)
    for n in range(STEPS):
        seis2d.runGpuSimulationStep(steps, n, c, -1)
    want = results(steps, c, stored)
    assert np.abs(want[1]).max() > 0
    for n, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b), n
    cpu = oracle.CpuOracle2D(c, 32)
    for a, b in zip(got, cpu.run(0, STEPS, receivers=c.rcv_grid_idx)):
        d = np.linalg.norm(np.asarray(a, np.float64) - b)
        assert d <= ORACLE32_TOL * np.linalg.norm(np.asarray(b, np.float64))


def test_captured_run_replays(solver2d_lib, cuda_device):
    # A run captured into a graph of the caller's and replayed is the run made again: the
    # exchanges of every replay need numbers of their own.
    c = shot((120, 100), 12, 3, True, capi2d.EXPLOSIVE)
    fields = []
    for captured in (True, False):
        gpu = session(c)
        stream = torch.cuda.Stream()
        seis2d._check(capi2d.load().seis2d_set_stream(seis2d._session(gpu), stream.cuda_stream))
        seis2d.setRunMode(gpu, capi2d.RUN_PERSISTENT)
        seis2d.runGpuSimulationSteps(gpu, 0, 20, c)
        seis2d.synchronize(gpu)
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                seis2d.runGpuSimulationSteps(gpu, 20, 30, c)
            with torch.cuda.stream(stream):
                for _ in range(3):
                    graph.replay()
        else:
            for _ in range(3):
                seis2d.runGpuSimulationSteps(gpu, 20, 30, c)
        seis2d.synchronize(gpu)
        fields.append([seis2d.copyField(gpu, n) for n in capi2d.FIELDS[:10]])
    assert np.abs(fields[0][2]).max() > 0
    for a, b in zip(*fields):
        assert np.array_equal(a, b)
