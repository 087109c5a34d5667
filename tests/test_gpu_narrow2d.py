"""2-D grids narrower than a strip's block, which take as many warps as they have columns for: widths at the
edges of the warps, replayed and in single steps, with more receivers than the block has threads.
Against the CPU FP32 oracle by the bound of test_gpu_parity2d.py (1e-4 relative L2)."""
import numpy as np
import pytest

import oracle
from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu

ORACLE32_TOL = 1e-4
STEPS = 60
WIDTHS = [9, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129]


@pytest.mark.parametrize("nx", WIDTHS)
@pytest.mark.parametrize("scheme,src_type", [(1, capi2d.ROTATED_FORCE), (2, capi2d.EXPLOSIVE), (3, capi2d.SHEAR)])
def test_narrow_grid(nx, scheme, src_type, solver2d_lib, cuda_device):
    nz = 240
    npml = min(8, (nx - 9) // 2)
    up = scheme == 3 and npml >= 4
    source = (min(nx // 2 + 1, nx - 5), nz // 2)
    receivers = [(x, z) for z in range(nz // 2 - 20, nz // 2 + 20) for x in sorted({4, nx // 2, nx - 5})] + \
                [(x, nz // 2 + 3) for x in range(nx)]
    c = models2d.layered_context(nx, nz, npml, 5.0, 0.0005, STEPS,
                                 [(0, 2200.0, 1200.0, 1900.0), (nz // 2 + 5, 2600.0, 1500.0, 2100.0)], f0=60.0, src=source,
                                 src_type=src_type, src_angle=30.0, receivers=receivers, flag_type=scheme, up=up)
    cpu = oracle.CpuOracle2D(c, 32)
    want = cpu.run(0, STEPS, receivers=c.rcv_grid_idx)
    cpu.close()
    assert np.abs(want[1]).max() > 0
    runs = []
    for single in (True, False):
        gpu = seis2d.GPUSimData()
        seis2d.initializeGpuSimulation(gpu, c)
        seis2d.setRunMode(gpu, capi2d.RUN_GRAPH)
        seis2d.gatherBegin(gpu, 0, 1, STEPS)
        if single:
            for n in range(STEPS):
                seis2d.runGpuSimulationStep(gpu, n, c, -1)
        else:
            seis2d.runGpuSimulationSteps(gpu, 0, STEPS, c)
        vx, vz, taken = seis2d.gatherFetch(gpu, STEPS)
        assert taken == STEPS
        seis2d.releaseGpuSimulation(gpu)
        runs.append((vx[: c.num_rcv], vz[: c.num_rcv]))
    for a, b, w in zip(*runs, want):
        assert np.array_equal(a, b)
        assert np.linalg.norm(np.asarray(a, np.float64) - w) <= ORACLE32_TOL * np.linalg.norm(np.asarray(w, np.float64))
