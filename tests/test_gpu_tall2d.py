"""2-D grids with more strips of rows than a launch takes blocks along y (65,535): the last size with one
layer of blocks, the first ones with two, and past them, with the source and the receivers around
the seam between the layers and beyond 262,144 rows.  Against the CPU FP32 oracle by the bound of
test_gpu_parity2d.py (1e-4 relative L2), single steps and replayed ones."""
import numpy as np
import pytest

import oracle
from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

pytestmark = pytest.mark.gpu

ORACLE32_TOL = 1e-4
STEPS = 50


# Strips have four rows here; 262,144 rows of cells that are updated are 65,536 strips.
@pytest.mark.parametrize("nx,nz,npml,scheme,src_type,source", [
    (9, 262144, 0, 1, capi2d.VERTICAL_FORCE, 131070),     # 65,534 strips and the receivers' row
    (9, 262148, 0, 1, capi2d.EXPLOSIVE, 131074),          # 65,535
    (10, 262150, 0, 1, capi2d.ROTATED_FORCE, 262138),     # 65,536: one block of the second layer to spare
    (12, 270000, 1, 2, capi2d.SHEAR, 135004),
    (12, 270000, 1, 2, capi2d.VERTICAL_FORCE, 269980),
    (17, 300001, 4, 3, capi2d.EXPLOSIVE, 150003),
])
def test_tall_grid(nx, nz, npml, scheme, src_type, source, solver2d_lib, cuda_device):
    x = nx // 2
    receivers = [(x, z) for z in range(source - 40, min(source + 40, nz - 4), 3)] + [(x, nz - 5), (x, npml + 4)]
    c = models2d.layered_context(nx, nz, npml, 5.0, 0.0005, STEPS, [(0, 2200.0, 1200.0, 1900.0), (source, 2600.0, 1500.0, 2100.0)],
                                 f0=60.0, src=(x, source), src_type=src_type, src_angle=30.0, receivers=receivers,
                                 flag_type=scheme, up=scheme == 3)
    cpu = oracle.CpuOracle2D(c, 32)
    want = cpu.run(0, STEPS, receivers=c.rcv_grid_idx)
    names = capi2d.FIELDS[:15] if scheme == 2 else capi2d.FIELDS[:10]
    fields = [cpu.field(n) for n in range(len(names))]
    cpu.close()
    assert np.abs(want[1]).max() > 0
    for single in (True, False):
        gpu = seis2d.GPUSimData()
        seis2d.initializeGpuSimulation(gpu, c)
        seis2d.gatherBegin(gpu, 0, 1, STEPS)
        if single:
            for n in range(STEPS):
                seis2d.runGpuSimulationStep(gpu, n, c, -1)
        else:
            seis2d.runGpuSimulationSteps(gpu, 0, STEPS, c)
        vx, vz, taken = seis2d.gatherFetch(gpu, STEPS)
        assert taken == STEPS
        got = [seis2d.copyField(gpu, n) for n in names]
        seis2d.releaseGpuSimulation(gpu)
        for a, b in zip([vx[: c.num_rcv], vz[: c.num_rcv]] + got, list(want) + fields):
            d = np.linalg.norm(np.asarray(a, np.float64) - b)
            assert d <= ORACLE32_TOL * np.linalg.norm(np.asarray(b, np.float64))
