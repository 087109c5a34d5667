"""The first step of a 2-D persistent run as its tiles see it.  The tiles of one run are ordered
only by the halos that neighbours exchange, so in a run of one or two steps on a line of many
tiles the first tile finishes long before the last one has heard of it; each must still take
its wavelet sample and its gather row from the step that the run was given."""
import os
import re

import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import capi2d, models2d, seis2d

RESIDENT = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cmakepro_cuda_seissim_v2_b200",
                        "csrc", "seis2d_resident.cuh")


def test_a_persistent_run_only_reads_its_control_block():
    text = re.sub(r"//[^\n]*", "", open(RESIDENT).read())
    signature = re.search(r"\bresidentRun\(([^)]*)\)", text).group(1)
    assert re.search(r"const Control2D\*\s*ctl\b", signature), signature
    assert not re.search(r"\bctl->\w+\s*[-+*]?=[^=]", text)


STEPS = 60


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 2, 3])
def test_short_runs_on_a_line_of_tiles(count, solver2d_lib, cuda_device):
    # A source and receivers in the last tiles of the line.
    nx, nz = 2000, 9
    c = models2d.layered_context(nx, nz, 0, 5.0, 0.0005, STEPS, [(0, 2200.0, 1200.0, 1900.0)], f0=60.0, src=(nx - 9, 4),
                                 src_type=capi2d.VERTICAL_FORCE, receivers=[(x, 4) for x in range(nx - 40, nx - 4)],
                                 flag_type=1, up=False)
    results = []
    for persistent in (True, False):
        gpu = seis2d.GPUSimData()
        seis2d.initializeGpuSimulation(gpu, c)
        seis2d.gatherBegin(gpu, 0, 1, STEPS)
        seis2d.setRunMode(gpu, capi2d.RUN_PERSISTENT)
        if persistent:
            for first in range(0, STEPS, count):
                seis2d.runGpuSimulationSteps(gpu, first, count, c)
        else:
            for n in range(STEPS):
                seis2d.runGpuSimulationStep(gpu, n, c, -1)
        vx, vz, taken = seis2d.gatherFetch(gpu, STEPS)
        assert taken == STEPS
        results.append((vx, vz, seis2d.copyField(gpu, "vz_1")))
        seis2d.releaseGpuSimulation(gpu)
    assert np.abs(results[1][1]).max() > 0
    for a, b in zip(*results):
        assert np.array_equal(a, b)
