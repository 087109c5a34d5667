"""The passes update x-adjacent cells in pairs.  Where a pair is not whole: the last column of an
odd number of active columns, a slab edge between the two cells (odd CPML thickness), and an
upper x slab whose words start at an odd index (odd width).  Fields against the FP32 oracle, and
the 16-bit memory mode against the oracle's emulation of it, by the tolerances of the parity
tests (test_gpu_parity.py, test_gpu_bf16_cpml.py)."""
import numpy as np
import pytest

import oracle
from cmakepro_cuda_seissim_v2_b200 import capi, models3d, seis3d

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-5        # relative L2, FP32 fields against the FP32 oracle
EMULATION_TOL = 5e-6    # relative L2, 16-bit memories against their emulation (traces, early steps)


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def run(shot, storage, steps):
    s = seis3d.Session(shot.context, storage=storage)
    try:
        s.upload_model(shot.vp, shot.vs, shot.rho)
        s.set_receivers(shot.receivers)
        s.gather_begin(1, steps)
        s.run_steps(shot.source, 0, steps)
        return s.gather_fetch(), [s.field(k) for k in range(9)]
    finally:
        s.release()


def run_oracle(shot, memories, steps):
    lib = oracle.oracle_library()
    lib.oracle3d_set_psi_storage(memories)
    try:
        o = oracle.CpuOracle(shot.context, 32)
        o.upload_model(shot.vp, shot.vs, shot.rho)
        g = o.run_gather(shot.source, 0, steps, shot.receivers, 1)
        f = [o.field(k) for k in range(9)]
        o.close()
        return g, f
    finally:
        lib.oracle3d_set_psi_storage(0)


@pytest.mark.parametrize("nx,pml", [(16, 8), (17, 8), (17, 9), (31, 11), (32, 9), (33, 8), (50, 13)])
@pytest.mark.parametrize("kind", [capi.SOURCE_EXPLOSION, capi.SOURCE_FORCE])
def test_pairs_cut_by_edges(nx, pml, kind, cuda_device):
    shot = models3d.small_shot(nx=nx, ny=19, nz=21, pml=pml, steps=70, kind=kind)
    g, f = run(shot, capi.STORAGE_FP32, shot.steps)
    eg, ef = run_oracle(shot, 0, shot.steps)
    assert np.all(np.isfinite(g)) and rel_l2(g, eg) < FIELD_TOL
    for k in range(9):
        assert rel_l2(f[k], ef[k]) < FIELD_TOL, capi.FIELDS[k]


@pytest.mark.parametrize("nx,pml", [(17, 9), (32, 8)])
def test_pairs_of_16_bit_memories(nx, pml, cuda_device):
    shot = models3d.small_shot(nx=nx, ny=19, nz=21, pml=pml, steps=60)
    g, _ = run(shot, capi.STORAGE_BF16_CPML, shot.steps)
    eg, _ = run_oracle(shot, 2, shot.steps)
    assert rel_l2(g, eg) < EMULATION_TOL
