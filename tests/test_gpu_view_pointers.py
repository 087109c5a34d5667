"""Alignment of the device pointers of seis3d_get_views: unpitched sessions (the reference's layout) start
their fields and CPML memories where the allocation starts; pitched ones start the first updated
cell of every row on a 128-byte line.  Both hold the same bits after a run."""
import ctypes

import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import capi, models3d, seis3d

pytestmark = pytest.mark.gpu

STEPS = 40


def address(p):
    return ctypes.cast(p, ctypes.c_void_p).value


@pytest.mark.parametrize("storage", [capi.STORAGE_FP32, capi.STORAGE_BF16_CPML])
@pytest.mark.parametrize("nx", [36, 72])     # gx of 60 and 96: one of them a whole number of lines
def test_field_pointers(nx, storage, solver_lib, cuda_device):
    shot = models3d.small_shot(nx=nx, ny=30, nz=32, pml=8, steps=STEPS)
    gx, gy, gz = shot.context.gx3D, shot.context.gy3D, shot.context.gz3D
    assert gx == nx + 24
    fields = []
    for compact in (True, False):
        s = seis3d.Session(shot.context, compact_rows=compact, storage=storage)
        s.upload_model(shot.vp, shot.vs, shot.rho)
        s.run_steps(shot.source, 0, STEPS)
        v = s.views()
        pointers = list(v.field3D) + [v.inverseDensity3D, v.lambda3D, v.mu3D]
        if compact:
            assert v.pitch == gx
            assert all((p - pointers[0]) == 4 * k * gx * gy * gz for k, p in enumerate(pointers))
            assert pointers[0] % 256 == 0
            assert all(p % 256 == 0 for p in (address(v.cpml3D[a]) for a in range(3)))
        else:
            assert v.pitch % 32 == 0
            assert all((p + 16) % 128 == 0 for p in pointers)
        fields.append([s.field(k) for k in range(12)])
        s.release()
    assert np.abs(fields[0][2]).max() > 0
    for a, b in zip(*fields):
        assert np.array_equal(a, b)

