"""Slip walls: the ghost shell after a stepping call is the mirror of the interior, axis by axis
(edges and corners included), and the fields agree with the FP32 oracle by the parity tests'
tolerance (test_gpu_parity.py).  Sizes: the smallest sides, odd ones, one side above a tile."""
import numpy as np
import pytest

import oracle
from cmakepro_cuda_seissim_v2_b200 import capi, seis3d

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-5
# Axes (x, y, z) along which a field lies on half nodes: its images are odd there.
HALF = {"vx": (0,), "vy": (1,), "vz": (2,), "sxy": (0, 1), "syz": (1, 2), "sxz": (0, 2)}


def mirrored(field, half_axes):
    """The field [z][y][x] with its ghost shell rebuilt from its interior."""
    out = field.copy()
    for axis in range(3):
        f = np.moveaxis(out, 2 - axis, 0)
        half = int(axis in half_axes)
        high = f.shape[0] - 5
        sign = -1.0 if half else 1.0
        for d in range(1, 5):
            f[4 - d] = 0.0 if half and d == 1 else sign * f[4 + d - 1 - half]
        for d in range(1, 5):
            f[high + d] = sign * f[high + 1 - d - half]
        if half:
            f[high] = 0.0
    return out


@pytest.mark.parametrize("size", [(16, 16, 16), (17, 33, 19), (40, 18, 25)])
@pytest.mark.parametrize("kind", [capi.SOURCE_EXPLOSION, capi.SOURCE_FORCE])
@pytest.mark.parametrize("steps", [1, 70])
def test_walls_mirror_the_interior(size, kind, steps, cuda_device):
    nx, ny, nz = size
    c = seis3d.validate_context3D(seis3d.default_context(nx3D=nx, ny3D=ny, nz3D=nz, reflecting3D=1, freeSurface3D=0,
                                                         modelKind3D=capi.MODEL_GRADIENT))
    src = seis3d.default_source(x3D=nx // 2, y3D=ny // 2, z3D=nz // 2, kind3D=kind, direction3D=(0.3, -0.5, 0.8))
    s = seis3d.Session(c)
    s.run_steps(src, 30, steps)
    fields = [s.field(k) for k in range(9)]
    materials = [s.field(k) for k in (9, 10, 11)]
    s.release()
    for name, f in zip(capi.FIELDS, fields):
        assert np.array_equal(f, mirrored(f, HALF.get(name, ()))), name
    o = oracle.CpuOracle(c, 32)
    core = (slice(4, -4),) * 3
    b, lam, mu = (m[core] for m in materials)
    vp, vs, rho = np.sqrt((lam + 2 * mu) * b), np.sqrt(mu * b), 1 / b
    o.upload_model(vp, vs, rho)
    o.run_gather(src, 30, steps, np.array([(nx // 2, ny // 2, 1)], np.int32), 1)
    for k, name in enumerate(capi.FIELDS):
        e = o.field(k).astype(np.float64)
        assert np.linalg.norm(fields[k] - e) <= FIELD_TOL * max(np.linalg.norm(e), 1e-300), name
    o.close()
