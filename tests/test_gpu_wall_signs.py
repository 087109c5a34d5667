"""The images of slip walls to the bit, the signs of zeros included: after a run the ghost cells and the zero
planes of every field are what the reference's images, axis after axis (cuda/Cuda_Seis3D.cu:152-175),
make of the field's interior.  Restated here in numpy."""
import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import capi, models3d, seis3d

pytestmark = pytest.mark.gpu

RADIUS = 4


def half_nodes(field, axis):
    if field < 3:
        return field == axis
    return {6: axis != 2, 7: axis != 0, 8: axis != 1}.get(field, False)


def images(field, f):
    """`f` [z][y][x] with its images, x first, written one layer after the other."""
    f = f.copy()
    for axis in range(3):
        v = np.moveaxis(f, 2 - axis, 0)      # a view, the axis first
        high, half = v.shape[0] - RADIUS - 1, half_nodes(field, axis)
        for depth in range(1, RADIUS + 1):
            if half and depth == 1:
                v[RADIUS - depth] = 0.0
            else:
                low = v[RADIUS + depth - 1 - half]
                v[RADIUS - depth] = -low if half else low
            up = v[high + 1 - depth - half]
            v[high + depth] = -up if half else up
        if half:
            v[high] = 0.0
    return f


@pytest.mark.parametrize("size", [(24, 19, 17), (40, 33, 48)])
@pytest.mark.parametrize("kind", [capi.SOURCE_EXPLOSION, capi.SOURCE_FORCE])
def test_images_to_the_bit(size, kind, solver_lib, cuda_device):
    c = seis3d.validate_context3D(seis3d.default_context(nx3D=size[0], ny3D=size[1], nz3D=size[2], reflecting3D=1,
                                                         freeSurface3D=0))
    s = seis3d.Session(c)
    source = seis3d.default_source(x3D=size[0] // 2, y3D=size[1] // 3, z3D=size[2] // 2, kind3D=kind)
    s.run_steps(source, 0, 90)
    s.run_step(source, 90)
    for k in range(9):
        f = s.field(k)
        assert np.abs(f[RADIUS, RADIUS]).max() > 0
        expect = images(k, f)
        assert np.array_equal(f.view(np.int32), expect.view(np.int32)), capi.FIELDS[k]
    s.release()
