"""The device's check of a whole model (seis3d_upload_model) against the host's check of a plane
(seis3d_upload_model_plane), cell by cell at the edges of what is admissible, and the conversion
into every cell of the padded grid for the smallest and for ragged sides."""
import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import models3d, seis3d

pytestmark = pytest.mark.gpu


def edges():
    f = np.float32
    up, down = (lambda v: np.nextafter(f(v), f(np.inf))), (lambda v: np.nextafter(f(v), f(-np.inf)))
    base = (f(3000), f(1500), f(2200))
    for k, values in enumerate((
            (0.0, -0.0, 1e-40, -1.0, np.nan, np.inf, -np.inf, down(4000), 4000.0, up(4000), 4000.004, 4000.01, up(30000)),
            (0.0, -0.0, 1e-40, -1e-40, np.nan, np.inf, -np.inf, 3000.0, down(3000), up(3000)),
            (0.0, -0.0, 1e-40, np.nan, np.inf, 50000.0, up(50000), -5.0))):
        for v in values:
            yield tuple(f(v) if a == k else base[a] for a in range(3))
    rng = np.random.default_rng(3)
    for vs in rng.uniform(100, 3000, 60).astype(f):   # vp * vp at (4/3) vs * vs and a few ulp beside it
        vp = np.sqrt(f(4.0 / 3.0) * vs * vs).astype(f)
        for _ in range(int(rng.integers(0, 4))):
            vp = up(vp)
        for _ in range(int(rng.integers(0, 4))):
            vp = down(vp)
        yield vp, vs, f(2200)


def accepted(call):
    try:
        call()
        return True
    except seis3d.InvalidArgument:
        return False


def test_device_check_equals_host_check(solver_lib, cuda_device):
    nx, ny, nz = 21, 18, 17
    c = models3d.imported_context(nx, ny, nz, 10.0, 8, False, 4000.0, 10.0)
    s = seis3d.Session(c)
    seen = set()
    for cell in edges():
        model = [np.full((nz, ny, nx), v, np.float32) for v in (3000, 1500, 2200)]
        for a, v in zip(model, cell):
            a[nz - 1, ny - 1, nx - 1] = v
        plane = np.stack([a[nz - 1] for a in model], axis=-1)
        host = accepted(lambda: s.upload_model_plane(nz - 1, plane))
        assert accepted(lambda: s.upload_volumes(*model)) == host, cell
        seen.add(host)
    assert seen == {True, False}
    s.release()


@pytest.mark.parametrize("size,surface", [((16, 16, 16), False), ((128, 16, 17), True), ((131, 33, 130), False), ((257, 65, 64), True)])
def test_whole_grid_equals_plane_uploads(size, surface, solver_lib, cuda_device):
    nx, ny, nz = size
    rng = np.random.default_rng(nx)
    vp = rng.uniform(2000, 4000, (nz, ny, nx)).astype(np.float32)
    vs, rho = vp / np.float32(1.8), rng.uniform(1500, 3000, vp.shape).astype(np.float32)
    c = models3d.imported_context(nx, ny, nz, 10.0, 8, surface, float(vp.max()), 10.0)
    a, b = seis3d.Session(c), seis3d.Session(c)
    a.upload_model(vp, vs, rho)
    b.upload_volumes(vp, vs, rho)
    for k in (9, 10, 11):
        assert np.array_equal(a.field(k), b.field(k)), k
    a.release()
    b.release()
