"""Passes cut into z chunks of falling sizes (grids with enough planes per place on the device)
against one chunk per tile, which reads no plane of another CTA's: the same bits."""
import numpy as np
import pytest

from cmakepro_cuda_seissim_v2_b200 import models3d, seis3d

pytestmark = pytest.mark.gpu

STEPS = 2400   # the wave reaches the ends of the longest grid


def run(size, surface, z_chunk):
    nx, ny, nz = size
    vp = 2000.0 + 1500.0 * models3d.splitmix64_uniform(nx * ny * nz, 3).reshape(nz, ny, nx)
    vp, vs, rho = models3d.elastic_from_vp(vp)
    c = models3d.imported_context(nx, ny, nz, 10.0, 8, surface, float(vp.max()), 15.0)
    s = seis3d.Session(c, z_chunk=z_chunk)
    s.upload_volumes(vp, vs, rho)
    s.set_receivers([(x, ny // 2, z) for x in range(0, nx, 9) for z in (0, 7, 21, nz - 1)])
    s.gather_begin(1, STEPS)
    s.run_steps(seis3d.default_source(x3D=nx // 2, y3D=ny // 2, z3D=6 if surface else nz // 2), 0, STEPS)
    out = [s.gather_fetch()] + [s.field(k) for k in range(9)]
    planes = s.z_chunk()[1]
    s.release()
    return planes, out


# Loads of 8 to 40 planes per place of a B200 and beside its lower end (equal chunks there), with
# sides that leave ragged tiles and a last chunk of one plane.
@pytest.mark.parametrize("size,surface", [((75, 80, 100), False), ((80, 80, 130), True), ((100, 90, 101), True),
                                          ((40, 48, 500), False), ((129, 113, 120), True), ((200, 120, 133), False)])
def test_falling_chunks_equal_one_chunk(size, surface, solver_lib, cuda_device):
    planes, got = run(size, surface, 0)
    whole, want = run(size, surface, 4096)
    assert planes < whole
    assert np.abs(want[0]).max() > 0 and all(np.abs(f[k]).max() > 0 for f in want[1:] for k in (8, -9))
    for n, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b), n
