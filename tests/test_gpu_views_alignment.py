"""The output of the view extraction (2 floats per sample) may start at any float of a device buffer, on an
8-byte boundary or between two of them: the same samples, the same statistics, and nothing
written around them."""
import pytest
import torch

from cmakepro_cuda_seissim_v2_b200 import models3d, seis3d

pytestmark = pytest.mark.gpu

GUARD = -7.0


@pytest.mark.parametrize("volume", [False, True])
@pytest.mark.parametrize("component,material", [(0, 5), (4, 7), (6, 6)])
def test_output_at_any_float(volume, component, material, solver_lib, cuda_device):
    shot = models3d.small_shot(steps=40)
    s = seis3d.Session(shot.context)
    s.upload_model(shot.vp, shot.vs, shot.rho)
    s.run_steps(shot.source, 0, 40)
    layout = seis3d.make_view_layout3D(s.context)
    count = 2 * (layout.totalSamples3D if volume else layout.volumeOffset3D)
    slices = (s.context.nx3D // 2, s.context.ny3D // 3, s.context.nz3D // 2)
    results = []
    for offset in (0, 1, 2, 3):
        buffer = torch.full((count + 8,), GUARD, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        stats = s.extract_views(buffer.data_ptr() + 4 * offset, layout, slices, component, material, volume, True)
        host = buffer.cpu()
        assert (host[:offset] == GUARD).all() and (host[offset + count:] == GUARD).all()
        results.append((host[offset:offset + count], stats))
    assert results[0][0].abs().max() > 0
    for samples, stats in results[1:]:
        assert torch.equal(samples, results[0][0]) and stats == results[0][1]
    with pytest.raises(seis3d.InvalidArgument):      # not the address of a float
        s.extract_views(buffer.data_ptr() + 2, layout, slices, component, material, volume, True)
    s.release()
