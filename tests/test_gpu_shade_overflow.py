"""Volume rendering of a wave whose scaled value overflows: a diverging run over a small display scale
(1e-12, the scale before the first extraction).  Such a sample is drawn at full density, as the
shader's division makes it.  Against the CPU shader oracle by the bounds of test_gpu_shade.py."""
import numpy as np
import pytest
import torch

import oracle
from cmakepro_cuda_seissim_v2_b200 import capi, models3d, seis3d

pytestmark = pytest.mark.gpu

VOLUME_TOL, VOLUME_OUTLIERS, VOLUME_MAX = 1e-3, 0.005, 0.05
WIDTH, HEIGHT = 160, 120


# 1e25 stays finite, 1e27 overflows with the scale, 3e38 with the gain already.  `fall` 0 fills the
# volume; with 600 the wave is a blob that falls through all magnitudes to nothing.
@pytest.mark.parametrize("amplitude", [1e25, 1e27, 1e30, 3e38])
@pytest.mark.parametrize("fall", [0, 600])
@pytest.mark.parametrize("sign,component", [(1, 0), (-1, 0), (1, 3)])
def test_overflowing_wave_is_drawn(amplitude, fall, sign, component, solver_lib, cuda_device):
    shot = models3d.small_shot(steps=2)
    s = seis3d.Session(shot.context)
    layout = seis3d.make_view_layout3D(s.context)
    d = seis3d.default_display(component3D=component, materialRange3D=[1500.0, 4500.0], volumeRequestedWidth3D=WIDTH,
                               volumeRequestedHeight3D=HEIGHT)
    t, u, w, h = seis3d.make_display_uniforms(s.context, layout, d)
    assert u.scale3D == np.float32(1e-12)
    shape = (layout.volumeZ3D, layout.volumeY3D, layout.volumeX3D)
    z, y, x = (np.linspace(-1, 1, n, dtype=np.float64).reshape([-1 if a == k else 1 for a in range(3)])
               for k, n in enumerate(shape))
    views = np.zeros((layout.totalSamples3D, 2), np.float32)
    wave = sign * amplitude * np.exp(-fall * (x * x + y * y + z * z))
    views[layout.volumeOffset3D:, 0] = wave.astype(np.float32).ravel()
    views[:, 1] = 2500.0
    texels = views[layout.volumeOffset3D:].reshape(*shape, 2)
    assert np.isfinite(views).all()
    want = oracle.render_volume(texels, t, u, w, h)
    device = torch.from_numpy(views).cuda()
    out = torch.zeros(h * w * 4, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    s.render_volume(layout, device.data_ptr(), t, u, w, h, capi.PIXELS_RGBA32F, out.data_ptr())
    s.synchronize()
    got = out.cpu().numpy().reshape(h, w, 4)
    s.release()
    assert np.isfinite(want).all() and np.isfinite(got).all()
    # The wave shows against the same volume without a wave.
    calm = texels.copy()
    calm[..., 0] = 0
    assert (np.abs(want - oracle.render_volume(calm, t, u, w, h)).max(axis=-1) > 0.1).mean() > 0.005
    err = np.abs(got - want).max(axis=-1)
    assert err.max() <= VOLUME_MAX and (err > VOLUME_TOL).mean() <= VOLUME_OUTLIERS
