"""Where the normal speed is zero the level set does not move, whatever its slope: delta is 0 also
where the slope's square leaves FP32's range. Steps of 1e25 per pixel along x, y and both, speeds
of either sign beside the zeros, spacings of both stencil variants, images of one and of
several tiles."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [1.0, 8192.0])
@pytest.mark.parametrize("sy,sx", [(0.0, 1e25), (1e25, 0.0), (1e25, -1e25)])
@pytest.mark.parametrize("shape", [(5, 7), (20, 133), (700, 1100)])
def test_zero_speed(shape, sy, sx, spacing):
    L = importlib.import_module("c-version-lithography_b200")
    rows, cols = shape
    y = torch.arange(rows, device="cuda", dtype=torch.float32)[:, None]
    x = torch.arange(cols, device="cuda", dtype=torch.float32)[None, :]
    phi = (sy * spacing * y + sx * spacing * x).contiguous()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows)
    vn = torch.randint(-1, 2, shape, generator=gen, device="cuda").float()
    vn[0, 0], vn[rows // 2, cols // 2] = 0.0, -0.0
    delta = L.LevelSetUtils.evolve_normal_WENO_godunov(phi, vn, spacing, spacing).delta
    zero = vn == 0
    assert zero.any() and torch.all(delta[zero] == 0)
