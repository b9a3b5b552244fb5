"""The speed maximum and time step (speed_dt_kernel, csrc/levelset.cu) in its 16-byte passes: image
sizes that are multiples of four, with one full group of four loads per thread, with a group and
single loads behind it, with several groups, one image and a batch of one CTA each. The maximum,
or a value that is not finite, stands in the first and last value, in each component of a load, in
each load of a group and in the loads behind the groups; dt is the formula's, bit for bit."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DX, DY, CFL, B = 2.0, 1.5, 0.5, 0.01


def _dt(m):
    den = float(m) / DX + float(m) / DY + float(np.float32(B)) * (1 / DX ** 2 + 1 / DY ** 2) * 2.0
    return float(np.float32(CFL / den))


def _places(n, nimg):
    """Elements in every load of thread 0 and of the last thread, in the kernel's split."""
    ctas = min(-(-n // 4096), max(1, 1184 // nimg))
    stride = 4 * 256 * ctas
    at = {0, 1, 2, 3, n - 4, n - 3, n - 2, n - 1}
    for t in (0, 256 * ctas - 1):
        at.update(range(4 * t + 1, n, stride))
    at = sorted(at)
    return at if len(at) <= 24 else at[:12] + at[-12:]


@pytest.mark.parametrize("nimg,rows,cols", [(1, 64, 64), (1, 60, 128), (1, 2304, 2304), (600, 64, 68),
                                            (300, 100, 101)])
def test_maximum_and_non_finite(nimg, rows, cols):
    L = importlib.import_module("c-version-lithography_b200")
    n = rows * cols
    assert n % 4 == 0
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    phi = torch.rand(nimg, rows, cols, generator=gen, device="cuda")
    vn = torch.rand(nimg, rows, cols, generator=gen, device="cuda") - 0.5
    out = torch.empty_like(phi)
    img = nimg // 2
    flat = vn.view(nimg, n)[img]
    rest = [_dt(v) for v in vn.abs().amax(dim=(1, 2)).cpu().numpy()]

    def step():
        return L.LevelSetUtils.rk2_update_batch(phi, vn, DX, DY, CFL, B, out)
    assert list(step()) == rest
    for k, at in enumerate(_places(n, nimg)):
        was = flat[at].item()
        flat[at] = -3.25 if k % 2 else 3.25
        dts = list(step())
        assert dts == rest[:img] + [_dt(3.25)] + rest[img + 1:], at
        flat[at] = [float("nan"), float("inf"), -float("inf")][k % 3]
        with pytest.raises(L.LithoError):
            step()
        flat[at] = was
    assert list(step()) == rest
