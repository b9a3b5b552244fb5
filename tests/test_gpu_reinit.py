"""GPU parity of the chamfer re-initialisation (csrc/reinit.cu) at the edges of its tiling:
row blocks of 8, class words of 32 rows, 32-column bounds, the near and the far search, and
the row pairs staged at a time (all four, two, or one for the widest images)."""
import importlib

import numpy as np
import pytest

from oracle import levelset_oracle as lo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    p = importlib.import_module("c-version-lithography_b200")
    p.load_library()
    return p


def _case(shape, kind):
    rows, cols = shape
    rng = np.random.default_rng(rows * 31 + cols)
    if kind == "noise":
        return rng.standard_normal(shape)
    if kind == "sparse":       # few inside pixels: the far search
        phi = np.full(shape, -1.0)
        phi.reshape(-1)[rng.integers(0, rows * cols, 1 + rows * cols // 20000)] = 1.0
        return phi
    if kind == "holes":        # few outside pixels
        return -_case(shape, "sparse")
    phi = np.full(shape, -1.0)   # "corner": one inside pixel
    phi[-1, 0] = 1.0
    return phi


@pytest.mark.parametrize("kind", ["noise", "sparse", "holes", "corner"])
@pytest.mark.parametrize("shape", [(1, 1), (1, 70), (2, 33), (70, 1), (7, 31), (8, 32), (9, 64),
                                   (33, 65), (41, 97), (65, 129), (257, 300), (130, 1000),
                                   (20, 7000), (18, 13000), (17, 17000)])
def test_matches_opencv(L, shape, kind):
    """Against cv2.distanceTransform(DIST_L2, 5): the same minimum, so float rounding only.
    OpenCV adds float32 weights step by step, up to max(shape) of them: 1e-5 relative."""
    phi = _case(shape, kind)
    ref = lo.reinit_sdf(phi, 2.0, 2.0)
    ref = np.where(np.abs(ref) > 1e37, np.copysign(np.float32(3.4028235e38), ref), ref)
    got, mask = L.LevelSetUtils.reinit_sdf(phi, 2.0, 2.0, with_mask=True)
    got = got.double().cpu().numpy()
    assert np.all(np.abs(got - ref) <= 1e-5 * np.abs(ref) + 1e-6)
    assert np.array_equal(mask.double().cpu().numpy(), (got >= 0).astype(np.float64))


def test_tall_columns(L):
    """More rows than one chunk of staged class words holds (32768), with the classes far
    apart across the chunk border."""
    rows, cols = 70001, 5
    phi = np.full((rows, cols), -1.0)
    phi[[3, 32767, 69990], [0, 4, 2]] = 1.0
    ref = lo.reinit_sdf(phi, 1.0, 1.0)
    got = L.LevelSetUtils.reinit_sdf(phi, 1.0, 1.0).double().cpu().numpy()
    assert np.all(np.abs(got - ref) <= 1e-5 * np.abs(ref) + 1e-6)


@pytest.mark.parametrize("threads_shape", [(24, 40, 3), (300, 301, 5)])
def test_batch_is_single(L, threads_shape):
    """Every image of a batch as alone, bit for bit, with a level and the printed mask."""
    r, c, b = threads_shape
    rng = np.random.default_rng(r)
    phi = torch.tensor(rng.random((b, r, c)), dtype=torch.float32, device="cuda")
    mask = torch.empty_like(phi)
    out = L.LevelSetUtils.reinit_sdf_batch(phi, 1.5, 1.5, level=0.5, mask_out=mask)
    for i in range(b):
        one = L.LevelSetUtils.reinit_sdf_batch(phi[i:i + 1].clone(), 1.5, 1.5, level=0.5)
        assert torch.equal(out[i], one[0])
    assert torch.equal(mask, (out >= 0).float())
