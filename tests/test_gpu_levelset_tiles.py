"""GPU parity of the level-set stencil (csrc/levelset.cu) at the edges of its tiling: 2 x 2
pixel blocks, 64-column tiles of 8 or 32 rows, odd and unaligned rows, and the maximum
speed's vector and scalar passes."""
import importlib

import numpy as np
import pytest

from oracle import levelset_oracle as lo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# FP32 against FP64: the bound of the random fields in test_gpu_levelset.py.
TOL = 2e-5


@pytest.fixture(scope="module")
def L():
    p = importlib.import_module("c-version-lithography_b200")
    p.load_library()
    return p


def _fields(rows, cols, seed):
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:rows, 0:cols].astype(np.float64)
    phi = 20.0 * np.sin(0.05 * xx + 0.3) * np.cos(0.043 * yy) + 0.5 * rng.standard_normal((rows, cols))
    vn = rng.standard_normal((rows, cols))
    vn[rng.random((rows, cols)) < 0.1] = 0.0      # no motion: |grad phi| does not matter
    return phi.astype(np.float32), vn.astype(np.float32)


def _close(got, want):
    got = got.double().cpu().numpy()
    assert np.max(np.abs(got - want)) <= TOL * np.max(np.abs(want))


@pytest.mark.parametrize("shape", [(3, 4), (4, 3), (8, 64), (9, 65), (7, 63), (16, 66), (31, 129),
                                   (33, 68), (5, 200), (200, 5)])
def test_edges_match_oracle(L, shape):
    phi, vn = _fields(*shape, seed=sum(shape))
    dx, dy, cfl, b = 2.0, 1.5, 0.5, 0.01
    e = L.LevelSetUtils.evolve_normal_WENO_godunov(phi, vn, dy, dx)
    _close(e.delta, lo.evolve_normal_weno_godunov(phi.astype(np.float64), vn.astype(np.float64), dy, dx)[0])
    _close(L.LevelSetUtils.evolve_kappa(phi, dx, dy, b), lo.evolve_kappa(phi.astype(np.float64), dx, dy, b))
    got, mask, dt = L.LevelSetUtils.rk2_update(phi, vn, dx, dy, cfl, b)
    want, want_dt = lo.lsm_rk2_update(phi.astype(np.float64), vn.astype(np.float64), dx, dy, cfl, b)
    _close(got, want)
    assert abs(dt - want_dt) <= 1e-6 * want_dt
    assert torch.equal(mask, (got >= 0).float())


@pytest.mark.parametrize("batch,rows,cols,shift", [(3, 40, 64, 0), (40, 300, 260, 0), (40, 300, 260, 1),
                                                   (40, 301, 257, 0)])
def test_batch_is_single(L, batch, rows, cols, shift):
    """Every image of a batch as alone, bit for bit: tall tiles against single-pass ones,
    16-byte rows against rows that start one float off (shift)."""
    n = batch * rows * cols
    f = [_fields(rows, cols, s) for s in range(batch)]

    def put(k):
        base = torch.empty(n + 4, device="cuda")[shift:shift + n].view(batch, rows, cols)
        base.copy_(torch.from_numpy(np.stack([x[k] for x in f])))
        return base
    phi, vn = put(0), put(1)
    out, mask = torch.empty_like(phi), torch.empty_like(phi)
    dts = L.LevelSetUtils.rk2_update_batch(phi, vn, 1.0, 1.0, 0.5, 0.01, out, mask_out=mask)
    for i in range(0, batch, 13):
        one, m, dt = L.LevelSetUtils.rk2_update(phi[i].clone(), vn[i].clone(), 1.0, 1.0, 0.5, 0.01)
        assert torch.equal(out[i], one) and torch.equal(mask[i], m) and dts[i] == dt


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("at", [0, 1023, 4095, 4109])
def test_non_finite_speed(L, bad, at):
    """A non-finite speed anywhere is reported, in the vector passes and in their rest."""
    phi, vn = _fields(41, 100, 3)
    vn = np.concatenate([vn.reshape(-1), np.zeros(10, np.float32)]).reshape(411, 10)
    phi = np.resize(phi, vn.shape)
    vn.reshape(-1)[at] = bad
    with pytest.raises(L.LithoError):
        L.LevelSetUtils.rk2_update(phi, vn, 1.0, 1.0, 0.5, 0.01)
