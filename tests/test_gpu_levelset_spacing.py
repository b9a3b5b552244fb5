"""The level-set stencil (csrc/levelset.cu) with spacings far from 1, as of lengths in metres:
outside 2^-12 .. 2^12 it divides every difference by the spacing first. Against the FP64 oracle
on both sides of either border and far beyond, on images with one and with several tiles and
with pixels of every border case. And a power of two in the spacing, the signed distance and
nothing else changes no rounding of a step without curvature: bit for bit the step of spacing 1,
single, batched and in update windows."""
import importlib

import numpy as np
import pytest

from oracle import levelset_oracle as lo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# FP32 against FP64: the bound of the random fields in test_gpu_levelset.py.
TOL = 2e-5
CFL = 0.5


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
    vn[rng.random((rows, cols)) < 0.1] = 0.0
    return phi.astype(np.float32), vn.astype(np.float32)


def _close(got, want):
    got = got.double().cpu().numpy()
    assert np.max(np.abs(got - want)) <= TOL * np.max(np.abs(want))


@pytest.mark.parametrize("shape", [(3, 4), (9, 65), (33, 68), (300, 257)])
@pytest.mark.parametrize("scale", [1e-15, 1e-12, 1e-9, 0.99 / 4096, 1.01 / 4096, 4090.0, 4100.0, 1e9])
def test_spacings_match_oracle(L, scale, shape):
    phi, vn = _fields(*shape, seed=sum(shape))
    phi = phi * np.float32(scale)
    dx, dy = scale, 0.999 * scale
    p64, v64 = phi.astype(np.float64), vn.astype(np.float64)
    e = L.LevelSetUtils.evolve_normal_WENO_godunov(phi, vn, dy, dx)
    _close(e.delta, lo.evolve_normal_weno_godunov(p64, v64, dy, dx)[0])
    for b in (0.01, 0.01 * scale):
        _close(L.LevelSetUtils.evolve_kappa(phi, dx, dy, b), lo.evolve_kappa(p64, dx, dy, b))
    b = 0.01 * scale
    got, mask, dt = L.LevelSetUtils.rk2_update(phi, vn, dx, dy, CFL, b)
    want, want_dt = lo.lsm_rk2_update(p64, v64, dx, dy, CFL, b)
    _close(got, want)
    assert abs(dt - want_dt) <= 1e-6 * want_dt
    assert torch.equal(mask, (got >= 0).float())


@pytest.mark.parametrize("shape", [(3, 4), (33, 68), (300, 257)])
def test_power_of_two(L, shape):
    s = 2.0 ** -40
    phi, vn = (torch.from_numpy(a).cuda() for a in _fields(*shape, seed=1))
    U = L.LevelSetUtils
    for f in (s, 1 / s):
        assert torch.equal(U.evolve_normal_WENO_godunov(phi * f, vn, f, f).delta,
                           U.evolve_normal_WENO_godunov(phi, vn, 1.0, 1.0).delta)
    one, mask1, dt1 = U.rk2_update(phi, vn, 1.0, 1.0, CFL, 0.0)
    got, mask, dt = U.rk2_update(phi * s, vn, s, s, CFL, 0.0)
    assert torch.equal(got, one * s) and torch.equal(mask, mask1) and dt == dt1 * s
    phis, vns = (torch.stack([a, a.flip(0), -a]) for a in (phi, vn))
    out, want = torch.empty_like(phis), torch.empty_like(phis)
    dts = U.rk2_update_batch(phis * s, vns, s, s, CFL, 0.0, out)
    want_dts = U.rk2_update_batch(phis, vns, 1.0, 1.0, CFL, 0.0, want)
    assert torch.equal(out, want * s) and np.array_equal(np.array(dts), np.array(want_dts) * s)


def test_power_of_two_in_windows(L):
    FC = importlib.import_module("c-version-lithography_b200.fullchip")
    wl = importlib.import_module("c-version-lithography_b200.workloads")
    s = 2.0 ** -40
    rng = np.random.default_rng(4)
    target = np.kron(rng.random((10, 10)) < 0.5, np.ones((20, 20))).astype(np.float32)
    res = []
    for dx in (1.0, s):
        ctx = L.Context()
        part = FC.Partition(200, 200, 2, 2, 40, 16, ctx=ctx)
        band, r0, c0, w, wss = wl.synthetic_socs_band(K=4, nk=15)
        cache = L.ImagingCache.from_band(part.tile_size, band, r0, c0, w, wss, ctx=ctx)
        opt = FC.FullChipLSMOptions(iterations=4, dx=dx, dy=dx, curvature_weight=0.0, reinit_interval=3,
                                    gradient_options=FC.MicroGradientOptions(loss_type="PEPenalty"))
        r = FC.FullChipLSMOptimizer(part, cache, 0.225, 50.0).optimize(target, target, opt)
        res.append((r.local_phi.clone() / dx, [(h.loss, h.min_dt / dx, h.max_dt / dx) for h in r.history]))
        ctx.close()
    assert torch.equal(res[0][0], res[1][0]) and res[0][1] == res[1][1]
