"""GPU parity of the level-set stencil (csrc/levelset.cu) on images of at most 32 columns, which take
narrow tiles, and on the first widths beyond: odd and even, one tile and several rows of tiles, the
divided variant too, against the FP64 oracle; a batch bit for bit as its images alone, and the
full-chip step's update windows in narrow micro tiles."""
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
    vn[rng.random((rows, cols)) < 0.1] = 0.0
    return phi.astype(np.float32), vn.astype(np.float32)


def _close(got, want):
    got = got.double().cpu().numpy()
    assert np.max(np.abs(got - want)) <= TOL * np.max(np.abs(want))


@pytest.mark.parametrize("spacing", [1.0, 1e-9])
@pytest.mark.parametrize("shape", [(3, 3), (16, 16), (15, 31), (17, 32), (16, 33), (48, 5), (33, 30),
                                   (700, 32)])
def test_matches_oracle(L, shape, spacing):
    phi, vn = _fields(*shape, seed=sum(shape))
    phi = phi * np.float32(spacing)
    dx, dy, cfl, b = 2.0 * spacing, 1.5 * spacing, 0.5, 0.01 * spacing
    p64, v64 = phi.astype(np.float64), vn.astype(np.float64)
    e = L.LevelSetUtils.evolve_normal_WENO_godunov(phi, vn, dy, dx)
    _close(e.delta, lo.evolve_normal_weno_godunov(p64, v64, dy, dx)[0])
    _close(L.LevelSetUtils.evolve_kappa(phi, dx, dy, b), lo.evolve_kappa(p64, dx, dy, b))
    got, mask, dt = L.LevelSetUtils.rk2_update(phi, vn, dx, dy, cfl, b)
    want, want_dt = lo.lsm_rk2_update(p64, v64, dx, dy, cfl, b)
    _close(got, want)
    assert abs(dt - want_dt) <= 1e-6 * want_dt
    assert torch.equal(mask, (got >= 0).float())


@pytest.mark.parametrize("batch,rows,cols", [(1000, 16, 16), (700, 40, 31)])
def test_batch_is_single(L, batch, rows, cols):
    f = [_fields(rows, cols, s) for s in range(batch)]
    phi, vn = (torch.from_numpy(np.stack([x[k] for x in f])).cuda() for k in (0, 1))
    out, mask = torch.empty_like(phi), torch.empty_like(phi)
    dts = L.LevelSetUtils.rk2_update_batch(phi, vn, 1.0, 1.0, 0.5, 0.01, out, mask_out=mask)
    for i in range(0, batch, 97):
        one, m, dt = L.LevelSetUtils.rk2_update(phi[i].clone(), vn[i].clone(), 1.0, 1.0, 0.5, 0.01)
        assert torch.equal(out[i], one) and torch.equal(mask[i], m) and dts[i] == dt


def test_update_windows(L):
    """Micro tiles of 30^2: the step of every tile inside its window, the old phi outside."""
    FC = importlib.import_module("c-version-lithography_b200.fullchip")
    import ctypes
    ctx = L.Context()
    part = FC.Partition(44, 44, 2, 2, 4, 2, ctx=ctx)
    n, ts = part.num_tiles, part.tile_size
    assert ts == 30
    phi, speed = (torch.from_numpy(np.stack(a)).cuda() for a in zip(*[_fields(ts, ts, s) for s in range(n)]))
    out, mask = torch.empty_like(phi), torch.empty_like(phi)
    lo_dt, hi_dt = ctypes.c_double(), ctypes.c_double()
    ctx._check(ctx.lib.litho_fullchip_lsm_step(
        ctx.handle, part.handle, phi.data_ptr(), speed.data_ptr(), 1.0, 1.0, 0.5, 0.01, 0, 0, 4,
        out.data_ptr(), mask.data_ptr(), ctypes.byref(lo_dt), ctypes.byref(hi_dt)))
    ctx.synchronize()
    for t in range(n):
        r = (ctypes.c_int * 16)()
        ctx._check(ctx.lib.litho_partition_tile_rects(part.handle, t, r))
        y0, y1, x0, x1 = r[12:16]
        p, v = phi[t].cpu().numpy(), np.zeros((ts, ts), np.float32)
        v[y0:y1, x0:x1] = speed[t].cpu().numpy()[y0:y1, x0:x1]
        # two stages on windowed images, the first one's result outside the window being phi
        p64, v64 = p.astype(np.float64), v.astype(np.float64)
        m = float(np.max(np.abs(v64)))
        dt = 0.5 / (m + m + 0.01 * 2.0 * 2.0)

        def stage(f):
            g = f + dt * (lo.evolve_kappa(f, 1.0, 1.0, 0.01)
                          - lo.evolve_normal_weno_godunov(f, v64, 1.0, 1.0)[0])
            keep = np.zeros((ts, ts), bool)
            keep[y0:y1, x0:x1] = True
            return g, keep
        g, keep = stage(p64)
        p1 = np.where(keep, g, p64)
        g, keep = stage(p1)
        want = np.where(keep, 0.5 * p64 + 0.5 * g, p64)
        _close(out[t], want)
        assert torch.equal(out[t][~torch.from_numpy(keep).cuda()], phi[t][~torch.from_numpy(keep).cuda()])
    ctx.close()
