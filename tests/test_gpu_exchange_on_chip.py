"""The exchange with the persistent fused kernel, which reads the layout and forms the loss
windows itself, against the per-tile schedule, which takes extracted targets and window
images: the same split-BF16 products and epilogue arithmetic per pixel, so raw and exchanged
gradients agree bit for bit; the FP64 loss sums add FP32 sums over other groups of pixels
(1e-6 relative, as in test_gpu_tc_schedule.py). Cases: layouts smaller than a tile (the
periodic rows wrap inside a 32-row segment), odd layouts, every loss region and both loss
types, and a raw buffer that the caller leaves to the library."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    p = importlib.import_module("c-version-lithography_b200")
    p.load_library()
    return p


@pytest.mark.parametrize("loss", ["PE", "PEPenalty"])
@pytest.mark.parametrize("region", ["Core", "CoreGuard"])
@pytest.mark.parametrize("H,W,rows,cols,halo,guard", [(40, 56, 2, 1, 40, 8), (301, 203, 2, 3, 33, 9),
                                                      (512, 512, 2, 2, 64, 16)])
def test_matches_per_tile_schedule(L, loss, region, H, W, rows, cols, halo, guard):
    FC = importlib.import_module("c-version-lithography_b200.fullchip")
    wl = importlib.import_module("c-version-lithography_b200.workloads")
    band, r0, c0, w, wss = wl.synthetic_socs_band(K=6, nk=21)
    rng = np.random.default_rng(H)
    target = torch.tensor(rng.random((H, W)) < 0.4, dtype=torch.float32, device="cuda")
    out = {}
    for sched in ("per_tile", "persistent"):
        ctx = L.Context()
        ctx.set_precision("bf16x3")
        ctx.set_tc_schedule(sched)
        part = FC.Partition(H, W, rows, cols, halo, guard, ctx=ctx)
        cache = L.ImagingCache.from_band(part.tile_size, band, r0, c0, w, wss, ctx=ctx)
        masks = part.extract_all(target) * 0.9
        ex = FC.MicroGradientExchange(part, cache, 0.225, 50.0)
        r = ex.compute(masks, target, FC.MicroGradientOptions(
            loss_type=loss, loss_region=region, enable_cept=True, enable_grad_fusion=True))
        out[sched] = (r.raw_gradients.clone(), r.mask_gradients.clone(),
                      [(t.pe_loss, t.penalty_loss, t.loss) for t in r.locals])
        ctx.close()
    a, b = out["per_tile"], out["persistent"]
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    assert a[0].abs().max().item() > 0.0
    for x, y in zip(a[2], b[2]):
        for u, v in zip(x, y):
            assert abs(u - v) <= 1e-6 * max(abs(u), 1e-12)
