"""Results do not depend on what the context's scratch memory held before a call: every path on image
sizes that are no multiple of its tiles, where tiles and operands reach past the image's edge, after
a level-set update that left the scratch full of zeros and after one that left it full of NaN. Bit
for bit, losses and norms included."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [67, 130, 131, 257])
@pytest.mark.parametrize("mode", ["fp32", "per_tile", "persistent"])
def test_scratch_contents_do_not_matter(mode, N):
    L = importlib.import_module("c-version-lithography_b200")
    FC = importlib.import_module("c-version-lithography_b200.fullchip")
    WL = importlib.import_module("c-version-lithography_b200.workloads")
    ctx = L.Context()
    if mode != "fp32":
        ctx.set_precision("bf16x3")
        ctx.set_tc_schedule(mode)
    band, r0, c0, w, wss = WL.synthetic_socs_band(K=5, nk=13)
    cache = L.ImagingCache.from_band(N, band, r0, c0, w, wss, ctx=ctx)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(N)
    B = 5
    x = torch.rand(B, N, N, generator=gen, device="cuda")
    t = (torch.rand(B, N, N, generator=gen, device="cuda") > 0.5).float()
    img, opt = L.Imaging(cache), L.CTMOptimizer(cache, t[0], 0.225, 50.0, iterations=1)
    gradient = L.Gradient(cache, 0.225, 50.0)
    part = FC.Partition(N, N + 4, 2, 1, 20, 3, ctx=ctx)   # micro tiles of about half the height
    tiles = L.ImagingCache.from_band(part.tile_size, band, r0, c0, w, wss, ctx=ctx)
    target = (torch.rand(N, N + 4, generator=gen, device="cuda") > 0.5).float()
    masks = part.extract_all(target) * 0.9
    exchange = FC.MicroGradientExchange(part, tiles, 0.225, 50.0)
    big = torch.empty(48, 1024, 1024, device="cuda")
    still = torch.zeros_like(big)
    out = torch.empty_like(big)

    def fill(value):   # the update's first stage is its scratch: phi where the speed is zero
        big.fill_(value)
        L.LevelSetUtils.rk2_update_batch(big, still, 1.0, 1.0, 0.5, 0.0, out, ctx=ctx)

    def results(value):
        got = []
        fill(value)
        r = img.compute(x[0], 0.225, 50.0)
        got += [r.aerial_image.clone(), r.wafer_image.clone()]
        wafer, field = r.wafer_image.clone(), img.get_electric_field()
        fill(value)
        got += [gradient.pe_gradient_with_penalty(wafer, t[0], field, 2.0, 0.01).clone(), gradient.last_loss]
        fill(value)
        loss, g, norm = opt.evaluate(3.0 * x[0])
        got += [loss, g.clone(), norm]
        fill(value)
        losses, g = L.pe_gradient_batch(cache, x, t, 0.225, 50.0)
        got += [list(losses), g.clone()]
        fill(value)
        losses, g, norms = L.ctm_evaluate_batch(cache, 3.0 * x, t, 0.225, 50.0)
        got += [list(losses), g.clone(), list(norms)]
        for metrics in (False, True):
            fill(value)
            e = exchange.compute(masks, target, FC.MicroGradientOptions(
                loss_type="PEPenalty", enable_cept=True, collect_core_metrics=metrics))
            got += [e.raw_gradients.clone(), e.mask_gradients.clone(), e.loss]
        return got
    for a, b in zip(results(0.0), results(float("nan"))):
        if isinstance(a, torch.Tensor):
            assert torch.isfinite(a).all() and torch.equal(a, b)
        else:
            assert np.all(np.isfinite(a)) and a == b
    ctx.close()
