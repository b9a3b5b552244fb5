"""Batches over wide bands, whose row-grouped small-grid kernels fit one CTA per SM and choose their rows
per CTA by the waves that they take: every image of a batch as alone, bit for bit, for both
kernels on either side of that rule and with rows left over in the last CTA."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nc", [(43, 43), (47, 48), (40, 64), (58, 58), (64, 61)])
@pytest.mark.parametrize("batch", [4, 9, 16])
def test_batch_is_single(nr, nc, batch):
    L = importlib.import_module("c-version-lithography_b200")
    N, K = 150, 4
    rng = np.random.default_rng(nr * 100 + nc)
    band = (rng.standard_normal((K, nr, nc)) + 1j * rng.standard_normal((K, nr, nc))) * 0.5 / np.sqrt(nr * nc)
    ctx = L.Context()
    ctx.set_precision("bf16x3")
    cache = L.ImagingCache.from_band(N, band, -(nr // 2), -(nc // 2), 0.8 ** np.arange(K), 1.0, ctx=ctx)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(batch)
    x = 3.0 * torch.rand(batch, N, N, generator=gen, device="cuda")
    t = (torch.rand(batch, N, N, generator=gen, device="cuda") > 0.5).float()
    losses, grads, norms = L.ctm_evaluate_batch(cache, x, t, 0.225, 50.0)
    assert torch.isfinite(grads).all() and grads.abs().max() > 0
    for b in range(0, batch, 3):
        loss, g, norm = L.CTMOptimizer(cache, t[b], 0.225, 50.0, iterations=1).evaluate(x[b].clone())
        assert torch.equal(grads[b], g) and losses[b] == loss and norms[b] == norm
    ctx.close()
