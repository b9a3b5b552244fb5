"""The persistent tensor-core pipelines against the per-tile kernels over band sizes, square and
not: row counts that are no multiple of the 8-column groups or of 16, operands with and without a
half-full last atom, the smallest ones, and those that do not fit beside each other in shared
memory (2 x 43 and 2 x 48 rows). Same products in the same order: bit for bit, but for the FP64
loss and norm sums (FP32 over 32 pixels in the pipelines): 1e-6 relative."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nc", [(3, 3), (8, 8), (13, 13), (21, 21), (32, 32), (39, 40), (40, 40),
                                   (43, 43), (48, 48), (9, 45), (45, 9)])
def test_schedules_agree(nr, nc):
    L = importlib.import_module("c-version-lithography_b200")
    WL = importlib.import_module("c-version-lithography_b200.workloads")
    N, B = 1030, 6   # 486 tiles: three or four in turn per CTA
    nk = max(nr, nc)
    band, _, _, w, wss = WL.synthetic_socs_band(K=5, nk=nk)
    a, b = (nk - nr) // 2, (nk - nc) // 2
    band = np.ascontiguousarray(band[:, a:a + nr, b:b + nc])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(nr * 64 + nc)
    x = torch.rand(B, N, N, generator=gen, device="cuda")
    t = (torch.rand(B, N, N, generator=gen, device="cuda") > 0.5).float()
    out = []
    for sched in ("per_tile", "persistent"):
        ctx = L.Context()
        ctx.set_precision("bf16x3")
        ctx.set_tc_schedule(sched)
        cache = L.ImagingCache.from_band(N, band, -(nr // 2), -(nc // 2), w, wss, ctx=ctx)
        losses, grads = L.pe_gradient_batch(cache, x, t, 0.225, 50.0)
        closs, cgrads, norms = L.ctm_evaluate_batch(cache, 3.0 * x, t, 0.225, 50.0)
        out.append((grads.clone(), cgrads.clone(), np.array([losses, closs, norms])))
        ctx.close()
    (g0, c0, s0), (g1, c1, s1) = out
    assert torch.isfinite(g0).all() and g0.abs().max() > 0
    assert torch.equal(g0, g1) and torch.equal(c0, c1)
    assert np.all(np.abs(s0 - s1) <= 1e-6 * np.abs(s0))
