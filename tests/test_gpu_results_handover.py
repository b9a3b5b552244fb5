"""Results and status of a call reach the host through pinned memory that its last kernel
writes, and the reduction header is cleared there: a call that saw a non-finite input must not
colour the next one, in any order of the entry points that share the header."""
import importlib

import numpy as np
import pytest
import torch

L = importlib.import_module("c-version-lithography_b200")
WL = importlib.import_module("c-version-lithography_b200.workloads")

pytestmark = pytest.mark.gpu
N = 64


def _calls(precision):
    ctx = L.Context(stream=torch.cuda.Stream())
    ctx.set_precision(precision)
    band, r0, c0, w, wss = WL.synthetic_socs_band(K=6, nk=13)
    cache = L.ImagingCache.from_band(N, band, r0, c0, w, wss, ctx=ctx)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    x = torch.rand(40, N, N, generator=gen, device="cuda")
    t = (x > 0.5).float()
    torch.cuda.synchronize()
    opt = L.CTMOptimizer(cache, t[0], 0.225, 50.0, iterations=1)
    img = L.Imaging(cache)
    return {
        "ctm": lambda v: opt.evaluate(v[0])[0],
        "ctm_batch": lambda v: L.ctm_evaluate_batch(cache, v, t, 0.225, 50.0)[0],
        "pe_batch": lambda v: L.pe_gradient_batch(cache, v, t, 0.225, 50.0)[0],
        "imaging": lambda v: float(img.compute(v[0], 0.225, 50.0).aerial_image.sum()),
        "rk2": lambda v: L.LevelSetUtils.rk2_update(t[0], v[0], 1.0, 1.0, 0.5, 0.01, ctx=ctx)[2],
        "rk2_batch": lambda v: L.LevelSetUtils.rk2_update_batch(
            t, v, 1.0, 1.0, 0.5, 0.01, torch.empty_like(t), ctx=ctx),
        "dt": lambda v: L.LevelSetUtils.evolution_term(t[0], v[0], 1.0, 1.0, 0.5, 0.01, ctx=ctx)[1],
    }, x


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
def test_every_call_starts_from_a_clear_header(precision):
    calls, x = _calls(precision)
    bad = x.clone()
    bad[0, 3, 5] = float("nan")
    torch.cuda.synchronize()
    want = {}
    for name, call in calls.items():    # each twice: the graph path too, then once more
        want[name] = call(x)
        for _ in range(3):
            assert np.array_equal(call(x), want[name]), name
    for first, call in calls.items():
        for second, other in calls.items():
            with pytest.raises(L.LithoError):
                call(bad)
            assert np.array_equal(other(x), want[second]), (first, second)
