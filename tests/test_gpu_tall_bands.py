"""GPU parity of the FP32 path (csrc/band_dft.cu) for bands with many rows, whose row twiddles
and synthesis operands do not fit in a CTA's shared memory and are taken in pieces: on both
sides of the limits (226 and 227 rows for the synthesis), one, two and three pieces, and each
column variant that hands over to the pieces by its number of tiles and columns. Against the
FP64 oracle at the FP32 mode's tolerances (aerial 1e-5 of peak, gradient 1e-4 relative L2, PE
1e-5 relative); in split BF16 such bands run the same kernels, bit for bit."""
import importlib

import numpy as np
import pytest

from oracle import imaging_oracle as io

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _band(nr, nc, K):
    """A pass at DC and random sidelobes over the whole band."""
    rng = np.random.default_rng(nr * 1000 + nc)
    band = rng.standard_normal((K, nr, nc)) + 1j * rng.standard_normal((K, nr, nc))
    band *= 0.5 / np.sqrt(nr * nc)
    band[0, nr // 2, nc // 2] += 1.0
    return band, -(nr // 2), -(nc // 2), 0.5 ** np.arange(K), 1.5


@pytest.mark.parametrize("nr,nc,N", [(200, 9, 256), (200, 9, 1280), (200, 35, 700), (165, 49, 1280),
                                     (226, 5, 384), (227, 5, 385), (300, 5, 1283), (460, 3, 512)])
def test_forward_and_adjoint(nr, nc, N):
    L = importlib.import_module("c-version-lithography_b200")
    wl = importlib.import_module("c-version-lithography_b200.workloads")
    band, r0, c0, w, wss = _band(nr, nc, 2)
    rng = np.random.default_rng(N)
    target = (rng.random((N, N)) < 0.4).astype(np.float64)
    theta = io.initialize_theta(target) + 0.2 * rng.standard_normal((N, N))
    oc = io.OracleCache(N=N, kernels=list(wl.band_to_dense(band, r0, c0, N)),
                        source_ws=np.array([wss]), eigenvalues=tuple(w))
    ref = io.ctm_evaluate(theta, target, oc, 0.225, 50.0)
    out = []
    for precision in ("fp32", "bf16x3"):
        ctx = L.Context()
        ctx.set_precision(precision)
        cache = L.ImagingCache.from_band(N, band, r0, c0, w, wss, ctx=ctx)
        got = L.Imaging(cache).compute(ref["mask"], 0.225, 50.0)
        peak = np.max(ref["aerial"])
        assert np.max(np.abs(got.aerial_image.double().cpu().numpy() - ref["aerial"])) <= 1e-5 * peak
        opt = L.CTMOptimizer(cache, target, 0.225, 50.0, iterations=1)
        loss, g, norm = opt.evaluate(torch.tensor(theta, dtype=torch.float32, device="cuda"))
        out.append((got.aerial_image.clone(), g.clone()))
        g = g.double().cpu().numpy()
        assert abs(loss - ref["loss"]) <= 1e-5 * ref["loss"]
        assert np.linalg.norm(g - ref["grad_theta"]) <= 1e-4 * ref["grad_norm"]
        assert abs(norm - ref["grad_norm"]) <= 1e-4 * ref["grad_norm"]
        ctx.close()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
