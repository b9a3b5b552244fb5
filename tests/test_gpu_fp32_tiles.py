"""GPU parity of the FP32 tile analysis and row synthesis (csrc/band_dft.cu) at the edges of
their tilings (64- and 128-pixel tiles, 32-column blocks, rows whose length is no multiple of
four) and on both sides of the column split's size rule, for narrow, odd, even and wide bands,
against the FP64 oracle. Tolerances of the FP32 mode (aerial 1e-5 of peak, gradient 1e-4
relative L2, PE 1e-5 relative)."""
import importlib

import numpy as np
import pytest

from oracle import imaging_oracle as io

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nk", [(63, 21), (64, 21), (65, 21), (127, 35), (130, 8), (257, 52),
                                  (700, 35), (768, 35), (1280, 35), (1283, 9)])
def test_forward_and_adjoint(N, nk):
    L = importlib.import_module("c-version-lithography_b200")
    wl = importlib.import_module("c-version-lithography_b200.workloads")
    K = 3
    band, r0, c0, w, wss = wl.synthetic_socs_band(K=K, nk=nk)
    rng = np.random.default_rng(N)
    target = (rng.random((N, N)) < 0.4).astype(np.float64)
    theta = io.initialize_theta(target) + 0.2 * rng.standard_normal((N, N))
    oc = io.OracleCache(N=N, kernels=list(wl.band_to_dense(band, r0, c0, N)),
                        source_ws=np.array([wss]), eigenvalues=tuple(w))
    ref = io.ctm_evaluate(theta, target, oc, 0.225, 50.0)
    cache = L.ImagingCache.from_band(N, band, r0, c0, w, wss)
    got = L.Imaging(cache).compute(ref["mask"], 0.225, 50.0)
    peak = np.max(ref["aerial"])
    assert np.max(np.abs(got.aerial_image.double().cpu().numpy() - ref["aerial"])) <= 1e-5 * peak
    opt = L.CTMOptimizer(cache, target, 0.225, 50.0, iterations=1)
    loss, g, norm = opt.evaluate(torch.tensor(theta, dtype=torch.float32, device="cuda"))
    g = g.double().cpu().numpy()
    assert abs(loss - ref["loss"]) <= 1e-5 * ref["loss"]
    assert np.linalg.norm(g - ref["grad_theta"]) <= 1e-4 * ref["grad_norm"]
    assert abs(norm - ref["grad_norm"]) <= 1e-4 * ref["grad_norm"]
