"""litho_ctx_reserve against what the calls that it is for allocate, device and pinned memory
alike. Runs without a GPU, in a child process whose CUDA runtime is tests/fake_cudart: the
library's host side as it is, no kernel run, every allocation counted."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, importlib, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
fake = ctypes.CDLL(sys.argv[2])
allocs = ctypes.c_int.in_dll(fake, "fake_allocs")
lib = importlib.import_module("c-version-lithography_b200").load_library()
N, K, nk, batch = 64, 3, 9, int(sys.argv[4])
ctx, cache = ctypes.c_void_p(), ctypes.c_void_p()
assert lib.litho_ctx_create(0, ctypes.c_void_p(1), ctypes.byref(ctx)) == 0
assert lib.litho_ctx_set_precision(ctx, {"fp32": 0, "bf16x3": 1}[sys.argv[3]]) == 0
assert lib.litho_ctx_enable_graphs(ctx, 0) == 0
kb = np.ones((K, nk, nk, 2))
pd = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
w = np.ones(K)
assert lib.litho_cache_create_band(ctx, N, K, nk, nk, -4, -4, pd(kb), pd(w), 3.0, ctypes.byref(cache)) == 0
images = np.zeros((4, batch, N, N), np.float32)
x, y, z, m = (a.ctypes.data for a in images)
res = np.zeros((2, 2 * batch))
assert lib.litho_ctx_reserve(ctx, cache, batch) == 0
reserved = allocs.value
calls = {
    "ctm_evaluate_batch": lambda: lib.litho_ctm_evaluate_batch(
        ctx, cache, batch, x, y, 0.225, 50.0, z, pd(res[0]), pd(res[1])),
    "pe_gradient_batch": lambda: lib.litho_pe_gradient_batch(
        ctx, cache, batch, x, y, 0.225, 50.0, z, pd(res[0])),
    "rk2_update_batch": lambda: lib.litho_lsm_rk2_update_batch(
        ctx, batch, N, N, x, y, 1.0, 1.0, 0.5, 0.01, z, m, pd(res[0])),
    "pe_gradient_batch_device": lambda: lib.litho_pe_gradient_batch_device(
        ctx, cache, batch, x, y, 0.225, 50.0, 1.0, z, res.ctypes.data),
    "rk2_update_batch_device": lambda: lib.litho_lsm_rk2_update_batch_device(
        ctx, batch, N, N, x, y, 1.0, 1.0, 0.5, 0.01, z, m, res.ctypes.data),
}
for name, call in calls.items():
    before = allocs.value
    assert call() == 0, name
    print(name, allocs.value - before)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not shutil.which("gcc"):
        pytest.skip("gcc is missing")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-Wall", "-Werror",
                    os.path.join(ROOT, "tests", "fake_cudart", "fake_cudart.c"), "-o", so], check=True)
    return so


@pytest.mark.parametrize("batch", [1, 16, 19, 100])
@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
def test_reserved_calls_allocate_nothing(fake, precision, batch):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, fake, precision, str(batch)],
                       env={**os.environ, "LD_PRELOAD": fake}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    took = dict(line.split() for line in r.stdout.splitlines())
    assert len(took) == 5 and set(took.values()) == {"0"}, took
