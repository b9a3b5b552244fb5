"""Device memory that the full-chip exchange holds per tile: nothing where its fused kernel forms
targets and windows itself and the caller takes the raw gradients, else a tile image for each of
targets, two windows and raw gradients that it needs; grown when a later call needs more, and not
taken again. Runs without a GPU, in a child process whose CUDA runtime is tests/fake_cudart."""
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
sizes = (ctypes.c_size_t * 4096).in_dll(fake, "fake_sizes")
L = importlib.import_module("c-version-lithography_b200")
lib = L.load_library()
pd = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
ctx, cache, part = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
assert lib.litho_ctx_create(0, ctypes.c_void_p(1), ctypes.byref(ctx)) == 0
assert lib.litho_ctx_set_precision(ctx, 1) == 0
assert lib.litho_partition_create(ctx, 192, 192, 2, 2, 16, 4, ctypes.byref(part)) == 0
n, ts = 4, 128
kb, w = np.ones((3, 9, 9, 2)), np.ones(3)
assert lib.litho_cache_create_band(ctx, ts, 3, 9, 9, -4, -4, pd(kb), pd(w), 3.0, ctypes.byref(cache)) == 0
images = np.zeros((4, n, ts, ts), np.float32)
x, y, m, t = (a.ctypes.data for a in images)
totals, res = np.zeros(3), np.zeros(17 * n)
o = L.ExchangeOptionsC(1, 0, 1.0, 1.0, 0.01, 1, 1, 1.0, 1, 0, 1.0, 1.0)
for arg in sys.argv[3:]:
    schedule, raw, metrics = arg.split("-")
    assert lib.litho_ctx_set_tc_schedule(ctx, {"auto": 0, "tile": 1}[schedule]) == 0
    e = L.ExchangeEpeC(1.0, 2, 1.0, int(metrics), None, None, 0)
    before = allocs.value
    st = lib.litho_exchange_compute_epe(ctx, part, cache, x, y, 0.225, 50.0, ctypes.byref(o), ctypes.byref(e),
                                        t if raw == "raw" else None, m, pd(res), pd(totals))
    assert st == 0, (st, lib.litho_ctx_last_error(ctx))
    per = n * ts * ts * 4
    print(sum(sizes[i] // per for i in range(before, allocs.value) if sizes[i] % per == 0 and sizes[i] // per < 5))
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not shutil.which("gcc"):
        pytest.skip("gcc is missing")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-Wall", "-Werror",
                    os.path.join(ROOT, "tests", "fake_cudart", "fake_cudart.c"), "-o", so], check=True)
    return so


# schedule - raw gradients - Core metrics of successive calls, images per tile each of them takes
@pytest.mark.parametrize("calls,images", [
    (["auto-raw-0", "auto-raw-0"], [0, 0]),
    (["auto-own-0", "auto-own-0", "auto-raw-0"], [1, 0, 0]),
    (["tile-raw-0", "auto-raw-0", "auto-own-0"], [3, 0, 0]),
    (["auto-raw-0", "tile-own-0", "tile-raw-0"], [0, 4, 0]),
    (["auto-own-0", "auto-raw-1"], [1, 3]),
])
def test_images_per_tile(fake, calls, images):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, fake, *calls],
                       env={**os.environ, "LD_PRELOAD": fake}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-400:]
    assert [int(v) for v in r.stdout.split()] == images
