"""A call of which a kernel launch fails reports LITHO_ERR_CUDA, leaves no error behind in the CUDA
runtime that the caller's next check of it would take for its own, and the next call works: each
launch of each call fails in turn, once. Runs without a GPU, in a child process whose CUDA runtime is
tests/fake_cudart (no kernel runs)."""
import os
import subprocess
import sys

import pytest

from test_alloc_failures import CHILD, ROOT, fake  # noqa: F401  (the calls and the runtime)

LOOP = r"""
launch_fail = ctypes.c_int.in_dll(fake, "fake_launch_fail")
last = ctypes.c_int.in_dll(fake, "fake_last")
for name, call in calls.items():
    k = 1
    while True:
        ctx, cache, part = fresh()
        launch_fail.value = k
        st = call(ctx, cache, part)
        hit = launch_fail.value == 0
        launch_fail.value = 0
        if not hit:
            assert st == 0, (name, st)
            break
        print(name, k, st, last.value, flush=True)
        assert st == 5, (name, k, st)
        assert last.value == 0, (name, k, "an error left behind")
        assert call(ctx, cache, part) == 0, (name, k)
        k += 1
    assert k > 3, name
"""


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
def test_calls_recover_from_failed_launches(fake, precision):  # noqa: F811
    setup = CHILD[:CHILD.index("for name, call in calls.items():")]
    r = subprocess.run([sys.executable, "-c", setup + LOOP, ROOT, fake, precision],
                       env={**os.environ, "LD_PRELOAD": fake}, capture_output=True, text=True)
    assert r.returncode == 0, (r.stdout[-300:], r.stderr[-300:])
