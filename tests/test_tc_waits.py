"""The waits of the persistent tensor-core pipelines (csrc/tc3.cu) give up after a limit, and the
kernel is to return then. Their roles use warp-wide instructions between the waits (tcgen05.ld,
shuffles, votes, __syncwarp), so a warp has to give up as a whole: a lane that left its loop alone
would leave the others waiting for it at the next of these instructions, without a limit. A wait
that runs out cannot be arranged in the kernels from outside, so the source is read: every wait
goes through pwait_warp, which votes on each test and on each reason to give up, and none is made
by some of a warp's lanes."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "c-version-lithography_b200", "csrc", "tc3.cu")
WAITS = ("pwait_warp", "epi_take", "collect2")


def _code():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _function(code, name):
    at = re.search(r"__device__ __forceinline__ bool %s\(.*?\)\s*\{" % name, code, re.S)
    depth, i = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(code[i], 0)
        i += 1
    return code[at.end():i]


def test_every_wait_is_a_whole_warps():
    code = _code()
    wait = _function(code, "pwait_warp")
    # each test of the barrier, of the failure flag and of the clock is the warp's
    assert wait.count("mbar_try_wait") == len(re.findall(r"__all_sync\(ALL, tc::mbar_try_wait\(", wait)) == 2
    assert len(re.findall(r"if \(__any_sync\(ALL, (?:\*fail|clock64\(\) - t0 > )", wait)) == 2
    rest = code.replace(wait, "")
    assert "mbar_try_wait" not in rest
    assert not re.search(r"\bpwait\(", rest)
    # the only other waits are those for copies and MMAs in flight after a failure, after the
    # loops, where no warp-wide instruction follows
    tails = re.findall(r"if \(\*vfail\) \{(.*?)\n    \}", rest, re.S)
    assert len(tails) == 3 and sum(t.count("mbar_wait(") for t in tails) == rest.count("mbar_wait(")


def test_no_wait_is_made_by_some_lanes():
    code = _code()
    calls = 0
    for name in WAITS:
        for m in re.finditer(r"\b%s(?:<\d>)?\(" % name, code):
            start = max(code.rfind(c, 0, m.start()) for c in ";{}")
            before = code[start + 1:m.start()]
            # the condition of a block that the call opens: if (...) { double t[2]; if (take(...
            opened = code[max(code.rfind("if (", 0, start), 0):m.start()] if "double t" in code[start - 30:start] else ""
            if "bool" in before:
                continue
            calls += 1
            assert "lane" not in before and "threadIdx" not in before, before
            assert not re.match(r"if \([^{]*lane", opened), opened
    assert calls >= 30
