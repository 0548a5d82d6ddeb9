"""Kernels that are set up while the launch before them still runs
(launch_after) wait for it before they touch what it writes, and promise
nothing about that data: a const __restrict__ parameter is read-only for the
life of a kernel, which is not so up to the wait.  Checked on the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "emsolvers_gb300", "csrc")


def _closing(s, i, o, c):
    n = 0
    while True:
        n += (s[i] == o) - (s[i] == c)
        if n == 0:
            return i
        i += 1


def _kernels(path):
    """(name, parameter list, body) of every kernel of a source file."""
    s = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__global__\s+void\s+", s):
        i = m.end()
        if s.startswith("__launch_bounds__", i):
            i = _closing(s, s.index("(", i), "(", ")") + 1
        a = s.index("(", i)
        b = _closing(s, a, "(", ")")
        body = s.index("{", b)
        yield s[i:a].strip(), s[a + 1:b], s[body:_closing(s, body, "{", "}") + 1]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_kernels_launched_ahead_wait_and_promise_nothing(path):
    kernels = {name: (params, body) for name, params, body in _kernels(path)}
    ahead = set(re.findall(r"launch_after\((\w+_kernel)\b", open(path).read()))
    for name in ahead:
        assert "wait_for_last()" in kernels[name][1], name + " is launched ahead and does not wait"
    for name, (params, body) in kernels.items():
        if "wait_for_last()" in body:
            assert "__restrict__" not in params, name


def test_captures_end_on_every_path():
    """Only Sim::capture begins a stream capture: it ends it also when a launch
    inside fails, which would leave the handle's stream capturing."""
    for path in glob.glob(os.path.join(CSRC, "*")):
        text = open(path).read()
        assert text.count("cudaStreamBeginCapture(") == (1 if path.endswith("ems_internal.hpp") else 0), path
