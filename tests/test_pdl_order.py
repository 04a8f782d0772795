"""Every kernel launched with programmatic stream serialization waits for its
predecessor on every way out: a return before griddepcontrol.wait would end the
kernel, and release its successor, while the predecessor's predecessor still
runs (host-side check of the kernels' source)."""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "wamca-gpu-mi_gb300", "csrc", "*.cu")))


def _kernels(src):
    src = re.sub(r"//[^\n]*", "", src)
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^{;]*\)\s*\{", src):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[at], 0)
            at += 1
        yield m.group(1), src[m.end():at - 1]


def _early_returns(body):
    """Returns that no pdl_wait of an enclosing scope precedes (lambdas' own returns have values)."""
    waited, bad = [False], []
    for t in re.finditer(r"[{}]|\bpdl_wait\(\)|\breturn\s*;", body):
        if t.group() == "{":
            waited.append(waited[-1])
        elif t.group() == "}":
            waited.pop()
        elif t.group().startswith("return"):
            if not waited[-1]:
                bad.append(body[max(0, t.start() - 80):t.end()])
        else:
            waited[-1] = True
    return bad


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_return_before_the_wait(path):
    for name, body in _kernels(open(path).read()):
        if "pdl_launch_dependents()" in body:
            assert "pdl_wait()" in body, name
            assert not _early_returns(body), (name, _early_returns(body))


def test_the_kernels_are_found():
    names = {n for p in SOURCES for n, b in _kernels(open(p).read()) if "pdl_launch_dependents()" in b}
    assert {"k_sweep", "k_sweep_dvnd", "k_sweep_dvnd2", "k_sweep_dvnd_wide", "k_merge", "k_merge_solo", "k_merge_one",
            "k_total_select", "k_total_finish"} <= names
