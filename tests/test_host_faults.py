"""The engine's host code on a fake CUDA runtime (tests/fake_cuda.h): failing
launches and allocations, and calls on a capturing stream."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_tile_count import _cuda_include

CSRC = os.path.join(ROOT, "wamca-gpu-mi_gb300", "csrc")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host") / "host_faults")
    # Uninitialised locals hold a pattern, not what the stack had.
    cmd = ["g++", "-std=c++17", "-O0", "-ftrivial-auto-var-init=pattern", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
           "-I", _cuda_include(), os.path.join(ROOT, "tests", "host_faults.cpp"), os.path.join(CSRC, "mlp_engine.cpp"),
           os.path.join(CSRC, "mlp_capi.cpp"), "-o", out, "-ldl", "-lpthread"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    return out


def _run(exe, check):
    r = subprocess.run([exe, check], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)


def test_failed_batch_result(exe):
    _run(exe, "batch_result")


def test_sweeps_on_a_capturing_stream(exe):
    _run(exe, "captured_sweeps")


def test_constructor_memory(exe):
    _run(exe, "constructor_memory")


def test_constructor_rule(exe):
    _run(exe, "constructor_rule")


def test_without_the_small_search(exe):
    _run(exe, "no_small_search")
