"""CPU tests of the kept device blocks (ruai_malloc / ruai_free): block_pool.cpp runs them against a stand-in for the CUDA runtime."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("block_pool") / "block_pool")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(CUDA, "include"), "-o", out, os.path.join(HERE, "block_pool.cpp")], check=True)
    return out


@pytest.mark.parametrize("scenario", [
    "reuse", "last context", "limit", "out of memory",
    "free in a capture", "capture of another context", "request in a capture",
    "freed twice", "freed through another device", "address of a block that cudaFree took",
    "trim during a wait", "out of memory during a wait",
    "used by another stream", "limit with work going on",
    "host memory out",
])
def test_scenario(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
