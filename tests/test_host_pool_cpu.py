"""The library's host threads: every part of every job runs once and before the call
returns, over many short jobs whose part counts change, from one caller and from
several."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pool") / "pool")
    subprocess.run(["g++", "-std=c++17", "-O2", "-march=x86-64-v2", "-I", os.path.join(CUDA, "include"),
                    os.path.join(HERE, "native", "pool_host.cpp"), "-o", out, "-lpthread"], check=True)
    return out


@pytest.mark.parametrize("jobs,callers", [(100000, 1), (20000, 3)])
def test_parts_run_once(exe, jobs, callers):
    r = subprocess.run([exe, str(jobs), str(callers)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and int(r.stdout) == 0
