"""The pinned staging buffer grows by half its size, and asks for the exact size
where the grown one cannot be pinned."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def hbuf(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("hbuf") / "hbuf")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(CUDA, "include"),
                    os.path.join(HERE, "native", "hbuf_host.cpp"), "-o", exe], check=True)

    def run(limit, *sizes):
        r = subprocess.run([exe, str(limit)] + [str(s) for s in sizes], check=True,
                           capture_output=True, text=True)
        return [int(x) for x in r.stdout.split()]
    return run


@pytest.mark.parametrize("limit,sizes,want", [
    (1 << 20, [1, 1000, 1200, 100], [256, 1000, 1500, 1500]),       # by half
    (1300, [1000, 1200], [1000, 1200]),                             # the exact size
    (1300, [1000, 1301, 900], [1000, -1, 900]),                     # refused, usable afterwards
])
def test_growth(hbuf, limit, sizes, want):
    assert hbuf(limit, *sizes) == want
