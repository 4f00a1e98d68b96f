"""Bins of the row top-K's histogram: never falling with the similarity, over all
non-negative floats, those outside the admitted range included."""
import ctypes as C
import os
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))


def test_bins_never_fall(tmp_path):
    so = str(tmp_path / "libbins.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared",
                    os.path.join(HERE, "native", "sim_bins_host.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    sims = np.concatenate([[0.0, 1e-30, 0.03125, 0.039, 0.5, 1.0 - 1e-6, 1.0, 1.0001, 2.0, 1e30],
                           np.linspace(0.0, 1.2, 5001)]).astype(np.float32)
    sims = np.unique(np.concatenate([sims, np.nextafter(sims, np.float32(3e38)),
                                     np.nextafter(sims, np.float32(0))]))
    bins = [lib.host_sim_bin(int(b)) for b in sims.view(np.uint32)]
    assert bins[0] == 0 and bins[-1] == lib.host_bins() - 1
    assert all(a <= b for a, b in zip(bins, bins[1:]))
    assert lib.host_sim_bin(int(np.float32(1.0).view(np.uint32))) == lib.host_bins() - 1
