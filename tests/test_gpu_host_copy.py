"""Pageable host memory through the pinned slots: sizes around a slot (8 MB) and
below the direct limit (1 MB), in and out, against plain numpy and the oracle."""
import numpy as np
import pytest

from rabbitbin_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb,m", [(10, 20, 17), (400, 2622, 40), (1024, 1024, 130),
                                     (1025, 2049, 130), (60, 9000, 257)])
def test_pageable_in_and_out(gpu_ctx, na, nb, m):
    rng = np.random.default_rng(na + nb)
    base = rng.integers(1, 2**62, size=(7, m), dtype=np.uint64)

    def rows(n):
        own = rng.integers(1, 2**62, size=(n, m), dtype=np.uint64)
        return np.where(rng.random((n, m)) < 0.5, base[rng.integers(0, 7, n)], own)
    A, B = rows(na), rows(nb)
    got = gpu_ctx.pmh_compare("jaccard_weighted", A, B)
    want = np.empty((na, nb))
    for i in range(na):
        want[i] = (A[i] == B).sum(axis=1) / np.float64(m)
    assert np.array_equal(got, want)
    regs = rng.random((nb, m))
    other = rng.random((nb, m))
    assert np.array_equal(gpu_ctx.pmh_merge_registers(regs, other), np.minimum(regs, other))


# one chunk, and several of 4 MB with contigs across their cuts
@pytest.mark.parametrize("n,length", [(700, 900), (9001, 1500)])
def test_winner_chunks(gpu_ctx, orc, n, length):
    rng = np.random.default_rng(n)
    lens = rng.integers(length // 2, length * 3 // 2, size=n)
    offs = np.zeros(n + 1, np.int64)
    offs[1:] = np.cumsum(lens)
    buf = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, size=int(offs[-1]))].tobytes()
    got = gpu_ctx.build_pmh_winners(buf, offs, api.default_params(m=300))
    assert np.array_equal(got, orc.build_winners(buf, offs, m=300))
