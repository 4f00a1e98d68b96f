"""Pinned result memory is bounded: no block above what the pool keeps (4 GB), and no
more than that held by callers at a time; a call whose result gets none fills plain
memory with the same values."""
import numpy as np
import pytest

from rabbitbin_b200 import api

pytestmark = pytest.mark.gpu
GB = 1 << 30


def test_bounds(gpu_ctx):
    L, h = gpu_ctx._L, gpu_ctx._h
    assert not L.rbg_result_alloc_on(h, 4 * GB + 1)
    assert not L.rbg_result_alloc(4 * GB + 1)
    assert not L.rbg_result_alloc_on(None, 1 << 20)
    rng = np.random.default_rng(5)
    A, B = rng.random((300, 40)), rng.random((700, 40))
    B[::9] = A[rng.integers(0, 300, len(B[::9]))]
    want = gpu_ctx.pmh_compare("jaccard", A, B).copy()      # (not held)
    held = []
    try:
        for _ in range(2):
            held.append(L.rbg_result_alloc_on(h, 2 * GB - 5))
        assert all(held)
        assert not L.rbg_result_alloc_on(h, 1 << 20)         # 4 GB are held
        assert not L.rbg_result_alloc(1 << 20)
        got = gpu_ctx.pmh_compare("jaccard", A, B)           # 1.7 MB, plain memory
        assert got.flags.owndata and np.array_equal(got, want)
    finally:
        for p in held:
            L.rbg_result_free(p)
    p = L.rbg_result_alloc_on(h, 1 << 20)
    assert p
    L.rbg_result_free(p)
