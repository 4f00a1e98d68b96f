"""Sketch comparisons (rbg_pmh_compare) around the kernel's tiles (64 rows a
side, 16 registers a chunk), with unset registers, NaN and zeros of both signs,
and a result large enough to leave in parts: the counted matches, exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(rng, n, m, weighted):
    if weighted:
        r = rng.integers(0, 6, (n, m)).astype(np.uint64) << np.uint64(31)   # 0: unset
        return r | (r != 0) * rng.integers(0, 2, (n, m)).astype(np.uint64)
    r = rng.choice([0.0, -0.0, 1.5, 2.0 ** -40, np.inf, np.nan, -np.inf], (n, m))
    return np.where(rng.random((n, m)) < 0.3, rng.integers(1, 4, (n, m)).astype(np.float64), r)


@pytest.mark.parametrize("na,nb,m", [(1, 1, 2), (63, 65, 15), (64, 64, 16), (65, 63, 17),
                                     (130, 129, 33), (1, 300, 1000), (1100, 2100, 31)])
@pytest.mark.parametrize("metric", ["jaccard_weighted", "jaccard"])
def test_tile_edges(gpu_ctx, na, nb, m, metric):
    rng = np.random.default_rng(na * nb + m)
    A, B = (_rows(rng, n, m, metric == "jaccard_weighted") for n in (na, nb))
    got = gpu_ctx.pmh_compare(metric, A, B)
    unset = 0 if metric == "jaccard_weighted" else np.inf
    cnt = np.zeros((na, nb), np.int64)
    for k in range(m):
        cnt += (A[:, k][:, None] == B[:, k][None, :]) & (A[:, k] != unset)[:, None]
    assert np.array_equal(got, cnt / m)
