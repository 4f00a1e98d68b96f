"""Sketch comparisons of few rows, in tiles of 16 and 32 rows a side: sizes around the
tiles and their chunks of 64 and 32 registers, and on both sides of the sizes where
the tile changes; the counted matches, exactly."""
import numpy as np
import pytest

from test_gpu_query_tiles import _rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb,m", [(1, 1, 1000), (15, 17, 63), (16, 16, 64), (17, 15, 65), (16, 4000, 20),
                                     (17, 3300, 33), (32, 3300, 31), (33, 3300, 32), (320, 320, 40),
                                     (321, 320, 40), (630, 641, 5), (640, 640, 5), (4000, 3, 7)])
@pytest.mark.parametrize("metric", ["jaccard_weighted", "jaccard"])
def test_few_rows(gpu_ctx, na, nb, m, metric):
    rng = np.random.default_rng(na * nb + m)
    A, B = (_rows(rng, n, m, metric == "jaccard_weighted") for n in (na, nb))
    got = gpu_ctx.pmh_compare(metric, A, B)
    unset = 0 if metric == "jaccard_weighted" else np.inf
    cnt = np.zeros((na, nb), np.int64)
    for k in range(m):
        cnt += (A[:, k][:, None] == B[:, k][None, :]) & (A[:, k] != unset)[:, None]
    assert np.array_equal(got, cnt / m)
