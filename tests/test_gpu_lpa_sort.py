"""Incidence lists at the sizes where their sort changes its way (registers of a
warp in steps up to 512 arcs, shared memory up to 4,096, global memory above),
parallel edges included, against the restated propagation."""
import numpy as np
import pytest

from oracle import lpa

pytestmark = pytest.mark.gpu

DEGREES = (1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512, 513, 700, 4096, 4097)


@pytest.mark.parametrize("sync", [False, True])
@pytest.mark.parametrize("rule", ["fisher", "sum"])
def test_hub_degrees(gpu_ctx, rule, sync):
    rng = np.random.default_rng(7)
    n = 5000
    h = len(DEGREES)
    src, dst = [], []
    for v, deg in enumerate(DEGREES):
        nbr = rng.choice(np.arange(h, n), deg - deg // 16, replace=False)
        nbr = np.concatenate([nbr, nbr[: deg // 16]])          # parallel edges
        src.append(np.full(deg, v))
        dst.append(rng.permutation(nbr))
    src.append(rng.integers(h, n, 6000))
    dst.append(rng.integers(h, n, 6000))
    src, dst = np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)
    keep = src != dst
    src, dst = src[keep], dst[keep]
    flip = rng.random(len(src)) < 0.5
    src, dst = np.where(flip, dst, src), np.where(flip, src, dst)
    w = rng.uniform(0.5, 0.99, len(src)).astype(np.float32)
    order = rng.permutation(n).astype(np.uint32)
    want = lpa.label_propagation(n, src, dst, w, order, rule=lpa.RULES[rule], synchronous=sync)
    got, _ = gpu_ctx.label_propagation(n, src, dst, w, node_order=order, rule=rule,
                                       synchronous=sync)
    assert (got == want).all(), int((got != want).sum())
