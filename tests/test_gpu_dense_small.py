"""The dense regime around the size where it leaves the register compare for the
tensor cores: the restated graph on both sides, alone and in one batch."""
import numpy as np
import pytest

from rabbitbin_b200.synth import make_assembly
from test_gpu_parity import _graph_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 97, 256, 511, 512, 513])
def test_few_contigs(gpu_ctx, orc, n):
    assert _graph_case(gpu_ctx, orc, 3, n, 5, seed=500 + n)["path"] == 1


def test_few_contigs_in_a_batch(gpu_ctx):
    asms = []
    for i, n in enumerate([513, 1, 512, 97, 700, 2]):
        a = make_assembly(3, n, 5, seed=600 + i)
        seqcat, offs = a.concat()
        asms.append((seqcat, offs, a.depth))
    got, _ = gpu_ctx.bin_batch(asms)
    for g, a in zip(got, asms):
        want = gpu_ctx.bin_graph(*a)
        for k in ("src", "dst", "scomp", "score"):
            assert np.array_equal(g[k], want[k]), k
