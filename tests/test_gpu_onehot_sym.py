"""The dense regime's symmetric pass (counts of the tiles on and above the
diagonal, both orientations stored, then the top-K of each row of counts)
against the list pass, which scores every ordered pair: sizes around the tile
sides and the column ranges of the selection, few registers (many equal
similarities at the cut), and contigs without abundance."""
import numpy as np
import pytest

from rabbitbin_b200 import api
from rabbitbin_b200.synth import make_assembly

pytestmark = pytest.mark.gpu


def _graphs(gpu_ctx, monkeypatch, a, depth, params):
    monkeypatch.delenv("RBG_ONEHOT_CAP", raising=False)
    seqcat, offs = b"".join(a.seqs), np.cumsum([0] + [len(s) for s in a.seqs])
    got = gpu_ctx.bin_graph(seqcat, offs, depth, params)
    monkeypatch.setenv("RBG_ONEHOT_CAP", "1024")           # the list pass
    want = gpu_ctx.bin_graph(seqcat, offs, depth, params)
    return got, want


@pytest.mark.parametrize("n", [1, 2, 31, 97, 128, 129, 255, 257, 511, 513, 1025, 2049, 4096, 4097,
                               8193, 9000, 17000])
@pytest.mark.parametrize("m,K", [(16, 20), (250, 200)])
def test_symmetric_counts_equal_lists(gpu_ctx, monkeypatch, n, m, K):
    a = make_assembly(max(2, n // 40), n, 3, seed=n + m)
    depth = a.depth.copy()
    depth[::7] = 0.0                                       # rows of equal ranks
    p = api.default_params(m=m, max_edges=K, force_path=1)
    got, want = _graphs(gpu_ctx, monkeypatch, a, depth, p)
    assert got["path"] == want["path"] == 1
    assert got["sim_cutoff"] == want["sim_cutoff"]
    for k in ("src", "dst", "scomp", "score"):
        assert np.array_equal(got[k], want[k]), k
