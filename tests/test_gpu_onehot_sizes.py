"""The dense regime on the tensor cores against the integer register compare, at sizes
that reach it (above 512 contigs): around the tiles of 128 and 256, at the last
column of each selection kernel and past it, and on both sides of the hand-over from
the matrix of counts to the lists (32,768 contigs)."""
import numpy as np
import pytest

from rabbitbin_b200 import api

pytestmark = pytest.mark.gpu


def _assembly(n, seed):
    """Contigs of 400 bases, each one of 60 base sequences with up to 80 changes."""
    rng = np.random.default_rng(seed)
    pool = rng.choice(list(b"ACGT"), size=(60, 400)).astype(np.uint8)
    buf = pool[rng.integers(0, 60, n)]
    hits = rng.integers(0, 81, n)
    at = rng.integers(0, 400, size=(n, 80))
    to = rng.choice(list(b"ACGT"), size=(n, 80)).astype(np.uint8)
    r, k = np.nonzero(np.arange(80)[None, :] < hits[:, None])
    buf[r, at[r, k]] = to[r, k]
    depth = rng.poisson(np.exp(rng.normal(2.0, 1.0, size=(5, 3)))[rng.integers(0, 5, n)])
    depth = depth.astype(np.float32)
    depth[::7] = 0.0                                       # contigs without abundance
    return buf.tobytes(), np.arange(n + 1, dtype=np.int64) * 400, depth


def _check(gpu_ctx, monkeypatch, n, m, K):
    seqcat, offs, depth = _assembly(n, n + m)
    p = api.default_params(m=m, max_edges=K, force_path=1)
    for env in ("RBG_ONEHOT_CAP", "RBG_DENSE_ALU"):
        monkeypatch.delenv(env, raising=False)
    got = gpu_ctx.bin_graph(seqcat, offs, depth, p)
    monkeypatch.setenv("RBG_DENSE_ALU", "1")
    want = gpu_ctx.bin_graph(seqcat, offs, depth, p)
    assert got["path"] == want["path"] == 1 and len(want["src"]) > n
    assert got["sim_cutoff"] == want["sim_cutoff"] and got["b0"] == want["b0"]
    for k in ("src", "dst", "scomp", "score"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("n", [513, 641, 767, 768, 769, 1024, 8192, 16384, 24576, 24577, 32768, 32769])
@pytest.mark.parametrize("m,K", [(24, 448), (250, 200)])
def test_counts_equal_register_compare(gpu_ctx, monkeypatch, n, m, K):
    _check(gpu_ctx, monkeypatch, n, m, K)


@pytest.mark.parametrize("n", [4097, 8193, 16385, 24577])
@pytest.mark.parametrize("K", [320, 321, 400, 448])
def test_many_neighbours(gpu_ctx, monkeypatch, n, K):
    """512 and 1,024 groups of columns a row (K up to 320, and above)."""
    _check(gpu_ctx, monkeypatch, n, 120, K)
