"""The sketch kernels' splits: registers over several CTAs (few contigs), a CTA
or a warp per contig in the k-mer count, and the 5-mer counting around invalid
bases, against the restated oracle."""
import numpy as np
import pytest

from rabbitbin_b200 import api

pytestmark = pytest.mark.gpu


def _seqs(rng, n, lo, hi, p_n=0.0):
    out = []
    for L in rng.integers(lo, hi, size=n):
        a = np.frombuffer(b"ACGTacgt", np.uint8)[rng.integers(0, 8, size=L)].copy()
        if p_n:
            a[rng.random(L) < p_n] = ord("N")
        out.append(a.tobytes())
    return out


def _check(ctx, orc, seqs, **kw):
    offs = np.zeros(len(seqs) + 1, np.int64)
    offs[1:] = np.cumsum([len(s) for s in seqs])
    buf = b"".join(seqs)
    p = api.default_params(**kw)
    got = ctx.build_pmh_winners(buf, offs, p)
    want = orc.build_winners(buf, offs, m=p.m, k=p.k, gc_norm=p.gc_norm)
    assert np.array_equal(got, want)


# register ranges: one CTA, uneven ranges, a range per 16 registers, several
# 256-register chunks in one range
@pytest.mark.parametrize("n,m", [(1, 2), (1, 17), (31, 496), (33, 500), (33, 4096), (300, 1000),
                                 (5000, 250)])
def test_register_split(gpu_ctx, orc, n, m):
    _check(gpu_ctx, orc, _seqs(np.random.default_rng(n + m), n, 30, 2600), m=m)


# a CTA per contig up to 20,000 contigs, a warp per contig above; lengths
# around a word (16 bases), a warp step (512) and a CTA step (4,096)
@pytest.mark.parametrize("n", [64, 20000, 20001])
@pytest.mark.parametrize("k,gc", [(4, 1), (4, 2), (3, 1)])
def test_count_forms(gpu_ctx, orc, n, k, gc):
    rng = np.random.default_rng(7 * n + k)
    seqs = _seqs(rng, n - 12, 3, 120, p_n=0.02)
    seqs += _seqs(rng, 12, 1, 2)
    for i, L in enumerate([15, 16, 17, 511, 512, 513, 4095, 4096, 4097, 9000, 2, 4]):
        seqs[5 * i] = _seqs(rng, 1, L, L + 1, p_n=0.01 if i % 2 else 0.0)[0]
    _check(gpu_ctx, orc, seqs, m=64, k=k, gc_norm=gc)
