"""Candidate lists of the symmetric pass: their size does not carry over from a
small assembly, nearly all of whose pairs pass the prune, to a large one at the
same sample count; and an assembly whose lists would take more than a quarter of
the device's memory is counted first."""
import gc

import numpy as np
import pytest
import torch

import oracle
from rabbitbin_b200 import api
from rabbitbin_b200.synth import make_assembly

pytestmark = pytest.mark.gpu
S = 6


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def dense_and_large():
    dense = make_assembly(1, 2600, S, seed=71, median_len=2600.0, max_len=3000)
    large = make_assembly(60, 26001, S, seed=72, median_len=2600.0, max_len=3000)
    return [(a.concat() + (a.depth, api.default_params(force_path=2))) for a in (dense, large)]


def _run(ctx, case, batch):
    if batch:
        return ctx.bin_batch([case])[0][0]
    return ctx.bin_graph(*case)


def _taken(cases, batch):
    """Device bytes a new context takes for the last case, after the others."""
    gc.collect()
    ctx = api.Context(0)
    try:
        for c in cases[:-1]:
            _run(ctx, c, batch)
        before = _free()
        g = _run(ctx, cases[-1], batch)
        return before - _free(), g
    finally:
        ctx.close()


@pytest.mark.parametrize("batch", [False, True])
def test_dense_small_assembly_does_not_size_a_large_one(dense_and_large, batch):
    dense, large = dense_and_large
    alone, want = _taken([large], batch)
    after, got = _taken([dense, large], batch)
    for k in ("src", "dst", "scomp", "score"):
        assert np.array_equal(got[k], want[k]), k
    # every pair of 26,001 contigs is 1.4 GB of entries; buffers kept from the dense
    # assembly make the second call's own share smaller, not larger
    assert after <= alone + (256 << 20)


@pytest.mark.parametrize("S,list_bytes", [(6, None), (6, 4 << 20), (12, None), (12, 4 << 20)])
def test_dense_assembly_graph(orc, monkeypatch, S, list_bytes):
    """A dense assembly alone, streamed behind its input (12 samples) and in a batch:
    the graph of the oracle when its lists overflow (first call), when they are
    sized from the fraction seen (second) and when they are counted first (a bound
    of 4 MB, where every pair takes 13.5 MB)."""
    if list_bytes:
        monkeypatch.setenv("RBG_LIST_BYTES", str(list_bytes))
    a = make_assembly(1, 2600, S, seed=73, median_len=4000.0, max_len=6000)
    buf, offs = a.concat()
    p = api.default_params(force_path=2)
    w = orc.build_winners(buf, offs)
    want = oracle.sorted_edges(orc.run_graph(oracle.default_params(2600, 500, S, force_path=2), w,
                                             a.depth))
    case = (buf, offs, a.depth, p)
    ctx = api.Context(0)
    try:
        for _ in range(2):
            for g in [ctx.bin_graph(*case)] + ctx.bin_batch([case] * 2)[0]:
                for x, k in zip(want, ("src", "dst", "scomp", "score")):
                    assert np.array_equal(g[k], x), k
    finally:
        ctx.close()


def test_streamed_pair_list_within_its_bound(monkeypatch):
    """A streamed pass lists every survivor of the prune.  Where they outgrow the
    list, it grows only within the bound of the lists; the pairs are scored after
    the copy from then on otherwise, with a list of the admitted pairs alone."""
    a = make_assembly(40, 3000, 12, seed=74, median_len=4000.0, max_len=6000)
    depth = a.depth.copy()
    rows = [a.depth[a.genome_of == g] for g in range(4)]         # 40 genomes, 4 coverages
    for i in range(a.n):
        r = rows[a.genome_of[i] & 3]
        depth[i] = r[i % len(r)]
    buf, offs = a.concat()
    case = (buf, offs, depth, api.default_params(force_path=2))
    monkeypatch.setenv("RBG_PAIR_CAP", "1024")

    def taken():
        gc.collect()
        before = _free()
        ctx = api.Context(0)
        try:
            got = [ctx.bin_graph(*case) for _ in range(2)]
            return before - _free(), got
        finally:
            ctx.close()

    taken()                                                      # modules load
    most, want = taken()
    monkeypatch.setenv("RBG_LIST_BYTES", str(16 << 20))
    least, got = taken()
    for g in got:
        for k in ("src", "dst", "scomp", "score"):
            assert np.array_equal(g[k], want[0][k]), k
    # about 1.1 M survivors: 45 MB with a quarter to spare
    assert least <= most - (12 << 20)


def test_nearby_sizes_share_their_fraction():
    """An assembly of twice the contigs of one seen before takes no second pass: its
    first call launches what its second does."""
    ctx = api.Context(0)
    try:
        def launches(n):
            # 20 genomes: about 0.7 M pairs of one genome at 5,200 contigs, below the 1 M
            # that the pair list holds at first
            a = make_assembly(20, n, 5, seed=7, median_len=2600.0, max_len=3000)
            ctx.stage(*a.concat(), a.depth)
            p = api.default_params(force_path=2)
            return [ctx.run_resident(p)["kernel_launches"] for _ in range(2)]
        first, later = launches(2600)
        assert first > later                                # lists overflowed, and the pass ran again
        first, later = launches(5200)
        assert first == later
    finally:
        ctx.close()
