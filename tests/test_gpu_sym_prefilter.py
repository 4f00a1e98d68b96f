"""The tensor-core prefilter of the symmetric pass against the restated oracle:
S at the ends of its K steps (the bias column's place), row and column counts
off its 128 x 256 tiles, and candidates so dense that a warp's item outgrows
its entry buffer."""
import numpy as np
import pytest

import oracle
from rabbitbin_b200 import api
from rabbitbin_b200.synth import make_assembly

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,N,S", [(30, 2561, 15), (30, 2700, 16), (30, 2688, 31), (30, 2815, 32),
                                   (30, 2817, 63), (1, 2600, 3), (2, 3001, 4)])
def test_prefilter_graph(gpu_ctx, orc, G, N, S):
    asm = make_assembly(G, N, S, seed=900 + N + S, median_len=3000.0)
    buf, offs = asm.concat()
    w = orc.build_winners(buf, offs)
    want = orc.run_graph(oracle.default_params(N, 500, S, force_path=2), w, asm.depth)
    p = api.default_params(force_path=2)
    ws, wd, wsc, wsw = oracle.sorted_edges(want)
    called = gpu_ctx.bin_graph(buf, offs, asm.depth, p)
    gpu_ctx.stage(buf, offs, asm.depth)
    gpu_ctx.run_resident(p)
    for got in (called, gpu_ctx.fetch_graph()):
        assert got["b0"] == want["b0"] and got["sim_cutoff"] == want["sim_cutoff"]
        assert np.array_equal(got["src"], ws) and np.array_equal(got["dst"], wd)
        assert np.array_equal(got["scomp"], wsc) and np.array_equal(got["score"], wsw)


@pytest.mark.parametrize("m", [17, 250, 255, 256, 500, 700, 1030])
def test_register_planes(gpu_ctx, orc, m):
    """Register compares on bit planes: short repeats leave few elements in a
    contig, so many registers are won by elements of large U (codes above the
    low planes'); m around the lanes a survivor takes (8, 16, 32) and above
    32 groups of 32 registers."""
    rng = np.random.default_rng(m)
    N = 2600
    seqs = []
    for i in range(N):
        if i % 3 == 0:
            unit = bytes(rng.choice(list(b"ACGT"), size=1 + i % 7))
            seqs.append((unit * 400)[:400])
        else:
            seqs.append(bytes(rng.choice(list(b"ACGT"), size=300 + i % 200)))
        if i % 501 == 0:
            seqs[-1] = b"NN"                      # no registers at all
    offs = np.zeros(N + 1, np.int64)
    offs[1:] = np.cumsum([len(s) for s in seqs])
    buf = b"".join(seqs)
    depth = rng.poisson(np.exp(rng.normal(2.0, 1.0, size=(4, 10)))[rng.integers(0, 4, N)])
    depth = depth.astype(np.float32)
    w = orc.build_winners(buf, offs, m=m)
    want = orc.run_graph(oracle.default_params(N, m, 10, force_path=2), w, depth)
    ws, wd, wsc, wsw = oracle.sorted_edges(want)
    got = gpu_ctx.bin_graph(buf, offs, depth, api.default_params(m=m, force_path=2))
    assert got["b0"] == want["b0"] and got["sim_cutoff"] == want["sim_cutoff"]
    assert np.array_equal(got["src"], ws) and np.array_equal(got["dst"], wd)
    assert np.array_equal(got["scomp"], wsc) and np.array_equal(got["score"], wsw)
