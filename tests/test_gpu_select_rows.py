"""Row top-K of the symmetric pass by histogram: rows with more keys than the
tie buffer holds in one similarity bin (few distinct similarities at small m),
several register counts in a bin (large m), K at its limits; and the scan of
the row counts at its tile sizes."""
import numpy as np
import pytest

import oracle
from rabbitbin_b200 import api
from rabbitbin_b200.synth import make_assembly

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,N,S,m,K", [(1, 2600, 3, 16, 200), (1, 2600, 12, 8, 448),
                                       (2, 4097, 5, 40, 1), (3, 2601, 10, 2000, 33),
                                       (2, 2600, 20, 500, 448)])
def test_select_rows(gpu_ctx, orc, G, N, S, m, K):
    asm = make_assembly(G, N, S, seed=77 + N + m, median_len=2600.0, max_len=4000)
    buf, offs = asm.concat()
    w = orc.build_winners(buf, offs, m=m)
    want = orc.run_graph(oracle.default_params(N, m, S, force_path=2, max_edges=K), w, asm.depth)
    ws, wd, wsc, wsw = oracle.sorted_edges(want)
    p = api.default_params(m=m, force_path=2, max_edges=K)
    gpu_ctx.stage(buf, offs, asm.depth)
    gpu_ctx.run_resident(p)
    for got in (gpu_ctx.fetch_graph(), gpu_ctx.bin_graph(buf, offs, asm.depth, p),
                gpu_ctx.bin_batch([(buf, offs, asm.depth, p)])[0][0]):
        assert got["b0"] == want["b0"] and got["sim_cutoff"] == want["sim_cutoff"]
        assert np.array_equal(got["src"], ws) and np.array_equal(got["dst"], wd)
        assert np.array_equal(got["scomp"], wsc) and np.array_equal(got["score"], wsw)


# row counts around the scan's tile (2,048 rows) and its steps (512)
@pytest.mark.parametrize("N", [1, 511, 512, 513, 2047, 2048, 2049, 4096])
def test_row_scan_sizes(gpu_ctx, orc, N):
    rng = np.random.default_rng(N)
    offs = np.arange(N + 1, dtype=np.int64) * 300
    pool = rng.choice(list(b"ACGT"), size=(5, 300)).astype(np.uint8)
    buf = pool[rng.integers(0, 5, N)].copy()
    at = rng.integers(0, 300, size=(N, 4))
    buf[np.arange(N)[:, None], at] = ord("A")
    buf = buf.tobytes()
    w = orc.build_winners(buf, offs, m=100)
    want = orc.run_graph(oracle.default_params(N, 100, 0, max_edges=20), w, np.zeros((N, 0)))
    ws, wd, wsc, wsw = oracle.sorted_edges(want)
    got = gpu_ctx.bin_graph(buf, offs, np.zeros((N, 0), np.float32),
                            api.default_params(m=100, max_edges=20))
    assert got["sim_cutoff"] == want["sim_cutoff"]
    assert np.array_equal(got["src"], ws) and np.array_equal(got["dst"], wd)
    assert np.array_equal(got["scomp"], wsc) and np.array_equal(got["score"], wsw)
