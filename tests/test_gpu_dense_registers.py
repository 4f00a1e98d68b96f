"""Few contigs at many registers: the register compare takes them while its rows fit
the shared memory (m up to 3,520), the one-hot pass from there on; alone and in
a batch, against the restated graph."""
import numpy as np
import pytest

import oracle
from rabbitbin_b200 import api
from rabbitbin_b200.synth import make_assembly

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [3520, 3521, 3528, 3529, 3536, 3600, 4000, 4095])
@pytest.mark.parametrize("n", [97, 512])
def test_many_registers(gpu_ctx, orc, n, m):
    a = make_assembly(4, n, 3, seed=n + m, median_len=2600.0, max_len=4000)
    buf, offs = a.concat()
    w = orc.build_winners(buf, offs, m=m)
    want = orc.run_graph(oracle.default_params(n, m, 3, max_edges=448), w, a.depth)
    edges = oracle.sorted_edges(want)
    p = api.default_params(m=m, max_edges=448)
    for got in [gpu_ctx.bin_graph(buf, offs, a.depth, p)] + gpu_ctx.bin_batch([(buf, offs, a.depth, p)] * 2)[0]:
        assert got["b0"] == want["b0"] and got["sim_cutoff"] == want["sim_cutoff"]
        for x, k in zip(edges, ("src", "dst", "scomp", "score")):
            assert np.array_equal(got[k], x), k
