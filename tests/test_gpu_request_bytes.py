"""The server's admission estimate covers the device memory that a request takes:
an assembly of the symmetric pass, with its register planes, padded rows,
candidate and pair lists."""
import gc

import pytest
import torch

from rabbitbin_b200 import api
from rabbitbin_b200.synth import make_assembly

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("S", [6, 20])
def test_estimate_covers_the_buffers(S):
    p = api.default_params(m=1000)
    small = make_assembly(2, 100, S, seed=80, median_len=2600.0, max_len=3000)
    big = make_assembly(120, 60000, S, seed=81, median_len=2600.0, max_len=3000)
    buf, offs = big.concat()
    gc.collect()
    ctx = api.Context(0)
    try:
        ctx.bin_graph(*small.concat(), small.depth, p)           # tables and small buffers
        before = _free()
        for _ in range(2):
            want = ctx.bin_graph(buf, offs, big.depth, p)
        taken = before - _free()
    finally:
        ctx.close()
    srv = api.Server(workers=1)
    try:
        g, st = srv.wait(srv.submit(buf, offs, big.depth, p))
    finally:
        srv.close()
    assert len(g["src"]) == len(want["src"])
    assert taken <= st["est_bytes"], (taken, st["est_bytes"])
