"""Few contigs split over two ranks: the register compare on a rank's rows (up to 512
contigs, its first row at any place), the one-hot pass above; against the whole graph."""
import datetime
import os

import numpy as np
import pytest
import torch.multiprocessing as mp

from rabbitbin_b200 import api, shard
from rabbitbin_b200.synth import make_assembly
from test_gpu_shard import _free_port

pytestmark = pytest.mark.gpu


def _rank_main(rank, world, port, n, cut, outdir):
    import torch.distributed as dist
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("gloo", rank=rank, world_size=world,
                            timeout=datetime.timedelta(seconds=120))
    asm = make_assembly(5, n, 3, seed=n, median_len=2600.0, max_len=4000)
    buf, offs = asm.concat()
    lo, hi = [(0, cut), (cut, n)][rank]
    ctx = api.Context(0)
    g = ctx.bin_graph_sharded(buf[offs[lo]:offs[hi]], offs[lo:hi + 1] - offs[lo], asm.depth[lo:hi],
                              rank, world, shard.host_allgather())
    np.savez(os.path.join(outdir, f"rank{rank}.npz"), cutoff=g["sim_cutoff"],
             **{k: g[k] for k in ("src", "dst", "scomp", "score")})
    ctx.close()
    dist.barrier()
    dist.destroy_process_group()


@pytest.mark.parametrize("n,cut", [(300, 37), (512, 256), (513, 1)])
def test_two_ranks_few_contigs(gpu_ctx, tmp_path, n, cut):
    mp.spawn(_rank_main, args=(2, _free_port(), n, cut, str(tmp_path)), nprocs=2, join=True)
    asm = make_assembly(5, n, 3, seed=n, median_len=2600.0, max_len=4000)
    buf, offs = asm.concat()
    want = gpu_ctx.bin_graph(buf, offs, asm.depth)
    parts = [np.load(tmp_path / f"rank{r}.npz") for r in range(2)]
    assert all(float(z["cutoff"]) == want["sim_cutoff"] for z in parts)
    for k in ("src", "dst", "scomp", "score"):
        assert np.array_equal(np.concatenate([z[k] for z in parts]), want[k]), k
