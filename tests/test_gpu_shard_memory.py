"""A sharded eigensolve in which one rank cannot have the eigensolver's buffers: every rank then takes
the memory-lean variant (the two issue different collectives).  The shortage is injected on the host, in
one rank's thread; both ranks end with the eigenvalues of the solve on one rank.

Tolerance: the stopping rule, |dE| <= 1e-10 |E| a run, twice that between two."""
import os
import sys
from datetime import timedelta

import numpy as np
import pytest
import torch.multiprocessing as mp

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_alloc_failure import fail_alloc
from test_gpu_lanczos import context
from test_gpu_shard import _free_port

pytestmark = pytest.mark.gpu

N, K = 3333, 4


def _rank_main(rank, world, port, short, first, out):
    import torch
    import torch.distributed as dist
    torch.cuda.set_device(0)
    dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{port}", rank=rank,
                            world_size=world, timeout=timedelta(seconds=60))
    from vhci_b200 import shard
    from vhci_b200 import api

    class Counting(shard.Comm):
        sizes = []

        def _allreduce(self, user, buf, count):
            self.sizes.append(int(count))
            return super()._allreduce(user, buf, count)

    comm = Counting(device="cuda")
    res = {"code": 0}
    with context(N, K, 0) as v:
        v.set_comm(comm)
        v.build_h()
        if rank == short:
            fail_alloc(first)
        try:
            res["E"] = v.eigs(K).tolist()
        except api.VhciError as e:
            res["code"] = e.code
        res["failed"] = fail_alloc(0, 0) >= first if rank == short else False
    res["errors"], res["sizes"] = list(comm.errors), comm.sizes
    out[rank] = res
    if not comm.errors:
        dist.barrier()
    dist.destroy_process_group()


@pytest.mark.parametrize("short", [0, 1])
def test_ranks_take_the_same_variant(short):
    with context(N, K, 0) as v:
        ref = v.eigs(K)
    world = 2
    with mp.get_context("spawn").Manager() as m:
        out = m.dict()
        mp.spawn(_rank_main, args=(world, _free_port(), short, 1, out), nprocs=world, join=True)
        res = dict(out)
    assert res[short]["failed"]
    for r in range(world):
        assert not res[r]["errors"] and res[r]["code"] == 0, res[r]
        assert (np.abs(np.array(res[r]["E"]) - ref) <= 2e-10 * np.abs(ref)).all()
    assert res[0]["sizes"] == res[1]["sizes"]  # the same collectives in the same order
    assert res[0]["E"] == res[1]["E"]
