"""The projected matrix of a sharded block Lanczos run: the Ritz pairs that rank 0 hands round have to
be eigenpairs of the matrix summed from the coefficients of both Gram-Schmidt passes, as on one rank.

The collectives' results are recorded on the way: the coefficients of each pass (two sums after every
gathered vector block) give T = Q^T H Q of the first cycle, and the vectors and values that follow must
satisfy T y = theta y.  With FP32 gathers the coefficients against the older blocks, which only the second
pass has, are the gathers' noise, about 1e-8 of ||H||; a T without them misses by that much.

Tolerance: a dense eigensolver's residual is a small multiple of m 2^-53 ||T|| (m = 48): 10 of them make
5e-14; 1e-13 is allowed."""
import os
import sys
from datetime import timedelta

import numpy as np
import pytest
import torch.multiprocessing as mp

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_lanczos import context
from test_gpu_shard import _free_port

pytestmark = pytest.mark.gpu

N, K, BLOCK = 3333, 4, 16


def _recorder(shard):
    import torch

    class Recorder(shard.Comm):
        def __init__(self):
            self.log = []
            super().__init__(device="cuda")

        def _allreduce(self, user, buf, count):
            r = super()._allreduce(user, buf, count)
            self.log.append(shard._view(buf, int(count), torch.float64, "cuda").cpu().numpy().copy())
            return r

        def _allgather(self, user, send, recv, nbytes):
            self.log.append(None)
            return super()._allgather(user, send, recv, nbytes)

    return Recorder()


def _rank_main(rank, world, port, precision, out):
    import torch
    import torch.distributed as dist
    torch.cuda.set_device(0)
    dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{port}", rank=rank,
                            world_size=world, timeout=timedelta(seconds=300))
    from vhci_b200 import shard
    comm = _recorder(shard)
    with context(N, K, precision) as v:
        v.set_comm(comm)
        E = v.eigs(K)
    out[rank] = {"E": E.tolist(), "errors": list(comm.errors), "log": comm.log if rank == 0 else None}
    dist.barrier()
    dist.destroy_process_group()


def _first_cycle(log):
    """T (from both passes), theta and the Ritz coefficients of the first cycle."""
    ld = (2 * (K + 8) + 2 * BLOCK + BLOCK + 15) // 16 * 16
    T = np.zeros((ld, ld))
    at = [i for i, x in enumerate(log) if x is None]
    m = 0
    for i in at:
        first, second = log[i + 1], log[i + 2]
        mm = m + BLOCK
        rows = first.size // BLOCK
        T[mm - rows:mm, m:mm] += first.reshape(BLOCK, rows).T
        T[:mm, m:mm] += second.reshape(BLOCK, mm).T
        m = mm
        rest = log[i + 3:]
        j = next((j for j, x in enumerate(rest) if x is None or x.size == ld * m), None)
        if j is not None and rest[j] is not None:  # the vectors, then the values
            return T[:m, :m], rest[j + 1], rest[j].reshape(m, ld).T[:m]
    raise AssertionError("no projected solution in the recorded sums")


@pytest.mark.parametrize("precision", [0, 1])
def test_ritz_pairs_belong_to_both_passes(precision):
    with context(N, K, precision) as v:
        ref = v.eigs(K)
    world = 2
    with mp.get_context("spawn").Manager() as m:
        out = m.dict()
        mp.spawn(_rank_main, args=(world, _free_port(), precision, out), nprocs=world, join=True)
        res = dict(out)
    assert not res[0]["errors"] and not res[1]["errors"]
    assert res[0]["E"] == res[1]["E"]
    T, theta, Y = _first_cycle(res[0]["log"])
    T = np.triu(T) + np.triu(T, 1).T
    nk = K + 8
    R = T @ Y[:, :nk] - Y[:, :nk] * theta[:nk]
    assert np.abs(R).max() <= 1e-13 * np.abs(T).sum(1).max()
    # both runs stop at residuals of 1e-10 |theta| (FP32 gathers: 1e-7 of the scale, then the FP64 sweep)
    bound = 2 * (1e-10 if precision == 0 else 1e-7) * np.abs(T).sum(1).max()
    assert np.abs(np.array(res[0]["E"]) - ref).max() <= bound
