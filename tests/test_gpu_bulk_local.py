"""Bulk allgather with all ranks on one GPU: the one-read form against the ring of bulk copies (which a traced communicator
keeps), 16- and 32-byte grids, pieces with a rest, blocks in place."""
import pytest
import torch

import configurable_hierarchical_allreduce_algorithms_b200 as chb
from configurable_hierarchical_allreduce_algorithms_b200.parallel.comm import Communicator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [2, 3, 8])
def test_local_form_equals_the_ring(cuda, P):
    # around one piece of 32 KiB (16 KiB with 16-byte vectors), and several with a rest
    for n in (4, 8, 12, 4092, 8188, 8192, 8196, 50004):
        comm = Communicator.emulated(P, scratch_bytes=1 << 20, user_bytes=(P + 1) * n * 4 + 8192)
        xs, ys = comm.empty(n, torch.float32), comm.empty(n * P, torch.float32)
        for r, x in enumerate(xs):
            x.copy_(torch.randn(n, device="cuda"))
        want = torch.cat(list(xs))
        for traced in (0, 4):
            comm.enable_trace(traced)
            for y in ys:
                y.zero_()
            chb.all_gather(comm, xs, out=ys, algo="bulk")
            assert all(torch.equal(y, want) for y in ys), (n, traced)
            slots = [y[r * n:(r + 1) * n] for r, y in enumerate(ys)]           # in place: only the peers' blocks move
            for r, y in enumerate(ys):
                y.zero_()
                slots[r].copy_(xs[r])
            chb.all_gather(comm, slots, out=ys, algo="bulk")
            assert all(torch.equal(y, want) for y in ys), (n, traced)
        assert comm.status(1)["launches"] == 4
        comm.check()
        comm.close()


def us(fn):
    fn()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


@pytest.mark.parametrize("n", [4 << 20, (4 << 20) + 8])
def test_a_given_number_of_ctas_is_kept(cuda, n):
    """One CTA a rank takes all pieces, several of them share them; the caller who asks for few leaves the other SMs free, so
    the call takes many times as long (16 SMs of 148 at most)."""
    P = 4
    comm = Communicator.emulated(P, scratch_bytes=1 << 20, user_bytes=(P + 1) * n * 2 + 8192)
    xs, ys = comm.empty(n, torch.bfloat16), comm.empty(n * P, torch.bfloat16)
    for x in xs:
        x.copy_(torch.randn(n, device="cuda"))
    want = torch.cat(list(xs))
    for nctas in (1, 3, 4, 1000):
        for y in ys:
            y.zero_()
        chb.all_gather(comm, xs, out=ys, algo="bulk", nctas=nctas)
        assert all(torch.equal(y, want) for y in ys), nctas
    few, many = [us(lambda: chb.all_gather(comm, xs, out=ys, algo="bulk", nctas=k)) for k in (1, 0)]
    assert few > 2 * many, (few, many)
    comm.check()
    comm.close()
