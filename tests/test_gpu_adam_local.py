"""Reduce-scatter + AdamW with all ranks on one GPU: the form without barriers against the per-rank kernel (which a traced
communicator keeps), bit for bit, around one CTA's 1024 elements and with more ranks than one batch of loads."""
import pytest
import torch

from configurable_hierarchical_allreduce_algorithms_b200.ops import fused
from configurable_hierarchical_allreduce_algorithms_b200.parallel.comm import Communicator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 2, 8, 11])
@pytest.mark.parametrize("n", [4, 1020, 1024, 1028, 40004])
def test_local_form_equals_the_barrier_kernel(cuda, P, n):
    comm = Communicator.emulated(P, scratch_bytes=1 << 20, user_bytes=P * n * 4 + 4096)
    g = torch.Generator(device="cuda").manual_seed(n)
    grads = comm.empty(P * n, torch.float32)
    grads = grads if P > 1 else [grads]
    for x in grads:
        x.copy_(torch.randn(P * n, generator=g, device="cuda"))
    start = [[torch.randn(n, generator=g, device="cuda").abs() for _ in range(P)] for _ in range(3)]
    one = lambda xs: xs if P > 1 else xs[0]
    got = []
    for traced in (0, 4):
        comm.enable_trace(traced)
        w, m, v = [[x.clone() for x in s] for s in start]
        p = [torch.zeros(n, dtype=torch.bfloat16, device="cuda") for _ in range(P)]
        for step in (1, 2):
            fused.reduce_scatter_adam(comm, one(list(grads)), one(w), one(m), one(v), one(p), lr=1e-2, weight_decay=0.1,
                                      step=step, grad_scale=1.0 / P, use_multimem=False)
        got.append([torch.cat(x).view(torch.uint8) for x in (w, m, v, p)])
    assert all(torch.equal(a, b) for a, b in zip(*got))
    comm.check()
    comm.close()


@pytest.mark.parametrize("P", [1, 4])
def test_a_given_number_of_ctas_is_kept(cuda, P):
    """The same bits from one CTA a rank, from several and from all; few of them leave the other SMs free, so the call takes
    many times as long (4 SMs of 148 at most)."""
    n = 1_000_004
    comm = Communicator.emulated(P, scratch_bytes=1 << 20, user_bytes=P * n * 4 + 4096)
    grads = comm.empty(P * n, torch.float32)
    grads = list(grads) if P > 1 else [grads]
    for x in grads:
        x.copy_(torch.randn(P * n, device="cuda"))
    start = [[torch.randn(n, device="cuda").abs() for _ in range(P)] for _ in range(3)]
    one = lambda xs: xs if P > 1 else xs[0]
    got, times = {}, {}
    for nctas in (0, 1, 3, 100_000):
        w, m, v = [[x.clone() for x in s] for s in start]
        p = [torch.zeros(n, dtype=torch.bfloat16, device="cuda") for _ in range(P)]
        best = float("inf")
        for step in range(1, 6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            fused.reduce_scatter_adam(comm, one(grads), one(w), one(m), one(v), one(p), lr=1e-2, weight_decay=0.1, step=step,
                                      grad_scale=1.0 / P, use_multimem=False, nctas=nctas)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        got[nctas], times[nctas] = [torch.cat(x).view(torch.uint8) for x in (w, m, v, p)], best
    for nctas in (1, 3, 100_000):
        assert all(torch.equal(a, b) for a, b in zip(got[0], got[nctas])), nctas
    assert times[1] > 2 * times[0], times
    comm.check()
    comm.close()
