"""fp8 wire reduce-scatter with all ranks on one GPU: the form without a wire buffer gives the bits of the wire kernel
(which a traced communicator keeps), for full and partial warps of groups, zeros, infinities and NaN, and in place."""
import pytest
import torch

from configurable_hierarchical_allreduce_algorithms_b200.ops import fused
from configurable_hierarchical_allreduce_algorithms_b200.parallel.comm import Communicator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [2, 3, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_local_form_equals_the_wire_kernel(cuda, P, dtype):
    comm = Communicator.emulated(P, scratch_bytes=8 << 20, user_bytes=4096)
    g = torch.Generator(device="cuda").manual_seed(11)
    for n in (128, 256, 384, 640, 128 * 37, 128 * 5000):
        ins = [(torch.randn(n * P, generator=g, device="cuda") * 10 ** (i - 2)).to(dtype) for i in range(P)]
        ins[0][:128] = 0
        ins[1][n - 1] = float("inf")
        ins[1][0] = float("nan")
        got = fused.reduce_scatter_fp8(comm, ins, scale=0.3)
        comm.enable_trace(4)
        want = fused.reduce_scatter_fp8(comm, ins, scale=0.3)
        comm.enable_trace(0)
        for r in range(P):
            assert torch.equal(got[r].view(torch.uint8), want[r].view(torch.uint8)), (n, r)
        # into the rank's own block of its input
        bufs = [x.clone() for x in ins]
        outs = fused.reduce_scatter_fp8(comm, bufs, out=[b[r * n:(r + 1) * n] for r, b in enumerate(bufs)], scale=0.3)
        for r in range(P):
            assert torch.equal(outs[r].view(torch.uint8), want[r].view(torch.uint8)), (n, r)
    comm.check()
    comm.close()
