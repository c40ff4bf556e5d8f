"""Element loops of a pull step on pointers that do not share an alignment: blocks of odd length put every source and
destination of a reduce-scatter on another residue.  Integer-valued inputs, so every order of summation is exact."""
import pytest
import torch

import configurable_hierarchical_allreduce_algorithms_b200 as chb
from configurable_hierarchical_allreduce_algorithms_b200.parallel.comm import Communicator

pytestmark = pytest.mark.gpu

# around the vector (4 - 16 elements), the head and tail of the shifted loop, a warp's 32 * 2 vectors and a CTA's pass
LENGTHS = (1, 7, 15, 16, 17, 31, 33, 47, 49, 63, 65, 255, 513, 1031, 8191, 40009)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.int32, torch.float64, torch.int64, torch.uint8])
def test_spans_on_any_alignment(cuda, dtype):
    P = 3
    comm = Communicator.emulated(P, scratch_bytes=8 << 20, user_bytes=4096)
    g = torch.Generator(device="cuda").manual_seed(7)
    for i, n in enumerate(LENGTHS):
        skew = i % 5                       # the views start off the allocation's grid as well
        ins = [torch.randint(0, 9, (P * n + 8,), generator=g, device="cuda", dtype=torch.int32).to(dtype)[skew + r:][:P * n]
               for r in range(P)]
        wide = torch.stack([x.to(torch.float64) for x in ins])
        outs = [torch.zeros(n + 2, dtype=dtype, device="cuda")[1:1 + n] for _ in range(P)]
        for op, want in (("sum", wide.sum(0)), ("max", wide.max(0).values)):
            chb.reduce_scatter(comm, ins, out=outs, op=op, algo="radix_batch:pull")
            for r in range(P):
                assert torch.equal(outs[r].to(torch.float64), want[r * n:(r + 1) * n]), (n, op, r)
        blocks = [x[:n] for x in ins]
        full = [torch.zeros(P * n + 2, dtype=dtype, device="cuda") for _ in range(P)]
        chb.all_gather(comm, blocks, out=[f[1:1 + P * n] for f in full], algo="radix_batch:pull")
        for f in full:
            assert torch.equal(f[1:1 + P * n], torch.cat(blocks)), n
            assert f[0] == 0 and f[-1] == 0, n          # nothing outside the result is written
    comm.check()
    comm.close()
