"""The kernels of one rank per GPU, with all ranks emulated on one.

Without an execution-mode suffix an emulated world runs in lockstep or in the local forms.  A traced communicator keeps the
per-rank kernels (its stamps describe ranks that signal each other), and so does a suffix: the calls of
``test_gpu_emulated.py`` once more, that way."""
import pytest
import torch

import configurable_hierarchical_allreduce_algorithms_b200 as chb
import test_gpu_emulated as emulated
from configurable_hierarchical_allreduce_algorithms_b200.parallel.comm import Communicator

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comms(cuda):
    made = {}

    def get(P):
        if P not in made:
            made[P] = Communicator.emulated(P, scratch_bytes=96 << 20, user_bytes=32 << 20)
            made[P].enable_trace(4)
        return made[P]

    yield get
    for c in made.values():
        c.close()


def test_schedules_on_the_per_rank_kernels(comms):
    for case in emulated.AR_CASES:
        emulated.test_allreduce_programs(comms, *case)
    for P in (2, 3, 4, 6, 8):
        emulated.test_three_collectives_radix_batch(comms, P)
    emulated.test_all_to_all_and_gather(comms)
    emulated.test_large_multi_cta_and_scale(comms)
    emulated.test_symmetric_buffers_zero_copy(comms)
    emulated.test_auto_choice_and_reference_signatures(comms)
    assert comms(8).read_trace(1, 0)[0][1] > 0              # somebody left stamps


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.int32, torch.float64, torch.int64])
def test_types_and_operations_on_the_per_rank_kernels(comms, dtype):
    for op in ("sum", "max", "min"):
        emulated.test_dtypes_ops(comms, dtype, op)


@pytest.mark.parametrize("P", [2, 4, 8])
def test_the_ring_of_bulk_copies(comms, P):
    emulated.test_bulk_copy_allgather(comms, P)


@pytest.mark.parametrize("mode", [":pull", ":ll"])
@pytest.mark.parametrize("algo", ["pairwise", "ring", "recursive_halving", "recursive_doubling", "radix", "radix_block", "radix_batch"])
def test_reduce_scatter_baselines(comms, algo, mode):
    for P in (4, 6, 8):
        n = 257
        ins = emulated.make_inputs(P, n * P, torch.float32)
        exp = emulated.ref_reduce(ins, "sum")
        outs = chb.reduce_scatter(comms(P), ins, algo=algo + mode, k=3, b=2)
        for r in range(P):
            emulated.check(outs[r], exp[r * n:(r + 1) * n], torch.float32, P)
        comms(P).check()


@pytest.mark.parametrize("mode", [":pull", ":ll"])
@pytest.mark.parametrize("algo", ["k_brucks", "ring", "recursive_doubling", "linear", "radix_batch"])
def test_allgather_baselines(comms, algo, mode):
    for P in (4, 8):
        blocks = emulated.make_inputs(P, 1001, torch.bfloat16)
        outs = chb.all_gather(comms(P), blocks, algo=algo + mode, k=3)
        for r in range(P):
            assert torch.equal(outs[r], torch.cat(blocks))
        comms(P).check()
