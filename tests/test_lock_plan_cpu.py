"""The lockstep form of a step program (one grid runs all ranks): its rewriting (copies read through, copies folded into
the step that produces their data, dead scratch dropped, rounds assigned anew) gives the pull form's results bit for bit,
on float inputs that do not add exactly, for every algorithm and every lowering, with the steps of a round in any order."""
import numpy as np
import pytest

import configurable_hierarchical_allreduce_algorithms_b200 as chb

CASES = [(coll, algo) for coll in ("allreduce", "reduce_scatter", "allgather", "alltoall", "gather")
         for algo in chb.list_algorithms(coll)]
LOWERINGS = [dict(), dict(in_symmetric=True), dict(out_symmetric=True), dict(in_symmetric=True, out_symmetric=True),
             dict(in_place=True)]


@pytest.mark.parametrize("coll,algo", CASES)
def test_lockstep_equals_the_pull_form(coll, algo):
    rng = np.random.default_rng(11)
    ran = 0
    for P, k, b in ((2, 2, 1), (3, 2, 1), (4, 2, 2), (6, 2, 3), (6, 3, 2), (8, 2, 1), (8, 2, 4), (8, 4, 2), (8, 8, 8), (5, 4, 1), (12, 3, 4)):
        for n in (1, 37):
            count = n * P if coll == "allreduce" else n
            for low in LOWERINGS:
                if low.get("in_place") and coll not in ("allreduce", "alltoall"):
                    continue            # one buffer as input and output: equal lengths
                try:
                    p = chb.Program(coll, algo, P, count, k, b, **low)
                except ValueError:
                    continue
                ins = [rng.standard_normal(p.in_elems).astype(np.float32) for _ in range(P)]
                alias = bool(low.get("in_place"))
                want = p.simulate([x.copy() for x in ins], alias=alias)
                for rewrite in (0, 1, 2):
                    got = p.simulate_lock(ins, seed=ran, rewrite=rewrite, alias=alias)
                    for r in range(P if coll != "gather" else 1):
                        assert got[r].tobytes() == want[r].tobytes(), (P, k, b, n, low, rewrite, r)
                ran += 1
    assert ran


def test_rewriting_removes_the_passes_it_is_for():
    # flat allreduce: every element read once from each rank and stored once on each, in one round
    P, n = 8, 8 * 100
    for low in (dict(), dict(in_symmetric=True, out_symmetric=True)):
        i = chb.Program("allreduce", "radix_batch", P, n, 2, 1, **low).lock_info()
        assert (i["rounds"], i["reads"], i["stores"]) == (1, P * n, P * n), (low, i)
    # allgather: every block read once
    i = chb.Program("allgather", "radix_batch", P, 100, 2, 1).lock_info()
    assert (i["rounds"], i["reads"], i["stores"]) == (1, P * 100, P * P * 100)
    # hierarchical allreduce: rounds and traffic of the reductions only
    p = chb.Program("allreduce", "radix_batch", P, n, 2, 4)
    assert p.lock_info()["rounds"] < p.lock_info(rewrite=0)["rounds"]
    assert p.lock_info()["stores"] < p.lock_info(rewrite=0)["stores"] // 2 + P * n
    # a pairwise and a ring reduce-scatter add in a chain: one step a rank where nothing is rounded in between
    for algo in ("pairwise", "ring"):
        i = chb.Program("reduce_scatter", algo, P, 100, 2, 1).lock_info()
        assert (i["rounds"], i["reads"], i["stores"]) == (1, P * P * 100, P * 100), (algo, i)


@pytest.mark.parametrize("dtype", [np.float32, np.int32, np.float64])
@pytest.mark.parametrize("algo", ["ring", "radix_batch", "recursive_doubling", "reduce_scatter_allgather"])
def test_in_place_on_different_16_byte_grids(algo, dtype):
    """Joined chains of an in-place allreduce store to several of their own operands; with the ranks' buffers on different
    16-byte grids no single vector loop serves those, and none may be read after it has been overwritten."""
    rng = np.random.default_rng(5)
    several = 0
    for P, k, b in ((3, 2, 1), (4, 2, 2), (4, 4, 1), (8, 4, 2), (8, 2, 2), (8, 4, 4), (8, 2, 1), (12, 3, 4), (16, 4, 4)):
        for low in (dict(in_place=True), dict(in_place=True, in_symmetric=True, out_symmetric=True)):
            p = chb.Program("allreduce", algo, P, 37 * P, k, b, **low)
            ins = [rng.standard_normal(p.in_elems) * 9 for _ in range(P)]
            ins = [x.astype(dtype) for x in ins]
            want = p.simulate([x.copy() for x in ins], alias=True)
            for skew in ([r % 4 for r in range(P)], [0] * (P - 1) + [1], [(3 * r + 1) % 4 for r in range(P)]):
                for rewrite in (0, 1, 2):
                    got = p.simulate_lock(ins, seed=k, rewrite=rewrite, alias=True, skew=skew)
                    for r in range(P):
                        assert got[r].tobytes() == want[r].tobytes(), (P, k, b, low, skew, rewrite, r)
                several += 1
    assert several


@pytest.mark.parametrize("P", [2, 3, 8, 16])
def test_flat_schedule_without_a_program(P):
    """The tables that a CTA writes for itself: the entries and costs of the plan they describe, and the line kernels'
    result (operands in rank order), around a grain of 2048 elements."""
    rng = np.random.default_rng(P)
    for n in (1, 7, 2047, 2048, 2049, 5001):
        xs = [rng.standard_normal(n * P).astype(np.float32) for _ in range(P)]
        total = xs[0].copy()
        for x in xs[1:]:
            total = total + x
        for seed in (0, 5):
            for got in chb.Program.simulate_flat("allreduce", xs, seed=seed):
                assert got.tobytes() == total.tobytes()
            for r, got in enumerate(chb.Program.simulate_flat("reduce_scatter", xs, seed=seed)):
                assert got.tobytes() == total[r * n:(r + 1) * n].tobytes()
            blocks = [x[:n].copy() for x in xs]
            for got in chb.Program.simulate_flat("allgather", blocks, seed=seed):
                assert got.tobytes() == np.concatenate(blocks).tobytes()


@pytest.mark.parametrize("coll,algo,P,k,b,block,dtype,grid16,lockstep", [
    # many rounds that the rewriting keeps: faster with flagged lines (16 ranks unless said otherwise)
    ("reduce_scatter", "ring", 16, 2, 1, 1248, 1, True, False), ("reduce_scatter", "pairwise", 16, 2, 1, 1248, 1, False, False),
    ("allreduce", "recursive_doubling", 16, 2, 1, 40, 0, True, False), ("allreduce", "recursive_doubling", 16, 2, 1, 40, 0, False, False),
    ("reduce_scatter", "recursive_halving", 16, 2, 1, 160, 1, False, False), ("alltoall", "tuna", 16, 2, 1, 40, 1, True, False),
    # one round, few rounds, or much data: faster in lockstep
    ("allreduce", "radix_batch", 8, 2, 1, 1248, 0, False, True), ("allreduce", "ring", 8, 2, 1, 4096, 0, True, True),
    ("allreduce", "radix_batch", 8, 4, 2, 131072, 0, True, True), ("allreduce", "radix_batch", 8, 8, 8, 1, 0, True, True),
    ("allreduce", "radix_batch", 8, 2, 4, 128, 0, True, True), ("alltoall", "linear", 8, 2, 1, 160, 0, True, True),
    ("reduce_scatter", "radix_batch", 8, 4, 2, 1248, 1, True, True)])
def test_lockstep_where_it_is_faster_than_flagged_lines(coll, algo, P, k, b, block, dtype, grid16, lockstep):
    p = chb.Program(coll, algo, P, block * P if coll == "allreduce" else block, k, b, in_symmetric=True, out_symmetric=True)
    assert p.lock_preferred(dtype, grid16) == lockstep
