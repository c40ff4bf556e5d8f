"""All ranks of an emulated world in one grid (the way a schedule without an execution-mode suffix runs there), against
the pull interpreter: bit for bit, on floats that do not add exactly, for aligned and odd lengths, skewed buffers, in
place, and mixed with the per-rank kernels on one communicator."""
import pytest
import torch

import configurable_hierarchical_allreduce_algorithms_b200 as chb
from configurable_hierarchical_allreduce_algorithms_b200.parallel.comm import Communicator

pytestmark = pytest.mark.gpu

FNS = {"allreduce": chb.all_reduce, "reduce_scatter": chb.reduce_scatter, "allgather": chb.all_gather, "alltoall": chb.all_to_all}


def lengths(coll, P, n):
    return {"allreduce": (n * P, n * P), "reduce_scatter": (n * P, n), "allgather": (n, n * P), "alltoall": (n * P, n * P)}[coll]


@pytest.mark.parametrize("P,k,b", [(2, 2, 1), (3, 2, 1), (8, 2, 1), (8, 4, 2), (8, 2, 4), (6, 3, 2), (16, 4, 4)])
@pytest.mark.parametrize("coll", list(FNS))
def test_lockstep_equals_pull(cuda, coll, P, k, b):
    comm = Communicator.emulated(P, ll_bytes=64 << 10, scratch_bytes=16 << 20, user_bytes=4096)
    g = torch.Generator(device="cuda").manual_seed(3)
    names = ["tuna", "linear"] if coll == "alltoall" else ["radix_batch", "ring"]
    # one element, a grain of 2048 elements and its neighbours, several grains with a rest
    for i, n in enumerate((1, 31, 2047, 2048, 2049, 40013)):
        for dtype in (torch.float32, torch.bfloat16) if n > 1 else (torch.float32, torch.float64, torch.uint8):
            n_in, n_out = lengths(coll, P, n)
            skew = [(i + r * (i % 2)) % 3 for r in range(P)]      # ranks on different 16-byte grids every second time
            src = [torch.rand(n_in + 4, generator=g, device="cuda").mul_(9).to(dtype) for _ in range(P)]
            ins = [s[a:a + n_in] for s, a in zip(src, skew)]
            full = [torch.zeros(n_out + 4, dtype=dtype, device="cuda") for _ in range(P)]
            outs = [f[a:a + n_out] for f, a in zip(full, skew)]
            for name in names:
                kw = dict(k=k, b=b)
                if coll in ("allreduce", "reduce_scatter") and dtype.is_floating_point:
                    kw["scale"] = 0.37
                want = FNS[coll](comm, ins, algo=name + ":pull", **kw)
                for f in full:
                    f.zero_()
                FNS[coll](comm, ins, out=outs, algo=name, **kw)
                for r in range(P):
                    assert torch.equal(outs[r], want[r]), (name, n, dtype, r)
                    assert not full[r][:skew[r]].any() and not full[r][skew[r] + n_out:].any()     # nothing around it
    comm.check()
    comm.close()


def test_bytes_wrap_after_every_step(cuda):
    """A chain of byte additions is not joined: its partial sums wrap, which a scale brings to light."""
    P, n = 4, 5000
    comm = Communicator.emulated(P, scratch_bytes=4 << 20, user_bytes=4096)
    src = [torch.randint(0, 256, (P * n,), device="cuda", dtype=torch.int32).to(torch.uint8) for _ in range(P)]
    for name in ("ring", "pairwise"):
        want = chb.reduce_scatter(comm, src, algo=name + ":pull", scale=0.5)
        got = chb.reduce_scatter(comm, src, algo=name, scale=0.5)
        assert all(torch.equal(a, b) for a, b in zip(got, want)), name
    comm.check()
    comm.close()


def test_lockstep_in_place_and_overlapping_buffers(cuda):
    P, n = 4, 5003
    comm = Communicator.emulated(P, scratch_bytes=4 << 20, user_bytes=4096)
    src = [torch.randn(n * P, device="cuda") for _ in range(P)]
    want = chb.all_reduce(comm, src, algo="radix_batch:pull", k=2, b=2)
    bufs = [s.clone() for s in src]
    chb.all_reduce(comm, bufs, out=bufs, algo="radix_batch", k=2, b=2)
    assert all(torch.equal(x, y) for x, y in zip(bufs, want))
    # reduce-scatter into the rank's own block of its input: known to no schedule, so it stays with the interpreter
    want = chb.reduce_scatter(comm, src, algo="radix_batch:pull")
    bufs = [s.clone() for s in src]
    outs = chb.reduce_scatter(comm, bufs, out=[b[r * n:(r + 1) * n] for r, b in enumerate(bufs)], algo="radix_batch")
    assert all(torch.equal(x, y) for x, y in zip(outs, want))
    # allgather of blocks that already lie in their slots
    full = [torch.zeros(n * P, device="cuda") for _ in range(P)]
    for r in range(P):
        full[r][r * n:(r + 1) * n] = src[r][:n]
    chb.all_gather(comm, [f[r * n:(r + 1) * n] for r, f in enumerate(full)], out=full, algo="radix_batch", k=2, b=2)
    cat = torch.cat([s[:n] for s in src])
    assert all(torch.equal(f, cat) for f in full)
    comm.check()
    comm.close()


def test_lockstep_mixes_with_the_per_rank_kernels(cuda):
    """Launch counters, epochs and sequence numbers: lockstep, pull, push and one-shot launches in any order, traced
    launches in between, and replays of a captured launch."""
    P, n = 8, 8 * 1000
    comm = Communicator.emulated(P, scratch_bytes=4 << 20, user_bytes=4096)
    src = [torch.randint(-9, 9, (n,), device="cuda", dtype=torch.int32) for _ in range(P)]
    want = torch.stack(src).sum(0)
    outs = [torch.zeros_like(s) for s in src]
    before = comm.status(5)["launches"]
    for i in range(3):
        for algo in ("radix_batch", "radix_batch:pull", "ring", "ll", "radix_batch:ll", "recursive_doubling"):
            chb.all_reduce(comm, src, out=outs, algo=algo, k=2, b=4)
            assert all(torch.equal(o, want) for o in outs), algo
    assert comm.status(5)["launches"] - before == 18
    comm.enable_trace(16)                                   # stamps describe ranks that signal each other
    chb.all_reduce(comm, src, out=outs, algo="recursive_doubling")
    assert comm.read_trace(2, 3)[-1][1] > 0
    comm.enable_trace(0)
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        chb.all_reduce(comm, src, out=outs, algo="radix_batch", k=2, b=4, stream=side)
    for i in range(3):
        src[0].add_(1)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[6], torch.stack(src).sum(0))
    comm.check()
    comm.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_pull_with_many_small_ctas(cuda, dtype):
    """Pulled vectors beyond 4 MiB spread an emulated rank over four CTAs an SM: same bits as with a given number of
    large ones, on aligned and odd lengths, private (nothing is staged) and registered buffers."""
    P = 4
    comm = Communicator.emulated(P, scratch_bytes=64 << 20, user_bytes=32 << 20)
    for n in ((5 << 20) // dtype.itemsize, (5 << 20) // dtype.itemsize + 4):      # the second one: slices off the grid
        src = [torch.randn(n, device="cuda").to(dtype) for _ in range(P)]
        reg = comm.empty(n, dtype)
        for x, y in zip(reg, src):
            x.copy_(y)
        for k, b in ((2, 1), (2, 2)):
            want = chb.all_reduce(comm, src, algo="radix_batch:pull", k=k, b=b, nctas=7)
            for ins in (src, reg):
                got = chb.all_reduce(comm, ins, algo="radix_batch:pull", k=k, b=b)
                assert all(torch.equal(x, y) for x, y in zip(got, want)), (n, k, b)
    comm.check()
    comm.close()
    # the scratch that the general lowering asks for is asked for here as well
    small = Communicator.emulated(P, scratch_bytes=1 << 20, user_bytes=4096)
    with pytest.raises(chb.CollectiveError):
        chb.all_reduce(small, [torch.zeros(1 << 20, device="cuda") for _ in range(P)], algo="radix_batch:pull", k=2, b=2)
    small.close()


@pytest.mark.parametrize("P", [2, 3, 8])
def test_automatic_small_calls_equal_the_line_kernels(cuda, P):
    """`auto` in an emulated world: the bits of the flagged-line kernels, on odd lengths, for every type and operation;
    in place and on misaligned buffers the line kernels and programs themselves run."""
    comm = Communicator.emulated(P, ll_bytes=1 << 20, scratch_bytes=8 << 20, user_bytes=4096)
    g = torch.Generator(device="cuda").manual_seed(P)
    for dtype in (torch.float32, torch.bfloat16, torch.float16, torch.int32, torch.float64, torch.uint8):
        for n in (1, 7, 2049, 15001):       # (blocks up to the 128 KiB where every table and rule still picks the lines)
            src = [torch.rand(n * P, generator=g, device="cuda").mul_(9).to(dtype) for _ in range(P)]
            for op, scale in (("sum", 1.0), ("sum", 0.5), ("max", 1.0)):
                whole = [s[:n] for s in src]
                assert all(torch.equal(a, b) for a, b in zip(chb.all_reduce(comm, whole, op=op, scale=scale),
                                                             chb.all_reduce(comm, whole, op=op, scale=scale, algo="ll")))
            got, want = chb.reduce_scatter(comm, src), chb.reduce_scatter(comm, src, algo="ll")
            assert all(torch.equal(a, b) for a, b in zip(got, want)), (dtype, n)
            blocks = [s[:n] for s in src]
            assert all(torch.equal(a, torch.cat(blocks)) for a in chb.all_gather(comm, blocks))
            bufs = [s[:n].clone() for s in src]
            chb.all_reduce(comm, bufs, out=bufs)
            assert all(torch.equal(a, b) for a, b in zip(bufs, chb.all_reduce(comm, blocks, algo="ll"))), (dtype, n)
    ins = [torch.randn(4097, device="cuda")[1:] for _ in range(P)]
    full = torch.stack(ins).sum(0)
    for y in chb.all_reduce(comm, ins):
        torch.testing.assert_close(y, full, rtol=1e-5, atol=1e-5 * P)
    comm.check()
    comm.close()


@pytest.mark.parametrize("P,algo,k,b", [(3, "ring", 2, 1), (4, "ring", 2, 1), (8, "ring", 2, 1), (4, "radix_batch", 2, 2), (8, "radix_batch", 4, 2),
                                        (8, "radix_batch", 2, 2), (8, "radix_batch", 4, 4), (8, "radix_batch", 2, 1)])
def test_in_place_on_different_16_byte_grids(cuda, P, algo, k, b):
    """Steps that store to several of their own operands, which skewed buffers keep from one vector loop: one CTA, a
    cluster and the whole grid, against the pull interpreter, and nothing written around the buffers."""
    comm = Communicator.emulated(P, scratch_bytes=24 << 20, user_bytes=4096)
    g = torch.Generator(device="cuda").manual_seed(7)
    for n in (24 * P, 2049 * P, 150_001 * P):
        for dtype in (torch.float32, torch.int32) if n > 24 * P else (torch.float32, torch.float64, torch.bfloat16):
            for skew in ([r % 4 for r in range(P)], [0] * (P - 1) + [1]):
                src = [torch.rand(n, generator=g, device="cuda").mul_(99).to(dtype) for _ in range(P)]
                want = chb.all_reduce(comm, src, algo=algo + ":pull", k=k, b=b)
                full = [torch.zeros(n + 4, dtype=dtype, device="cuda") for _ in range(P)]
                bufs = [f[a:a + n] for f, a in zip(full, skew)]
                for x, s in zip(bufs, src):
                    x.copy_(s)
                chb.all_reduce(comm, bufs, out=bufs, algo=algo, k=k, b=b)
                for r in range(P):
                    assert torch.equal(bufs[r], want[r]), (n, dtype, skew, r)
                    assert not full[r][:skew[r]].any() and not full[r][skew[r] + n:].any()
    comm.check()
    comm.close()


def test_automatic_in_place_on_the_rows_of_an_odd_matrix(cuda):
    comm = Communicator.emulated(8, scratch_bytes=80 << 20, user_bytes=4096)
    m = torch.randn(8, 2_000_001, device="cuda")
    want = chb.all_reduce(comm, list(m.clone()), algo="ring:pull")
    chb.all_reduce(comm, list(m), out=list(m))
    assert all(torch.equal(x, y) for x, y in zip(m, want))
    comm.check()
    comm.close()


@pytest.mark.parametrize("coll", ["allreduce", "allgather"])
def test_skewed_destinations_around_the_longest_element_wise_span(cuda, coll):
    """One CTA a rank, so that a step of the round is one span: element by element up to 8192 elements, a pass for each
    destination beyond."""
    P = 3
    comm = Communicator.emulated(P, ll_bytes=64 << 10, scratch_bytes=4 << 20, user_bytes=4096)
    for blk in (8191, 8192, 8193, 10241):
        n_in, n_out = lengths(coll, P, blk)
        for dtype in (torch.float32, torch.bfloat16):
            ins = [torch.randn(n_in + 2, device="cuda").to(dtype)[r:r + n_in] for r in range(P)]
            full = [torch.zeros(n_out + 4, dtype=dtype, device="cuda") for _ in range(P)]
            outs = [f[r:r + n_out] for r, f in enumerate(full)]
            want = FNS[coll](comm, ins, algo="radix_batch:pull")
            FNS[coll](comm, ins, out=outs, algo="radix_batch", nctas=1)
            for r in range(P):
                assert torch.equal(outs[r], want[r]), (blk, dtype, r)
                assert not full[r][:r].any() and not full[r][r + n_out:].any()
    comm.check()
    comm.close()


def test_first_call_of_a_length_may_be_captured(cuda):
    """Automatic small calls need no schedule that lasts: the first call of a new length is captured, and its replay
    survives more other lengths than the program cache holds."""
    P, n = 8, 3001
    comm = Communicator.emulated(P, ll_bytes=1 << 20, scratch_bytes=8 << 20, user_bytes=4096)
    src = [torch.randn(n * P, device="cuda") for _ in range(P)]
    blocks = [s[:n].clone() for s in src]
    ar, rs = [torch.zeros(n, device="cuda") for _ in range(P)], [torch.zeros(n, device="cuda") for _ in range(P)]
    ag = [torch.zeros(n * P, device="cuda") for _ in range(P)]

    def calls(m):
        chb.all_reduce(comm, [b[:m] for b in blocks], out=[x[:m] for x in ar])
        chb.reduce_scatter(comm, [s[:m * P] for s in src], out=[x[:m] for x in rs])
        chb.all_gather(comm, [b[:m] for b in blocks], out=[x[:m * P] for x in ag])

    calls(n - 1)                                            # (loads the kernels)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        calls(n)
    for m in range(16, 1516):                               # (the smallest ones belong to another row of the tuned table)
        calls(m)
    for x in ar + rs + ag:
        x.zero_()
    graph.replay()
    full = chb.all_reduce(comm, src, algo="ll")             # operands in rank order, as here
    for r in range(P):
        assert torch.equal(ar[r], full[0][:n]) and torch.equal(rs[r], full[0][r * n:(r + 1) * n])
        assert torch.equal(ag[r], torch.cat(blocks))
    comm.check()
    comm.close()


def test_a_captured_call_keeps_to_tables_that_are_there(cuda):
    """Recursive doubling of 512 elements runs in lockstep on aligned buffers and with flagged lines on skewed ones: captured
    on skewed buffers after calls on aligned ones it stays in lockstep, where no table has to be uploaded."""
    P, n = 8, 512
    p = chb.Program("allreduce", "recursive_doubling", P, n, 2, 1, in_symmetric=True, out_symmetric=True)
    assert p.lock_preferred(0, True) and not p.lock_preferred(0, False)
    comm = Communicator.emulated(P, scratch_bytes=4 << 20, user_bytes=4096)
    src = [torch.randn(n + 1, device="cuda") for _ in range(P)]
    chb.all_reduce(comm, [s[:n].clone() for s in src], algo="recursive_doubling")
    chb.all_reduce(comm, [s[1:3] for s in src], algo="recursive_doubling")      # (loads the kernel for other alignments)
    ins, outs = [s[1:] for s in src], [torch.zeros(n + 1, device="cuda")[1:] for _ in range(P)]
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        chb.all_reduce(comm, ins, out=outs, algo="recursive_doubling")
    graph.replay()
    want = chb.all_reduce(comm, ins, algo="recursive_doubling:pull")
    assert all(torch.equal(x, y) for x, y in zip(outs, want))
    comm.check()
    comm.close()
