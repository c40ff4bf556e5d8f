"""What the performance of this library is measured on.

Every case is one call (or one optimizer step) that a user's program makes through the public entry points, with
all ranks of the world emulated on one GPU (``Communicator.emulated``), or in a world of one rank.  Kinds:

``collective``  all_reduce / reduce_scatter / all_gather / all_to_all on P ranks.  ``count`` is the length of the
                vector for an allreduce and of one block for the others; ``registered`` says that the buffers come
                from the peer-visible region (``comm.empty``), as the data-parallel wrapper's do.
``fp8``         reduce-scatter with the fp8 wire format, blocks of ``count`` elements.
``shard``       sharded optimizer step: reduce-scatter fused with AdamW on shards of ``count`` elements, then the
                in-place allgather of the bf16 parameters.
``bucket``      data-parallel gradient bucket in a world of one rank: fill from bf16 gradients, allreduce, AdamW.
"""
import math

import torch

import configurable_hierarchical_allreduce_algorithms_b200 as chb
from configurable_hierarchical_allreduce_algorithms_b200.ops import fused

MIB = 1 << 20
DTYPE = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16, "int32": torch.int32}
SIZE = {"fp32": 4, "bf16": 2, "fp16": 2, "int32": 4}
HYPER = {"lr": 3e-4, "betas": (0.9, 0.95), "eps": 1e-8, "weight_decay": 0.1, "step": 10}
MAX_VECTOR = 64 * MIB      # bytes of one rank's long vector in the drawn collectives


def _coll(coll, algo, P, count, dtype="fp32", k=2, b=1, op="sum", scaled=False, registered=False):
    return {"kind": "collective", "coll": coll, "algo": algo, "P": P, "count": count, "dtype": dtype, "k": k, "b": b,
            "op": op, "scaled": scaled, "registered": registered}


def listed():
    cases = {
        # the smallest message of the allreduce sweep's tuned table: a handful of scalars (a loss, a norm, a flag)
        "allreduce 32 B": _coll("allreduce", "auto", 8, 8),
        # latency-bound tensor-parallel sized activations
        "allreduce 32 KiB bf16": _coll("allreduce", "auto", 8, 16 << 10, "bf16"),
        # a vector whose length the ranks do not divide (odd, fp16): one rank short of 1 MiB
        "allreduce 1 MiB odd fp16": _coll("allreduce", "auto", 8, (512 << 10) - 1, "fp16"),
        # hierarchical schedule at a middle size, as the (k, b) sweeps run it
        "allreduce 4 MiB k4 b2": _coll("allreduce", "radix_batch", 8, 1 << 20, k=4, b=2),
        # one 25 MB gradient bucket of the data-parallel path, registered buffers, 1/P fused
        "allreduce 25 MiB bucket": _coll("allreduce", "auto", 8, 25 * MIB // 4, scaled=True, registered=True),
        # two-level schedule on ordinary (staged) buffers at a bandwidth-bound size
        "allreduce 64 MiB bf16 k2 b4": _coll("allreduce", "radix_batch:pull", 8, 32 << 20, "bf16", k=2, b=4),
        # reduce-scatter of blocks with an odd length: no block but the first is aligned
        "reduce-scatter odd bf16": _coll("reduce_scatter", "radix_batch", 8, 1_000_003, "bf16", k=4, b=2),
        # parameter allgather of a sharded model, registered buffers
        "allgather 8 MiB bf16": _coll("allgather", "auto", 8, 4 << 20, "bf16", registered=True),
        # gradient reduce-scatter with the compressed wire format
        "fp8 reduce-scatter bf16": {"kind": "fp8", "P": 8, "count": 4 << 20, "dtype": "bf16", "scaled": True},
        # one sharded optimizer step (a slice of the 1.3B decoder's parameters on 8 ranks)
        "sharded AdamW step": {"kind": "shard", "P": 8, "count": 2 << 20},
        # one bucket of a GPT-2-medium-shaped decoder (width 1024): MLP weight, projection, biases
        "gradient bucket": {"kind": "bucket", "width": 1024, "accumulate": False},
        # the benchmark's default: 1 GiB of fp32 in a world of one rank
        "allreduce 1 GiB one rank": _coll("allreduce", "auto", 1, 256 << 20, registered=True),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("allreduce", "reduce_scatter", "allgather", "alltoall", "one", "fp8", "shard", "bucket"),
                       (6, 3, 3, 1, 1, 2, 2, 2))[0]
    P = rng.choice((2, 4, 4, 8, 8, 8, 3, 6))
    if kind == "fp8":
        return {"kind": "fp8", "P": P, "count": 128 * _log(rng, 8, 32 << 10), "dtype": rng.choice(("bf16", "fp32")),
                "scaled": rng.random() < 0.7}
    if kind == "shard":
        return {"kind": "shard", "P": rng.choice((1, 2, 4, 8)), "count": 64 * _log(rng, 64, 32 << 10)}
    if kind == "bucket":
        return {"kind": "bucket", "width": _log(rng, 64, 1024), "accumulate": rng.random() < 0.5}
    if kind == "one":
        return _coll("allreduce", "auto", 1, _log(rng, 64, 128 << 20), rng.choice(("fp32", "bf16")), registered=True)
    dtype = rng.choice(("fp32", "fp32", "bf16", "bf16", "fp16", "int32"))
    nbytes = _log(rng, 32, MAX_VECTOR)                     # the long vector of one rank
    count = max(1, nbytes // SIZE[dtype] // P)             # one block; odd ones are the rule
    if rng.random() < 0.5:
        count = (count + 15) // 16 * 16                    # ... and half of the blocks are 32-byte multiples
    op = "sum" if kind in ("allgather", "alltoall") or rng.random() < 0.8 else rng.choice(("max", "min"))
    b = rng.choice([d for d in (1, 2, 3, 4, 8) if P % d == 0])
    k = rng.choice((2, 3, 4, 8))
    if kind == "allreduce":
        algo = rng.choice(("auto", "auto", "auto", "radix_batch", "radix_batch", "ring", "recursive_doubling",
                           "reduce_scatter_allgather"))
        if algo == "auto" and rng.random() < 0.4:
            count = count * P + rng.randrange(P)           # any length
        else:
            count = count * P
    elif kind == "reduce_scatter":
        algo = rng.choice(("auto", "auto", "radix_batch", "radix_batch", "pairwise", "recursive_halving"))
    elif kind == "allgather":
        algo = rng.choice(("auto", "auto", "radix_batch", "k_brucks", "ring"))
    else:
        algo = rng.choice(("tuna", "linear"))
    scaled = op == "sum" and dtype != "int32" and kind in ("allreduce", "reduce_scatter") and rng.random() < 0.3
    return _coll(kind, algo, P, count, dtype, k, b, op, scaled, rng.random() < 0.5)


def _lens(case):
    """Elements of one rank's input and output."""
    P, n = case["P"], case["count"]
    return {"allreduce": (n, n), "reduce_scatter": (n * P, n), "allgather": (n, n * P), "alltoall": (n * P, n * P)}[case["coll"]]


def _values(g, n, dtype):
    """Uniform in [-1, 1), or small integers."""
    if dtype == torch.int32:
        return torch.randint(0, 97, (n,), generator=g, device="cuda", dtype=dtype)
    return torch.rand(n, generator=g, device="cuda").mul_(2.0).sub_(1.0).to(dtype)


def _inputs(case, seed):
    """The values that prepare() hands to the call; exact() starts from the same ones."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "collective":
        return [_values(g, _lens(case)[0], DTYPE[case["dtype"]]) for _ in range(case["P"])]
    if kind == "fp8":
        return [_values(g, case["P"] * case["count"], DTYPE[case["dtype"]]) for _ in range(case["P"])]

    def normal(n, s):
        return torch.randn(n, generator=g, device="cuda") * s

    if kind == "shard":
        P, n = case["P"], case["count"]
        grads = [normal(P * n, 1e-2) for _ in range(P)]
        return grads, [normal(n, 2e-2) for _ in range(P)], [normal(n, 1e-3) for _ in range(P)], \
            [normal(n, 1e-2).square() for _ in range(P)]
    shapes = _bucket(case)
    n = sum((s + 3) // 4 * 4 for s in shapes)
    return [normal(s, 1e-2).bfloat16() for s in shapes], normal(n, 1e-2), normal(n, 2e-2), normal(n, 1e-3), normal(n, 1e-2).square()


def _bucket(case):
    """Parameters of one bucket in the order in which backward reaches them."""
    d = case["width"]
    return [4 * d * d, d, d * d, 3 * d]


def _one(comm, xs):
    return xs if comm.nlocal > 1 else xs[0]


def _registered(comm, numel, dtype):
    t = comm.empty(numel, dtype)
    views = [x.view(-1) for x in (t if comm.nlocal > 1 else [t])]
    for x in views:
        x.owner = comm      # the memory is the communicator's: a result that is kept keeps it too
    return views


def prepare(case, seed):
    xs = _inputs(case, seed)
    kind, P = case["kind"], case.get("P", 1)
    if kind == "collective":
        dtype = DTYPE[case["dtype"]]
        n_in, n_out = _lens(case)
        esz = SIZE[case["dtype"]]
        user = (n_in + n_out) * esz + 4096 if case["registered"] else 4096
        comm = chb.Communicator.emulated(P, ll_bytes=(4 * MIB if P > 1 else 4096), user_bytes=user,
                                         scratch_bytes=5 * max(n_in, n_out) * esz + 64 * 1024 if P > 1 else MIB)
        if case["registered"]:
            ins, outs = _registered(comm, n_in, dtype), _registered(comm, n_out, dtype)
            for dst, src in zip(ins, xs):
                dst.copy_(src)
        else:
            ins, outs = xs, [torch.empty(n_out, dtype=dtype, device="cuda") for _ in range(P)]
        kw = {"algo": case["algo"], "k": case["k"], "b": case["b"]}
        if case["coll"] in ("allreduce", "reduce_scatter"):
            kw.update(op=case["op"], scale=1.0 / P if case["scaled"] else 1.0)
        fn = {"allreduce": chb.all_reduce, "reduce_scatter": chb.reduce_scatter, "allgather": chb.all_gather,
              "alltoall": chb.all_to_all}[case["coll"]]
        return {"kind": kind, "comm": comm, "fn": fn, "x": _one(comm, ins), "out": _one(comm, outs), "kw": kw}
    if kind == "fp8":
        n = case["count"]
        comm = chb.Communicator.emulated(P, scratch_bytes=P * n + P * n // 32 + 4096, user_bytes=4096)
        out = [torch.empty(n, dtype=DTYPE[case["dtype"]], device="cuda") for _ in range(P)]
        return {"kind": kind, "comm": comm, "x": xs, "out": out, "scale": 1.0 / P if case["scaled"] else 1.0}
    if kind == "shard":
        grads, w, m, v = xs
        n = case["count"]
        comm = chb.Communicator.emulated(P, scratch_bytes=4 * P * n + MIB, user_bytes=P * n * 6 + 8192)
        flat_g, flat_p = _registered(comm, P * n, torch.float32), _registered(comm, P * n, torch.bfloat16)
        for dst, src in zip(flat_g, grads):
            dst.copy_(src)
        shards = [flat_p[r][r * n:(r + 1) * n] for r in range(P)]
        return {"kind": kind, "comm": comm, "grad": _one(comm, flat_g), "w": _one(comm, w), "m": _one(comm, m),
                "v": _one(comm, v), "shard": _one(comm, shards), "param": _one(comm, flat_p), "scale": 1.0 / P}
    grads, acc0, w, m, v = xs
    n = acc0.numel()
    comm = chb.Communicator.emulated(1, scratch_bytes=MIB, user_bytes=8 * n + 8192)
    (acc,), (red,) = _registered(comm, n, torch.float32), _registered(comm, n, torch.float32)
    acc.copy_(acc0)
    items, off = [], 0
    for t in grads:
        items.append((t, off, not case["accumulate"]))
        off += (t.numel() + 3) // 4 * 4
    return {"kind": kind, "comm": comm, "items": items, "acc": acc, "red": red, "w": w, "m": m, "v": v,
            "param": torch.zeros(n, dtype=torch.bfloat16, device="cuda")}


def run(state):
    comm, kind = state["comm"], state["kind"]
    if kind == "collective":
        return state["fn"](comm, state["x"], out=state["out"], **state["kw"])
    if kind == "fp8":
        return fused.reduce_scatter_fp8(comm, state["x"], out=state["out"], scale=state["scale"])
    if kind == "shard":
        fused.reduce_scatter_adam(comm, state["grad"], state["w"], state["m"], state["v"], state["shard"],
                                  grad_scale=state["scale"], **HYPER)
        chb.all_gather(comm, state["shard"], out=state["param"])
        return {k: state[k] for k in ("w", "m", "v", "param")}
    fused.bucket_fill(state["acc"], state["items"])
    chb.all_reduce(comm, state["acc"], out=state["red"])
    fused.adam_flat(state["red"], state["w"], state["m"], state["v"], state["param"], **HYPER)
    return {k: state[k] for k in ("acc", "red", "w", "m", "v", "param")}


def work(case):
    kind, P = case["kind"], case.get("P", 1)
    if kind == "collective":
        n_in, n_out = _lens(case)
        reduces = case["coll"] in ("allreduce", "reduce_scatter")
        return {"bytes": P * (n_in + n_out) * SIZE[case["dtype"]], "flops": (P - 1) * n_in if reduces else 0}
    if kind == "fp8":
        n, esz = case["count"], SIZE[case["dtype"]]
        return {"bytes": P * P * n * esz + P * n * esz, "flops": (P - 1) * P * n}
    if kind == "shard":
        n = P * case["count"]                              # all shards: state read and written, parameters gathered
        return {"bytes": P * 4 * n + 24 * n + P * 2 * n, "flops": (P - 1) * n + 20 * n}
    n = sum(_bucket(case))
    return {"bytes": (36 + (4 if case["accumulate"] else 0)) * n, "flops": 20 * n}


def tolerance(case):
    kind = case["kind"]
    if kind == "collective":
        copies = case["coll"] in ("allgather", "alltoall") or case["op"] != "sum" or case["dtype"] == "int32" or case["P"] == 1
        return "exact" if copies else {"rel": {"fp32": 5e-7, "fp16": 1.5e-3, "bf16": 1.5e-2}[case["dtype"]]}
    if kind == "fp8":       # another rounding of a scale moves a few values to the next e4m3 step
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
    return {"rel": 7e-3}    # the bf16 parameters; the fp32 state is far closer


def _adam(g, w, m, v):
    """AdamW in 64 bits: new master, moments."""
    b1, b2 = HYPER["betas"]
    m = b1 * m + (1 - b1) * g
    v = b2 * v + (1 - b2) * g * g
    step = (m / (1 - b1 ** HYPER["step"])) / ((v / (1 - b2 ** HYPER["step"])).sqrt() + HYPER["eps"])
    return w - HYPER["lr"] * (step + HYPER["weight_decay"] * w), m, v


def _sum64(xs):
    total = xs[0].double()
    for x in xs[1:]:
        total += x
    return total


def exact(case, seed):
    xs = _inputs(case, seed)
    kind, P = case["kind"], case.get("P", 1)
    if kind == "collective":
        if case["coll"] == "allgather":
            full = torch.cat(xs).double()
            return [full] * P if P > 1 else full
        if case["coll"] == "alltoall":
            n = case["count"]
            return [torch.cat([x[r * n:(r + 1) * n] for x in xs]).double() for r in range(P)]
        if case["op"] == "sum":
            full = _sum64(xs) * (1.0 / P if case["scaled"] else 1.0)
        else:
            full = xs[0].double()
            for x in xs[1:]:
                full = (torch.maximum if case["op"] == "max" else torch.minimum)(full, x.double())
        if case["coll"] == "reduce_scatter":
            n = case["count"]
            return [full[r * n:(r + 1) * n] for r in range(P)]
        return [full] * P if P > 1 else full
    if kind == "fp8":       # what the call approximates: the sum of the unquantised blocks
        full = _sum64(xs) * (1.0 / P if case["scaled"] else 1.0)
        n = case["count"]
        return [full[r * n:(r + 1) * n] for r in range(P)]
    if kind == "shard":
        grads, w, m, v = xs
        n = case["count"]
        full = _sum64(grads) / P
        new = [_adam(full[r * n:(r + 1) * n], w[r].double(), m[r].double(), v[r].double()) for r in range(P)]
        flat = torch.cat([x[0] for x in new])
        out = {"w": [x[0] for x in new], "m": [x[1] for x in new], "v": [x[2] for x in new], "param": [flat] * P}
        return out if P > 1 else {k: x[0] for k, x in out.items()}
    grads, acc0, w, m, v = xs
    acc, off = acc0.double(), 0
    for t in grads:
        slot = acc[off:off + t.numel()]
        slot.copy_(slot + t.double() if case["accumulate"] else t.double())
        off += (t.numel() + 3) // 4 * 4
    new_w, new_m, new_v = _adam(acc, w.double(), m.double(), v.double())
    return {"acc": acc, "red": acc, "w": new_w, "m": new_m, "v": new_v, "param": new_w}
