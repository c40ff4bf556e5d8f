"""Gradient bucket fill around its block of 4096 elements and its groups of eight, empty tensors among the others."""
import pytest
import torch

from configurable_hierarchical_allreduce_algorithms_b200.ops import fused

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("skew", [0, 1])
def test_block_and_group_edges(cuda, dtype, skew):
    sizes = [1, 7, 8, 9, 0, 4088, 4095, 4096, 4097, 8192, 8199, 100_000]
    g = torch.Generator(device="cuda").manual_seed(1)
    grads = [torch.randn(n + skew, generator=g, device="cuda").to(dtype)[skew:] for n in sizes]
    for overwrite in (True, False):
        offs, off = [], 0
        for n in sizes:
            offs.append(off)
            off += (n + 3) // 4 * 4 + 4                     # gaps, which stay as they are
        bucket = torch.randn(off, generator=g, device="cuda")
        want = bucket.clone()
        for t, o in zip(grads, offs):
            want[o:o + t.numel()] = t.float() if overwrite else want[o:o + t.numel()] + t.float()
        fused.bucket_fill(bucket, [(t, o, overwrite) for t, o in zip(grads, offs)])
        assert torch.equal(bucket, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("skew", [2, 4, 6, 8])
def test_views_at_every_alignment(cuda, dtype, skew):
    """Sources that start two to eight elements into their allocation: 16-bit ones on an 8-byte boundary keep vector loads
    (and their speed), the others go element by element."""
    sizes = [1, 8, 4095, 4096, 4097, 100_003]
    g = torch.Generator(device="cuda").manual_seed(skew)
    grads = [torch.randn(n + skew, generator=g, device="cuda").to(dtype)[skew:] for n in sizes]
    for overwrite in (True, False):
        offs = [sum((m + 3) // 4 * 4 for m in sizes[:i]) for i in range(len(sizes))]
        bucket = torch.randn(offs[-1] + sizes[-1], generator=g, device="cuda")
        want = bucket.clone()
        for t, o in zip(grads, offs):
            want[o:o + t.numel()] = t.float() if overwrite else want[o:o + t.numel()] + t.float()
        fused.bucket_fill(bucket, [(t, o, overwrite) for t, o in zip(grads, offs)])
        assert torch.equal(bucket, want)


def test_eight_byte_aligned_sources_are_as_fast(cuda):
    n = 32 << 20                                            # 192 MB in and out: beyond L2
    raw = torch.randn(n + 8, device="cuda").bfloat16()
    bucket = torch.empty(n, device="cuda")
    times = []
    for skew in (0, 4):
        items, best = [(raw[skew:skew + n], 0, True)], float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            fused.bucket_fill(bucket, items)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] < 1.3 * times[0], times
