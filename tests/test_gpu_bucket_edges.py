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
