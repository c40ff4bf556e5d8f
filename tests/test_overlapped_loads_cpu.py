"""Kernels whose CTAs may be placed while their producer still runs read nothing through pointers that promise the compiler
unchanging memory (`const ... * __restrict__`); tables that are uploaded once are the exception."""
import re
from pathlib import Path

import configurable_hierarchical_allreduce_algorithms_b200 as chb

KERNELS = Path(chb.__file__).parent / "csrc" / "kernels"
NEVER_WRITTEN = {"blob"}


def functions(text):
    """(name, parameters, body) of every function with a body."""
    for m in re.finditer(r"\b(\w+)\(([^()]*(?:\([^()]*\)[^()]*)*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(2), text[m.end():i]


def test_no_read_only_promise_in_overlapped_kernels():
    seen = 0
    for f in sorted(KERNELS.glob("*.cu")):
        found = {name: (params, body) for name, params, body in functions(f.read_text())}
        overlapped = [n for n, (_, body) in found.items() if "dependent_launch();" in body]
        called = {n for n in found if any(re.search(rf"\b{n}\s*[<(]", found[k][1]) for k in overlapped)}
        for name in set(overlapped) | called:
            for pointer in re.findall(r"const[^,]*\*\s*__restrict__\s+(\w+)", found[name][0]):
                assert pointer in NEVER_WRITTEN, f"{f.name}: {name}({pointer})"
        seen += len(overlapped)
    assert seen >= 8


def test_tables_have_arrived_before_a_launch_reads_them():
    """A blocking copy from pageable memory may return before its last part is on the device, and launches on non-blocking
    streams do not wait for it: uploads that kernels read go through the helper that waits."""
    for f in sorted(KERNELS.parent.rglob("*.cu")):
        if "tools" not in f.parts:
            assert not re.search(r"\bcudaMemcpy\([^;]*HostToDevice", f.read_text()), f.name
    helper = next(body for name, _, body in functions((KERNELS.parent / "symm" / "comm.h").read_text()) if name == "upload_table")
    assert helper.index("cudaMemcpyHostToDevice") < helper.index("cudaStreamSynchronize")
