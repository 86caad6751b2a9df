"""What stands in front of a kernel's wait on the preceding grid, read from the sources: a kernel that lets its dependents in
before it has its tensor memory, or that reads the preceding kernel's output before the wait, hangs or races on a device."""
import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parents[1] / "dgpp_b200" / "csrc" / "kernels"


def kernels():
    for f in sorted(SRC.glob("*.cu")) + sorted(SRC.glob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
            depth, i = 0, text.index("{", m.end())
            for j in range(i, len(text)):
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                if depth == 0:
                    break
            yield m.group(1), text[i:j]


KERNELS = dict(kernels())
ALLOCATING = {name: body for name, body in KERNELS.items() if re.search(r"\btmem_alloc(_pair)?\(", body)}


def test_allocating_kernels_are_found():
    assert len(ALLOCATING) >= 13 and "attn_prefill_tc_kernel" in ALLOCATING and "gemm_tc_pair_kernel" in ALLOCATING


@pytest.mark.parametrize("name", sorted(ALLOCATING))
def test_dependents_are_let_in_behind_the_allocation(name):
    """The release of the next grid (`pdl_wait` carries it) stands behind the allocation, a barrier of the block between them."""
    body = ALLOCATING[name]
    alloc = re.search(r"\btmem_alloc(_pair)?\(", body).start()
    release = re.search(r"\b(pdl_wait|pdl_launch_dependents)\(\)", body)
    assert release is not None and release.start() > alloc
    between = body[alloc:release.start()]
    assert "__syncthreads()" in between or "cluster_barrier()" in between


@pytest.mark.parametrize("name", ["attn_decode_tc_kernel", "mla_decode_tc_kernel"])
def test_selection_lists_are_read_behind_the_wait(name):
    """The list of selected tokens or blocks is the output of the kernel before."""
    body = KERNELS[name]
    assert re.search(r"\bpdl_wait(_only)?\(\)", body).start() < re.search(r"= p\.sel \+", body).start()
