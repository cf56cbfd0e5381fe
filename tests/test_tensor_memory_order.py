"""Kernels that use tensor memory let their dependents start only after their own allocation.

tcgen05.alloc has no time limit: a dependent that takes the columns first and then waits for this kernel would never be waited out.
Read from the sources: such an order is not to be tried on a GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kungfu_b200", "csrc")


def _bodies():
    """(file, text) of every top-level definition that allocates tensor memory, comments removed."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                text = re.sub(r"//[^\n]*", "", f.read())
            for body in re.split(r"\n}", text):
                if "tcgen05.alloc" in body:
                    yield name, body


def test_the_kernels_are_found():
    assert {name for name, _ in _bodies()} >= {"gemm_tc.cu", "attention_prefill_tc.cu", "grouped_tc.cu"}
    assert sum(1 for _ in _bodies()) >= 6


@pytest.mark.parametrize("name,body", [pytest.param(n, b, id=f"{n}-{i}") for i, (n, b) in enumerate(_bodies())])
def test_dependents_start_after_the_allocation(name, body):
    alloc, trigger = body.index("tcgen05.alloc"), [m.start() for m in re.finditer(r"kf_pdl_trigger\(\)", body)]
    assert len(trigger) == 1, f"{name}: {len(trigger)} triggers beside one allocation"
    met = body.find("__syncthreads()", alloc)
    assert alloc < met < trigger[0], f"{name}: the dependent launch is triggered before every warp knows of the allocation"
