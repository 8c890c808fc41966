"""CPU check of an ordering that no run shows: a kernel's dependents may start only behind its tensor-memory allocation."""
import glob
import os
import re

import pytest

import __graft_entry__ as entry

SOURCES = sorted(glob.glob(os.path.join(entry.PKG_DIR, "csrc", "*.cu")))
TRIGGER = re.compile(r"md_pdl_launch_dependents\(\);|griddepcontrol\.launch_dependents")


def kernels_with_tensor_memory():
    for path in SOURCES:
        for body in open(path).read().split("__global__")[1:]:
            if "tcgen05.alloc" in body:
                yield os.path.basename(path), body


def test_kernels_with_tensor_memory_are_found():
    assert {f for f, _ in kernels_with_tensor_memory()} == {"attention_latent_tc.cu", "attention_tc.cu", "gemm_pair.cu",
                                                            "gemm_skinny.cu", "gemm_tc.cu"}


@pytest.mark.parametrize("name,body", list(kernels_with_tensor_memory()), ids=lambda v: v if v.endswith(".cu") else "")
def test_dependents_start_behind_the_allocation(name, body):
    """A CTA of the dependent grid that allocated first would keep the columns until this grid has ended, and this grid would wait
    for them: the trigger stands behind the allocation and the barrier that makes it known to the whole CTA."""
    triggers = [m.start() for m in TRIGGER.finditer(body)]
    allocated = body.index("__syncthreads();", body.index("tcgen05.alloc"))
    assert triggers and min(triggers) > allocated, name
