"""Tensor memory and programmatic dependent launch, checked in the sources.

A CTA that allocates tensor memory waits until its SM has the columns.  If the kernel were to let the next one start
before that (any one thread's griddepcontrol.launch_dependents counts for its CTA), a CTA of the next kernel could take
the columns and then wait for this kernel to complete, which waits for the columns: neither ends.  Such a stop cannot be
tested by running it, so the order is checked where it is written down."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "gpt.c_b200", "csrc")


def code(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def kernels():
    """(file, text from one __global__ to the next) of every kernel."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for body in re.split(r"\b__global__\b", code(path))[1:]:
            yield os.path.basename(path), body


def test_next_kernel_is_let_start_by_the_thread_that_has_allocated():
    allocating = [(f, body) for f, body in kernels() if re.search(r"\btmem_alloc", body)]
    assert {f for f, _ in allocating} == {"attn_fwd_sm100.cu", "attn_bwd_sm100.cu", "linear_sm100.cu", "linear_split_sm100.cu"}
    for f, body in allocating:
        assert len(re.findall(r"\btmem_alloc_then_launch_dependents\(", body)) == 1, f
        assert not re.search(r"launch_dependents\(|launch_dependents;", body.replace("tmem_alloc_then_launch_dependents(", "")), \
            f"{f}: the next kernel is let start by something else than the allocation"


def test_allocation_comes_before_the_signal():
    headers = {os.path.basename(p): code(p) for p in glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.cu"))}
    assert [f for f, text in sorted(headers.items()) if "tcgen05.alloc" in text] == ["tc05.cuh"]
    text = headers["tc05.cuh"]
    body = text[text.index("tmem_alloc_then_launch_dependents("):]
    body = body[:body.index("\n}")]
    assert text.count("tcgen05.alloc") == 1 and 0 < body.index("tcgen05.alloc") < body.index("pdl_launch_dependents();")
