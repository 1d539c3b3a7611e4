"""Kernels that may start before the previous one of their stream has completed: what they read is only visible to a kernel
that has waited for it itself, so each of them waits, whatever its arguments.  Read from the sources: a kernel that does not
is a race on memory, which a run may or may not show."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "gpt.c_b200", "csrc")
WAIT = re.compile(r"^    (?:tc05::)?pdl_wait\(\);", re.M)  # a statement of the kernel's own block, under no condition
START = re.compile(r"pdl_launch_dependents\(\)|tmem_alloc_then_launch_dependents\(")


def kernels():
    """(name, body) of every kernel that lets the next one of the stream start early, or is launched that way itself."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        for m in re.finditer(r"__global__.*?\b(\w+_kernel)\(", text, re.S):
            name, body = m.group(1), text[m.end():text.index("\n}\n", m.end())]
            if START.search(body) or re.search(r"launch_\w*after_previous\([^;]*\b%s\b" % name, text):
                found.append((name, body))
    return found


def test_kernels_are_found():
    names = [n for n, _ in kernels()]
    assert {"linear_gemm_kernel", "linear_split_kernel", "bias_grad_kernel", "attn_fwd_kernel", "attn_bwd_kernel",
            "attn24_fwd_kernel", "attn24_bwd_kernel", "split_kernel", "ln_forward_kernel"} <= set(names)


@pytest.mark.parametrize("name,body", kernels(), ids=lambda v: v if len(v) < 64 else "")
def test_kernel_waits_for_the_one_before_it(name, body):
    assert WAIT.search(body), f"{name} can read what the previous kernel of the stream wrote without having waited for it"
