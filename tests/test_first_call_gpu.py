"""The first call of a process may be one that a stream captures: it may neither allocate nor synchronise."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SCRIPT = """
import sys
import torch
import __graft_entry__ as entry

pkg = entry.load_package()
L = pkg.lib()
name, C = sys.argv[1], int(sys.argv[2])
x = torch.randn(5, C, device="cuda")
y, targets, loss = torch.empty_like(x), torch.zeros(5, device="cuda"), torch.zeros(1, device="cuda")
w = torch.randn(64, C, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    st = torch.cuda.current_stream().cuda_stream
    if name == "xent":
        rc = L.xent_sm100_forward(x.data_ptr(), targets.data_ptr(), y.data_ptr(), loss.data_ptr(), 5, C, st)
    else:
        rc = L.linear_sm100_forward(x.data_ptr(), w.data_ptr(), None, y.data_ptr(), None, 5, 64, C, st)
assert rc == 0, rc
graph.replay()
assert pkg.device_status() == 0
if name == "xent":
    assert (y - torch.log_softmax(x.double(), -1)).abs().max().item() <= 1e-4
else:
    want = x.double() @ w.double().T
    got = y.flatten()[:5 * 64].view(5, 64)
    assert ((got - want).abs() <= 2.0 ** -8 * (x.abs().double() @ w.abs().double().T)).all()
"""


@pytest.mark.parametrize("name,C", [("xent", 50257), ("xent", 1000), ("linear", 768)])
def test_first_call_under_capture(name, C):
    r = subprocess.run([sys.executable, "-c", SCRIPT, name, str(C)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
