"""A captured split-BF16 SGEMM whose workspace holds its pieces but not the sums of its K ranges (GPU):
it is accepted, over all of K.  In a process of its own, whose workspace no other call has grown."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch
import eigen_b200 as eb

def operands(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a = torch.rand((k, m), device="cuda", generator=g) * 2 - 1
    b = torch.rand((n, k), device="cuda", generator=g) * 2 - 1
    return a, b, torch.zeros((n, m), device="cuda")

eb.set_sgemm_method(eb.METHOD_EMULATED)
eb.set_tile_n(256)
s = torch.cuda.Stream()
# 148 tiles of 128 x 256 and one K chunk: no K ranges, a workspace of the pieces alone (8.8 MB)
m, n, k = 128 * 37, 1024, 256
a, b, c = operands(m, n, k)
assert eb.sgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m, stream=s.cuda_stream) == eb.EB2_OK
s.synchronize()
# 32 tiles in two K ranges: 6.3 MB of pieces and 8.4 MB of sums
m, n, k = 1024, 1024, 512
a, b, c = operands(m, n, k)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=s):
    rc = eb.sgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m, stream=s.cuda_stream)
    splits = eb.last_call_info()["splits"]
assert rc == eb.EB2_OK, eb.last_error()
assert splits == 1, splits
graph.replay()
torch.cuda.synchronize()
exact = b.double() @ a.double()
err = float((c.double() - exact).norm() / exact.norm())
assert err < 2.5e-7, err
# a direct call has room for the ranges
assert eb.sgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m, stream=s.cuda_stream) == eb.EB2_OK
assert eb.last_call_info()["splits"] == 2
s.synchronize()
err = float((c.double() - exact).norm() / exact.norm())
assert err < 2.5e-7, err
graph.replay()  # the workspace that the graph holds is still there
torch.cuda.synchronize()
print("done")
"""


def test_captured_call_without_room_for_the_ranges():
    root = Path(__file__).resolve().parents[1]
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
