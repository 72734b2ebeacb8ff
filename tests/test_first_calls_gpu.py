"""The first call of a process where a program may make it: inside a stream capture, and on several threads at once."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

CAPTURED = """
import torch
from litinfer_b200 import kernels as K
a, w, out = torch.randn(ROWS, 256, device="cuda"), torch.randn(300, 256, device="cuda"), torch.zeros(ROWS, 300, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    K.linear(a, w, None, out)
g.replay()
torch.cuda.synchronize()
# float32 sums of 256 products of numbers about 1, in two orders
assert float((out.double() - a.double() @ w.double().T).abs().max()) < 1e-3
"""

THREADS = """
import threading, torch
from litinfer_b200 import kernels as K
K.library()
a, w = torch.randn(3, 256, device="cuda"), torch.randn(300, 256, device="cuda")
outs, failed = [torch.zeros(3, 300, device="cuda") for _ in range(16)], []
torch.cuda.synchronize()
start = threading.Barrier(16)
def work(out):
    start.wait()
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            K.linear(a, w, None, out)
            torch.cuda.current_stream().synchronize()
    except Exception as e:
        failed.append(e)
threads = [threading.Thread(target=work, args=(o,)) for o in outs]
[t.start() for t in threads]
[t.join() for t in threads]
start = threading.Barrier(1)
outs.append(torch.zeros(3, 300, device="cuda"))
late = threading.Thread(target=work, args=(outs[-1],))
late.start()
late.join()
assert not failed, failed
assert all(torch.equal(o, outs[0]) for o in outs)
"""

FORM_CAPTURED = """
import torch
from litinfer_b200 import kernels as K
g = torch.Generator(device="cuda").manual_seed(1)
w = (torch.randn(1536, 8960, generator=g, device="cuda") * 8960 ** -0.5).to(torch.bfloat16)
a = torch.randn(64, 8960, generator=g, device="cuda").to(torch.bfloat16)
one, out = torch.zeros(1, 1536, device="cuda"), torch.zeros(64, 1536, device="cuda")
K.linear(a[:1], w, None, one)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    K.linear(a, w, None, out)
graph.replay()
torch.cuda.synchronize()
assert float((out - a.float() @ w.float().T).abs().max()) < 1e-4
"""


def run(program):
    r = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("rows", [3, 40])
def test_float32_product_captured_before_any_other_call(rows):
    run(CAPTURED.replace("ROWS", str(rows)))


def test_float32_product_first_called_by_many_threads():
    run(THREADS)


def test_another_form_of_the_streaming_product_first_called_inside_a_capture():
    """Its workspace is there from a call with one token; its limits and its depth are asked for inside the capture."""
    run(FORM_CAPTURED)

