"""Convolution calls under stream capture, each as the first of its process: what a
first call prepares must not end the capture."""
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import sys
import torch
from skewengine_gb300 import surrogate as sur
call, mode = sys.argv[1:]
g = torch.Generator(device="cuda").manual_seed(1)
x = torch.randn((2, 40, 48, 64), generator=g, device="cuda").to(torch.bfloat16)
w = torch.randn((64, sur.kpad(64)), generator=g, device="cuda").to(torch.bfloat16)
y = torch.randn((2, 40, 48, 64), generator=g, device="cuda").to(torch.bfloat16)
def run():
    if call == "forward":
        return [sur.conv3x3(x, w, None, True)]
    if call == "relu":
        return list(sur.relu_grad(x, y))
    return list(sur.conv3x3_backward(x, w, y, x))
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode=mode):
    got = run()
graph.replay()
torch.cuda.synchronize()
for a, b in zip(got, run()):
    # (The weight gradient's atomics add in any order.)
    assert torch.equal(a, b) or (call == "backward" and torch.allclose(a, b, rtol=1e-3, atol=1e-3)), call
print("captured")
"""


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("call", ["forward", "backward", "relu"])
def test_first_call_of_a_process_under_capture(gpu_lib, call, mode):
    p = subprocess.run([sys.executable, "-c", CODE, call, mode], capture_output=True, text=True, timeout=300, cwd=ROOT,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert p.returncode == 0 and "captured" in p.stdout, p.stderr[-2000:]
