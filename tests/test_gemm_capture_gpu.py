"""A prefill GEMM kernel whose first launch in the process is inside a stream capture (every split and epilogue is its own
kernel, and the shared-memory limit of one is raised at its first use)."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch
import qwen35x_b200 as q
torch.manual_seed(0)
w = q.Nvfp4Weight.from_device(*q.quantize_weight(torch.randn((512, 4096), device="cuda")))
cases = []
for m in (8, 130, 100):  # split in 8 and in 1, then a split again
    a = q.quantize_activations(torch.randn((m, 4096), device="cuda").to(torch.bfloat16))
    cases.append((m, a, torch.empty((m, 512), dtype=torch.bfloat16, device="cuda")))
torch.cuda.synchronize()
stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.stream(stream):
    with torch.cuda.graph(graph, stream=stream):
        for m, a, out in cases:
            q.gemm_w4a4(w, *a, m, out=out)
    graph.replay()
    stream.synchronize()
    for m, a, out in cases:
        assert torch.equal(out, q.gemm_w4a4(w, *a, m)), m
assert q.gemm_default_status() == 0
"""


def test_first_launch_inside_a_capture():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
