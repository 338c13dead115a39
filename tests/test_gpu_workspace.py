"""The scratch buffer behind the Python entry points: allocated by the first call that needs one, so a capture is refused
for such a call and for no other, and kept for the graphs that were captured with it.  Each case is a process of its own: the buffer lives as long as the process."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

HEAD = """
import torch
import tiny_vllm_b200
from tiny_vllm_b200.quantization.cuda import (apply_int8_weight_only_linear, apply_w8a8_linear, reserve_workspace,
                                              quantize_activation_int8, w8a8_int32_accumulators, w8a8_linear_dynamic)
def problem(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    q = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8, generator=g)
    return x, q, torch.rand(N, device="cuda", generator=g) * 1e-3
def captured(fn):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = fn()
    return graph, y
"""

NEEDS_NONE = """
x, q, s = problem(128, 512, 8192)          # few tiles of a long K: split over a cluster, not through memory
xq, a_s = quantize_activation_int8(x)
torch.cuda.synchronize()
calls = [lambda: w8a8_linear_dynamic(x, q, s, None), lambda: w8a8_int32_accumulators(xq, q),
         lambda: apply_w8a8_linear(xq, a_s, q, s, out_dtype=torch.bfloat16)]
graphs = [captured(f) for f in calls]
for (graph, y), f in zip(graphs, calls):
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, f())
"""

NEEDS_SOME = """
x, q, s = problem(3000, 2048, 2048)        # W8A16 prefill: the expanded weights
fn = lambda: apply_int8_weight_only_linear(x, q, s)
torch.cuda.synchronize()
try:
    captured(fn)
except RuntimeError as e:
    assert "during CUDA graph capture" in str(e), e
else:
    raise AssertionError("the capture was not refused")
reserve_workspace(1 << 20, "cuda")
graph, y = captured(fn)
graph.replay()
torch.cuda.synchronize()
assert torch.equal(y, fn())
"""


OUTGROWN = """
x, q, s = problem(3000, 2048, 2048)
fn = lambda: apply_int8_weight_only_linear(x, q, s)
expect = fn()
graph, y = captured(fn)                    # holds the address of the buffer of that moment
x2, q2, s2 = problem(3000, 8192, 8192)     # 128 MiB of expanded weights: more than the buffer has
apply_int8_weight_only_linear(x2, q2, s2)
others = [torch.full((4 << 20,), 7, dtype=torch.uint8, device="cuda") for _ in range(64)]   # from freed blocks first
graph.replay()
torch.cuda.synchronize()
assert all(bool((t == 7).all()) for t in others), "the graph wrote into another tensor"
assert torch.equal(y, expect)
"""


WIDE = """
x, q, s = problem(700, 24576, 2048)        # W8A16 at 513 to 1023 tokens of wide layers: none either
fn = lambda: apply_int8_weight_only_linear(x, q, s)
torch.cuda.synchronize()
graph, y = captured(fn)                    # without a call before it
graph.replay()
torch.cuda.synchronize()
expect = fn()
assert torch.equal(y, expect)
x2, q2, s2 = problem(700, 24576, 2064)
expect2 = apply_int8_weight_only_linear(x2, q2, s2)
a, b = torch.cuda.Stream(), torch.cuda.Stream()
torch.cuda.synchronize()
for _ in range(20):                        # two streams at once share nothing
    with torch.cuda.stream(a):
        ya = fn()
    with torch.cuda.stream(b):
        yb = apply_int8_weight_only_linear(x2, q2, s2)
    torch.cuda.synchronize()
    assert torch.equal(ya, expect) and torch.equal(yb, expect2)
"""


@pytest.mark.parametrize("body", [NEEDS_NONE, NEEDS_SOME, OUTGROWN, WIDE],
                         ids=["needs-none", "needs-some", "outgrown", "wide-layers"])
def test_capture_in_a_fresh_process(body):
    r = subprocess.run([sys.executable, "-c", HEAD + body], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
