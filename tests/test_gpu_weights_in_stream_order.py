"""Weights written in stream order directly before the call that uses them: the GEMM kernels read weights before they
wait for their predecessor, so whoever writes them must have ended by then."""
import pytest
import torch

from tests.gpu_util import bits, device_status_ok
import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200.quantization.cuda import (apply_int8_weight_only_linear, quantize_activation_int8,
                                              w8a8_linear_dynamic)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("writer", ["quantiser", "copy", "torch"])
@pytest.mark.parametrize("scheme", ["w8a8", "w8a16"])
@pytest.mark.parametrize("M,N,K", [(1, 1024, 1024), (8, 4096, 1024), (16, 6144, 4096), (40, 1024, 3072),
                                   (300, 4096, 1024), (700, 6144, 4096), (8, 24576, 4096),
                                   (1100, 2048, 2048), (1, 6144, 4096)])
def test_weights_written_by_the_work_ahead(M, N, K, scheme, writer):
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    fn = w8a8_linear_dynamic if scheme == "w8a8" else apply_int8_weight_only_linear
    w16 = torch.empty(N, K, device="cuda", dtype=torch.bfloat16)
    w8, s = torch.empty(N, K, device="cuda", dtype=torch.int8), torch.empty(N, device="cuda")
    new8, new_s = torch.empty_like(w8), torch.empty_like(s)

    def step():
        y0 = fn(x, w8, s, None)          # a kernel of the library that lets its successor start at once
        if writer == "quantiser":
            w, scale = quantize_activation_int8(w16)
        else:
            w, scale = w8, s
            if writer == "copy":
                w.copy_(new8)
                scale.copy_(new_s)
            else:
                torch.add(new_s, 0.0, out=scale)
                torch.mul(new8, 1, out=w)
        return y0, fn(x, w, scale, None)

    def fresh():
        w16.copy_(torch.randn(N, K, device="cuda", generator=gen))
        q, qs = quantize_activation_int8(w16)
        new8.copy_(q)
        new_s.copy_(qs)
        torch.cuda.synchronize()
        expect = fn(x, q, qs, None)
        torch.cuda.synchronize()
        return expect

    fresh()
    w8.copy_(new8)
    s.copy_(new_s)
    step()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _, y = step()
    for _ in range(4):                # new weights each time: a read of the old ones shows
        expect = fresh()
        graph.replay()
        assert torch.equal(bits(y), bits(expect))
        assert torch.equal(bits(step()[1]), bits(expect))
    assert device_status_ok()
