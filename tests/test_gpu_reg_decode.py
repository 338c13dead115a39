"""Decode kernels that hold the weights in registers: each split of K, ragged channels and tokens, the
in-kernel quantisation, and chains in which every launch reads what the one before it wrote (the
weights are fetched ahead of that launch's end, the activations must not be)."""
import pytest
import torch

from oracle import quant_linear_oracle as O
from tests.gpu_util import bits, device_status_ok, forced_path, knobs
import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200.quantization.cuda import (apply_int8_weight_only_linear, apply_w8a8_linear,
                                              w8a8_int32_accumulators, w8a8_linear_dynamic)

pytestmark = pytest.mark.gpu

# K at the edges of the register splits (512, 1024, 1536, 2048, 3072, 4096), channels at tile edges
SHAPES = [(8, 16), (33, 512), (96, 528), (1000, 1040), (4096, 1024), (72, 1536), (1021, 1552), (256, 2064),
          (1024, 3072), (40, 3088), (264, 4096)]


@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("N,K", SHAPES)
def test_both_schemes(M, N, K, oracle_c_lib):
    dtype = torch.bfloat16 if (M + N) % 2 else torch.float16
    q, s = O.make_weight(N, K, seed=N + K)
    x = O.make_activation(M, K, seed=M, dtype=dtype)
    xq, a_s = O.quantize_per_row_dynamic(x)
    b = (torch.randn(N, generator=torch.Generator().manual_seed(M)) * 0.1).to(dtype)
    with forced_path("mma"), knobs(BULK_DECODE=1):
        acc = w8a8_int32_accumulators(xq.cuda(), q.cuda())
        y8 = apply_w8a8_linear(xq.cuda(), a_s.cuda(), q.cuda(), s.cuda(), b.cuda(), out_dtype=dtype)
        yd = w8a8_linear_dynamic(x.cuda(), q.cuda(), s.cuda(), b.cuda())   # in one kernel for few values
        y16 = apply_int8_weight_only_linear(x.cuda(), q.cuda(), s.cuda(), b.cuda())
    ref = O.w8a8_int32_accumulators(xq, q)
    assert torch.equal(acc.cpu(), ref)
    expect = bits(O.w8a8_native_epilogue(ref, a_s, s, b, dtype))
    assert torch.equal(bits(y8.cpu()), expect) and torch.equal(bits(yd.cpu()), expect)
    m = O.tensor_metrics(O.w8a16_native_reference(x, q, s, b), y16)
    assert m["relative_l2"] <= 4e-3 and m["cosine_similarity"] >= 0.9999, m
    assert device_status_ok()


@pytest.mark.parametrize("M", [1, 16, 40, 300])
@pytest.mark.parametrize("scheme", ["w8a8", "w8a16"])
def test_dependent_chains_in_a_graph(M, scheme):
    # decode and mid-size kernels start before their predecessor has ended: replayed as a graph, 40 layers
    # that feed each other give what they give with a synchronisation after each
    K = 1024
    gen = torch.Generator(device="cuda").manual_seed(M)
    ws = [torch.randint(-127, 128, (K, K), device="cuda", dtype=torch.int8, generator=gen) for _ in range(40)]
    s = torch.full((K,), 1 / (73 * K ** 0.5), device="cuda")
    x0 = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    fn = w8a8_linear_dynamic if scheme == "w8a8" else apply_int8_weight_only_linear

    def run(sync):
        x = x0
        for w in ws:
            x = fn(x, w, s, None)
            if sync:
                torch.cuda.synchronize()
        return x

    expect = run(True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = run(False)
    for _ in range(5):
        y.zero_()
        graph.replay()
        assert torch.equal(bits(y), bits(expect))
    assert device_status_ok()
