"""Chains in which every linear reads what the one before it wrote, for each kernel family: captured in a graph, where
kernels start before their predecessors have ended, they give what they give with a synchronisation after each."""
import pytest
import torch

from tests.gpu_util import bits, device_status_ok, forced_path, knobs
import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200.quantization.cuda import apply_int8_weight_only_linear, w8a8_linear_dynamic

pytestmark = pytest.mark.gpu

LAYERS = 12
FAMILIES = {  # forced path, knobs, token counts
    "register-streaming": ("mma", {"NO_REG": 1, "BULK_DECODE": 1}, (1, 16, 40)),
    "ring": ("mma", {"BULK_DECODE": 2}, (1, 16)),
    "registers": ("mma", {"BULK_DECODE": 1}, (2, 16)),
    "mid": ("umma", {}, (16, 100, 300)),
    "persistent": ("umma", {"NO_MID": 1, "NO_PAIR": 1, "NO_TS": 1}, (40, 300)),
    "persistent-swap": ("umma_swap", {}, (40, 200)),
    "tensor-memory-weights": ("umma", {"NO_MID": 1, "NO_PAIR": 1}, (300,)),
    "pair": (None, {"NO_MID": 1, "PAIR_MIN_TILES": 1, "W8A16_PAIR_MIN_M": 512}, (600,)),
}
CASES = [(f, M, K) for f, (_, _, Ms) in FAMILIES.items() for M in Ms for K in (1024, 2112, 4096)]


@pytest.mark.parametrize("scheme", ["w8a8", "w8a16"])
@pytest.mark.parametrize("family,M,K", CASES)
def test_graph_equals_one_at_a_time(family, M, K, scheme):
    path, settings, _ = FAMILIES[family]
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    ws = [torch.randint(-127, 128, (K, K), device="cuda", dtype=torch.int8, generator=gen) for _ in range(LAYERS)]
    s = torch.full((K,), 1 / (73 * K ** 0.5), device="cuda")     # keeps the variance
    x0 = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    fn = w8a8_linear_dynamic if scheme == "w8a8" else apply_int8_weight_only_linear

    def run(sync):
        x = x0
        for w in ws:
            x = fn(x, w, s, None)
            if sync:
                torch.cuda.synchronize()
        return x

    with forced_path(path), knobs(**settings):
        expect = run(True)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = run(False)
    assert torch.isfinite(expect.float()).all() and 0.1 < expect.float().std() < 10
    for _ in range(4):
        y.zero_()
        graph.replay()
        assert torch.equal(bits(y), bits(expect))
    assert device_status_ok()
