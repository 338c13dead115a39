"""TMA descriptors of the kernels for tens to hundreds of tokens: encoded on the first pass over a weight, so a call
makes those that its kernel reads and no other, and a full table loses its oldest entries only."""
import pytest
import torch

from tests.gpu_util import device_status_ok, mid_plan
import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200 import _lib
from tiny_vllm_b200.quantization.cuda import apply_int8_weight_only_linear, apply_w8a8_linear

pytestmark = pytest.mark.gpu

TABLE = 8192


def encoded(fn):
    before = _lib.lib().b200q_debug_maps_encoded()
    fn()
    return _lib.lib().b200q_debug_maps_encoded() - before


def linear(op, M, N, K):
    q = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8)
    s = torch.rand(N, device="cuda")
    if op == _lib.OP_W8A16:
        x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
        return lambda w=q: apply_int8_weight_only_linear(x, w, s)
    xq = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8)
    a_s = torch.rand(M, device="cuda")
    return lambda w=q: apply_w8a8_linear(xq, a_s, w, s, out_dtype=torch.bfloat16)


@pytest.mark.parametrize("op", [_lib.OP_W8A8, _lib.OP_W8A16], ids=["w8a8", "w8a16"])
@pytest.mark.parametrize("K,pairs", [(1024, 1),     # whole blocks: 3-D maps of both operands
                                     (1040, 2),     # whole chunks and a partial block: 2-D maps too
                                     (48, 1)])      # less than a block: 2-D maps alone
def test_a_call_makes_the_descriptors_that_it_reads(op, K, pairs):
    M, N = 64, 264
    assert mid_plan(op, M, N, K) is not None
    fn = linear(op, M, N, K)
    assert encoded(fn) == 2 * pairs        # activations and weights
    assert encoded(fn) == pairs            # the weights' are kept
    assert device_status_ok()


def test_a_full_table_keeps_the_newer_descriptors():
    M, N, K = 64, 8, 128
    assert mid_plan(_lib.OP_W8A8, M, N, K) is not None
    fn = linear(_lib.OP_W8A8, M, N, K)
    weights = torch.randint(-127, 128, (TABLE + 8, N, K), device="cuda", dtype=torch.int8)
    for w in weights:
        fn(w)
    torch.cuda.synchronize()
    assert encoded(lambda: [fn(w) for w in weights[8:]]) == TABLE      # the activations' alone
    assert encoded(lambda: fn(weights[0])) == 2                        # the oldest had to go
    assert device_status_ok()
