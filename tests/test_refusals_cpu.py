"""What the Python entry points say about dense tensors that the native call did not take (no GPU: a stand-in that takes
nothing, and the check for CUDA tensors off)."""
import pytest
import torch

import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200 import _lib
from tiny_vllm_b200.quantization import cuda as Q


class TakesNothing:
    def __getattr__(self, name):
        return lambda *args: None


@pytest.fixture(autouse=True)
def no_gpu(monkeypatch):
    monkeypatch.setattr(Q, "_native", TakesNothing)
    monkeypatch.setattr(Q, "_require_cuda", lambda *tensors: None)


def tensors(M=4, N=8, K=20):
    return {"x": torch.zeros(M, K, dtype=torch.bfloat16), "xq": torch.zeros(M, K, dtype=torch.int8),
            "a_s": torch.ones(M), "w": torch.zeros(N, K, dtype=torch.int8), "s": torch.ones(N)}


CALLS = {
    "quantise": lambda t: Q.quantize_activation_int8(t["x"]),
    "norm": lambda t: Q.add_rmsnorm_quantize_int8(t["x"], torch.ones(20, dtype=torch.bfloat16), 1e-6),
    "silu": lambda t: Q.silu_mul_quantize_int8(t["x"]),
    "w8a16": lambda t: Q.apply_int8_weight_only_linear(t["x"], t["w"], t["s"]),
    "w8a8": lambda t: Q.apply_w8a8_linear(t["xq"], t["a_s"], t["w"], t["s"], out_dtype=torch.bfloat16),
    "i32": lambda t: Q.w8a8_int32_accumulators(t["xq"], t["w"]),
}


@pytest.mark.parametrize("name", CALLS)
def test_a_shape_is_named(name):
    with pytest.raises(_lib.B200QError, match=r"unsupported shape.*M=4.*[KI]=(20|10)") as e:
        CALLS[name](tensors())
    assert e.value.code == _lib.ERR_UNSUPPORTED_SHAPE


@pytest.mark.parametrize("name", ["w8a16", "w8a8", "i32"])
def test_tensors_on_two_devices_are_named(name):
    t = tensors()
    t["w"] = t["w"].to("meta")
    with pytest.raises(RuntimeError, match="must be on one GPU"):
        CALLS[name](t)
