"""Row-wise kernels at every split of a row over threads and chunks: the same codes and scales as the
stand-alone quantiser on the value formed, and sums of squares that do not depend on the split."""
import pytest
import torch

from oracle import quant_linear_oracle as O
from tests.gpu_util import bits, device_status_ok
import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200.quantization.cuda import (add_rmsnorm_quantize_int8, quantize_activation_int8,
                                              silu_mul_quantize_int8)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16, 272, 1024, 1040, 3072, 4112, 12288])
def test_results_do_not_depend_on_the_number_of_rows(K):
    dtype = torch.bfloat16 if K % 32 else torch.float16
    M = 300 * 1024 // K * 8 * 4 + 3          # more than three waves of one-chunk threads
    g = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    res = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (1 + 0.2 * torch.randn(K, device="cuda", generator=g)).to(dtype)
    q, s = quantize_activation_int8(x)
    nq, ns, nres, normed = add_rmsnorm_quantize_int8(x, w, 1e-6, res, return_normed=True)
    gate_up = torch.cat([x, res], dim=1)
    aq, as_, act = silu_mul_quantize_int8(gate_up, return_act=True)
    for rows in (slice(0, 5), slice(M - 3, M), slice(0, M // 3)):
        part = [quantize_activation_int8(x[rows]), add_rmsnorm_quantize_int8(x[rows], w, 1e-6, res[rows], True),
                silu_mul_quantize_int8(gate_up[rows], True)]
        assert torch.equal(part[0][0], q[rows]) and torch.equal(part[0][1], s[rows])
        assert torch.equal(part[1][0], nq[rows]) and torch.equal(part[1][1], ns[rows])
        assert torch.equal(bits(part[1][2]), bits(nres[rows])) and torch.equal(bits(part[1][3]), bits(normed[rows]))
        assert torch.equal(part[2][0], aq[rows]) and torch.equal(bits(part[2][2]), bits(act[rows]))
    ref = O.quantize_per_row_dynamic(x[:40].cpu())
    assert torch.equal(q[:40].cpu(), ref[0]) and torch.equal(s[:40].cpu().flatten(), ref[1].flatten())
    ref = O.quantize_per_row_dynamic(normed[-40:].cpu())
    assert torch.equal(nq[-40:].cpu(), ref[0]) and torch.equal(ns[-40:].cpu().flatten(), ref[1].flatten())
    assert device_status_ok()
