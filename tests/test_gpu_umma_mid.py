"""The tcgen05 kernel for tens to hundreds of tokens (two CTAs per SM, K split over a cluster whose
CTAs share the reduction): edges of its tiles, K tails, every tile width, cluster and ring shape."""
import pytest
import torch

from oracle import quant_linear_oracle as O
from tests.gpu_util import bits, device_status_ok, forced_path, knobs, mid_plan
import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200 import _lib
from tiny_vllm_b200.quantization.cuda import (apply_int8_weight_only_linear, apply_w8a8_linear,
                                              select_path, w8a8_int32_accumulators)

pytestmark = pytest.mark.gpu

SHAPES = [  # (M, N, K): one row of a tile, ragged everything, several token tiles, long and short K
    (1, 8, 1024), (17, 72, 1040), (33, 264, 1616), (77, 4096, 1024), (128, 768, 4096),
    (129, 1000, 528), (300, 1024, 3072), (512, 264, 2112), (40, 136, 96), (1500, 640, 1184), (20, 128, 16),
]


def takes(op, M, N, K, cluster, bn):
    """Every CTA of the cluster gets a chunk of 1, 2 or 4 K blocks; W8A16 clusters in two CTAs per SM at most."""
    if cluster is None or cluster == 1:
        return True
    if op == _lib.OP_W8A16 and -(-M // bn) * -(-N // 128) * cluster > 2 * 148:
        return False
    blocks = -(-K // (128 if op == _lib.OP_W8A8 else 64))
    chunks = [-(-blocks // kc) for kc in (1, 2, 4)]
    return any(-(-c // cluster) * (cluster - 1) < c for c in chunks)


@pytest.mark.parametrize("cluster,bn", [(None, None), (1, 32), (2, 64), (4, 128), (8, 64), (1, 256)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_both_schemes(M, N, K, cluster, bn, oracle_c_lib):
    dtype = torch.bfloat16 if M % 2 else torch.float16
    q, s = O.make_weight(N, K, seed=N + K)
    x = O.make_activation(M, K, seed=M, dtype=dtype)
    xq, a_s = O.quantize_per_row_dynamic(x)
    b = (torch.randn(N, generator=torch.Generator().manual_seed(M)) * 0.1).to(dtype)
    args = {k: v for k, v in (("CLUSTER", cluster), ("BN", bn)) if v is not None}
    # (a tile and cluster that do not fit a shape fall back to the family's persistent kernel)
    with forced_path("umma"), knobs(**args):
        assert select_path(_lib.OP_W8A8, M, N, K) == "umma_i8_tokens128"
        for op, tile in ((_lib.OP_W8A8, "channels"), (_lib.OP_W8A16, "tokens")):
            plan = mid_plan(op, M, N, K)         # ... and which ones these are is known
            assert (plan is not None) == takes(op, M, N, K, cluster, bn), (op, plan)
            assert plan is None or cluster is None or (plan["cluster"], plan[tile]) == (cluster, bn), (op, plan)
        ref = O.w8a8_int32_accumulators(xq, q)
        assert torch.equal(w8a8_int32_accumulators(xq.cuda(), q.cuda()).cpu(), ref)
        y = apply_w8a8_linear(xq.cuda(), a_s.cuda(), q.cuda(), s.cuda(), b.cuda(), out_dtype=dtype)
        assert torch.equal(bits(y.cpu()), bits(O.w8a8_native_epilogue(ref, a_s, s, b, dtype)))
        y = apply_int8_weight_only_linear(x.cuda(), q.cuda(), s.cuda(), b.cuda())
        m = O.tensor_metrics(O.w8a16_native_reference(x, q, s, b), y)
        assert m["relative_l2"] <= 4e-3 and m["cosine_similarity"] >= 0.9999, m
        again = apply_int8_weight_only_linear(x.cuda(), q.cuda(), s.cuda(), b.cuda())
        assert torch.equal(bits(y), bits(again))     # sums in a fixed order
    assert device_status_ok()


@pytest.mark.parametrize("M,N,K,bn", [(1100, 4104, 272, None), (12, 16384, 2064, None), (2048, 1032, 1040, 192),
                                      (50, 264, 1616, 16), (97, 1000, 528, 48), (200, 136, 2112, 96),
                                      (64, 9728, 2560, None), (33, 12296, 1040, None),
                                      (33, 16384, 528, None), (255, 1000, 208, 256)])
def test_w8a16_more_than_one_wave_and_every_token_tile(M, N, K, bn):
    # several waves of tiles, matrices too large for the ring kernel from 9 tokens on, the other tile widths
    q, s = O.make_weight(N, K, seed=N + K)
    x = O.make_activation(M, K, seed=M, dtype=torch.bfloat16)
    with knobs(**({} if bn is None else {"BN": bn})):
        assert select_path(_lib.OP_W8A16, M, N, K) == "umma_f16_expand_tokens128"
        plan = mid_plan(_lib.OP_W8A16, M, N, K)
        assert plan is not None and (bn is None or plan["tokens"] == bn), plan
        y = apply_int8_weight_only_linear(x.cuda(), q.cuda(), s.cuda())
    m = O.tensor_metrics(O.w8a16_native_reference(x, q, s, None), y)
    assert m["relative_l2"] <= 4e-3 and m["cosine_similarity"] >= 0.9999, m
    assert device_status_ok()


@pytest.mark.parametrize("M,N,K,path", [(200, 24584, 528, "umma_i8_pair_tokens256"), (300, 24584, 528, "umma_i8_tokens128"),
                                        (450, 12288, 2064, "umma_i8_pair_tokens256"), (129, 9728, 2048, "umma_i8_pair_tokens256"),
                                        (450, 6144, 1024, "umma_i8_tokens128")])
def test_w8a8_beyond_one_wave_takes_the_pair_kernel_where_rounding_tokens_up_costs_no_wave(M, N, K, path, oracle_c_lib):
    assert select_path(_lib.OP_W8A8, M, N, K) == path
    assert mid_plan(_lib.OP_W8A8, M, N, K) is None    # beyond one wave the name means the persistent kernel
    q, s = O.make_weight(N, K, seed=N + K)
    xq, a_s = O.quantize_per_row_dynamic(O.make_activation(M, K, seed=M, dtype=torch.bfloat16))
    ref = O.w8a8_int32_accumulators(xq, q)
    y = apply_w8a8_linear(xq.cuda(), a_s.cuda(), q.cuda(), s.cuda(), None, out_dtype=torch.bfloat16)
    assert torch.equal(bits(y.cpu()), bits(O.w8a8_native_epilogue(ref, a_s, s, None, torch.bfloat16)))
    assert torch.equal(w8a8_int32_accumulators(xq.cuda(), q.cuda()).cpu(), ref)
    assert device_status_ok()


@pytest.mark.parametrize("M,N,K", [(257, 24584, 1040), (385, 16384, 1024)])
def test_w8a16_beyond_the_mid_sizes_takes_the_tensor_memory_kernel(M, N, K):
    assert select_path(_lib.OP_W8A16, M, N, K) == "umma_f16_tmem_weights_channels256"
    q, s = O.make_weight(N, K, seed=N + K)
    x = O.make_activation(M, K, seed=M, dtype=torch.bfloat16)
    y = apply_int8_weight_only_linear(x.cuda(), q.cuda(), s.cuda())
    m = O.tensor_metrics(O.w8a16_native_reference(x, q, s, None), y)
    assert m["relative_l2"] <= 4e-3 and m["cosine_similarity"] >= 0.9999, m
    assert device_status_ok()


@pytest.mark.parametrize("M,N,K", [(513, 16384, 1040), (700, 12296, 2064), (1023, 9728, 2560), (513, 22016, 1024),
                                   (830, 9728, 2560), (512, 16384, 1040)])
def test_w8a16_to_1023_tokens_takes_one_route_whatever_the_workspace(M, N, K):
    assert select_path(_lib.OP_W8A16, M, N, K) == "umma_f16_tmem_weights_channels256"
    L = _lib.lib()
    assert L.b200q_workspace_bytes(_lib.OP_W8A16, M, N, K) == 0
    q, s = O.make_weight(N, K, seed=N + K)
    x = O.make_activation(M, K, seed=M, dtype=torch.bfloat16)
    b = (torch.randn(N, generator=torch.Generator().manual_seed(M)) * 0.1).to(torch.bfloat16)
    dev = [t.cuda() for t in (x, q, s, b)]
    y = apply_int8_weight_only_linear(*dev)
    m = O.tensor_metrics(O.w8a16_native_reference(x, q, s, b), y)
    assert m["relative_l2"] <= 4e-3 and m["cosine_similarity"] >= 0.9999, m
    ws = torch.full((2 * N * K + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(y)
    rc = L.b200q_w8a16_gemm(*[t.data_ptr() for t in (*dev, out)], M, N, K, _lib.DTYPE_BF16, ws.data_ptr(), ws.numel(),
                            torch.cuda.current_stream().cuda_stream)
    assert rc == _lib.OK and torch.equal(bits(out), bits(y)) and bool((ws == 0x5A).all())
    with knobs(W8A16_PAIR_MIN_M=512):           # the kernel of larger calls
        y_pair = apply_int8_weight_only_linear(*dev)
    assert O.tensor_metrics(y_pair, y)["relative_l2"] <= 2e-3
    assert device_status_ok()
