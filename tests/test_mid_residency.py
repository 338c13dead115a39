"""Plans of the tcgen05 kernels for tens to hundreds of tokens (host code, no GPU).  A CTA of a cluster that waits for
tensor memory held by another such CTA never ends, so the ones that fit an SM together may not need more than it has."""
import re
from pathlib import Path

import pytest

from tests.gpu_util import knobs, mid_plan
import tiny_vllm_b200  # noqa: F401
from tiny_vllm_b200 import _lib, build as b200_build

SM_SHARED, CTA_RESERVED = 228 * 1024, 1024    # bytes per SM; bytes the runtime adds to every CTA
SM_COLUMNS = 512                              # of tensor memory
MAX_CTAS = 2                                  # of these kernels on an SM, by registers

COMMON = (Path(__file__).resolve().parent.parent / "tiny-vllm_b200" / "csrc" / "common.h").read_text()
PAIR_SHARED = int(re.search(r"kPairSmem = (\d+) \* 1024", COMMON).group(1)) * 1024    # the CTA-pair kernel, all 512 columns

TOKENS = [1, 8, 16, 17, 24, 33, 40, 48, 64, 77, 96, 128, 129, 200, 256, 384, 512, 700, 1024, 1500, 2048]
CHANNELS = [8, 72, 128, 264, 440, 512, 640, 768, 1024, 1536, 2048, 3072, 3968, 4096, 6144, 9728, 12288, 24576]
INNER = [16, 96, 528, 896, 1024, 1536, 2048, 2112, 2944, 3072, 4096, 8192, 12288]


@pytest.mark.parametrize("forced", [{}, {"CLUSTER": 2}, {"CLUSTER": 4, "BN": 64}, {"CLUSTER": 8, "BN": 256}],
                         ids=["chosen", "cluster2", "cluster4-bn64", "cluster8-bn256"])
@pytest.mark.parametrize("op", [_lib.OP_W8A8, _lib.OP_W8A16], ids=["w8a8", "w8a16"])
def test_clusters_never_wait_for_tensor_memory(op, forced):
    b200_build.build()
    seen = 0
    with knobs(**forced):
        for M in TOKENS:
            for N in CHANNELS:
                for K in INNER:
                    p = mid_plan(op, M, N, K)
                    if p is None or p["cluster"] == 1:
                        continue
                    seen += 1
                    # with another CTA of its own kernel, and of any other plan (256 columns at least stay free, or
                    # nothing that has dynamic shared memory fits)
                    fit = min(MAX_CTAS, SM_SHARED // (p["shared"] + CTA_RESERVED))
                    assert fit >= 1 and fit * p["columns"] <= SM_COLUMNS, (M, N, K, p)
                    left = SM_SHARED - p["shared"] - CTA_RESERVED
                    assert p["columns"] <= SM_COLUMNS // 2 or left <= CTA_RESERVED, (M, N, K, p)
                    assert p["shared"] + PAIR_SHARED + 2 * CTA_RESERVED > SM_SHARED, (M, N, K, p)
    assert seen > 50


@pytest.mark.parametrize("M,N,K,deep", [(129, 4096, 12288, True), (256, 2560, 9728, True), (200, 2048, 6144, True),
                                        (128, 4096, 12288, False), (256, 4096, 4096, False), (256, 1024, 3072, False),
                                        (256, 4096, 1024, False)])
def test_w8a8_rings_leave_room_for_the_quantiser_unless_rows_are_long(M, N, K, deep):
    b200_build.build()
    plan = mid_plan(_lib.OP_W8A8, M, N, K)
    assert (plan["shared"] > 218 * 1024) == deep, plan
