"""Rules of the kernels that start while their predecessor in the stream still runs (programmatic dependent launch),
checked on the sources: what they break shows on a GPU only now and then."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tiny-vllm_b200" / "csrc"
# what a kernel of this library reads that the kernel before it may have written
PRODUCED = {"x", "xq", "a_s", "a_scales", "residual", "residual_in", "gate_up", "p0", "p1", "src"}
OVERLAPPED = re.compile(r"\blaunch_(overlapped|maybe_overlapped|clustered|mid_kernel)\b|\bB200Q_ROWS_DISPATCH\b")


def code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def sources():
    # headers go into several files; a .cu that launches in plain stream order alone is exempt
    return [p for p in sorted(CSRC.iterdir())
            if p.suffix == ".cuh" or p.suffix == ".cu" and OVERLAPPED.search(code(p))]


def argument(text, start):
    depth = 0
    for i in range(start, len(text)):
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        if depth == 0:
            return text[start + 1:i]
    raise AssertionError("unbalanced parentheses")


@pytest.mark.parametrize("path", sources(), ids=lambda p: p.name)
def test_no_non_coherent_load_of_what_the_predecessor_writes(path):
    # such a load counts as one of constant memory: the compiler may move it ahead of griddepcontrol.wait
    text = code(path)
    for m in re.finditer(r"__ldg\s*\(|ld\.global\.nc", text):
        assert m.group(0).startswith("__ldg"), path.name
        names = set(re.findall(r"[A-Za-z_]\w*", argument(text, m.end() - 1)))
        assert not names & PRODUCED, (path.name, argument(text, m.end() - 1))
    for name in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", text):
        assert name not in PRODUCED, (path.name, name)


def test_the_rule_covers_the_kernels():
    names = {p.name for p in sources()}
    assert {"gemm_mma_decode.cu", "gemm_umma.cu", "w8a8_device.cuh", "gemm_umma_pair.cu", "gemm_umma_mid.cu",
            "gemm_umma_mid_w8a16.cu", "gemm_reg_decode.cu", "gemm_bulk_decode.cu", "act_quant.cu"} <= names


def test_the_stand_alone_quantiser_holds_its_successors_back():
    # its rows may be weights, which the GEMM kernels read ahead of their wait; only inside
    # b200q_w8a8_dynamic_gemm is it known that they are not
    quantiser = code(CSRC / "act_quant.cu")
    triggers = re.findall(r"[^;{}]*grid_launch_dependents\(\)", quantiser)
    assert triggers and all(re.search(r"if \(early\)", t) for t in triggers), triggers
    api = code(CSRC / "api.cu")
    body = {name: re.search(rf"\bint {name}\([^)]*\) \{{(.*?)\n\}}", api, re.S).group(1)
            for name in ("b200q_act_quant_i8", "b200q_w8a8_dynamic_gemm")}
    early = {name: argument(text, text.index("run_act_quant(") + len("run_act_quant")).split(",")[-2].strip()
             for name, text in body.items()}
    assert early == {"b200q_act_quant_i8": "false", "b200q_w8a8_dynamic_gemm": "true"}
