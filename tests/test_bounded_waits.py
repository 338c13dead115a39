"""How the kernels give up a wait that ran out, read from their sources (nothing here runs on a GPU).

A bounded mbarrier wait can end differently for the lanes of one warp, and differently for the warps of a CTA.  So
* a warp that waits together votes, or its lanes keep the answer in a flag of their own and go on together: the flag
  stands in no condition around an instruction of the warp, only beside the one lane that signals or issues;
* a loop that meets a barrier of several warps is not left when a wait runs out: the others would wait for good;
* a TMA producer waits for its copies in flight before it ends.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tiny-vllm_b200" / "csrc"
SOURCES = [p for p in sorted(CSRC.glob("*.cu*")) if p.name != "ptx_sm100.cuh" and "mbar_wait" in p.read_text()]
ONE_LANE = re.compile(r"\blane == 0\b|\bproduce\(")       # produce(): under `lane < kPipes`, a ring per lane
BARRIER = re.compile(r"named_bar_sync|consumer_barrier|__syncthreads|cluster_wait|cluster_sync_all")
WAIT = r"ptx::mbar_wait\([^;]*\)"


def code_of(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def blocks(code):
    """(what stands before the brace, its position, that of the closing one) of every block."""
    stack, out = [], []
    for i, c in enumerate(code):
        if c == "{":
            head = max(code.rfind(e, 0, i) for e in (";", "{", "}"))
            loop = code.rfind("for (", 0, i)
            if loop > 0 and code.count("(", loop, i) == code.count(")", loop, i) and code.count("{", loop, i) == 0:
                head = min(head, loop - 1)
            stack.append((code[head + 1:i].strip(), i))
        elif c == "}":
            before, start = stack.pop()
            out.append((before, start, i))
    return out


def enclosing(found, at):
    return [b for b in found if b[1] < at < b[2]]


def conditions(code):
    """Of every if, while and for: what stands in its parentheses and what follows them."""
    for m in re.finditer(r"\b(?:if|while|for) \(", code):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(code[i], 0)
            i += 1
        yield code[m.end():i - 1], code[i:i + 400]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_a_warp_goes_on_or_gives_up_as_one(path):
    code = code_of(path)
    found = blocks(code)
    for m in re.finditer(r"ptx::mbar_wait(_cluster)?\(", code):
        inside = enclosing(found, m.start())
        if any(ONE_LANE.search(b[0]) for b in inside):
            continue
        begin = max(code.rfind(e, 0, m.start()) for e in (";", "{", "}")) + 1
        before, statement = code[begin:m.start()], code[begin:code.index(";", m.start()) + 1]
        vote = before.rfind("ptx::warp_all(")
        if vote >= 0 and before.count("(", vote) > before.count(")", vote):
            continue
        flag = (re.fullmatch(r"\s*if \(ok && [^()]*\) ok = %s;" % WAIT, statement)
                or re.fullmatch(r"\s*if \((?:alive)\)\s*alive = %s;" % WAIT, statement)
                or re.fullmatch(r"\s*if \((?:[^()]* && )?!%s\) ok = false;" % WAIT, statement))
        assert flag, statement
        name = "alive" if "alive" in statement else "ok"
        scope = next(b for b in sorted(inside, key=lambda b: -b[1]) if f"bool {name} = true;" in code[b[1]:b[2]])
        for cond, then in conditions(code[scope[1]:scope[2]]):
            if not re.search(r"\b%s\b" % name, cond):
                continue
            waits_only = re.match(r"\s*%s = %s;" % (name, WAIT), then)
            one_lane = re.match(r"(?:ptx::elect_one\(\)|lane == \w+) && %s$" % name, cond)
            own_count = re.match(r"%s && \+\+\w+ == " % name, cond)      # the lane's own place in the ring
            # a template argument: true in the form without the vote, and the flag is the warp's in the other
            no_branch = cond == "X_SMEM || alive" and re.search(r"if constexpr \(X_SMEM\) \{\s*if \(alive\) alive = %s;" % WAIT, code)
            voted = re.match(r"\s*alive = ptx::warp_all\(", then)
            assert waits_only or one_lane or own_count or no_branch or voted, cond
    for m in re.finditer(r"(?<!void )\bproduce\(&", code):
        assert re.search(r"if \(lane < kPipes\)\s*$", code[:m.start()])


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_warp_leaves_the_others_at_a_barrier(path):
    code = code_of(path)
    loops = [b for b in blocks(code) if b[0].startswith("for")]
    for _, start, end in loops:
        if not BARRIER.search(code[start:end]):
            continue
        inner = [b for b in loops if start < b[1] and b[2] < end and not BARRIER.search(code[b[1]:b[2]])]
        for m in re.finditer(r"mbar_wait\w*\(", code[start:end]):
            at = start + m.start()
            if any(b[1] < at < b[2] for b in inner):
                continue
            statement = code[code.rfind(";", 0, at):code.find(";", at)]
            assert "break" not in statement and "return" not in statement, statement


@pytest.mark.parametrize("path", [p for p in SOURCES if "tma_load" in p.read_text()], ids=lambda p: p.name)
def test_a_producer_that_gives_up_waits_for_its_copies(path):
    assert re.search(r"if \((rank == 0 && |ptx::elect_one\(\) && )?\*abort_flag != 0\) ptx::drain_ring\(", code_of(path))
