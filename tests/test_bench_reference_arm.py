"""``bench.py --impl reference``: a line of the reference's own code, or one that says why there is none."""
import argparse
import json
import types

import pytest

import bench
from oracle import build_ref


@pytest.fixture
def args(monkeypatch):
    monkeypatch.setattr(bench, "TOKENS", 16)
    return argparse.Namespace(gpus=1, steps=1, warmup=0)


def test_without_a_mirror_it_is_unavailable(args, monkeypatch, capsys):
    monkeypatch.setattr(build_ref, "load_reference", lambda: None)
    bench.run_reference_arm(args)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_with_a_mirror_its_functions_are_timed(args, monkeypatch, capsys):
    calls = []
    stand_in = types.SimpleNamespace(
        utils=types.SimpleNamespace(quantize_int8_per_row_dynamic=lambda x: calls.append("quantise") or (x, None)),
        cuda=types.SimpleNamespace(w8a8_linear_fallback=lambda *a: calls.append("linear")))
    monkeypatch.setattr(build_ref, "load_reference", lambda: stand_in)
    bench.run_reference_arm(args)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["value"] > 0 and line["cpu_baseline"]["kind"] == "reference"
    assert calls == ["quantise", "linear"] * len(bench.PROJECTIONS)
