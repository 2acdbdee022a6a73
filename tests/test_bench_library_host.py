"""bench.py builds the group-type library only for the mode whose launches use it."""
import importlib.util
import os

import pytest

from qsv_b200 import engine

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("mode", ["auto", "eager", "off", "coarse", "library"])
def test_library_is_built_where_it_is_used(mode, monkeypatch):
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    built = []
    monkeypatch.setattr(engine, "jit_prepare_library", lambda programs: built.append(programs) or 7)
    info = bench._build_library(mode, lambda: [("segment", 16)])
    assert built == ([[("segment", 16)]] if mode == "library" else [])
    assert (info is None) == (mode != "library") and (info is None or info["types"] == 7)


def test_no_other_call_builds_it():
    text = open(os.path.join(ROOT, "bench.py")).read()
    assert text.count("jit_prepare_library") == 1
