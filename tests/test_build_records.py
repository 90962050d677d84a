"""When the in-tree libraries are rebuilt: their records name what they were built from, and a failed build leaves the old
file and its record to be found out of date again."""
import subprocess
import sys

import pytest
import torch

from tagseq2tagseq_b200 import build as b


@pytest.fixture(autouse=True)
def built():
    b.build_library()


def test_another_pytorch_makes_the_operators_unusable(monkeypatch):
    assert b.unusable() == []
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert b.unusable() == [b.TORCH_LIB]


def test_failed_build_is_not_taken_for_a_success(monkeypatch):
    with open(b.TORCH_LIB, "rb") as fh:
        before = fh.read()
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    monkeypatch.setattr(b, "_torch_flags", lambda: ["-not-an-option", "none.cpp"])
    for _ in range(2):
        with pytest.raises(RuntimeError, match="torch operators failed to build"):
            b.build_library()
    with open(b.TORCH_LIB, "rb") as fh:
        assert fh.read() == before
    assert b.unusable() == [b.TORCH_LIB]


def test_import_needs_no_built_library():
    code = f"""
import importlib.util, sys
spec = importlib.util.spec_from_file_location("tagseq2tagseq_b200.build", {b.__file__!r})
build = importlib.util.module_from_spec(spec)
spec.loader.exec_module(build)
build.TORCH_LIB += ".missing"
build.build_library = None
sys.modules["tagseq2tagseq_b200.build"] = build
from tagseq2tagseq_b200 import _lib, synth
assert synth.make_pack(1, 50, 10, 2, 30).seq_len == 50 and _lib._OPS is None
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=b.HERE + "/..")
