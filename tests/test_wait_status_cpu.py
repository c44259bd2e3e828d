"""Waits that run out reach the host: no device wait goes without a status word, the models hand theirs to the ops whose kernels
wait, and every code has its text."""
import re
from pathlib import Path

import pytest

import ninfer_fusion_b200
from ninfer_fusion_b200._lib import StatusWord, load_native, native_available

PKG = Path(ninfer_fusion_b200.__file__).resolve().parent
SOURCES = sorted(p for p in (PKG / "csrc").rglob("*") if p.suffix in (".cu", ".cuh"))


def calls(text, name):
    """Argument texts of each call of `name` in `text`."""
    for m in re.finditer(rf"\b{name}\(", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        yield text[m.end():end - 1]


@pytest.mark.parametrize("wait", ["mbar_wait", "wait_counter"])
def test_every_wait_has_a_status_word(wait):
    seen = 0
    for path in SOURCES:
        for args in calls(path.read_text(), wait):
            seen += 1
            assert "status" in args and "nullptr" not in args, f"{path.name}: {wait}({args})"
    assert seen > 5


@pytest.mark.parametrize("file,op", [("layered.py", "mlstm"), ("hybrid.py", "gdn_recurrent")])
def test_models_pass_their_status_word(file, op):
    found = list(calls((PKG / "models" / file).read_text(), rf"ops\.{op}"))
    assert found and all("self.status.tensor" in args for args in found)
    if native_available():
        schema = getattr(load_native(), op).default._schema
        assert [a.name for a in schema.arguments][-1] == "status"


def test_every_status_code_has_a_text():
    codes = {int(c) for path in SOURCES for c in re.findall(r"\bkStatus\w+ = (\d+)", path.read_text())}
    assert codes - {0} == set(StatusWord.CODES)
