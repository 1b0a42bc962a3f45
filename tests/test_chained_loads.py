"""No kernel reads what its predecessor may still be writing with a non-coherent load (CPU).

Steps of a run or rollout overlap: a step starts while the one before it runs.
``__ldg`` (``ld.global.nc``) is defined only for data that is read-only for the whole
kernel, so it may touch static fields, a network's bias and the finished states
of a rollout, and nothing that a step or reverse step writes.
"""

from __future__ import annotations

import re

from conftest import PKG_ROOT

# Arguments of __ldg that name memory no step writes: bed, n^2, the rain multiplier, the
# strip edges' bed and n^2, a layer's bias, and load2's planes of a finished state.
STATIC = re.compile(r"(d|p\.d)\.(bed|nm|mult|edge_static)\b|bias\b|q$")


def _arguments(text: str, name: str):
    for m in re.finditer(re.escape(name) + r"\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_non_coherent_loads_only_of_what_no_step_writes():
    seen = 0
    for path in sorted((PKG_ROOT / "csrc").glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        assert "ld.global.nc" not in text
        for arg in _arguments(text, "__ldg"):
            plain = re.sub(r"^reinterpret_cast<[^>]*>\((.*)\)$", r"\1", arg.strip())
            assert STATIC.match(plain), f"{path.name}: __ldg({arg})"
            seen += 1
    assert seen


def test_reverse_step_reads_lambda_with_ordinary_loads():
    """load2's non-coherent form is for finished states: dL/dU comes from the reverse step before."""
    text = (PKG_ROOT / "csrc" / "swe_adjoint.cuh").read_text()
    used = re.findall(r"load2<VEC, (true|false)>\(p\.(\w+)\.", text)
    assert {s for f, s in used if f == "true"} == {"in", "d", "next"}
    assert [f for f, s in used if s == "lam"] == ["false"] * 3
