"""What the sources of kernels launched as programmatic dependents must and must not hold (common/pdl.cuh): such a kernel is
running while the kernel before it still writes its inputs, which no run on a GPU shows reliably when it goes wrong."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "meshslice_b200" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def _matching(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        if depth == 0:
            return i
    raise AssertionError("unbalanced source")


def functions(text, qualifier):
    """{name: (parameters, body)} of the functions that carry ``qualifier``."""
    out = {}
    for m in re.finditer(qualifier + r"\b[^;{}]*?(\w+)\(", text):
        name, at = m.group(1), m.end() - 1
        while name in ("__launch_bounds__", "__cluster_dims__"):
            nxt = re.compile(r"\s*[^;{}(]*?(\w+)\(").match(text, _matching(text, at, "()") + 1)
            name, at = nxt.group(1), nxt.end() - 1
        close = _matching(text, at, "()")
        brace = text.find("{", close)
        if text[close + 1:brace].strip():
            continue                                             # a declaration
        out[name] = (text[at:close + 1], text[brace:_matching(text, brace, "{}") + 1])
    return out


SOURCES = [CSRC / "ops/ops.cu", CSRC / "ops/attention.cu", CSRC / "gemm/sm100_gemm2.cu"]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_inputs_of_dependent_kernels_are_read_coherently(path):
    """A const __restrict__ pointer, or a load that asks for it, may go through the non-coherent path and be moved over the
    wait.  Only kernels that are launched plainly, and so never wait, may have them."""
    text = _code(path)
    kernels = functions(text, "__global__")
    waiting = {n for n, (_, body) in kernels.items() if "grid_wait()" in body}
    assert waiting
    for name in waiting:
        assert "__restrict__" not in kernels[name][0] + kernels[name][1], name
    for name, (params, body) in functions(text, "__device__").items():
        assert "__restrict__" not in params, name
    assert not re.search(r"__ldg\(|__ldcs\(|ld\.global\.nc", "".join(b for n, (_, b) in kernels.items() if n in waiting)
                         + "".join(b for _, b in functions(text, "__device__").values()))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_dependent_launches_wait(path):
    """What launch_dependent() launches waits for the grids before it."""
    text = _code(path)
    kernels = functions(text, "__global__")
    launched = set(re.findall(r"launch_dependent\((\w+_kernel)\b", text)) & set(kernels)
    assert launched or "auto kernel" in text
    for name in launched:
        assert "grid_wait()" in kernels[name][1], name


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_dependent_kernels_wait_before_they_touch_memory(path):
    """A grid sees the writes of the grids before it only after a wait of its own: one that every thread comes to, with no load
    or copy in front of it and no other wait that a kernel's order could rest on."""
    text = _code(path)
    for name, (_, body) in functions(text, "__device__").items():
        assert "grid_wait()" not in body, name
    for name, (_, body) in functions(text, "__global__").items():
        if "grid_wait()" not in body:
            continue
        waits = []
        for m in re.finditer(r"grid_wait\(\);", body):
            before = body[:m.start()]
            leads = re.search(r"[;{}]\s*$", before) is not None          # a statement of its own, not the branch of an if
            if leads and before.count("{") - before.count("}") == 1:
                waits.append(before)
        assert len(waits) == 1, name
        assert not re.search(r"load_tile|bulk_g2s|tma_load|cp_async16|__ldcs|ld_stream", waits[0]), name


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_kernels_of_a_row_exchange_do_not_let_the_next_one_start(path):
    """A trigger counts in a plainly launched grid too: the next kernel would hold SMs while this one waits for other GPUs."""
    for name, (params, body) in functions(_code(path), "__global__").items():
        if "RowExchange" in params and "grid_trigger()" in body:
            assert body.count("grid_trigger()") == body.count("if (ex.n == 0) grid_trigger();") == 1, name
