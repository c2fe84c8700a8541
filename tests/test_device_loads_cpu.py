"""Source checks on the device code's memory accesses that no run can pin.

A pass kernel launched with the programmatic-serialisation attribute starts
while its predecessor still writes the images that it is about to read; only
`griddepcontrol.wait` stands between.  A load may be moved above that wait when
the source lets the compiler take it for a pure function: inline assembly
without `volatile` and a "memory" clobber, or a load declared read-only for the
kernel's lifetime (`__ldg`, `const __restrict__`).  Whether one build's scheduling does
so shows in no test result, so the sources are checked."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "glscv_gb300" / "csrc"
DEVICE_SOURCES = sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")))


def _code(path: Path) -> str:
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def _asm_statements(code: str):
    """(volatile?, text in the parentheses) of every asm statement."""
    for m in re.finditer(r"\basm\b\s*(volatile)?\s*\(", code):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = code[i]
            if c == '"' and code[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (c == "(") - (c == ")")
            i += 1
        yield bool(m.group(1)), code[m.end():i - 1]


@pytest.mark.parametrize("path", DEVICE_SOURCES, ids=lambda p: p.name)
def test_asm_memory_accesses_are_ordered(path):
    """Every inline instruction that reads or writes memory is volatile and
    names memory, so it stays behind the dependency wait and the barriers."""
    access = re.compile(r"\b(ld|st|atom|red|cp|multimem|tcgen05\.(ld|st|cp))\.")
    for volatile, text in _asm_statements(_code(path)):
        if access.search(text):
            assert volatile and '"memory"' in text, text.strip()


@pytest.mark.parametrize("path", [p for p in DEVICE_SOURCES if re.search(
    r"pdl_enter\(\)|griddepcontrol\.wait", _code(p)) or p.name == "fft_kernels.cuh"], ids=lambda p: p.name)
def test_images_are_not_declared_read_only(path):
    """In the kernels with a dependency wait only the constant tables (uploaded
    when the context is created) are read through the read-only path."""
    code = _code(path)
    for m in re.finditer(r"__ldg\(\s*(\w+)|__restrict__\s+(\w+)", code):
        assert (m.group(1) or m.group(2)) in ("g_dft", "g_tw"), m.group(0)
