"""Kernels that start beside their predecessor read nothing of its before the
wait. A memory clobber does not hold back loads through `const __restrict__`
pointers or inline loads the compiler may take for pure functions of their
address, so the wait hands an index through and every use of it must take the
result; an inline memory access must be volatile with a memory clobber."""
import re

import pytest

from conftest import PKG

SOURCES = sorted((PKG / "csrc").glob("*.cu*"))


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_waits_pass_an_index_through(path):
    text = code(path)
    for m in re.finditer(r"\basm\b[^;]*?griddepcontrol\.wait.*?\)\s*;", text, re.S):
        assert re.search(r':\s*"\+[rl]"\(', m.group(0)), m.group(0)
    for m in re.finditer(r"\bpdl_(?:wait|enter)\s*\(", text):
        line = text[text.rfind("\n", 0, m.start()) + 1:text.find("\n", m.start())]
        if "__device__" in line:
            continue
        # an argument, and a result that is used
        assert not re.match(r"\s*pdl_\w+\(", line), line
        assert text[m.end():].lstrip()[0] != ")", line


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_inline_memory_accesses_are_ordered(path):
    for m in re.finditer(r'\basm\b(\s+volatile)?\s*\(\s*"(ld|st)\..*?\)\s*;', code(path), re.S):
        assert m.group(1) and '"memory"' in m.group(0), m.group(0)
