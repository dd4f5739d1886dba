"""Inline assembly that reads or writes memory, or orders it, says so to the
compiler: without the "memory" clobber plain accesses to the same words may be
moved across it (CPU-only: reads the sources)."""
from __future__ import annotations

import glob
import os
import re

import pytest

from conftest import REPO

FILES = sorted(glob.glob(os.path.join(REPO, "oncolytica_b200", "csrc", "*.cu*")))
ACCESS = re.compile(r"(?<![\w.])(ld|st|red|atom|cp|mbarrier|barrier|fence|griddepcontrol)\.")


def _asm_statements(text: str):
    """Each asm statement, from its keyword to the closing parenthesis."""
    for m in re.finditer(r"\basm\b(\s+volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if c == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (c == "(") - (c == ")")
            i += 1
        yield text.count("\n", 0, m.start()) + 1, text[m.start():i]


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_asm_accesses_are_memory_clobbers(path):
    bad = [f"{os.path.basename(path)}:{line}" for line, stmt in _asm_statements(open(path).read())
           if ACCESS.search(stmt) and '"memory"' not in stmt]
    assert not bad, bad
