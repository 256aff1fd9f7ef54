"""Inline PTX that reads or writes shared or global memory must be volatile with a "memory" clobber: to the compiler any
other asm is a function of its operands, which it may move across the waits and barriers that make the data valid (a
kernel launched early must not read before griddepcontrol.wait, a ring stage not before its mbarrier) or merge across a
store."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ffnoml_gb300", "csrc")
MEMORY = re.compile(r"\b(ld|st)\.(global|shared|weak|relaxed|acquire|release)|\bcp\.async|\bred\.|\batom\.|\bmbarrier\."
                    r"|\bbar\.(sync|red)|\bgriddepcontrol\.|\bfence\.")


def _statements(path):
    text = open(path).read()
    for m in re.finditer(r"\basm\b\s*(volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if c == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (c == "(") - (c == ")")
            i += 1
        yield text.count("\n", 0, m.start()) + 1, bool(m.group(1)), text[m.end():i - 1]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_memory_accesses_are_ordered(path):
    loose = [line for line, volatile, body in _statements(path)
             if MEMORY.search(body) and not (volatile and '"memory"' in body)]
    assert not loose, f"{os.path.basename(path)}: asm at lines {loose}"


def test_the_accesses_are_found():
    found = [body for p in glob.glob(os.path.join(CSRC, "*.cu*")) for _, _, body in _statements(p) if MEMORY.search(body)]
    assert len(found) >= 20
