"""Rules that the CUDA sources keep and no run can show: inline assembly that synchronises the lanes of a
warp or the threads of a block, or touches memory, is volatile.  Without it the compiler may move a
statement into the branch that uses its result, where lanes that a full-mask collective waits for never come."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gtrap_gb300" / "csrc"
FILES = sorted(p.name for p in CSRC.glob("*.cu*"))


def _asm_statements(text):
    """(line, volatile or not, body) of every asm statement."""
    for m in re.finditer(r"\basm\b\s*(volatile|__volatile__)?\s*\(", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        yield text.count("\n", 0, m.start()) + 1, bool(m.group(1)), text[m.end():end - 1]


@pytest.mark.parametrize("name", FILES)
def test_collectives_and_memory_in_assembly_are_volatile(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for line, volatile, body in _asm_statements(text):
        if re.search(r"\.sync|barrier|\bbar\.|\bld\.|\bst\.|\bred\.|\batom\.|cp\.async|fence", body):
            assert volatile, "%s:%d: %s" % (name, line, body)
