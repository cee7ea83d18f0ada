"""Inline assembly that touches memory must stay where it stands: a statement that is not volatile,
or does not clobber memory, may be moved across a barrier or merged with another, since the
compiler sees only its register operands."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "invariantbitpacking_b200", "csrc")
# instructions that read or write memory, or order such accesses
TOUCHES = re.compile(r"\b(ld|st|red|atom|cp\.async|griddepcontrol|fence|membar|mbarrier)\b[.\s]")


def statements(text):
    for m in re.finditer(r"\basm\b\s*(volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if quoted:
                i += c == "\\"
                quoted = c != '"'
            elif c == '"':
                quoted = True
            else:
                depth += (c == "(") - (c == ")")
            i += 1
        yield bool(m.group(1)), text[m.end():i - 1]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))),
                         ids=os.path.basename)
def test_memory_assembly_is_volatile_and_clobbers_memory(path):
    for volatile, body in statements(open(path).read()):
        if TOUCHES.search("".join(re.findall(r'"((?:[^"\\]|\\.)*)"', body.split(":")[0]))):
            assert volatile and '"memory"' in body, body
