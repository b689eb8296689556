"""Rules of the tensor-memory instructions that no result shows, checked on
the CUDA source.

A tensor-memory load fills its registers only once tcgen05.wait::ld has
returned, and that wait names no register: a load and its wait stand in one
asm statement, so that no use of the registers can be placed between them.

A kernel launched with programmatic stream serialisation takes tensor memory
only after griddepcontrol.wait: the kernel before it may take its own after
it let this one in, and the two would wait for each other."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "inmsom_elfs_b200" / "csrc"


def _asm_statements(text):
    """The text of every asm statement, comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\basm\b(?:\s+volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            ch = text[i]
            if ch == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (ch == "(") - (ch == ")")
            i += 1
        yield text[m.end():i - 1]


def test_tensor_memory_loads_wait_in_their_own_statement():
    loads = [a for f in sorted(CSRC.glob("*.cu*")) for a in _asm_statements(f.read_text()) if "tcgen05.ld." in a]
    assert loads
    for a in loads:
        assert "tcgen05.wait::ld.sync.aligned;" in a[a.index("tcgen05.ld."):], a


def test_tensor_memory_is_taken_after_the_stream_wait():
    seen = 0
    for f in sorted(CSRC.glob("*.cu*")):
        order = [k for a in _asm_statements(f.read_text()) for k in ("griddepcontrol.wait", "tcgen05.alloc") if k in a]
        if "tcgen05.alloc" in order:
            seen += 1
            assert "griddepcontrol.wait" in order[:order.index("tcgen05.alloc")], f.name
    assert seen
