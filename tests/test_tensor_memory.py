"""Rules of the tensor-memory instructions that no result shows while the
compiler happens to keep them, checked on the CUDA source: a tensor-memory
load fills its registers only once tcgen05.wait::ld has returned, and that
wait names no register, so that a load and its wait stand in one asm
statement (a use of the registers cannot be placed between them)."""
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
