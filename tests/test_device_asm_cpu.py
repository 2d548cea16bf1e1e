"""Inline assembly that touches memory which a running kernel may write is
volatile and declares it (a "memory" clobber), so the compiler keeps it in its
place among stores and barriers. Only loads through the read-only path
(ld.global.nc, ld.const) may be treated as functions of their address."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pyre_gb300" / "csrc"
ACCESS = re.compile(r'"\s*(ld|st|red|atom|cp)\.(?!global\.nc|const|param)')


def _asm_statements():
    for f in sorted(CSRC.glob("*.cu*")):
        text = f.read_text()
        for m in re.finditer(r"\basm\b", text):
            end = text.index(");", m.start())
            yield f.name, " ".join(text[m.start():end + 2].split())


def test_memory_assembly_is_ordered():
    statements = list(_asm_statements())
    assert any(ACCESS.search(s) for _, s in statements)
    for name, s in statements:
        if ACCESS.search(s):
            assert re.match(r"asm volatile\b", s) and '"memory"' in s, f"{name}: {s}"
