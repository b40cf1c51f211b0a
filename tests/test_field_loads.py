"""Fields and state are never read with read-only loads.

The step kernels begin while the kernel before them still writes (they wait
for it first of all), and the one-launch kernels step several times: a load
through the read-only path (``__ldg``, the policies' ``ldc``) is for data that
no kernel writes during a launch.  The sources are read: no such load may name
a field, an adjoint, a state array or the recorded increments, and the cell
kernels' field loads go through ``ldf``.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "gmes_gb300" / "csrc"
WRITTEN = re.compile(r"\b(?:g|gi|t|u|v)\.(?:f|l|aux|tmp|phi|hist|mon|grad|tf_field)\b")


def _read_only_loads(text):
    """The argument text of every read-only load."""
    for m in re.finditer(r"(?:__ldg|\bP::ldc?|\bldc)\(", text):
        depth, q = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[q], 0)
            q += 1
        yield text[:m.start()].count("\n") + 1, text[m.end():q - 1]


def test_written_arrays_take_plain_loads():
    found = [(p.name, line, arg)
             for p in sorted(CSRC.glob("gmes_*.cu*"))
             for line, arg in _read_only_loads(p.read_text())
             if WRITTEN.search(arg)]
    assert found == []


def test_cell_kernels_read_fields_with_plain_loads():
    text = (CSRC / "gmes_cell.cuh").read_text()
    body = re.search(r"P::R ldf\(.*?\n}\n", text, re.S).group(0)
    assert "P::ldw(" in body and "P::ld(" not in body and "ldc(" not in body
    internal = (CSRC / "gmes_internal.cuh").read_text()
    assert internal.count("ldw(const T* p) { return *p; }") == 2  # FP64, FP32
    assert re.search(r"ldw\(const T\* p\) \{\s+const float2 v = \*p;", internal)
