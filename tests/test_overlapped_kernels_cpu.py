"""Kernels that start before their predecessor has ended (griddepcontrol) must not promise, by
__restrict__, that a buffer stays unchanged while they run unless no kernel writes it: such loads
may be moved before the wait or served by the read-only path.  Checked on the sources."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "parallel_admm_b200" / "csrc"
# parameters that no kernel of their stream writes
CONSTANT = {"elems", "start", "cols", "vals", "diag", "b"}


def _kernels():
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            if text[i:].lstrip()[0] != "{":
                continue
            depth, j = 1, text.index("{", i) + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
            yield m.group(1), params, text[i:j]


def test_no_restrict_on_what_a_predecessor_writes():
    seen, bad = 0, []
    for name, params, body in _kernels():
        if "ADMM_PDL_" not in body and "griddepcontrol" not in body:
            continue
        seen += 1
        names = re.findall(r"__restrict__\s+(\w+)", params)
        bad += [f"{name}: {p}" for p in names if p not in CONSTANT]
    assert seen > 30 and not bad, bad
