"""Kernels that are brought up while the one before them on the stream still
runs (launch_ordered): what that one may write is not read through pointers
whose loads the compiler may move before the wait."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "kiraray_gb300" / "csrc"

# written before the kernel before: trees by builds, views and constants when
# a frame begins, by launches that nothing overlaps
OLDER = {"nodes", "tris", "views", "fc"}


def _kernels():
    """(file, name, parameter list, body's first statement) of every kernel."""
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            first = text[text.index("{", i) + 1:].lstrip().split(";")[0]
            yield f.name, m.group(1), params, first


def test_ordered_kernels_read_no_fresh_data_as_invariant():
    ordered = [k for k in _kernels() if k[3] == "stream_order()"]
    assert len(ordered) >= 14
    for file, name, params, _ in ordered:
        for p in re.split(r",(?![^<]*>)", params):
            if re.search(r"\bconst\b.*\*\s*__restrict__", p):
                assert p.split()[-1].lstrip("*") in OLDER, (file, name, p.strip())


def test_ordered_launches_start_with_the_wait():
    """What launch_ordered starts begins with stream_order()."""
    first = {name: f for _, name, _, f in _kernels()}
    n = 0
    for f in sorted(CSRC.glob("*.cu")):
        for m in re.finditer(r"launch_ordered\(([^;]*?)(\bk_\w+)", f.read_text()):
            assert first[m.group(2)] == "stream_order()", (f.name, m.group(2))
            n += 1
    assert n >= 14
