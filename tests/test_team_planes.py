"""The two box tests of compressed nodes, a lane's (visit_node) and a team's
(team_child): one form of the planes, so that one error bound covers both."""
import re
from pathlib import Path

import numpy as np

SRC = (Path(__file__).resolve().parents[1] / "kiraray_gb300" / "csrc" / "accel_device.cuh").read_text()


def _body(name):
    start = SRC.index(name + "(")
    start = SRC.index("{", start)
    depth, i = 1, start + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(SRC[i], 0)
        i += 1
    return SRC[start:i]


def test_same_offsets_and_slack():
    lane, team = _body("void visit_node"), _body("bool team_child")
    for what in (r"fmaf\((-\d+)\.f, ad[xyz]", r"fabsf\(ad[xyz]\) \* ([\d.]+)f", r"fabsf\(tmax\) \* ([\d.e-]+)f"):
        a, b = set(re.findall(what, lane)), set(re.findall(what, team))
        assert a == b and len(a) == 1, (what, a, b)


def test_team_planes_are_exact():
    base, shift = re.search(r"__uint_as_float\((0x[0-9A-F]+)u \| \(q << (\d+)\)\)", _body("bool team_child")).groups()
    q = np.arange(256, dtype=np.uint32)
    planes = (np.uint32(int(base, 16)) | (q << np.uint32(int(shift)))).view(np.float32)
    assert np.array_equal(planes, 1024 + q.astype(np.float32))
