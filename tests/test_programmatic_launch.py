"""Kernels that let the next launch begin early (griddepcontrol.launch_dependents)
have to wait for the grid before them on every path: the grid after them waits for
them alone, so one that ended without waiting would let it overtake the one before."""
import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).parents[1] / "biomedisa_gb300" / "csrc").glob("*.cu"))
WAIT, LAUNCH = "griddepcontrol.wait", "griddepcontrol.launch_dependents"


def _kernels(text):
    """(name, body) of every __global__ function, comments removed."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        at = text.index("{", text.index(")", m.end()))
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield m.group(1), text[at:end]


FOUND = [(p.name, n, b) for p in SOURCES for n, b in _kernels(p.read_text()) if LAUNCH in b]


def test_kernels_are_found():
    assert sum(p.read_text().count(LAUNCH + ";") for p in SOURCES) == len(FOUND) >= 3


@pytest.mark.parametrize("name,body", [(f"{f}:{n}", b) for f, n, b in FOUND], ids=[n for _, n, _ in FOUND])
def test_every_path_waits(name, body):
    waits = [m.end() for m in re.finditer(re.escape(WAIT) + r'[^"]*"[^;]*;', body)]
    # the wait that all threads pass: one that no return follows at once
    plain = [e for e in waits if not re.match(r"\s*return\b", body[e:])]
    assert plain, name
    for m in re.finditer(r"\breturn\b", body[:plain[0]]):
        assert any(e <= m.start() and not body[e:m.start()].strip() for e in waits), (name, body[:m.end()][-80:])
