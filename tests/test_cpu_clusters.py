"""Kernels that run as thread-block clusters, read as text: every access to
another CTA's shared memory stands between two cluster barriers.  A CTA's shared
memory exists for its peers only from its start (the barrier before the first
access) to its exit (the barrier after the last one)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "qdsim_b200" / "csrc"
REMOTE = "map_shared_rank("
BARRIER = "cluster.sync()"


def _closing(text, at):
    """Index just past the brace that closes the one at text[at]."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced braces")


def _kernels():
    out = []
    for f in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__cluster_dims__\(.*?\)\s*(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
            start = text.index("{", m.end())
            out.append(pytest.param(text[start:_closing(text, start)], id=f"{f.name}:{m.group(1)}"))
    return out


def _accesses(body):
    """Positions of remote accesses: direct ones and calls of lambdas that make one."""
    names, spans = [], []
    for m in re.finditer(r"auto\s+(\w+)\s*=\s*\[[^\]]*\]", body):
        start = body.index("{", m.end())
        end = _closing(body, start)
        spans.append((m.start(), end))
        if REMOTE in body[start:end]:
            names.append(m.group(1))
    words = [re.escape(REMOTE)] + [rf"\b{n}\(" for n in names]
    hits = [m.start() for m in re.finditer("|".join(words), body)]
    return [h for h in hits if not any(a <= h < b for a, b in spans)]


def test_there_are_cluster_kernels():
    assert _kernels()


@pytest.mark.parametrize("body", _kernels())
def test_remote_shared_memory_is_used_between_cluster_barriers(body):
    hits = _accesses(body)
    assert hits
    assert body.index(BARRIER) < min(hits)
    assert body.rindex(BARRIER) > max(hits)
