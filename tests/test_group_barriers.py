"""A CTA that gave up waiting at a group barrier must leave the tile there (CPU, by the source).

Provoking the ten-second wait on a GPU to see the other outcome (a walk over words nobody wrote) is out of the question, so
this reads the kernel: in the DAG phase the statement after every group barrier, and after every loop that holds one, must
be the test that leaves.
"""

from __future__ import annotations

import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LEAVES = re.compile(r"\s*if \(left\(\)\) \{\s*break;\s*\}")


def closing(text, at):
    """Index after the bracket that closes the one at text[at]."""
    pairs, depth = {"(": ")", "{": "}"}, 0
    for i in range(at, len(text)):
        if text[i] in pairs:
            depth += 1
        elif text[i] in pairs.values():
            depth -= 1
            if depth == 0:
                return i + 1
    raise AssertionError("unbalanced")


def dag_phase():
    with open(os.path.join(ROOT, "neurograph_b200", "csrc", "sssp_kernels.cuh")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[text.index("tile_kernel(const __grid_constant__"):]
    body = body[:body.index("#undef NGX_GT")]
    return body[body.index("dag_low(dist, low"):body.index("const int my_src = s_src[lane];")]


def test_every_barrier_is_followed_by_the_way_out():
    body = dag_phase()
    ends = []
    for m in re.finditer(r"\b(sync0|sync|group_exclusive_scan)\(", body):
        end = closing(body, m.end() - 1)
        ends.append(body.index(";", end) + 1)
    assert len(ends) >= 12
    for end in ends:
        assert LEAVES.match(body, end), body[max(0, end - 120):end + 80]


def test_every_loop_with_a_barrier_is_followed_by_the_way_out():
    body = dag_phase()
    loops = 0
    for m in re.finditer(r"\bfor \(", body):
        head = closing(body, m.end() - 1)
        end = closing(body, body.index("{", head))
        if "sync0(" in body[head:end] or "sync([" in body[head:end]:
            loops += 1
            assert LEAVES.match(body, end), body[head:end + 80]
    assert loops == 4  # sigma and delta levels, with and without lists
