"""How many nodes a warp's traversal pops at a time (packet_trace, range_collect, k_cull_query,
k_containment, containment_many), restated: on trees whose nodes are all hit, down
to 20 complete levels, on lopsided ones of 64, and from one root or 32, the stack holds every
child; with nothing kept free it breaks off."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rayspace3d_gb300", "csrc")
RULE = re.compile(r"const int take = min\(min\(sp, 32\), max\((\w+) - kStackRoom - sp, 1\)\);")
LOOPS = {"rs_query_core.cuh": 2, "rs_join.cu": 3}


def _sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in LOOPS}


def _constant(name):
    for text in _sources().values():
        m = re.search(rf"constexpr int {name} = (\d+);", text)
        if m:
            return int(m[1])
    raise AssertionError(name)


def _stacks():
    """Stack sizes of all loops that pop several nodes."""
    sizes = []
    for f, text in _sources().items():
        names = RULE.findall(text)
        assert len(names) == LOOPS[f] == len(re.findall(r"const int take = ", text)), f
        sizes += [_constant(n) for n in names]
    return sorted(set(sizes))


def _most(size, room, roots, children):
    """Most entries on the stack of a traversal that hits every node (None: it broke off);
    children(level) are the inner children of a node of a level, as levels."""
    stack, most = [0] * roots, roots
    while stack:
        take = min(len(stack), 32, max(size - room - len(stack), 1))
        popped = stack[-take:]
        del stack[-take:]
        pushed = [c for p in popped for c in children(p)]
        if len(stack) + len(pushed) > size:
            return None
        stack += pushed
        most = max(most, len(stack))
    return most


@pytest.mark.parametrize("roots", [1, 32])
@pytest.mark.parametrize("levels", [10, 14, 18, 20])
def test_complete_trees(levels, roots):
    if levels > 18 and roots > 1:
        levels = 18
    room = _constant("kStackRoom")
    complete = lambda level: [level + 1] * (2 if level + 1 < levels else 0)
    for size in _stacks():
        assert _most(size, room, roots, complete) is not None
        if levels >= 18:
            assert _most(size, 0, roots, complete) is None


@pytest.mark.parametrize("roots", [1, 32])
def test_lopsided_trees(roots):
    """64 levels, an inner child beside each node of the long branch that has 6 complete levels of its own."""
    room = _constant("kStackRoom")
    assert room >= 64

    def children(node):
        level, side = node if isinstance(node, tuple) else (node, None)
        if side is not None:
            return [(level, side + 1)] * (2 if side < 6 else 0)
        return [level + 1, (level, 0)] if level < 63 else []
    for size in _stacks():
        assert _most(size, room, roots, children) is not None
