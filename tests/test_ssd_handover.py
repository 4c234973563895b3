"""The words in which the Mamba-2 scan on tcgen05 notes non-finite inputs of a chunk, between the warps that write them (make_xs) and the
warps of the same group that read them (outputs): the order that the kernel's barriers give, as a graph over all its roles, on the CPU.
The number of stages is read from the kernel's source.

The property: a warp reads the words of a step after every warp has written them, and they are written again only after every warp
has read them."""
import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parents[1] / "linearnexus_b200" / "csrc" / "dr_ssd_sm100.cuh").read_text()
WARPS = range(4)


def order(n1, steps, xs_stages, early):
    """Edges (before, after) of steps 0 .. steps - 1, the first n1 for their effect on the state alone.  ``early``: D is issued
    before G (the issuer picks either)."""
    edges, last = [], {}

    def node(role, what, *after):
        """A node of a role's program, behind the role's previous one and behind ``after``."""
        if role in last:
            edges.append((last[role], what))
        edges.extend((a, what) for a in after)
        last[role] = what

    def freed(it):
        return [("out" if it >= n1 else "xs", it, w) for w in WARPS]

    for it in range(steps):
        full, first = it >= n1, it == n1
        # copies: B, the next x, C
        if it == 0:
            node("copy", ("X", 0))
        node("copy", ("B", it), *([("D", it - 1)] if it else []))
        if it + 1 < steps:
            node("copy", ("X", it + 1), *(freed(it + 1 - xs_stages) if it + 1 >= xs_stages else []))
        if full:
            node("copy", ("C", it), *([] if first else [("Y1", it - 1)]))
        # scalars, two warps in turn
        node(("scal", it & 1), ("S", it), *(freed(it - xs_stages) + [("upd", it - xs_stages)] if it >= xs_stages else []))
        # xs of this step, then the outputs of the one before
        for w in WARPS:
            node(("grp", w), ("xs", it, w), ("S", it), ("X", it), *([("D", it - 1)] if it else []))
            if it > n1:
                node(("grp", w), ("out", it - 1, w), ("Y", it - 1))
        # issue
        def issue_d():
            node("issue", ("iD", it), ("B", it), *[("xs", it, w) for w in WARPS], *([("upd", it - 1)] if it else []))
        if early or not full:
            issue_d()
        if full:
            node("issue", ("G", it), ("B", it), ("C", it), *([] if first else [("Y", it - 1)]))
        if full and not early:
            issue_d()
        node("issue", ("D", it))
        if full:
            node("issue", ("Y1", it), ("pub", it), *([] if first else [("out", it - 1, w) for w in WARPS]))
            node("issue", ("iY", it), ("P", it))
            edges.append((("iY", it), ("Y", it)))
            node("p", ("P", it), ("S", it), ("G", it))
            node("state", ("pub", it), *([] if first else [("Y1", it - 1)]))
        node("state", ("upd", it), ("D", it))
    for w in WARPS:
        if steps > n1:
            node(("grp", w), ("out", steps - 1, w), ("Y", steps - 1))
    return edges


def unordered(n1, steps, xs_stages, word_stages, early):
    """A pair that should be ordered and is not, or None."""
    succ = {}
    for a, b in order(n1, steps, xs_stages, early):
        succ.setdefault(a, []).append(b)

    def reaches(a):
        seen, todo = {a}, [a]
        while todo:
            for b in succ.get(todo.pop(), ()):
                if b not in seen:
                    seen.add(b)
                    todo.append(b)
        return seen

    for it in range(n1, steps):
        for w in WARPS:
            written, read = reaches(("xs", it, w)), reaches(("out", it, w))
            for v in WARPS:
                if ("out", it, v) not in written:
                    return ("xs", it, w), ("out", it, v)
                if it + word_stages < steps and ("xs", it + word_stages, v) not in read:
                    return ("out", it, w), ("xs", it + word_stages, v)
    return None


def test_words_of_a_step_are_read_before_they_are_written_again():
    stages = int(re.search(r"kXs = (\d+);", SRC).group(1))
    word = re.search(r"auto bad_of = .*\(it % (\w+)\)", SRC)
    assert word and word.group(1) == "kXs"
    for n1, steps in ((0, 1), (0, 2), (0, 9), (4, 8), (5, 9)):
        for early in (False, True):
            assert unordered(n1, steps, stages, stages, early) is None


@pytest.mark.parametrize("word_stages,sound", [(2, False), (3, True), (4, True)])
def test_the_graph_tells_sound_from_unsound(word_stages, sound):
    """With two stages a warp can write the words of step it + 2 while another has yet to read those of step it."""
    assert (unordered(0, 9, 3, word_stages, True) is None) == sound
