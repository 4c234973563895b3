"""The hand-over of the RWKV kernel's stages between its staging groups and the warps that hold the state, explored on the CPU over
every order in which groups and state warps can proceed.  Constants and the kind of barrier are read from the kernel's source.

The property: when the state reaches block n, the block's stage holds block n, and a stage is only written after its last block was
consumed."""
import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parents[1] / "linearnexus_b200" / "csrc" / "dr_rwkv_chunk.cuh").read_text()


def explore(groups, stages, phases, nblk):
    """None, or a text that says what goes wrong.  ``phases``: an emptied stage is announced by a barrier with phases that a group
    waits for by parity; otherwise by a barrier without, which the state's arrival and ANY group's arrival complete together."""
    # state: next block of every group, whether it stands at its stage barrier, content of the stages, full flags,
    # next block of the consumer, arrivals (phases: completed phases of the stage; else: 0 / 1 arrival pending)
    start = (tuple(range(groups)), (None,) * stages, (False,) * stages, 0, (0,) * stages)
    seen, todo = {start}, [start]
    while todo:
        nxt, held, full, cons, empty = todo.pop()
        out = []
        if cons < nblk and full[cons % stages]:   # the state consumes a block and announces the stage empty
            s = cons % stages
            if held[s] != cons:
                return f"the state expects block {cons} and stage {s} holds {held[s]}"
            if not phases and empty[s] and cons + stages < nblk:
                return f"stage {s} announced empty twice"
            e = empty[s] + 1 if phases else int(cons + stages < nblk)
            out.append((nxt, held, full[:s] + (False,) + full[s + 1:], cons + 1, empty[:s] + (e,) + empty[s + 1:]))
        for i, blk in enumerate(nxt):
            if blk >= nblk:
                continue
            s = blk % stages
            if phases:   # a wait by parity returns once the current phase has the other parity
                free = blk < stages or (empty[s] & 1) != ((blk // stages - 1) & 1)
            else:
                free = blk < stages or empty[s] == 1
            if not free:
                continue
            if full[s] or (held[s] is not None and held[s] >= cons):
                return f"block {blk} is written over block {held[s]} before the state has read it"
            if held[s] is not None and blk != held[s] + stages:
                return f"stage {s} takes block {blk} after block {held[s]}"
            e = empty if phases or blk < stages else empty[:s] + (0,) + empty[s + 1:]
            out.append((nxt[:i] + (blk + groups,) + nxt[i + 1:], held[:s] + (blk,) + held[s + 1:],
                        full[:s] + (True,) + full[s + 1:], cons, e))
        if not out and (cons < nblk or any(b < nblk for b in nxt)):
            return f"nothing can proceed at block {cons}"
        for st in out:
            if st not in seen:
                seen.add(st)
                todo.append(st)
    return None


def group_counts():
    """The numbers of staging groups that the kernel is built with: every value that groups_of can take."""
    default = int(re.search(r"kGroups = (\d+), kRing", SRC).group(1))
    rule = re.search(r"constexpr int groups_of = (.*?);", SRC).group(1)
    values = [v.strip() for v in re.split(r"[?:]", rule)[1:]] or [rule.strip()]
    return sorted({default if v == "kGroups" else int(v) for v in values})


def test_rwkv_stage_handover_in_every_order():
    stages = int(re.search(r"kStages = (\d+)", SRC).group(1))
    counts = group_counts()
    assert len(counts) >= 2   # RWKV-6 on bf16 has its own
    for groups in counts:
        for nblk in (1, 2, 3, 4, 5, 8, 9, 20):
            assert explore(groups, stages, "bar_sync(kBarEmpty" not in SRC, nblk) is None


@pytest.mark.parametrize("groups,stages,phases,sound", [(3, 4, False, False), (3, 3, False, True), (3, 4, True, True), (3, 6, False, True),
                                                            (4, 4, True, True)])
def test_exploration_tells_sound_from_unsound(groups, stages, phases, sound):
    """Without phases a stage has to belong to one group (stages a multiple of the groups)."""
    assert (explore(groups, stages, phases, 20) is None) == sound
