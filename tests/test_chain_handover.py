"""The barriers of the backward's serial pass (chain_kernel) between the warp that issues products, the tensor pipe and the workers, explored on the
CPU over every order in which they can proceed.  How many barriers announce Y^T d_o is read from the kernel's source.

The property: nobody passes a wait before its phase is complete, and nobody waits for a phase that the barrier has left behind (a wait by parity then
returns only with the next one of that parity, which may never come)."""
import re
from pathlib import Path

SRC = (Path(__file__).resolve().parents[1] / "linearnexus_b200" / "csrc" / "dr_bwd_chunk.cuh").read_text()


def explore(slots, chunks, workers=2):
    """None, or a text that says what goes wrong.  A state: the issuer's step, products issued and completed (alternately Y^T d_o and N dS), the step of
    every worker.  Steps per chunk, issuer: issue Y^T d_o; wait for all workers, issue N dS; wait for the one; wait for the other.  Worker:
    announce dS; wait for Y^T d_o; wait for N dS."""
    def passes(done, n):   # a wait for phase n by parity, `done` phases complete: None when it passes too early
        if done & 1 == n & 1:
            return False
        return True if done > n else None
    start = (0, 0, 0, (0,) * workers)
    seen, todo = {start}, [start]
    while todo:
        issuer, issued, completed, work = todo.pop()
        y_done, d_done = (completed + 1) // 2, completed // 2
        on = lambda n: (y_done - n % slots + slots - 1) // slots   # phases complete of the barrier that chunk n's Y^T d_o arrives on
        out = []
        if completed < issued:
            out.append((issuer, issued, completed + 1, work))
        it, step = divmod(issuer, 4)
        if it < chunks:
            if step == 0:
                out.append((issuer + 1, issued + 1, completed, work))
            elif step == 1:
                if all(w > 3 * it for w in work):
                    out.append((issuer + 1, issued + 1, completed, work))
            else:
                ok = passes(on(it), it // slots) if step == 2 else passes(d_done, it)
                if ok is None:
                    return f"the issuer passes its wait in chunk {it} too early"
                if ok:
                    out.append((issuer + 1, issued, completed, work))
        for i, w in enumerate(work):
            it, step = divmod(w, 3)
            if it >= chunks:
                continue
            ok = True if step == 0 else passes(on(it), it // slots) if step == 1 else passes(d_done, it)
            if ok is None:
                return f"a worker passes its wait in chunk {it} too early"
            if ok:
                out.append((issuer, issued, completed, work[:i] + (w + 1,) + work[i + 1:]))
        if not out and (issuer < 4 * chunks or any(w < 3 * chunks for w in work)):
            return f"nothing can proceed: issuer in chunk {issuer // 4}, workers in {[w // 3 for w in work]}"
        for s in out:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def test_chain_handover_in_every_order():
    slots = int(re.search(r"bar_y\[(\d)\], bar_d", SRC).group(1))
    waits = re.findall(r"wait_bar\(ctl\.bar_y\[it & 1\], \(it >> 1\) & 1\)", SRC)
    assert slots == 2 and len(waits) == 2 and "mma_commit(tc::smem_u32(&ctl.bar_y[it & 1]))" in SRC
    assert explore(slots, 7) is None
    assert "nothing can proceed" in explore(1, 7)   # one barrier: a worker that is late by a product waits for good


def explore_terms(chunks, converters=2, workers=2):
    """The same for per-channel decays, where more warps turn N (in halves) and Y^T into terms.  Steps per chunk, issuer: all terms of Y: issue Y^T d_o;
    all terms of N's first half and all of dS: issue their products; the second half's: issue; wait for Y^T d_o.  Converter: wait for the chunk before's
    Y^T d_o, store Y; for its first products, store a half; for its last ones, store the other.  Worker as above.  Phases of a barrier that a
    group arrives on: the least that any of the group has done."""
    def passes(done, n):
        if done & 1 == n & 1:
            return False
        return True if done > n else None
    start = (0, 0, 0, (0,) * converters, (0,) * workers)
    seen, todo = {start}, [start]
    while todo:
        issuer, issued, completed, conv, work = todo.pop()
        done = [(completed + 2 - i) // 3 for i in range(3)]   # phases complete: Y^T d_o (of all chunks), first products, last products
        y_on = lambda n: (done[0] - n % 2 + 1) // 2           # of the barrier that chunk n's Y^T d_o arrives on
        stored = [min((c + 2 - i) // 3 for c in conv) for i in range(3)]
        ready = min((w + 2) // 3 for w in work)
        out, bad = [], None
        if completed < issued:
            out.append((issuer, issued, completed + 1, conv, work))
        it, step = divmod(issuer, 4)
        if it < chunks:
            needs = [passes(stored[step], it)] if step < 3 else [passes(y_on(it), it // 2)]
            if step == 1:
                needs.append(passes(ready, it))
            if None in needs:
                bad = "issuer"
            elif all(needs):
                out.append((issuer + 1, issued + (step < 3), completed, conv, work))
        for i, c in enumerate(conv):
            it, step = divmod(c, 3)
            if it < chunks:
                ok = True if it == 0 else passes(y_on(it - 1), (it - 1) // 2) if step == 0 else passes(done[step], it - 1)
                if ok is None:
                    bad = "converter"
                elif ok:
                    out.append((issuer, issued, completed, conv[:i] + (c + 1,) + conv[i + 1:], work))
        for i, w in enumerate(work):
            it, step = divmod(w, 3)
            if it < chunks:
                ok = True if step == 0 else passes(y_on(it), it // 2) if step == 1 else passes(done[2], it)
                if ok is None:
                    bad = "worker"
                elif ok:
                    out.append((issuer, issued, completed, conv, work[:i] + (w + 1,) + work[i + 1:]))
        if bad:
            return f"a wait of the {bad} passes too early"
        if not out and (issuer < 4 * chunks or any(x < 3 * chunks for x in conv + work)):
            return "nothing can proceed"
        for s in out:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def test_chain_handover_of_terms_in_every_order():
    # the waits of the model, in the kernel's words
    for text in ("wait_bar(ctl.full_l, it & 1);", "wait_bar(ctl.full_h[hf], it & 1);", "if (hf == 0) wait_bar(ctl.rdy, it & 1);",
                 "if (it > 0) { y_done(it - 1);", "wait_bar(hf ? ctl.bar_d : ctl.bar_e, (it - 1) & 1);"):
        assert text in SRC, text
    assert explore_terms(5) is None
