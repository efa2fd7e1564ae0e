"""Order of the forward attention kernel's accumulator: every schedule of its roles, with barriers that are waited for by parity, on a model of the kernel."""
import re
from pathlib import Path

import pytest

KERNEL = Path(__file__).resolve().parent.parent / "ferrotorch_b200" / "csrc" / "kernels" / "flash_fwd.cu"
WARPS = 2                                        # softmax warps; each arrives once a step


def one_barrier(j):
    return 0, j & 1


def two_barriers(j):
    return j & 1, (j >> 1) & 1


def explore(nblk, where, each_step):
    """Faults over all schedules: a softmax warp that touches the accumulator ahead of the products before it, or a schedule in which nobody can go on. ``where(j)``: barrier and parity of
    the products of step j; ``each_step``: whether a warp also waits for the products of step j - 2 at step j.

    State: V blocks that have arrived, next instruction of the issuing thread (S(0), then S(j + 1) and P.V(j) in turn), tensor operations completed (in order of issue), each warp's step
    and place in it, arrivals for P, and completed phases of the barriers (an arrival trails its operation by any time, in order of issue)."""
    ops = [("s", 0)] + [x for j in range(nblk) for x in ((("s", j + 1),) if j + 1 < nblk else ()) + (("pv", j),)]
    faults, seen, todo = set(), set(), []
    todo.append((0, 0, 0, 0, tuple(((0, "score"),) * WARPS)))

    def phases(signalled):
        """Completed phases of every barrier after the first ``signalled`` operations have arrived."""
        s, pv = [0, 0], [0, 0]
        for kind, j in ops[:signalled]:
            if kind == "s":
                s[j & 1] += 1
            else:
                pv[where(j)[0]] += 1
        return s, pv

    def passes(count, parity):
        return count & 1 != parity

    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        loaded, issued, done, signalled, warps = state
        s, pv = phases(signalled)
        nxt = []
        if loaded < nblk:
            nxt.append((loaded + 1, issued, done, signalled, warps))
        if issued < len(ops):
            kind, j = ops[issued]
            ready = kind == "s" or (loaded > j and all(w[0] > j for w in warps))
            if ready:
                nxt.append((loaded, issued + 1, done, signalled, warps))
        if done < issued:
            nxt.append((loaded, issued, done + 1, signalled, warps))
        if signalled < done:
            nxt.append((loaded, issued, done, signalled + 1, warps))
        products = sum(kind == "pv" for kind, _ in ops[:done])
        for i, (j, at) in enumerate(warps):
            def go(*place):
                nxt.append((loaded, issued, done, signalled, warps[:i] + (place,) + warps[i + 1:]))
            if at == "score" and j < nblk and passes(s[j & 1], (j >> 1) & 1):
                go(j, "behind" if each_step and j >= 2 else "sums")
            elif at == "behind":
                b, p = where(j - 2)
                if passes(pv[b], p):
                    go(j, "sums")
            elif at == "sums":
                go(j + 1, "score")                                   # the running maximum stays
                if j > 0:
                    go(j, "rescale")
            elif at == "rescale":
                b, p = where(j - 1)
                if passes(pv[b], p):
                    if products < j:
                        faults.add(("rescaled early", j))
                    go(j + 1, "score")
            elif at == "score" and j == nblk:
                b, p = where(nblk - 1)
                if passes(pv[b], p):
                    if products < nblk:
                        faults.add(("read early", j))
                    go(j, "end")
        if not nxt and any(w != (nblk, "end") for w in warps):
            faults.add(("stuck", warps))
        todo += nxt
    return faults


@pytest.mark.parametrize("nblk", [1, 2, 3, 4, 5, 6])
def test_no_schedule_reads_the_accumulator_early(nblk):
    assert not explore(nblk, two_barriers, True)


@pytest.mark.parametrize("nblk", [2, 3, 4])
def test_the_model_finds_a_wait_that_is_two_phases_behind(nblk):
    assert any(f[0] == "read early" for f in explore(nblk, one_barrier, False))


def test_the_kernel_keeps_the_rule_of_the_model():
    code = re.sub(r"//[^\n]*", "", KERNEL.read_text())
    assert "auto pv = [&](int j) { return wait(&pv_done[j & 1], (j >> 1) & 1); };" in code
    assert re.findall(r"umma_commit\(&?pv_done[^)]*\)", code) == ["umma_commit(&pv_done[j & 1])"]
    assert re.findall(r"\bpv\((.*?)\)", code) == ["j - 2", "j - 1", "nblk - 1"] and "const bool behind = j < 2 || pv(j - 2);" in code
    assert len(re.findall(r"wait\(&?pv_done", code)) == 1
