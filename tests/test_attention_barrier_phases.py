"""The hand-over of P between the softmax warps and the issuing thread of the attention forward, and who may touch O when, as
models on the CPU: every order that the waits allow.  A wait on parity p passes while the barrier's current phase has the other parity, so
a phase that completes twice before it is looked for is missed."""
import itertools

import pytest


def _faults(barriers: int, ahead: bool, blocks: int) -> int:
    """States in which the issuing thread is stuck, or takes a P that is not there."""
    faults, seen, todo = 0, set(), [(0, 0, 0)]          # P waits passed, S issued, blocks the softmax warps have arrived for
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        waited, scores, arrived = state
        steps = [(waited, scores, arrived + 1)] if arrived < scores else []
        if scores < min(waited + (2 if ahead else 1), blocks):
            steps.append((waited, scores + 1, arrived))               # S(j + 1), before or after PV(j)
        elif waited < blocks:
            phase = sum(b % barriers == waited % barriers for b in range(arrived))
            if phase % 2 != (waited // barriers) % 2:
                if arrived > waited:
                    steps.append((waited + 1, scores, arrived))
                else:
                    faults += 1
        faults += not steps and waited < blocks
        todo += steps
    return faults


@pytest.mark.parametrize("blocks", [1, 2, 3, 9])
def test_p_is_handed_over_once(blocks):
    assert _faults(2, True, blocks) == 0                # head_dim 64: scores one block ahead, two barriers
    assert _faults(2, False, blocks) == 0               # head_dim 128: scores after P V
    assert _faults(1, False, blocks) == 0
    assert (_faults(1, True, blocks) > 0) == (blocks > 1)     # one barrier is not enough ahead


def _overlaps(ordered: bool, ahead: bool, rescaled: tuple, snapshot: int | None) -> int:
    """States in which a product that accumulates into O may run while one of the two softmax warps of 32 rows works on its
    half of O's columns: in the blocks in which both rescale, or before the block at which the student output is written.
    Each half of P V writes ALL columns of O; the first waits for the warp with the first 64 keys only.  ``ordered``: the
    warps meet between rescaling and their P."""
    blocks = len(rescaled)
    warps = [[], []]
    for part, program in enumerate(warps):
        for i in range(blocks):
            program.append(("done", ("S", i)))
            if i == snapshot:
                program += [("done", ("PV", i - 1, 1))] if ahead else []
                program += [("meet",), ("meet",), ("take",), ("leave",)]         # l of the other thread; O is read
            program.append(("meet",))                                            # whether any row has to rescale
            if rescaled[i]:
                program += [("done", ("PV", i - 1, 1))] if ahead and i > 0 else []
                program += [("meet",), ("meet",)]                                # no wait has expired; the other thread's max
                if i > 0:
                    program += [("take",), ("leave",)] + ([("meet",)] if ordered else [])
            program.append(("arrive", i, part))
    issue = [("issue", ("S", 0))]
    for j in range(blocks):
        following = [("issue", ("S", j + 1))] if j + 1 < blocks else []
        issue += following if ahead else []
        for half in (0, 1):
            issue += [("arrived", j, half), ("issue", ("PV", j, half))]
        issue += [] if ahead else following
    queue = [op[1] for op in issue if op[0] == "issue"]

    faults, seen, todo = 0, set(), [(0, 0, 0, 0)]       # the warps' and the issuing thread's next step, products completed
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        pcs, t, done = state[:2], state[2], state[3]
        issued = sum(op[0] == "issue" for op in issue[:t])
        arrived = {op[1:] for w in (0, 1) for op in warps[w][:pcs[w]] if op[0] == "arrive"}
        at = [warps[w][pcs[w]] if pcs[w] < len(warps[w]) else ("end",) for w in (0, 1)]
        inside = any(op == ("leave",) for op in at)
        if inside and done < issued and queue[done][0] == "PV":
            faults += 1
        steps = [(*pcs, t, done + 1)] if done < issued else []
        if t < len(issue) and (issue[t][0] == "issue" or issue[t][1:] in arrived):
            steps.append((*pcs, t + 1, done))
        if at[0] == at[1] == ("meet",):
            steps.append((pcs[0] + 1, pcs[1] + 1, t, done))
        for w in (0, 1):
            if at[w][0] in ("take", "leave", "arrive") or (at[w][0] == "done" and at[w][1] in queue[:done]):
                steps.append((pcs[0] + (w == 0), pcs[1] + (w == 1), t, done))
        assert steps or (at == [("end",)] * 2 and done == len(queue)), "the hand-over is stuck"
        todo += steps
    return faults


@pytest.mark.parametrize("ahead", [False, True])           # head_dim 128, 64
@pytest.mark.parametrize("rescaled", list(itertools.product([False, True], repeat=4)))
def test_o_belongs_to_one_at_a_time(ahead, rescaled):
    for snapshot in (None, 2):
        assert _overlaps(True, ahead, rescaled, snapshot) == 0
        # without the meeting a late second warp still rescales while the first half of P V runs
        assert (_overlaps(False, ahead, rescaled, snapshot) > 0) == any(rescaled[1:])
