"""The hand-over of P between the softmax warps and the issuing thread of the attention forward, as a model on the CPU: every
order of the two that their waits allow.  A wait on parity p passes while the barrier's current phase has the other parity, so
a phase that completes twice before it is looked for is missed."""
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
