"""The two warps that fill one box of the SwiGLU epilogue (csrc/gemm.cu) as a model on the CPU: every order of their steps, and every
outcome of their waits once some role of the CTA has given up."""
import pytest


def _stuck(agreed: bool, tiles: int) -> int:
    """States in which a warp stands at the pair's barrier and its partner has left.  ``agreed``: what the waits for the accumulator
    returned is and-ed over the pair at a barrier, and both go by the result; else each warp goes by its own."""
    program = []
    for _ in range(tiles):
        program += ["wait"] + ([] if agreed else ["go"]) + ["meet"] + (["go"] if agreed else []) + ["meet"]
    faults, seen, todo = 0, set(), [(False, (0, True, False), (0, True, False))]     # abort flag; per warp: next step, result, left
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        abort, *warps = state
        op = [None if left else "end" if pc == len(program) else program[pc] for pc, _, left in warps]
        nxt = [] if abort else [(True, *warps)]                                      # another role gives up
        for w in (0, 1):
            pc, ok, left = warps[w]
            if op[w] == "wait":
                to = [(pc + 1, True, False)] + ([(pc + 1, False, False)] if abort else [])
            elif op[w] == "go":
                to = [(pc + 1, ok, False) if ok else (pc, ok, True)]
            else:
                continue
            nxt += [(abort, t, warps[1]) if w == 0 else (abort, warps[0], t) for t in to]
        if op == ["meet", "meet"]:
            both = warps[0][1] and warps[1][1] if agreed else None
            nxt.append((abort, *((pc + 1, ok if both is None else both, False) for pc, ok, _ in warps)))
        faults += "meet" in op and (None in op or "end" in op)
        todo += nxt
    return faults


@pytest.mark.parametrize("tiles", [1, 2, 5])
def test_a_pair_of_warps_leaves_together(tiles):
    assert _stuck(True, tiles) == 0
    assert _stuck(False, tiles) > 0
