"""The exchange between the two CTAs of a pair in row_chain.cu as a model, every order of its steps (no GPU): the warps of a CTA meet at
barriers and nowhere else, and sums that were sent arrive at any later time.  The number of buffers is read from the source."""
import pathlib
import re

import pytest

SOURCE = pathlib.Path(__file__).resolve().parents[1] / "axono_b200" / "csrc" / "row_chain.cu"
UNITS = 9


def buffers() -> int:
    return int(re.search(r"constexpr int kRecvs = (\d+);", SOURCE.read_text())[1])


def programs():
    """What the owners (they wait for the other CTA's sums and read them) and the senders of a CTA do, in their order."""
    owner, sender = [], []
    for n in range(UNITS):
        both = [("meet", 2 * n)] * (n > 0) + [("meet", 2 * n + 1)]  # partial sums of n - 1 have been read; those of n are there
        owner += both + [("read", n - 1)] * (n > 0)
        sender += both + [("send", n)]
    return owner + [("read", UNITS - 1)], sender


def overwritten(slots: int) -> bool:
    """Whether in some order sums arrive in a buffer whose last ones have not been read."""
    owner, sender = programs()
    # a state: places in the programs of (owner 0, sender 0, owner 1, sender 1), and the sums sent to CTA 0 and to CTA 1 that are under way
    start = (0, 0, 0, 0, frozenset(), frozenset())
    seen, todo = {start}, [start]

    def has(place, what, n):  # the owners of a place have done a step
        return any(step == (what, n) for step in owner[:place])

    def moves(state):
        for cta in (0, 1):
            o, s = state[2 * cta], state[2 * cta + 1]
            out = list(state)
            if o < len(owner) and owner[o][0] == "meet" and s < len(sender) and owner[o] == sender[s]:
                out[2 * cta], out[2 * cta + 1] = o + 1, s + 1
                yield tuple(out)
            if o < len(owner) and owner[o][0] == "read":
                n = owner[o][1]
                if ("send", n) in sender[:state[2 * (1 - cta) + 1]] and n not in state[4 + cta]:  # it has arrived
                    out = list(state)
                    out[2 * cta] = o + 1
                    yield tuple(out)
            if s < len(sender) and sender[s][0] == "send":
                out = list(state)
                out[2 * cta + 1] = s + 1
                out[4 + 1 - cta] = out[4 + 1 - cta] | {sender[s][1]}
                yield tuple(out)
            for n in state[4 + cta]:
                if n >= slots and not has(o, "read", n - slots):
                    raise OverflowError
                out = list(state)
                out[4 + cta] = out[4 + cta] - {n}
                yield tuple(out)

    try:
        while todo:
            for state in moves(todo.pop()):
                if state not in seen:
                    seen.add(state)
                    todo.append(state)
    except OverflowError:
        return True
    return False


@pytest.mark.parametrize("slots,bad", [(2, True), (3, True), (4, False)])
def test_the_model_tells_enough_buffers_from_too_few(slots, bad):
    assert overwritten(slots) == bad


def test_sums_are_read_before_others_take_their_place():
    assert not overwritten(buffers())
