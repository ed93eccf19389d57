"""What of row_chain.cu needs no GPU.  The exchange between the two CTAs of a pair as a model, every order of its steps: the warps of
a CTA meet at barriers and nowhere else, and sums that were sent arrive at any later time; the number of buffers is read from the
source.  What becomes of the exchange when a wait runs out, with barriers that count arrivals and bytes.  And where the chain is taken."""
import pathlib
import random
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


class Barrier:
    """One arrival and the bytes it announces per phase."""

    def __init__(self):
        self.phase, self.pending, self.bytes = 0, 1, 0

    def change(self, arrivals=0, expected=0, landed=0):
        assert self.pending >= arrivals, "an arrival too many"
        self.pending -= arrivals
        self.bytes += expected - landed
        if self.pending == 0 and self.bytes == 0:
            self.phase, self.pending = self.phase + 1, 1

    def ended(self, phase):  # what a wait on the phase's parity says
        return (self.phase & 1) != (phase & 1)


def run_pair(rng, arm_after_giving_up: bool) -> bool:
    """A pair in a random order of steps in which waits run out at random; whether every send of a CTA had landed when the other left."""
    slots = buffers()
    bars = [[Barrier() for _ in range(slots)] for _ in (0, 1)]
    under_way, left, gave_up = [[], []], [False, False], [False, False]
    met = [[0, 0], [0, 0]]
    lost = False

    def meet(cta, who, n):
        met[cta][who] = n
        while met[cta][1 - who] < n:
            yield

    def owners(cta):
        armed = 0

        def read(n):
            while not gave_up[cta] and not bars[cta][n % slots].ended(n // slots):
                if rng.random() < 0.02:
                    gave_up[cta] = True
                yield

        for n in range(UNITS):
            yield from meet(cta, 0, n + 1)
            if n:
                yield from read(n - 1)
            if arm_after_giving_up or not gave_up[cta]:
                bars[cta][n % slots].change(arrivals=1, expected=1)
                armed += 1
            yield
        yield from read(UNITS - 1)
        yield from meet(cta, 0, UNITS + 1)
        if gave_up[cta]:
            for i, bar in enumerate(bars[cta]):
                phases = (armed - i + slots - 1) // slots
                rest = (UNITS - i + slots - 1) // slots - phases
                if rest:
                    bar.change(expected=rest)
                yield
                while phases and not bar.ended(phases - 1):
                    yield
                if rest:
                    bar.change(arrivals=1)
                    while not bar.ended(phases):
                        yield
        left[cta] = True

    def senders(cta):
        for n in range(UNITS):
            yield from meet(cta, 1, n + 1)
            under_way[1 - cta].append(n)
            yield
        yield from meet(cta, 1, UNITS + 1)

    threads = [owners(0), senders(0), owners(1), senders(1)]
    for _ in range(200000):
        if rng.random() < 0.5:
            cta = rng.randrange(2)
            if under_way[cta]:
                n = under_way[cta].pop(rng.randrange(len(under_way[cta])))
                lost |= left[cta]
                if not left[cta]:
                    bars[cta][n % slots].change(landed=1)
        elif threads:
            t = rng.choice(threads)
            try:
                next(t)
            except StopIteration:
                threads.remove(t)
        elif not any(under_way):
            return not lost
    raise TimeoutError("a wait without an end")


def test_all_sums_have_landed_when_a_cta_leaves():
    for seed in range(3000):
        assert run_pair(random.Random(seed), arm_after_giving_up=False)


def test_barriers_armed_after_a_wait_ran_out_would_miscount():
    with pytest.raises(AssertionError, match="an arrival too many"):
        for seed in range(3000):
            run_pair(random.Random(seed), arm_after_giving_up=True)


@pytest.mark.parametrize("width,ff,next_,gains", [
    (2048, 6144, 4096, 1), (2048, 6144, 151936, 1), (4096, 12288, 6144, 1), (1024, 3072, 4096, 1), (512, 1536, 1024, 1), (128, 384, 256, 1),
    (1024, 3072, 151936, 0), (512, 1536, 32000, 0), (128, 512, 32000, 0)])
def test_the_chain_is_taken_where_it_was_measured_faster(width, ff, next_, gains):
    from axono_b200 import _capi

    lib = _capi.lib()
    assert lib.axb200_row_chain_supported(8, 2048, width, ff, next_, _capi.FLOAT16)
    assert lib.axb200_row_chain_gains(8, 2048, width, ff, next_, _capi.FLOAT16) == gains
    assert not lib.axb200_row_chain_gains(9, 2048, width, ff, next_, _capi.FLOAT16)
