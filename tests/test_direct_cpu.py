"""The protocol of the kernels that exchange without a step barrier (csrc/tc_direct.cuh), with the constants of that header, walked
through all interleavings of its roles: two CTAs of one storing warp each, their counting warps, stores and resets that are performed
late and in any order between fences."""
import os
import re

import pytest

from flashlstm_poc_b200 import _build

SOURCE = open(os.path.join(_build.CSRC, "tc_direct.cuh")).read()


def constant(name):
    return int(re.search(rf"\b{name} = (\d+)", SOURCE).group(1))


def missed_phase(slack, barriers, ahead, steps):
    """A state in which the counting warp waits for a phase that can no longer be told from the running one, or None.

    mbarrier t % barriers completes a phase when all warps have arrived for step t; a wait for phase n goes by parity and sees it
    exactly while n + 1 phases are complete."""
    resets = [t for t in range(steps) if t + ahead + 1 < steps]
    seen, todo = set(), [(0, 0)]  # steps the storing warps have reported, steps the counting warp has counted
    while todo:
        reported, counted = state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        if reported < len(resets) and counted >= reported - slack + 1:  # wait_performed(t - slack + 1) comes before step t's resets
            todo.append((reported + 1, counted))
        if counted < len(resets):
            bar, phase = counted % barriers, counted // barriers
            complete = len([t for t in resets[:reported] if t % barriers == bar])
            if complete > phase and (complete & 1) == (phase & 1):
                return state
            if complete > phase:
                todo.append((reported, counted + 1))
    assert (len(resets), len(resets)) in seen
    return None


def test_the_counting_warp_sees_every_phase():
    slack, ahead = constant("kResetSlack"), constant("kResetAhead")
    barriers = constant("kResetBarriers") if "kResetBarriers" in SOURCE else 1
    assert missed_phase(2, 1, 4, 20) is not None  # the walk finds a miss: two steps may report ahead of one mbarrier
    for steps in range(1, 30):
        assert missed_phase(slack, barriers, ahead, steps) is None


def wrong_exchange(slots, ahead, slack, steps):
    """A state in which a CTA takes an old word for a new one or a reset wipes out a word that has not been read, or None.

    Per CTA: its next step, the steps it has counted as reset, and the words of its slots: (step written or None) with the resets that
    are issued but not yet performed, which may take effect any time until they are counted.  Step t of a CTA: look at the others'
    words of step t - 1, wait for the resets of step t - slack, write slot t % slots, issue the reset of slot (t + ahead) % slots."""
    sent = steps - 1  # the last step sends nothing
    start = tuple((0, 0, (None,) * slots, ()) for _ in range(2))
    seen, todo = set(), [start]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        for me in range(2):
            step, counted, words, pending = state[me]
            other = state[1 - me]

            def push(new):
                todo.append((new, other) if me == 0 else (other, new))

            if step < steps:
                there = True
                if step > 0:
                    word = other[2][(step - 1) % slots]
                    if word is not None and word != step - 1:
                        return state
                    there = word == step - 1
                waits = step >= slack and step - slack + ahead + 1 < steps
                if there and (not waits or counted >= step - slack + 1):
                    new, late = list(words), pending
                    if step < sent:
                        if any(slot == step % slots for _, slot in pending):
                            return state  # a reset under way could overtake the word
                        new[step % slots] = step
                    if step + ahead + 1 < steps:
                        late = pending + ((step, (step + ahead) % slots),)
                    push((step + 1, counted, tuple(new), late))
            for i, (t, slot) in enumerate(pending):  # performed, in any order
                word = words[slot]
                if word is not None and other[0] <= word + 1:
                    return state  # the other CTA has not looked at it yet
                new = list(words)
                new[slot] = None
                push((step, counted, tuple(new), pending[:i] + pending[i + 1:]))
            if counted < step and counted + ahead + 1 < steps and all(t > counted for t, _ in pending):
                push((step, counted + 1, words, pending))
    assert any(all(cta[0] == steps for cta in state) for state in seen)
    return None


@pytest.mark.parametrize("steps", [1, 2, 5, 6, 9, 13, 20])
def test_slots_are_read_before_they_are_reset_and_reset_before_they_are_looked_at(steps):
    assert wrong_exchange(constant("kDirectSlots"), constant("kResetAhead"), constant("kResetSlack"), steps) is None


def test_the_walk_finds_exchanges_that_are_wrong():
    assert wrong_exchange(8, 1, 2, 20) is not None  # a slot is looked at before its reset is performed
    assert wrong_exchange(8, 7, 2, 20) is not None  # the slot of the step before is reset before it has been read everywhere
