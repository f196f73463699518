"""Phases of the mbarriers of the paired prefill kernel (csrc/tq_prefill_attn.cu), read from its source and stepped
through on the CPU.

A wait on a parity passes when the barrier's current phase has the other parity.  It cannot tell a phase that has not
completed from the one two before it, so a thread must not be able to sleep through two completions of a barrier.
"""

import itertools
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turboquant_b200", "csrc", "tq_prefill_attn.cu")


def _pair_kernel():
    text = open(SOURCE).read()
    body = text[text.index("tq_prefill_pair_kernel("):]
    return body[:body.index("typedef CUresult")]


def _finishes(waits, commits, seen_first):
    """A softmax warp polls `waits` [(barrier, parity)]; `commits` are the barriers that complete, in order, the first
    `seen_first` of them before the warp looks at all, the others while it waits.  Returns how many commits had completed
    when the last wait passed, None if one never does."""
    count = dict.fromkeys([b for b, _ in waits] + list(commits), 0)
    done = 0
    for b in commits[:seen_first]:
        count[b] += 1
        done += 1
    for b, parity in waits:
        while count[b] % 2 == parity:          # the current phase has this parity: not completed yet
            if done == len(commits):
                return None
            count[commits[done]] += 1
            done += 1
    return done


@pytest.mark.parametrize("w", [0, 1])
def test_last_products_are_seen_however_late_a_warp_looks(w):
    body = _pair_kernel()
    commit = re.findall(r"umma_commit\(bar_o \+ ([^)]+)\)", body)
    assert len(commit) == 1
    commits = [eval(commit[0], {"w": w, "odd": odd}) for odd in (0, 1)]      # the halves of the last key tile
    wait = r"wait_warp\(bar_o \+ ([^,]+), (\d)\)"
    lines = [line for line in body.splitlines() if re.search(wait, line)]
    assert len(lines) == 2                                                   # the rescale of the last half, the epilogue
    rescale, epilogue = ([(eval(e, {"w": w}), int(p)) for e, p in re.findall(wait, line)] for line in lines)
    for looked in range(3):
        # the epilogue passes once the products of both halves are complete, never earlier, and always
        assert _finishes(epilogue, commits, looked) == 2, (commits, epilogue, looked)
        # the rescale of the second half needs the first half's; the second's wait for this very warp
        if looked < 2:
            assert _finishes(rescale, commits, looked) == 1
    other = [eval(commit[0], {"w": 1 - w, "odd": odd}) for odd in (0, 1)]
    assert not set(commits) & set(other)


def test_every_barrier_has_its_own_place_and_is_initialised():
    body = _pair_kernel()
    names = {m[0]: int(m[1] or 0) for m in re.findall(r"\*(bar_\w+|free_\w+) = bars(?: \+ (\d+))?", body)}
    total = int(re.search(r"constexpr int PP_BARS = (\d+);", open(SOURCE).read()).group(1))
    used = list(itertools.chain(*([names[n] + i for i in range(c)] for n, c in (
        ("bar_q", 1), ("bar_k", 2), ("bar_v", 2), ("free_k", 2), ("free_v", 2), ("bar_o", 4), ("bar_s", 4), ("bar_p", 4)))))
    assert sorted(used) == list(range(total))
    first_arrivals = int(re.search(r"tq_mbar_init\(bars \+ i, i >= (\d+) \? PA_TOK : 1\)", body).group(1))
    assert first_arrivals == names["bar_p"]
