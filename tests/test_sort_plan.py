"""The sort's device-side plan of its passes, restated from sort_plan (sort_kernels.cuh):
whatever passes move keys, every one reads what the one before wrote, nothing reads and
writes one buffer at once, a separate source is never written, and the result ends in the
output (a single pass in place: in the first alternate, copied back by the caller)."""
import itertools

import pytest

SORT, COPY = 16, 32


def sort_plan(trivial, in_place):
    passes = len(trivial)
    moving = [p for p in range(passes) if not trivial[p] or passes == 1]
    m = len(moving)

    def to(j):
        if not in_place or m % 2 == 0:
            return 2 if (m - 1 - j) % 2 else 1
        return 3 if j == 1 else 2 if j == 0 or j % 2 else 1

    def part(p):
        if m == 0:
            return COPY | 0 | 1 << 2 if not in_place and p == passes - 1 else 0
        last = moving[-1]
        if in_place and m == 1 and passes > 1:
            if last < passes - 1:
                return SORT | 0 | 2 << 2 if p == last else COPY | 2 | 1 << 2 if p == passes - 1 else 0
            return SORT | 2 | 1 << 2 if p == last else COPY | 0 | 2 << 2 if p == 0 else 0
        if p not in moving:
            return 0
        j = moving.index(p)
        return SORT | (to(j - 1) if j else 0) | to(j) << 2

    return [part(p) for p in range(passes)]


@pytest.mark.parametrize("in_place", [True, False])
@pytest.mark.parametrize("passes", range(1, 9))
def test_every_plan_ends_in_the_output(passes, in_place):
    for trivial in itertools.product([0, 1], repeat=passes):
        route = sort_plan(trivial, in_place)
        # the content of the buffers: how many sorting passes went into it (None: nothing)
        held = {0: 0, 1: 0 if in_place else None, 2: None, 3: None}
        done = 0
        for p, r in enumerate(route):
            if r == 0:
                assert trivial[p]
                continue
            src, dst = r & 3, r >> 2 & 3
            assert held[src] == done and dst != src and dst != 0
            assert not (in_place and src == 0 and dst == 1)
            assert dst != 3 or passes >= 3
            if r & SORT:
                assert not trivial[p] or passes == 1
                done += 1
            else:
                assert trivial[p]
            held[dst] = done
            if in_place and dst == 1:
                held[0] = done
        assert done == sum(1 for t in trivial if not t) or passes == 1
        assert held[2 if in_place and passes == 1 else 1] == done
