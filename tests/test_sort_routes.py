"""The sort's plan of its passes, as the library computes it (sort_plan, sort_kernels.cuh): whatever
passes move keys, every one reads what the one before wrote, nothing reads and writes one buffer
at once, a separate source is never written, and the result ends in the output (a single pass in
place: in the first alternate, copied back by the caller)."""
import ctypes as C

import pytest

from redfox_b200 import rfx as R

SORT, COPY = 16, 32
R.LIB.rfx_test_sort_plan.restype = C.c_uint32
R.LIB.rfx_test_sort_plan.argtypes = [C.c_uint32] * 4


@pytest.mark.parametrize("in_place", [0, 1])
@pytest.mark.parametrize("passes", [*range(1, 11), 16])
def test_every_plan_ends_in_the_output(passes, in_place):
    for moving in range(0, 1 << passes, 1 if passes < 16 else 7):
        # the content of the buffers: how many passes that move keys went into each
        held = {0: 0, 1: 0 if in_place else None, 2: None, 3: None}
        done = 0
        for p in range(passes):
            r = R.LIB.rfx_test_sort_plan(moving, passes, in_place, p)
            moves = bool(moving >> p & 1) or passes == 1
            assert bool(r & SORT) == moves and r < 64 and not (r & SORT and r & COPY)
            if r == 0:
                continue
            src, dst = r & 3, r >> 2 & 3
            assert held[src] == done and dst not in (0, src) and not (in_place and src == 0 and dst == 1)
            assert dst != 3 or passes >= 3   # the second pair of alternates exists from three passes on
            done += moves
            held[dst] = done
            if in_place and dst == 1:
                held[0] = done
        assert done == (bin(moving).count("1") if passes > 1 else 1)
        assert held[2 if in_place and passes == 1 else 1] == done
