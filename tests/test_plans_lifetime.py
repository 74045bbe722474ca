"""Plans run on a stream of the caller's choice while PyTorch's allocator reuses freed memory in
the order of the current one: what an enqueued sort reads out of place has to live until the
plan ends.  CPU only, with operators that record what they were given."""
import weakref

import pytest
import torch

from redfox_b200 import plans as PL


class Operators:
    """Stand-ins for the operators of redfox_b200.rfx."""
    EQ = GE = LT = OPND_VAR = OPND_CONST = I8 = I32 = SET_INTERSECTION = SET_DIFFERENCE = 0

    def __init__(self):
        self.sorted_from = []

    @staticmethod
    def rows(width):
        return torch.zeros((4, width), dtype=torch.uint8)

    def select(self, *a, **k):
        return self.rows(8), 4

    def select_project(self, *a, **k):
        return self.rows(8), 4

    def project(self, *a, **k):
        return self.rows(4)

    def join_tuples_two_step(self, *a, **k):
        return self.rows(16), 4

    def set_op(self, op, a, b, **k):
        return a.clone()

    def sorted_copy(self, keys, values=None, **k):
        self.sorted_from.append(weakref.ref(keys))
        return keys.clone(), None

    def reduce_tuples(self, *a, **k):
        assert all(ref() is not None for ref in self.sorted_from)
        return None, None, None, 0


@pytest.mark.parametrize("resident", [True, False])
def test_three_relation_keeps_what_its_sorts_read(monkeypatch, resident):
    ops = Operators()
    monkeypatch.setattr(PL, "R", ops)
    f = ops.rows(16)
    PL.three_relation(ops.rows(8), ops.rows(16), f, None, None, f_sorted=f if resident else None)
    assert len(ops.sorted_from) == (2 if resident else 3)


def test_join_aggregate_keeps_what_its_sorts_read(monkeypatch):
    ops = Operators()
    monkeypatch.setattr(PL, "R", ops)
    strided = torch.zeros((8, 16), dtype=torch.uint8)[::2]
    PL.join_aggregate(ops.rows(8), strided)
    assert len(ops.sorted_from) == 2
