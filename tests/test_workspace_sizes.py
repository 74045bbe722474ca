"""Workspace sizes never fall as the input grows, so that one sized for the largest input
serves every smaller one: around the sizes where an operator changes its unit or tile."""
import pytest

from redfox_b200 import rfx as R


def _rises(size, edges):
    ns = sorted({max(1, n + d) for n in edges for d in (-1, 0, 1, 2)})
    sizes = [size(n) for n in ns]
    falls = [(a, b, x, y) for a, b, x, y in zip(ns, ns[1:], sizes, sizes[1:]) if y < x]
    assert not falls, falls


def test_reduce_f64():
    step = 32 * 148 * 256   # one unit of 256 elements per resident warp
    _rises(R.LIB.rfx_reduce_f64_workspace, [1, 255, 256, 257, 4096, 10**6, *(k * step for k in range(1, 18)),
                                            20_000_000, 60_000_000, (1 << 30) - 2])


@pytest.mark.parametrize("kb,vb", [(1, 0), (4, 0), (8, 0), (16, 0), (64, 0), (4, 4), (4, 8), (8, 4), (8, 8), (16, 16)])
@pytest.mark.parametrize("bits", [8, 16, 24, 0])
def test_sort(kb, vb, bits):
    tile = {1: 10240, 4: 10240, 8: 7168, 12: 5120, 16: 4608}.get(kb + vb, 2304)
    edges = [1, 31, 512, 65536, 10**6, 20_000_000, (1 << 30) - 2, *(k * tile for k in (1, 2, 99, 147, 148, 149, 371))]
    _rises(lambda n: R.LIB.rfx_sort_workspace(n, kb, vb, 0, min(bits, kb * 8) or kb * 8), edges)
