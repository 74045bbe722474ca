"""Radix sort against the oracle's stable LSD sort (bit-exact, stability included)."""
import numpy as np
import pytest

import oracle as O
from redfox_b200 import rfx as R

from helpers import to_np

pytestmark = pytest.mark.gpu


def _keys(n, kb, seed, hi_bits=None):
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 256, (n, kb), dtype=np.uint8)
    if hi_bits is not None:  # keep only the low `hi_bits` bits
        bits = np.unpackbits(a, axis=1, bitorder="little")
        bits[:, hi_bits:] = 0
        a = np.packbits(bits, axis=1, bitorder="little")
    return a


def _dev(a, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


SIZES = [0, 1, 2, 31, 33, 1000, 4095, 4096, 4097, 100003]


@pytest.mark.parametrize("kb", [1, 2, 4, 8, 16, 32, 64])
@pytest.mark.parametrize("n", SIZES)
def test_sort_keys_full_width(cuda, kb, n):
    keys = _keys(n, kb, seed=kb * 31 + n)
    end = min(kb * 8, 128)
    d = _dev(keys, cuda)
    R.sort_pairs(d, begin_bit=0, end_bit=end)
    exp = O.sort_pairs(keys, begin_bit=0, end_bit=end)
    assert np.array_equal(to_np(d), exp)
    assert R.device_status() == R.OK


@pytest.mark.parametrize("kb,vb", [(4, 4), (4, 8), (8, 8), (8, 16), (16, 16), (16, 4), (1, 2), (2, 1), (64, 16), (32, 8)])
@pytest.mark.parametrize("n", [5, 4097, 200001])
def test_sort_pairs_stable(cuda, kb, vb, n):
    keys = _keys(n, kb, seed=n + kb * 7 + vb, hi_bits=min(kb * 8, 12))  # many duplicates
    vals = np.random.default_rng(n).integers(0, 256, (n, vb), dtype=np.uint8)
    dk, dv = _dev(keys, cuda), _dev(vals, cuda)
    end = min(kb * 8, 40)
    R.sort_pairs(dk, dv, begin_bit=0, end_bit=end)
    ek, ev = O.sort_pairs(keys, vals, begin_bit=0, end_bit=end)
    assert np.array_equal(to_np(dk), ek) and np.array_equal(to_np(dv), ev)


@pytest.mark.parametrize("begin,end", [(3, 17), (64, 96), (100, 128), (8, 9)])
def test_sort_bit_range_of_packed_tuples(cuda, begin, end):
    n = 50000
    keys = _keys(n, 16, seed=begin * 1000 + end)
    d = _dev(keys, cuda)
    R.sort_pairs(d, begin_bit=begin, end_bit=end)
    assert np.array_equal(to_np(d), O.sort_pairs(keys, begin_bit=begin, end_bit=end))


def test_sort_wide_range_over_128_bits(cuda):
    n = 20000
    keys = _keys(n, 32, seed=3, hi_bits=200)
    d = _dev(keys, cuda)
    R.sort_pairs(d, begin_bit=0, end_bit=256)
    assert np.array_equal(to_np(d), O.sort_pairs(keys, begin_bit=0, end_bit=256))


def test_all_equal_keys_keep_input_order(cuda):
    import torch
    n = 300000
    keys = torch.full((n,), 7, dtype=torch.int32, device=cuda)
    vals = torch.arange(n, dtype=torch.int32, device=cuda)
    R.sort_pairs(keys, vals)
    assert torch.equal(vals, torch.arange(n, dtype=torch.int32, device=cuda))


def test_skip_trivial_passes_same_result(cuda):
    n = 1_000_003
    keys = _keys(n, 4, seed=11, hi_bits=18)
    vals = np.arange(n, dtype=np.uint32)
    a, av = _dev(keys, cuda), _dev(vals, cuda)
    b, bv = _dev(keys, cuda), _dev(vals, cuda)
    R.sort_pairs(a, av)
    R.sort_pairs(b, bv, flags=R.SORT_SKIP_TRIVIAL)
    ek, ev = O.sort_pairs(keys, vals)
    for k, v in ((a, av), (b, bv)):
        assert np.array_equal(to_np(k), ek) and np.array_equal(to_np(v), ev)


def test_large_sort_properties(cuda):
    """Full-size property check: sorted, and a permutation (value checksum) at 8M pairs."""
    import torch
    n = 8_000_000
    g = torch.Generator(device=cuda).manual_seed(5)
    keys = torch.randint(0, 2**31 - 1, (n,), dtype=torch.int64, device=cuda, generator=g)
    vals = torch.arange(n, dtype=torch.int64, device=cuda)
    k0 = keys.clone()
    R.sort_pairs(keys, vals)
    assert bool((keys[1:] >= keys[:-1]).all())
    assert int(vals.sum()) == n * (n - 1) // 2
    assert torch.equal(k0[vals], keys)


def test_reference_compatible_entries(cuda):
    import ctypes as C
    import torch
    n = 70000
    rng = np.random.default_rng(1)
    # b40c sort_pair: 18-bit keys in u32 containers, I64 values (value_type code 4)
    k = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    v = np.arange(n, dtype=np.uint64)
    dk, dv = _dev(k, cuda), _dev(v, cuda)
    torch.cuda.synchronize()
    assert R.LIB.rfx_b40c_sort_pair(C.c_void_p(dk.data_ptr()), C.c_void_p(dv.data_ptr()), n, 18, R.I64) == R.OK
    ek, ev = O.sort_pairs(k, v, begin_bit=0, end_bit=18)
    assert np.array_equal(to_np(dk), ek) and np.array_equal(to_np(dv), ev)
    # mgpu sort_key on 128-bit keys (I128): whole-key order, high limb first
    k128 = rng.integers(0, 256, (n, 16), dtype=np.uint8)
    dk = _dev(k128, cuda)
    torch.cuda.synchronize()
    assert R.LIB.rfx_mgpu_sort_key(C.c_void_p(dk.data_ptr()), n, R.I128) == R.OK
    assert np.array_equal(to_np(dk), O.sort_pairs(k128))
    # b40c sort_key with 37 bits in u64 containers
    k64 = rng.integers(0, 2**63, n, dtype=np.uint64)
    dk = _dev(k64, cuda)
    torch.cuda.synchronize()
    assert R.LIB.rfx_b40c_sort_key(C.c_void_p(dk.data_ptr()), n, 37) == R.OK
    assert np.array_equal(to_np(dk), O.sort_pairs(k64, begin_bit=0, end_bit=37))


# Tile sizes of the two pass kernels: the per-tile pass (3072 / 5120 / 6144 keys of 16 / 8
# / 4 bytes) and the pipelined onesweep pass (3072 / 6144 / 8192 by default); sizes around
# both, and sizes with many tiles per block (persistent grids).
ONESWEEP_SIZES = {16: [3071, 3072, 3073, 9217, 2_000_003], 8: [5119, 5120, 5121, 6145, 18_433, 3_000_001],
                  4: [6143, 6144, 6145, 8193, 24_577, 4_000_037]}


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("kb", [4, 8, 16])
def test_sort_pass_variants_match_oracle(cuda, kb, variant):
    """Every pass kernel variant (pinned through the tuner) gives the oracle's stable
    order, on whole keys and on bit ranges that leave payload bits outside the key."""
    try:
        R.tune_force(R.TUNE_SORT_PASS, variant)
        for n in ONESWEEP_SIZES[kb]:
            keys = _keys(n, kb, seed=n * 3 + kb)
            # whole keys; a range leaving payload bits; odd pass counts (3 and 5 digits),
            # which end in the caller's buffer through the second alternate buffer
            for begin, end in ((0, kb * 8), (kb * 4, kb * 8 - 3), (kb * 8 - 24, kb * 8), (kb * 8 - 40, kb * 8 - 1)):
                if begin < 0:
                    continue
                d = _dev(keys, cuda)
                R.sort_pairs(d, begin_bit=begin, end_bit=end)
                assert np.array_equal(to_np(d), O.sort_pairs(keys, begin_bit=begin, end_bit=end, threads=8)), (n, begin)
        assert R.device_status() == R.OK
    finally:
        R.tune_force(R.TUNE_SORT_PASS, -1)


def test_sort_unaligned_slice_uses_per_tile_pass(cuda):
    """A key array that starts 8 bytes into an allocation (not 16-byte aligned) is sorted by
    the per-tile pass with the same result."""
    import torch
    n = 100_001
    keys = _keys(n + 1, 8, seed=77)
    d = _dev(keys, cuda)
    sub = d[1:]
    assert sub.data_ptr() % 16 == 8
    R.sort_pairs(sub, begin_bit=0, end_bit=64)
    assert np.array_equal(to_np(sub), O.sort_pairs(keys[1:], begin_bit=0, end_bit=64))
    assert torch.equal(d[0], _dev(keys[0], cuda))


@pytest.mark.parametrize("kb,vb,begin,end", [(4, 0, 0, 8), (4, 0, 0, 16), (8, 8, 8, 32), (16, 0, 64, 96),
                                             (8, 4, 0, 64), (16, 16, 0, 128), (64, 0, 0, 200)])
@pytest.mark.parametrize("n", [1, 33, 100003])
def test_sort_from_leaves_input_and_matches_in_place(cuda, kb, vb, begin, end, n):
    """rfx_sort_pairs_from sorts the input into other buffers (one to four passes, values,
    keys over 128 bits) with the in-place sort's result and leaves the input as it was."""
    import torch
    keys = _keys(n, kb, seed=kb + vb + n + end)
    vals = _keys(n, vb, seed=7 + n) if vb else None
    dk = _dev(keys, cuda)
    dv = _dev(vals, cuda) if vb else None
    ok, ov = R.sorted_copy(dk, dv, begin_bit=begin, end_bit=end)
    assert np.array_equal(to_np(dk), keys)
    if vb:
        assert np.array_equal(to_np(dv), vals)
    ek = _dev(keys, cuda)
    ev = _dev(vals, cuda) if vb else None
    R.sort_pairs(ek, ev, begin_bit=begin, end_bit=end)
    assert torch.equal(ok, ek)
    if vb:
        assert torch.equal(ov, ev)
    assert R.device_status() == R.OK


def test_sort_from_all_trivial_and_overlap(cuda):
    """Every digit constant with the skip flag: the output is a copy of the input.  Input
    and output overlapping: rejected."""
    import torch
    keys = np.zeros((5000, 4), np.uint8)
    keys[:, 0] = np.arange(5000) % 256
    dk = _dev(keys, cuda)
    out = torch.empty_like(dk)
    s = R.Sorter(5000, 4, 0, 8, 32, device=cuda)
    s(out, None, 1, None, src_keys=dk)
    assert np.array_equal(to_np(out), keys)
    st = R.LIB.rfx_sort_pairs_from(R._ptr(dk), None, R._ptr(dk[100:]), None, 4000, 4, 0, 0, 32, 0, R._ptr(s.ws), s.wsb,
                                   R._stream())
    assert st == R.ERR_INVALID


# Keys per tile of the digit pass, by key and value bytes (SortTuning): 4 B 10240, up to 8 B
# 7168, up to 12 B 5120, up to 16 B 4608, up to 32 B 2304, up to 48 B 1536, above 1024.
TILE_KEYS = {(1, 0): 10240, (4, 0): 10240, (8, 0): 7168, (4, 4): 7168, (4, 8): 5120, (16, 0): 4608, (8, 8): 4608,
             (16, 16): 2304, (32, 0): 2304, (32, 16): 1536, (64, 16): 1024}
ABOVE_CLUSTER = 70_000   # rows the one-launch sort does not take


@pytest.mark.parametrize("kb,vb", sorted(TILE_KEYS))
@pytest.mark.parametrize("extra", [-1, 0, 1, 2 * 10240 + 17])
def test_sort_tile_edges_with_many_equal_digits(cuda, kb, vb, extra):
    """Whole tiles less a key, whole tiles, a key more, some tiles more; digits that straddle a
    32-bit word and digits that most of a warp's keys share, whose order must stay."""
    tile = TILE_KEYS[kb, vb]
    n = (ABOVE_CLUSTER // tile + 1) * tile + extra
    keys = _keys(n, kb, seed=n + kb)
    keys[:, (kb * 8 - 5) // 8] &= np.uint8(0x13)
    vals = np.random.default_rng(n).integers(0, 256, (n, vb), dtype=np.uint8) if vb else None
    for begin, end in ((0, min(kb * 8, 11)), (max(0, kb * 8 - 21), kb * 8 - 1)):
        dk, dv = R.sorted_copy(_dev(keys, cuda), _dev(vals, cuda) if vb else None, begin_bit=begin, end_bit=end)
        exp = O.sort_pairs(keys, vals, begin_bit=begin, end_bit=end) if vb else (O.sort_pairs(keys, begin_bit=begin,
                                                                                              end_bit=end), None)
        assert np.array_equal(to_np(dk), exp[0])
        if vb:
            assert np.array_equal(to_np(dv), exp[1])
    assert R.device_status() == R.OK


@pytest.mark.parametrize("moving", [[], [0], [1], [3], [0, 3], [0, 1, 2], [1, 2, 3], [0, 1, 2, 3]])
@pytest.mark.parametrize("kb,vb,n", [(4, 0, 20_011), (8, 4, 9_001), (16, 0, 70_001)])
def test_sort_skips_constant_digits_on_the_device(cuda, kb, vb, n, moving):
    """Constant digits in every place among four: in place and out of place, keys and values."""
    keys = np.full((n, kb), 0x5A, np.uint8)
    rng = np.random.default_rng(n + sum(moving))
    for b in moving:
        keys[:, kb - 4 + b] = rng.integers(0, 256, n, dtype=np.uint8)
    if kb > 4:
        keys[:, 0] = rng.integers(0, 256, n, dtype=np.uint8)   # payload: shows the order of equal keys
    vals = rng.integers(0, 256, (n, vb), dtype=np.uint8) if vb else None
    begin, end = (kb - 4) * 8, kb * 8
    exp = O.sort_pairs(keys, vals, begin_bit=begin, end_bit=end) if vb else (O.sort_pairs(keys, begin_bit=begin,
                                                                                          end_bit=end), None)
    a, av = _dev(keys, cuda), _dev(vals, cuda) if vb else None
    b, bv = R.sorted_copy(a, av, begin_bit=begin, end_bit=end)
    assert np.array_equal(to_np(a), keys)
    R.sort_pairs(a, av, begin_bit=begin, end_bit=end)
    for k, v in ((a, av), (b, bv)):
        assert np.array_equal(to_np(k), exp[0])
        if vb:
            assert np.array_equal(to_np(v), exp[1])
    assert R.device_status() == R.OK


# The one-launch sort takes inputs up to 16 slices of 64 KB or 4096 elements (ClusterTuning).
@pytest.mark.parametrize("kb,vb,most", [(1, 0, 65536), (4, 0, 65536), (8, 0, 65536), (4, 8, 65536), (16, 0, 65536),
                                        (16, 8, 43520), (64, 16, 12800)])
@pytest.mark.parametrize("n", [2, 31, 512, 513, 1025, 8193, "most", "above"])
def test_sort_small_inputs_in_one_cluster(cuda, kb, vb, most, n):
    """One block, every cluster size and its neighbours, the largest input and the first that
    takes the general passes; constant digits first, between and last; in and out of place."""
    n = most if n == "most" else most + 1 if n == "above" else n
    keys = _keys(n, kb, seed=n * 5 + kb)
    keys[:, kb // 2] &= np.uint8(0x81)
    keys[:, kb - 1] = 7
    vals = np.random.default_rng(n).integers(0, 256, (n, vb), dtype=np.uint8) if vb else None
    for begin, end in ((0, kb * 8), (max(0, kb * 8 - 24), kb * 8), (max(0, kb * 8 - 13), kb * 8 - 4)):
        a, av = _dev(keys, cuda), _dev(vals, cuda) if vb else None
        b, bv = R.sorted_copy(a, av, begin_bit=begin, end_bit=end)
        exp = O.sort_pairs(keys, vals, begin_bit=begin, end_bit=end) if vb else (O.sort_pairs(keys, begin_bit=begin,
                                                                                              end_bit=end), None)
        assert np.array_equal(to_np(a), keys)
        R.sort_pairs(a, av, begin_bit=begin, end_bit=end)
        for k, v in ((a, av), (b, bv)):
            assert np.array_equal(to_np(k), exp[0]), (begin, end)
            if vb:
                assert np.array_equal(to_np(v), exp[1]), (begin, end)
    assert R.device_status() == R.OK


@pytest.mark.parametrize("kb,vb", [(4, 0), (8, 0), (4, 4), (4, 8), (8, 4), (16, 0), (8, 8)])
@pytest.mark.parametrize("where", ["small tile", "last small", "first large"])
def test_sort_small_and_large_tiles(cuda, kb, vb, where):
    """The pass's small tiles (512 threads x 8, 6, 5 or 4 elements) at a tile's edge, the most
    elements that take them (148 large tiles) and one more."""
    small = 512 * {4: 8, 8: 6, 12: 5, 16: 4}[kb + vb]
    n = {"small tile": (ABOVE_CLUSTER // small + 1) * small + 1, "last small": 148 * TILE_KEYS.get((kb, vb), 5120),
         "first large": 148 * TILE_KEYS.get((kb, vb), 5120) + 1}[where]
    keys = _keys(n, kb, seed=n + kb)
    vals = np.random.default_rng(n).integers(0, 256, (n, vb), dtype=np.uint8) if vb else None
    begin, end = kb * 8 - 19, kb * 8
    dk, dv = R.sorted_copy(_dev(keys, cuda), _dev(vals, cuda) if vb else None, begin_bit=begin, end_bit=end)
    exp = (O.sort_pairs(keys, vals, begin_bit=begin, end_bit=end, threads=8) if vb
           else (O.sort_pairs(keys, begin_bit=begin, end_bit=end, threads=8), None))
    assert np.array_equal(to_np(dk), exp[0])
    if vb:
        assert np.array_equal(to_np(dv), exp[1])
    assert R.device_status() == R.OK


@pytest.mark.parametrize("kb,vb", [(4, 0), (8, 0), (4, 8), (16, 0)])
def test_smaller_inputs_in_the_workspace_of_more(cuda, kb, vb):
    """One workspace, sized for some more rows than take small tiles, serves the sizes on either
    side of that line."""
    line = 148 * TILE_KEYS[kb, vb]
    s = R.Sorter(line + 1, kb, vb, kb * 8 - 24, kb * 8)
    for n in (line + 1, line, line - 1, line // 2, 5):
        keys = _keys(n, kb, seed=n)
        vals = np.random.default_rng(n).integers(0, 256, (n, vb), dtype=np.uint8) if vb else None
        s.n = n
        dk, dv = _dev(keys, cuda), _dev(vals, cuda) if vb else None
        s(dk, dv)
        exp = (O.sort_pairs(keys, vals, begin_bit=s.begin, end_bit=s.end, threads=8) if vb
               else (O.sort_pairs(keys, begin_bit=s.begin, end_bit=s.end, threads=8), None))
        assert np.array_equal(to_np(dk), exp[0]), n
        if vb:
            assert np.array_equal(to_np(dv), exp[1]), n
    assert R.device_status() == R.OK


@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("count", [0, 1, 2, 3, 31, 255, 257, 511, 513, 1023, 4608, 7167, 10240])
def test_order_entries(cuda, count, threads):
    """The repair of a tile whose entries (digit << 16 | place in the tile) are out of order, which
    inputs bring about only if the hardware serves a warp's atomics out of lane order: equal digits
    exchanged within a warp's step, each digit's places turned round, one entry far off, none."""
    import ctypes as C
    rng = np.random.default_rng(count + threads)
    digit = np.sort(rng.integers(0, 40, count)).astype(np.uint32)
    want = digit << 16 | np.arange(count, dtype=np.uint32)
    swapped, turned, far = want.copy(), want.copy(), want.copy()
    for i in range(0, count - 31, 32):
        part = swapped[i:i + 32]
        for d in np.unique(part >> 16):
            m = part >> 16 == d
            part[m] = rng.permutation(part[m])
    for d in np.unique(digit):
        turned[digit == d] = turned[digit == d][::-1]
    if count > 2:
        far[0], far[-1] = want[-1], want[0]
    for got in (want, swapped, turned, far):
        dev = _dev(np.append(got, np.uint32(0xABCD)).view(np.int32), cuda)   # one more: not touched
        st = R.LIB.rfx_test_order_entries(R._ptr(dev), C.c_uint32(count), C.c_uint32(threads), R._stream())
        out = to_np(dev).view(np.uint32)
        assert st == R.OK and np.array_equal(out[:count], np.sort(want)) and out[count] == 0xABCD


@pytest.mark.parametrize("moving", [[], [0], [1], [3], [0, 3], [0, 1, 2], [1, 2, 3], [0, 1, 2, 3]])
@pytest.mark.parametrize("kb,vb,n", [(4, 0, 70_011), (8, 4, 70_001), (4, 1, 70_003), (8, 16, 70_001)])
def test_sort_skips_constant_digits_above_the_cluster_sort(cuda, kb, vb, n, moving):
    """Constant digits in every place among four, sizes that the digit passes take: keys and values
    in place and out of place, with 16-byte aligned arrays and with others."""
    rng = np.random.default_rng(n + sum(moving))
    keys = np.full((n + 1, kb), 0x5A, np.uint8)
    for b in moving:
        keys[:, kb - 4 + b] = rng.integers(0, 256, n + 1, dtype=np.uint8)
    if kb > 4:
        keys[:, 0] = rng.integers(0, 256, n + 1, dtype=np.uint8)   # payload: shows the order of equal keys
    vals = rng.integers(0, 256, (n + 1, vb), dtype=np.uint8) if vb else None
    begin, end = (kb - 4) * 8, kb * 8
    for first in (0, 1):
        hk, hv = keys[first:first + n], vals[first:first + n] if vb else None
        exp = O.sort_pairs(hk, hv, begin_bit=begin, end_bit=end) if vb else (O.sort_pairs(hk, begin_bit=begin,
                                                                                          end_bit=end), None)
        a, av = _dev(keys, cuda)[first:first + n], _dev(vals, cuda)[first:first + n] if vb else None
        b, bv = R.sorted_copy(a, av, begin_bit=begin, end_bit=end)
        assert np.array_equal(to_np(a), hk)
        R.sort_pairs(a, av, begin_bit=begin, end_bit=end)
        for k, v in ((a, av), (b, bv)):
            assert np.array_equal(to_np(k), exp[0]), first
            if vb:
                assert np.array_equal(to_np(v), exp[1]), first
    assert R.device_status() == R.OK


def test_a_small_sort_warms_up_for_a_captured_large_one():
    """In a process whose first call is a small sort (the one-launch form, which needs none of the
    device's lasting state), a larger one can be captured, as after any other first sort; a small
    one can be captured as the first call."""
    import os
    import subprocess
    import sys
    code = """
import torch
from redfox_b200 import rfx as R
def capture(n):
    k = torch.randint(0, 256, (n, 4), dtype=torch.uint8, device="cuda")
    o, s, g = torch.empty_like(k), R.Sorter(n, 4), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s(o, src_keys=k)
    g.replay()
    torch.cuda.synchronize()
    return k, o
pairs = [capture(5000)] if FIRST else []
R.sorted_copy(torch.randint(0, 256, (5000, 4), dtype=torch.uint8, device="cuda"))
pairs.append(capture(300000))
assert all(torch.equal(o, R.sorted_copy(k)[0]) for k, o in pairs)
"""
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for first in ("False", "True"):
        r = subprocess.run([sys.executable, "-c", code.replace("FIRST", first)], cwd=repo, capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, (first, r.stderr[-2000:])
