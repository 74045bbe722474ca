"""The work that a program on top of redfox_b200 has it do, as measurable cases.

Each case is a dict of plain values: `op` names the path, the rest its sizes and options.
The paths are the steps of a relational-algebra plan through the public entry points of
redfox_b200 -- the fused filter-aggregate scan, select, the radix sort, set operations, the
reductions of double values -- and whole plans: join + aggregate, the three-relation
pipeline and a captured batch of queries.  Sizes run from a few thousand rows, where
launches and host work count, to tens of millions.
"""
import math

import torch

from redfox_b200 import batch as B
from redfox_b200 import plans as PL
from redfox_b200 import rfx as R
from redfox_b200 import shapes as SH
from redfox_b200 import workloads as WL

SET_KINDS = {"union": R.SET_UNION, "difference": R.SET_DIFFERENCE, "intersection": R.SET_INTERSECTION}
F64_KINDS = {"sum": R.F64_SUM, "min": R.F64_MIN}


def listed():
    return [
        # the headline scan: a resident 60M-row fact table, filter + two products + 6 groups
        {"name": "aggregate_60M", "op": "aggregate", "n": 60_000_000, "cutoff": 2475},
        # a select that keeps almost every row of a wide table: the reporting query's first step
        {"name": "select_20M", "op": "select", "n": 20_000_000, "cutoff": 2475, "project": False},
        # a key list sorted before it enters the set operations
        {"name": "sort_u32_60M", "op": "sort", "n": 60_000_000, "key": 4, "value": 0, "begin": 0, "end": 32},
        # the kernel library's sort_pair: keys and a separate value column
        {"name": "sort_pairs_4M", "op": "sort", "n": 4_000_000, "key": 4, "value": 8, "begin": 0, "end": 32},
        # a small relation sorted on its join key: launches and latency
        {"name": "sort_rows_10K", "op": "sort", "n": 10_007, "key": 8, "value": 0, "begin": 32, "end": 64},
        # the plain plan at its own size: sort both sides, join, SUM and COUNT per key
        {"name": "join_aggregate_1Mx4M", "op": "join_aggregate", "nr": 1_000_000, "ns": 4_000_000,
         "domain": 1 << 18, "fused": False},
        # one short query of a mix, through the fused operator
        {"name": "join_aggregate_10Kx37K", "op": "join_aggregate", "nr": 10_000, "ns": 37_003,
         "domain": 2_500, "fused": True},
        # a whole plan: selects, two joins, set intersection and difference, reduce; skewed keys
        {"name": "three_relation_60M", "op": "three_relation", "n": 60_000_000, "resident": False},
        # a long sorted key list without the keys of another, both with duplicates
        {"name": "difference_60M_15M", "op": "set", "kind": "difference", "elem": 4, "na": 60_000_000,
         "nb": 15_000_000, "domain": 1 << 30},
        # two key lists of ordinary length merged
        {"name": "union_5M_2M", "op": "set", "kind": "union", "elem": 4, "na": 5_000_000, "nb": 2_000_000,
         "domain": 15_000_000},
        # SUM over a double column grouped by key (the shape of a join's output)
        {"name": "f64_sum_19M", "op": "f64", "kind": "sum", "n": 19_300_000, "groups": 256_000},
        # many queries of uneven sizes folded into one captured plan
        {"name": "batched_32", "op": "batched", "nq": 32, "lo": B.C3_MIN, "hi": B.C3_MAX, "sizes": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["aggregate", "select", "sort", "sort", "join_aggregate", "three_relation", "set", "set", "f64",
                     "batched"])
    if op == "aggregate":
        return {"op": op, "n": _log(rng, 4_000, 60_000_000), "cutoff": rng.randint(100, 2525)}
    if op == "select":
        return {"op": op, "n": _log(rng, 4_000, 20_000_000), "cutoff": rng.randint(100, 2525),
                "project": rng.random() < 0.5}
    if op == "sort":
        # key lists, packed rows on a key field of 12 to 32 bits, pairs
        key, value, top, most = rng.choice([(4, 0, 32, 60_000_000), (8, 0, 64, 20_000_000), (8, 0, 32, 60_000_000),
                                            (16, 0, 32, 60_000_000), (4, 4, 32, 60_000_000), (4, 8, 32, 40_000_000),
                                            (8, 8, 64, 15_000_000)])
        begin = {(8, 32): 32, (16, 32): 64}.get((key, top), 0)
        return {"op": op, "n": _log(rng, 4_000, most), "key": key, "value": value, "begin": begin,
                "end": begin + (top if rng.random() < 0.5 else rng.randint(12, top))}
    if op == "join_aggregate":
        nr = _log(rng, 4_000, 1_000_000)
        return {"op": op, "nr": nr, "ns": int(nr * rng.uniform(1.0, 4.0)), "domain": max(1, nr // rng.randint(1, 6)),
                "fused": rng.random() < 0.5}
    if op == "three_relation":
        return {"op": op, "n": _log(rng, 60_000, 60_000_000), "resident": rng.random() < 0.5}
    if op == "set":
        na = _log(rng, 4_000, 60_000_000)
        return {"op": op, "kind": rng.choice(sorted(SET_KINDS)), "elem": rng.choice([4, 4, 8]), "na": na,
                "nb": max(1, int(na * math.exp(rng.uniform(math.log(0.02), 0.0)))),
                "domain": min(1 << 30, int(na * rng.uniform(1.5, 20.0)))}
    if op == "f64":
        n = _log(rng, 4_000, 19_300_000)
        return {"op": op, "kind": rng.choice(sorted(F64_KINDS)), "n": n,
                "groups": max(1, int(n / math.exp(rng.uniform(math.log(4), math.log(1000)))))}
    return {"op": op, "nq": rng.randint(2, 32), "lo": B.C3_MIN, "hi": _log(rng, 100_000, 4_000_000),
            "sizes": rng.randint(2, 1 << 20)}


# ---------------------------------------------------------------------------- inputs
def _ints(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), dtype=torch.int64, device="cuda", generator=g)


def _rows16(hi, lo):
    """16-byte rows from their high and low 64-bit limbs."""
    return torch.stack((lo, hi), 1).view(torch.uint8)


def _wrap32(x):
    """The 32-bit patterns of values in [0, 2^32)."""
    return x.to(torch.int32)


def _sort_inputs(g, c):
    n, bits = c["n"], c["end"] - c["begin"]
    if c["key"] == 4:
        keys = _wrap32(_ints(g, 0, 1 << bits, n))
    elif c["key"] == 8 and c["begin"] == 0:
        keys = _ints(g, -(1 << 63), (1 << 63) - 1, n) if bits == 64 else _ints(g, 0, 1 << min(bits, 62), n)
    elif c["key"] == 8:
        keys = ((_ints(g, 0, 1 << bits, n) << 32) | _ints(g, 0, 1 << 32, n)).view(torch.uint8).view(n, 8)
    else:
        keys = _rows16(_ints(g, 0, 1 << bits, n), _ints(g, 100, 10_000_000, n))
    values = None
    if c["value"]:
        values = torch.arange(n, dtype=torch.int32 if c["value"] == 4 else torch.int64, device="cuda")
    return keys, values


def _fixed(*shape):
    """The generator of a case's key structure: which keys repeat and meet, the same for every
    seed, so that a result's size is the case's own.  The seed relabels the keys and draws
    the rest of the rows."""
    g = torch.Generator(device="cuda")
    return g.manual_seed(WL.SEED_BASE + sum((i + 1) * int(x) for i, x in enumerate(shape)))


def _relabel(g, n):
    return torch.randperm(n, dtype=torch.int64, device="cuda", generator=g)


def _join_keys(g, nr, ns, domain):
    """R's keys uniform in the domain, S's drawn from R's."""
    f = _fixed(nr, ns, domain)
    keys, pick, label = _ints(f, 0, domain, nr), _ints(f, 0, nr, ns), _relabel(g, domain)
    keys = label[keys]
    return keys, keys[pick]


def _join_inputs(g, nr, ns, domain):
    """R(key, payload) in 8-byte rows, S(fk, amount) in 16-byte rows."""
    rk, sk = _join_keys(g, nr, ns, domain)
    return ((rk << 32) | _ints(g, 0, 1 << 32, nr)).view(torch.uint8).view(nr, 8), _rows16(sk, _ints(g, 100, 10_000_000, ns))


def _three_relation_inputs(g, n3, resident):
    """D1(pk, segment), D2(pk, fk Zipf, date), F(fk, amount) and two sorted key lists, in the
    proportions of 1.5M : 15M : 60M : 5M : 2M rows."""
    n1, n2 = max(1, n3 // 40), max(1, n3 // 4)
    fx, label1, label2 = _fixed(n3), _relabel(g, n1), _relabel(g, n2)
    segment = _ints(fx, 0, 5, n1)[torch.argsort(label1)]
    d1 = ((torch.arange(n1, dtype=torch.int64, device="cuda") << 8) | segment).view(torch.uint8).view(n1, 8)
    cdf = torch.cumsum(1.0 / torch.arange(1, n1 + 1, dtype=torch.float64, device="cuda"), 0)
    u = torch.rand(n2, dtype=torch.float64, device="cuda", generator=fx) * cdf[-1]
    fk = torch.searchsorted(cdf, u, right=True).clamp_(max=n1 - 1)
    low = ((label1[fk] << 32) | _ints(fx, 0, 2526, n2))[torch.argsort(label2)]
    d2 = _rows16(torch.arange(n2, dtype=torch.int64, device="cuda"), low)
    fk = label2[_ints(fx, 0, n2, n3)]
    f = _rows16(torch.sort(fk).values if resident else fk, _ints(g, 100, 10_000_000, n3))
    lists = [_wrap32(torch.sort(label2[torch.unique(_ints(fx, 0, n2, max(1, n3 // k)))]).values) for k in (12, 30)]
    return d1, d2, f, lists[0], lists[1]


def _batch_inputs(g, sizes):
    """R and S of every query back to back, the query id folded into the key fields."""
    rs, ss = [], []
    for q, (nr, ns) in enumerate(sizes):
        rk, sk = _join_keys(g, nr, ns, max(1, nr // 4))
        rs.append((B.fold(rk, q) << 32) | _ints(g, 0, 1 << 32, nr))
        ss.append(torch.stack((_ints(g, 100, 10_000_000, ns), B.fold(sk, q)), 1))
    r, s = torch.cat(rs), torch.cat(ss)
    return r.view(torch.uint8).view(-1, 8), s.view(torch.uint8)


def _mirrored(values, top, seed):
    """Sorted values counted from the other end for every second seed."""
    return (top - values).flip(0) if seed % 2 else values


def _set_inputs(c, seed):
    """Two sorted lists with duplicates, shifted by the seed within 31 bits."""
    f, dt = _fixed(c["na"], c["nb"], c["domain"]), torch.int32 if c["elem"] == 4 else torch.int64
    shift = (seed * 7919) % (1 << 30)
    return [(_mirrored(torch.sort(_ints(f, 0, c["domain"], n)).values, c["domain"] - 1, seed) + shift).to(dt)
            for n in (c["na"], c["nb"])]


def _fact_rows(g, c, seed):
    """The fact table with every date equally often (field 0: bytes 34..37 of a row)."""
    rows = R.gen_uniform_rows(c["n"], SH.FACT_WIDTHS, seed, SH.FACT_LO, SH.FACT_HI)
    dates = (_relabel(g, c["n"]) % SH.FACT_HI[SH.F_DATE]).to(torch.int32)
    rows[:, 34:38] = dates.view(torch.uint8).view(-1, 4)
    return rows


def _sizes(c):
    return B.query_sizes(c["nq"], c["lo"], c["hi"], c["sizes"])


def _f64_inputs(c, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    keys = torch.sort(_ints(_fixed(c["n"], c["groups"]), 0, c["groups"], c["n"])).values
    return _wrap32(_mirrored(keys, c["groups"] - 1, seed)), _ints(g, 90_000, 10_500_001, c["n"]).to(torch.float64) / 100.0


def _predicate(c):
    return [(R.LE, (R.OPND_VAR, SH.F_DATE), (R.OPND_CONST, c["cutoff"]), R.I32)]


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    c, s = case, {"case": case}
    if c["op"] in ("aggregate", "select"):
        s["rows"] = _fact_rows(g, c, seed)
        if c["op"] == "aggregate":
            s["plan"] = R.FilterAggregate(c["n"], SH.FACT_WIDTHS, _predicate(c), WL.fact_ariths(),
                                          SH.FACT_GROUP_FIELDS, SH.FACT_GROUP_DOMAIN, SH.FACT_SUM_FIELDS)
    elif c["op"] == "sort":
        s["keys"], s["values"] = _sort_inputs(g, c)
    elif c["op"] == "join_aggregate":
        s["r"], s["s"] = _join_inputs(g, c["nr"], c["ns"], c["domain"])
    elif c["op"] == "three_relation":
        s["d1"], s["d2"], s["f"], s["in"], s["out"] = _three_relation_inputs(g, c["n"], c["resident"])
    elif c["op"] == "set":
        s["a"], s["b"] = _set_inputs(c, seed)
    elif c["op"] == "f64":
        s["keys"], s["values"] = _f64_inputs(c, seed)
    else:
        s["plan"] = B.BatchedPlan(*_batch_inputs(g, _sizes(c)))
        s["plan"].capture()
    return s


def run(state):
    s, c = state, state["case"]
    op = c["op"]
    if op == "aggregate":
        p = s["plan"]
        p.launch(s["rows"])
        return p.keys, p.sums, p.counts, p.ngroups
    if op == "select":
        if c["project"]:
            return R.select_project(s["rows"], SH.FACT_WIDTHS, _predicate(c), WL.fact_ariths()[:1], [8, 8, 64, 64],
                                    [SH.F_FLAG1, SH.F_FLAG2, SH.F_QTY, 7])[0]
        return R.select(s["rows"], SH.FACT_WIDTHS, _predicate(c))[0]
    if op == "sort":
        return R.sorted_copy(s["keys"], s["values"], c["begin"], c["end"])
    if op == "join_aggregate":
        return (PL.join_aggregate_fused if c["fused"] else PL.join_aggregate)(s["r"], s["s"])[:3]
    if op == "three_relation":
        return PL.three_relation(s["d1"], s["d2"], s["f"], s["in"], s["out"], f_sorted=s["f"] if c["resident"] else None)
    if op == "set":
        return R.set_op(SET_KINDS[c["kind"]], s["a"], s["b"])
    if op == "f64":
        return R.reduce_f64(s["keys"], s["values"], F64_KINDS[c["kind"]])
    s["plan"].replay()
    return s["plan"].result()


def work(case):
    """Each input read once, each output written once (expected sizes of uniform inputs)."""
    c, op = case, case["op"]
    if op == "aggregate":
        return {"bytes": 64.0 * c["n"], "flops": 0}
    if op == "select":
        kept = min(1.0, (c["cutoff"] + 1) / SH.FACT_HI[SH.F_DATE])
        return {"bytes": c["n"] * (64.0 + kept * (32.0 if c["project"] else 64.0)), "flops": 0}
    if op == "sort":
        return {"bytes": 2.0 * c["n"] * (c["key"] + c["value"]), "flops": 0}
    if op == "join_aggregate":
        return {"bytes": 8.0 * c["nr"] + 16.0 * c["ns"] + 16.0 * min(c["domain"], c["nr"]), "flops": 0}
    if op == "three_relation":
        n = c["n"]
        return {"bytes": 16.0 * n + 16.0 * (n // 4) + 8.0 * (n // 40) + 4.0 * (n // 12 + n // 30), "flops": 0}
    if op == "set":
        keep = {"union": c["na"] + c["nb"], "difference": c["na"], "intersection": 0}[c["kind"]]
        return {"bytes": float(c["elem"]) * (c["na"] + c["nb"] + keep), "flops": 0}
    if op == "f64":
        return {"bytes": 12.0 * c["n"] + 12.0 * min(c["groups"], c["n"]), "flops": 0}
    sizes = _sizes(c)
    return {"bytes": float(sum(8 * r + 16 * s + 16 * (r // 4) for r, s in sizes)), "flops": 0}


def exact(case, seed):
    """The double-valued results, each group's sum rounded once; the other paths give whole
    numbers and rows, which have no error to state."""
    if case["op"] != "f64":
        return None
    import numpy as np
    keys, values = _f64_inputs(case, seed)
    keys, values = keys.cpu().numpy(), values.cpu().numpy()
    starts = np.flatnonzero(np.concatenate(([True], keys[1:] != keys[:-1])))
    if case["kind"] == "min":
        return None, np.minimum.reduceat(values, starts), None
    ends, v = np.append(starts[1:], len(keys)).tolist(), values.tolist()
    return None, np.array([math.fsum(v[a:b]) for a, b in zip(starts.tolist(), ends)]), None
