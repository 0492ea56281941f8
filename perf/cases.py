"""Performance cases: the queries a program runs through this package's plan API.

A state holds what such a program keeps: an engine with its registered tables
and a prepared plan (or a prepared batch).  One pass executes it and takes the
result columns, ordered by their keys: a plan returns its rows in no particular
order, so a program that prints or compares them orders them first.  Every value
is a whole number or a byte, so results are exact.

Tables are drawn on the GPU from the seed and registered from host memory.
"""
import math

import numpy as np
import torch

from dogqc_b200 import scalar as scal
from dogqc_b200 import workloads
from dogqc_b200.database import Database, StringColumn, Table
from dogqc_b200.engine import Engine
from dogqc_b200.lowering import Lowering
from dogqc_b200.relational import Reduction, RelationalAlgebra
from dogqc_b200.types import Type

DAY0, DAYS = workloads.EPOCH_1992, workloads.DATE_RANGE
I, S, F, D, C = Type.INT, Type.STRING, Type.FLOAT, Type.DATE, Type.CHAR


def listed():
    return [
        # the smallest call: a dashboard tile over a small dimension and fact
        # table, where launches and host work count
        {"name": "join_agg_tiny", "kind": "join_agg", "rows": 6_000},
        # the headline benchmark: a filtered dimension of 1.5 M rows joined to
        # 6 M facts, grouped by 25 nations
        {"name": "join_agg", "kind": "join_agg", "rows": 6_000_000},
        # a pricing summary report (TPC-H Q1): one scan, six groups, eight aggregates
        {"name": "scan_agg", "kind": "scan_agg", "rows": 6_000_000},
        # a join on skewed keys where a probe row meets from none to many
        # thousands of build rows, then four filters and a count
        {"name": "expand", "kind": "expand", "rows": 16_777_216, "two_sided": False},
        # the largest: a three-way star join over 60 M facts into 750 k groups,
        # of which the few large ones are wanted (a HAVING clause)
        {"name": "star_having", "kind": "star", "rows": 60_000_000, "having": True},
        # the same join over an ordinary fact table, every group read back
        {"name": "star_groups", "kind": "star", "rows": 6_000_001, "having": False},
        # grouping by two variable-length strings that the result carries (TPC-H Q12)
        {"name": "string_group", "kind": "string_group", "rows": 6_000_000},
        # NOT LIKE over 1.5 M comments, an outer join and an aggregation over an
        # aggregation (TPC-H Q13)
        {"name": "like_outer", "kind": "like_outer", "rows": 1_500_000},
        # EXISTS and NOT EXISTS with conditions over three scans of 6 M lines (TPC-H Q21)
        {"name": "exists", "kind": "exists", "rows": 6_000_000},
        # a LIKE prefix, semi joins, a two-key table built from an aggregation and
        # string results (TPC-H Q20)
        {"name": "excess", "kind": "excess", "rows": 6_000_000},
        # substrings in an IN list and as a group key, a scalar subquery and an
        # anti join (TPC-H Q22): many short pipelines
        {"name": "substring_anti", "kind": "substring_anti", "rows": 1_500_000},
        # many small instances of one query in one batch
        {"name": "batch", "kind": "batch", "rows": 65_536, "instances": 48},
    ]


# rows of each kind's largest table that a drawn case may have
RANGES = {"join_agg": (3_000, 12_000_000), "scan_agg": (1_000, 24_000_000), "expand": (50_000, 16_000_000),
          "star": (400_000, 30_000_000), "string_group": (20_000, 6_000_000), "like_outer": (10_000, 1_500_000),
          "exists": (20_000, 6_000_000), "excess": (60_000, 6_000_000), "substring_anti": (10_000, 3_000_000),
          "batch": (2_000, 65_536)}


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    lo, hi = RANGES[kind]
    case = {"kind": kind, "rows": int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))}
    if kind == "expand":
        case["two_sided"] = rng.random() < 0.5  # the last filter compares a build with a probe attribute
    if kind == "star":
        case["having"] = case["rows"] > 6_000_000 or rng.random() < 0.5
    if kind == "batch":
        case["instances"] = rng.randint(4, 64)
    return case


# ------------------------------------------------------------------ tables --

class Draw(object):
    """Seeded columns, drawn on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def ints(self, lo, hi, n):
        """n whole numbers in [lo, hi)."""
        return torch.randint(lo, hi, (n,), device="cuda", generator=self.g)

    def perm(self, n):
        """1..n in random order."""
        return torch.randperm(n, device="cuda", generator=self.g) + 1

    def pick(self, values, n):
        return torch.as_tensor(values, device="cuda")[self.ints(0, len(values), n)]

    def uniform(self, n):
        return torch.rand(n, device="cuda", dtype=torch.float64, generator=self.g)

    def zipf(self, n, distinct):
        """Keys in 1..distinct with P(rank k) ~ 1/k and shuffled labels."""
        cdf = torch.cumsum(1.0 / torch.arange(1, distinct + 1, device="cuda", dtype=torch.float64), 0)
        idx = torch.searchsorted(cdf / cdf[-1].clone(), self.uniform(n)).clamp_(max=distinct - 1)
        return self.perm(distinct)[idx]


def _n(rows, share, least=1):
    return max(least, int(round(rows * share)))


def _i32(t):
    return t.to(torch.int32).cpu().numpy()


def _u32(t):
    return _i32(t).view(np.uint32)


def _i8(t):
    return t.to(torch.int8).cpu().numpy()


def _u64(t):
    return t.cpu().numpy().view(np.uint64)


def _strings(chars, mask):
    """The bytes of chars[i] where mask[i], row after row, as a string column."""
    offsets = torch.zeros(mask.shape[0] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(mask.sum(1), 0, out=offsets[1:])
    return StringColumn(chars[mask].cpu().numpy(), offsets.cpu().numpy().view(np.uint64))


def _words(vocabulary, picks, counts=None):
    """Row i: the words vocabulary[picks[i, :counts[i]]] with spaces between."""
    width = max(len(w) for w in vocabulary) + 1
    table = torch.zeros((len(vocabulary), width), dtype=torch.uint8)
    for i, w in enumerate(vocabulary):
        table[i, :len(w) + 1] = torch.tensor(list(w) + [32], dtype=torch.uint8)
    table = table.cuda()
    n, k = picks.shape
    chars = table[picks]
    mask = chars != 0
    count = torch.full((n,), k, device="cuda") if counts is None else counts
    word = torch.arange(k, device="cuda").expand(n, k)
    mask &= (word < count[:, None])[:, :, None]
    lens = torch.tensor([len(w) for w in vocabulary], device="cuda")
    last = count - 1
    rows = torch.arange(n, device="cuda")
    mask[rows, last, lens[picks[rows, last]]] = False  # no space after the last word
    return _strings(chars.reshape(n, -1), mask.reshape(n, -1))


def _digits(prefix, values, digits, n):
    """Row i: prefix, then values[i] in `digits` digits."""
    out = torch.empty((n, len(prefix) + digits), dtype=torch.uint8, device="cuda")
    out[:, :len(prefix)] = torch.tensor(list(prefix), dtype=torch.uint8, device="cuda")
    for j in range(digits):
        out[:, len(prefix) + j] = (values // 10 ** (digits - 1 - j) % 10 + 48).to(torch.uint8)
    return out


def _join_agg(d, rows):
    nd = _n(rows, 0.25)
    return {"dim": {"d_key": d.perm(nd), "d_segment": d.ints(0, 5, nd), "d_nation": d.ints(0, 25, nd)},
            "fact": {"f_fk": d.ints(1, nd + 1, rows), "f_measure": d.ints(1_000, 10_000_001, rows)}}


def _scan_agg(d, rows):
    return {"lineitem": {
        "l_quantity": d.ints(1, 51, rows), "l_extendedprice": d.ints(90_000, 10_500_001, rows),
        "l_discount": d.ints(0, 11, rows), "l_tax": d.ints(0, 9, rows), "l_shipdate": DAY0 + d.ints(0, DAYS, rows),
        "l_returnflag": d.pick(list(b"ANR"), rows), "l_linestatus": d.pick(list(b"FO"), rows)}}


def _expand(d, rows, two_sided=False):
    nb = _n(rows, 10 / 16.777216)
    distinct = _n(nb, 0.01, 16)
    build = {"r_key": d.zipf(nb, distinct)}
    for i in range(1, 5):
        build["r_f%d" % i] = d.ints(0, 100, nb)
    build["r_measure"] = d.ints(1, 1_000_001, nb)
    probe = {"s_key": d.ints(1, 2 * distinct + 1, rows)}
    if two_sided:
        probe["s_cut"] = d.ints(0, 3, rows)
    return {"r_build": build, "s_probe": probe}


def _star(d, rows):
    n1, n2, n3 = _n(rows, 1 / 40), _n(rows, 1 / 300), _n(rows, 1 / 6000)
    vocabulary = workloads.vocabulary()
    return {"dim1": {"d1_key": d.perm(n1), "d1_attr": d.ints(0, 100, n1)},
            "dim2": {"d2_key": d.perm(n2), "d2_words": d.ints(0, len(vocabulary), 5 * n2).reshape(n2, 5)},
            "dim3": {"d3_key": d.perm(n3), "d3_attr": d.ints(0, 100, n3)},
            "fact": {"f_fk1": d.ints(1, n1 + 1, rows), "f_fk2": d.ints(1, n2 + 1, rows),
                     "f_fk3": d.ints(1, n3 + 1, rows), "f_price": d.ints(90_000, 10_500_001, rows),
                     "f_disc": d.ints(0, 11, rows)}}


def _string_group(d, rows):
    return {"lineitem": {
        "l_extendedprice": d.ints(90_000, 10_500_001, rows), "l_receiptdate": DAY0 + d.ints(0, DAYS, rows),
        "mode": d.ints(0, len(workloads.C9_MODES), rows), "instruct": d.ints(0, len(workloads.C9_INSTRUCT), rows)}}


COMMENT = workloads.C14_WORDS + [b"special"]


def _like_outer(d, rows):
    """Customers, a third of them without orders; 1% of the comments hold
    'special' and, words later, 'requests' (and some of the others 'requests')."""
    nc = _n(rows, 0.1, 16)
    with_orders = torch.arange(1, nc + 1, device="cuda")
    with_orders = with_orders[with_orders % 3 != 0]
    count = d.ints(3, 13, rows)
    words = d.ints(0, len(workloads.C14_WORDS), 12 * rows).reshape(rows, 12)
    planted = d.ints(0, 100, rows) == 0
    words[:, 0] = torch.where(planted, len(COMMENT) - 1, words[:, 0])
    at = torch.arange(rows, device="cuda")
    request = workloads.C14_WORDS.index(b"requests")
    words[at, count - 1] = torch.where(planted, request, words[at, count - 1])
    return {"customer": {"c_custkey": torch.arange(1, nc + 1, device="cuda")},
            "orders": {"o_orderkey": torch.arange(1, rows + 1, device="cuda"),
                       "o_custkey": with_orders[d.ints(0, len(with_orders), rows)],
                       "words": words, "count": count, "planted": planted}}


def _exists(d, rows):
    no, ns = _n(rows, 0.25, 64), _n(rows, 1 / 600, 16)
    with_lines = torch.arange(1, no + 1, device="cuda")
    with_lines = with_lines[with_lines % 7 != 0]
    commit = DAY0 + d.ints(0, DAYS, rows)
    return {"orders": {"o_orderkey": d.perm(no), "o_orderstatus": d.pick(list(b"FOP"), no)},
            "lineitem": {"l_orderkey": with_lines[d.ints(0, len(with_lines), rows)],
                         "l_suppkey": d.ints(1, ns + 1, rows), "l_commitdate": commit,
                         "l_receiptdate": commit + d.ints(-30, 31, rows)}}


def _excess(d, rows):
    ns, npart = _n(rows, 1 / 600, 16), _n(rows, 1 / 30, 16)
    pk = torch.arange(1, npart + 1, device="cuda").repeat_interleave(4)
    i = torch.arange(4, device="cuda").repeat(npart)
    sk = (pk + i * (ns // 4 + (pk - 1) // ns)) % ns + 1
    ps = d.ints(0, 4 * npart, rows)
    return {"supplier": {"s_suppkey": torch.arange(1, ns + 1, device="cuda"), "s_nationkey": d.ints(0, 25, ns),
                         "address": d.ints(0, len(workloads.ALNUM), 40 * ns).reshape(ns, 40),
                         "length": d.ints(10, 41, ns)},
            "part": {"p_partkey": torch.arange(1, npart + 1, device="cuda"),
                     "names": d.ints(0, len(workloads.TPCH_COLORS), 5 * npart).reshape(npart, 5)},
            "partsupp": {"ps_partkey": pk, "ps_suppkey": sk, "ps_availqty": d.ints(1, 10_000, 4 * npart)},
            "lineitem": {"l_partkey": pk[ps], "l_suppkey": sk[ps], "l_quantity": d.ints(1, 51, rows),
                         "l_shipdate": DAY0 + d.ints(0, DAYS, rows)}}


def _substring_anti(d, rows):
    nc = _n(rows, 0.1, 64)
    with_orders = torch.arange(1, nc + 1, device="cuda")
    with_orders = with_orders[with_orders % 3 != 0]
    balance = torch.where(d.ints(0, 20, nc) == 0, 0, d.ints(1, 1_000_000, nc))
    return {"customer": {"c_custkey": d.perm(nc), "code": d.ints(10, 35, nc), "local": d.ints(0, 10 ** 10, nc),
                         "c_acctbal": balance},
            "orders": {"o_custkey": with_orders[d.ints(0, len(with_orders), rows)]}}


DRAWN = {"join_agg": _join_agg, "scan_agg": _scan_agg, "expand": _expand, "star": _star,
         "string_group": _string_group, "like_outer": _like_outer, "exists": _exists, "excess": _excess,
         "substring_anti": _substring_anti}


def _columns(case, seed):
    options = {"two_sided": case["two_sided"]} if case["kind"] == "expand" else {}
    return DRAWN[case["kind"]](Draw(seed), case["rows"], **options)


def _tables(case, t):
    """The host tables of the drawn columns `t`: (name, columns, types)."""
    kind = case["kind"]
    if kind == "join_agg":
        dim, fact = t["dim"], t["fact"]
        return [("dim", {k: _i32(v) for k, v in dim.items()}, {k: I for k in dim}),
                ("fact", {"f_fk": _i32(fact["f_fk"]), "f_measure": _u64(fact["f_measure"])},
                 {"f_fk": I, "f_measure": F})]
    if kind == "scan_agg":
        v = t["lineitem"]
        make = {I: _i32, F: _u64, D: _u32, C: _i8}
        types = {"l_quantity": I, "l_extendedprice": F, "l_discount": I, "l_tax": I, "l_shipdate": D,
                 "l_returnflag": C, "l_linestatus": C}
        return [("lineitem", {k: make[types[k]](v[k]) for k in types}, types)]
    if kind == "expand":
        b, p = t["r_build"], t["s_probe"]
        return [("r_build", {k: _u64(v) if k == "r_measure" else _i32(v) for k, v in b.items()},
                 {k: F if k == "r_measure" else I for k in b}),
                ("s_probe", {k: _i32(v) for k, v in p.items()}, {k: I for k in p})]
    if kind == "star":
        vocabulary = workloads.vocabulary()
        table = torch.tensor([list(w) + [32] for w in vocabulary], dtype=torch.uint8, device="cuda")
        text = table[t["dim2"]["d2_words"]].reshape(-1, 5 * 5)
        fact = t["fact"]
        return [("dim1", {k: _i32(v) for k, v in t["dim1"].items()}, {"d1_key": I, "d1_attr": I}),
                ("dim2", {"d2_key": _i32(t["dim2"]["d2_key"]), "d2_text": StringColumn.fixed(text.cpu().numpy())},
                 {"d2_key": I, "d2_text": S}),
                ("dim3", {k: _i32(v) for k, v in t["dim3"].items()}, {"d3_key": I, "d3_attr": I}),
                ("fact", {k: _u64(v) if k == "f_price" else _i32(v) for k, v in fact.items()},
                 {k: F if k == "f_price" else I for k in fact})]
    if kind == "string_group":
        v = t["lineitem"]
        cols = {"l_extendedprice": _u64(v["l_extendedprice"]), "l_receiptdate": _u32(v["l_receiptdate"]),
                "l_shipmode": _whole_words(workloads.C9_MODES, v["mode"]),
                "l_shipinstruct": _whole_words(workloads.C9_INSTRUCT, v["instruct"])}
        return [("lineitem", cols, {"l_extendedprice": F, "l_receiptdate": D, "l_shipmode": S, "l_shipinstruct": S})]
    if kind == "like_outer":
        o = t["orders"]
        return [("customer", {"c_custkey": _i32(t["customer"]["c_custkey"])}, {"c_custkey": I}),
                ("orders", {"o_orderkey": _i32(o["o_orderkey"]), "o_custkey": _i32(o["o_custkey"]),
                            "o_comment": _words(COMMENT, o["words"], o["count"])},
                 {"o_orderkey": I, "o_custkey": I, "o_comment": S})]
    if kind == "exists":
        o = t["orders"]
        return [("orders", {"o_orderkey": _i32(o["o_orderkey"]), "o_orderstatus": _i8(o["o_orderstatus"])},
                 {"o_orderkey": I, "o_orderstatus": C}),
                ("lineitem", {k: _i32(v) for k, v in t["lineitem"].items()}, {k: I for k in t["lineitem"]})]
    if kind == "excess":
        s, p = t["supplier"], t["part"]
        n = len(s["s_suppkey"])
        address = torch.from_numpy(workloads.ALNUM.copy()).cuda()[s["address"]]
        within = torch.arange(40, device="cuda") < s["length"][:, None]
        name = _digits(b"Supplier#", s["s_suppkey"], 9, n)
        return [("nation", {"n_nationkey": np.arange(25, dtype=np.int32),
                            "n_name": StringColumn.from_list(workloads.C15_NATIONS)}, {"n_nationkey": I, "n_name": S}),
                ("supplier", {"s_suppkey": _i32(s["s_suppkey"]), "s_nationkey": _i32(s["s_nationkey"]),
                              "s_name": _strings(name, torch.ones_like(name, dtype=torch.bool)),
                              "s_address": _strings(address, within)},
                 {"s_suppkey": I, "s_nationkey": I, "s_name": S, "s_address": S}),
                ("part", {"p_partkey": _i32(p["p_partkey"]), "p_name": _words(workloads.TPCH_COLORS, p["names"])},
                 {"p_partkey": I, "p_name": S}),
                ("partsupp", {k: _i32(v) for k, v in t["partsupp"].items()}, {k: I for k in t["partsupp"]}),
                ("lineitem", {k: _i32(v) for k, v in t["lineitem"].items()}, {k: I for k in t["lineitem"]})]
    c = t["customer"]
    n = len(c["c_custkey"])
    phone = torch.full((n, 15), ord("-"), dtype=torch.uint8, device="cuda")  # CC-AAA-BBB-CCCC
    phone[:, 0:2] = _digits(b"", c["code"], 2, n)
    phone[:, 3:6] = _digits(b"", c["local"] // 10 ** 7, 3, n)
    phone[:, 7:10] = _digits(b"", c["local"] // 10 ** 4 % 10 ** 3, 3, n)
    phone[:, 11:15] = _digits(b"", c["local"] % 10 ** 4, 4, n)
    return [("customer", {"c_custkey": _i32(c["c_custkey"]), "c_phone": StringColumn.fixed(phone.cpu().numpy()),
                          "c_acctbal": _i32(c["c_acctbal"])}, {"c_custkey": I, "c_phone": S, "c_acctbal": I}),
            ("orders", {"o_custkey": _i32(t["orders"]["o_custkey"])}, {"o_custkey": I})]


def _whole_words(vocabulary, picks):
    """Row i: vocabulary[picks[i]], which may hold spaces."""
    width = max(len(w) for w in vocabulary)
    table = torch.zeros((len(vocabulary), width), dtype=torch.uint8)
    for i, w in enumerate(vocabulary):
        table[i, :len(w)] = torch.tensor(list(w), dtype=torch.uint8)
    chars = table.cuda()[picks]
    return _strings(chars, chars != 0)


# ------------------------------------------------------------------- plans --

SHAPES = {"join_agg": "c1", "scan_agg": "c0", "string_group": "c9", "like_outer": "c17", "exists": "c12",
          "excess": "c18", "substring_anti": "c16"}
HAVING = 19    # the star join's wanted groups have more rows than that
ORDERS = 256   # more orders than a customer has


def _expand_plan(alg, two_sided):
    if not two_sided:
        return workloads.plan_c2(alg, scal, Type, Reduction)
    join = alg.join(("r_key", "s_key"), alg.scan("r_build"), alg.scan("s_probe"))
    node, cfg = join, {join.opId: {"selectivity": 50.0}}
    for i, (name, t) in enumerate((("r_f1", "90"), ("r_f2", "50"), ("r_f3", "10"), ("r_f4", None)), start=1):
        cut = scal.ConstExpr(t, Type.INT) if t else scal.AttrExpr("s_cut")
        node = alg.selection(scal.SmallerExpr(scal.AttrExpr(name), cut), node)
        cfg[node.opId] = {"selectivity": (90, 50, 10, 1)[i - 1] / 100.0}
    agg = alg.aggregation([], [(Reduction.COUNT, "", "cnt"), (Reduction.SUM, "r_measure", "sum_measure")], node)
    return agg, cfg


def _plan(case, db):
    alg = RelationalAlgebra(db)
    kind, rows = case["kind"], case["rows"]
    if kind == "star":
        groups = max(1024, rows // 60)
        plan, cfg = workloads.plan_c3(alg, scal, Type, Reduction, numgroups=groups)
        if case["having"]:
            plan = alg.selection(scal.LargerExpr(scal.AttrExpr("cnt"), scal.ConstExpr(str(HAVING), Type.INT)), plan)
            cfg[plan.opId] = {"selectivity": 0.001}
    elif kind == "expand":
        plan, cfg = _expand_plan(alg, case["two_sided"])
    elif kind == "like_outer":
        plan, cfg = workloads.plan_c17(alg, scal, Type, Reduction, numgroups=max(1024, rows // 10))
    else:
        plan, cfg = workloads.PLANS[SHAPES[kind]](alg, scal, Type, Reduction)
    return alg.resolveAlgebraPlan(plan, cfg)


class State(object):
    def __init__(self, case):
        self.case = case
        self.engine = Engine(0)
        self.plan = None

    def __del__(self):
        if self.plan is not None:
            self.plan.free()
        self.engine.close()


def _instances(case, seed):
    """The row counts of a batch's instances: log-uniform up to case["rows"]."""
    r = np.random.RandomState(seed % (1 << 32))
    lo = max(256, case["rows"] // 64)
    return np.exp(r.uniform(math.log(lo), math.log(case["rows"]), case["instances"])).astype(int)


def prepare(case, seed):
    state = State(case)
    if case["kind"] == "batch":
        lowerings = []
        for i, rows in enumerate(_instances(case, seed)):
            one = {"kind": "expand", "rows": int(rows), "two_sided": False}
            tables = [Table(n, c, t) for n, c, t in _tables(one, _expand(Draw(seed * 1000 + i), int(rows)))]
            lowering = Lowering(_plan(one, Database(tables)))
            for p in lowering.pipes:  # every instance scans tables of its own
                if p.table:
                    p.table = "%s@%d" % (p.table, i)
            for t in tables:
                state.engine.register_table(Table("%s@%d" % (t.name, i), t.columns, t.types))
            lowerings.append(lowering)
        state.plan = state.engine.prepare_batch(lowerings)
        return state
    db = Database([Table(*t) for t in _tables(case, _columns(case, seed))])
    state.engine.register_database(db)
    state.engine.registered.clear()  # the program keeps no host copy
    state.plan = state.engine.prepare(_plan(case, db))
    return state


def _padded(a, n):
    """`a` with zeros after it: how many rows a query keeps depends on the seed."""
    out = np.zeros(n, dtype=a.dtype)
    out[:len(a)] = a
    return out


def _string_rows(rows, cap):
    """The columns of at most cap rows; strings as their bytes and lengths."""
    out = [np.array([len(rows)])]
    for column in zip(*rows):
        if isinstance(column[0], bytes):
            text = b"".join(column)
            out.append([_padded(np.frombuffer(text, dtype=np.uint8), 48 * cap),
                        _padded(np.array([len(s) for s in column]), cap)])
        else:
            out.append(_padded(np.array(column).astype(np.int64), cap))
    return out


def _int64(column):
    return column.view(np.int64) if column.dtype == np.uint64 else column.astype(np.int64)


def run(state):
    kind = state.case["kind"]
    if kind == "batch":
        results = state.plan.execute()
        return [np.concatenate([_int64(r.columns[j]) for r in results]) for j in range(2)]
    result = state.plan.execute()
    if kind in ("string_group", "excess", "substring_anti"):  # few rows, ordered by their strings
        cap = {"string_group": 28, "excess": max(256, state.case["rows"] // 6_000), "substring_anti": 7}[kind]
        return _string_rows(sorted(result.rows()), cap)
    columns = [_int64(c) for c in result.columns]
    if kind == "exists":  # lines by supplier key
        out = np.zeros(_n(state.case["rows"], 1 / 600, 16) + 1, dtype=np.int64)
        out[columns[0]] = columns[1]
        return out
    if kind == "like_outer":  # customers by their orders
        out = np.zeros(ORDERS, dtype=np.int64)
        out[columns[0]] = columns[1]
        return out
    if kind == "scan_agg":
        order = np.lexsort((columns[1], columns[0]))
    elif kind == "expand":
        return columns
    elif kind == "star" and not state.case["having"]:  # by dimension key
        out = np.zeros((len(columns), _n(state.case["rows"], 1 / 40) + 1), dtype=np.int64)
        for j, c in enumerate(columns):
            out[j, columns[0]] = c
        return out
    else:
        order = np.argsort(columns[0])
    columns = [c[order] for c in columns]
    return [_padded(c, max(256, state.case["rows"] // 10_000)) for c in columns] if kind == "star" else columns


# -------------------------------------------------------------------- sizes --

def work(case):
    """Bytes: every column the query reads, once, at its stored width, and the
    result.  Strings: their bytes and 8-byte offsets (none at a fixed width)."""
    kind, n = case["kind"], case["rows"]
    if kind == "join_agg":
        b = _n(n, 0.25) * 12 + n * 12 + 25 * 16
    elif kind == "scan_agg":
        b = n * 26 + 6 * 66
    elif kind == "expand":
        b = _n(n, 10 / 16.777216) * 28 + n * (8 if case["two_sided"] else 4) + 12
    elif kind == "star":
        groups = 0.5 * _n(n, 1 / 40)
        b = _n(n, 1 / 40) * 8 + _n(n, 1 / 300) * 29 + _n(n, 1 / 6000) * 8 + n * 24
        b += 4_000 if case["having"] else groups * 24
    elif kind == "string_group":
        mode = sum(map(len, workloads.C9_MODES)) / len(workloads.C9_MODES)
        instruct = sum(map(len, workloads.C9_INSTRUCT)) / len(workloads.C9_INSTRUCT)
        b = n * (8 + 4 + 16 + mode + instruct) + 28 * 40
    elif kind == "like_outer":
        word = sum(map(len, COMMENT)) / len(COMMENT) + 1
        b = _n(n, 0.1, 16) * 4 + n * (4 + 4 + 8 + 7.5 * word) + 600
    elif kind == "exists":
        b = _n(n, 0.25, 64) * 5 + n * 16 + _n(n, 1 / 600, 16) * 8
    elif kind == "excess":
        part, supplier = _n(n, 1 / 30, 16), _n(n, 1 / 600, 16)
        colour = sum(map(len, workloads.TPCH_COLORS)) / len(workloads.TPCH_COLORS) + 1
        b = n * 16 + part * (4 + 8 + 5 * colour) + 4 * part * 12 + supplier * (8 + 16 + 18 + 25)
    elif kind == "substring_anti":
        b = _n(n, 0.1, 64) * (4 + 15 + 4) + n * 4 + 7 * 20
    else:  # the mean of log-uniform sizes
        lo = max(256, n // 64)
        mean = (n - lo) / math.log(n / lo) if n > lo else n
        b = case["instances"] * mean * (28 * 10 / 16.777216 + 4)
    return {"bytes": float(b), "flops": 0.0}


def tolerance(case):
    return "exact"


# -------------------------------------------------------------------- exact --

def _group(keys, n, *values):
    """Per key in 0..n-1: the count and the sums of the values."""
    out = [torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(1 + len(values))]
    out[0].index_add_(0, keys, torch.ones_like(keys))
    for o, v in zip(out[1:], values):
        o.index_add_(0, keys, v)
    return out


def _np(*tensors):
    return [t.cpu().numpy() for t in tensors]


def _exact_expand(t):
    b, p = t["r_build"], t["s_probe"]
    keep = (b["r_f1"] < 90) & (b["r_f2"] < 50) & (b["r_f3"] < 10)
    key, measure, f4 = b["r_key"][keep], b["r_measure"][keep], b["r_f4"][keep]
    n = int(max(b["r_key"].max(), p["s_key"].max())) + 1
    cnt = total = 0
    for cut in (0, 1, 2) if "s_cut" in p else (None,):
        probes = p["s_key"] if cut is None else p["s_key"][p["s_cut"] == cut]
        mine = f4 < (1 if cut is None else cut)
        times = torch.bincount(probes, minlength=n)[key[mine]]
        cnt += int(times.sum())
        total += int((times * measure[mine]).sum())
    return cnt, total


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        got = [_exact_expand(_expand(Draw(seed * 1000 + i), int(n))) for i, n in enumerate(_instances(case, seed))]
        return [np.array([g[j] for g in got], dtype=np.int64) for j in range(2)]
    t = _columns(case, seed)
    if kind == "join_agg":
        dim, fact = t["dim"], t["fact"]
        nation = torch.full((len(dim["d_key"]) + 1,), -1, device="cuda", dtype=torch.int64)
        chosen = dim["d_segment"] == 1
        nation[dim["d_key"][chosen]] = dim["d_nation"][chosen]
        g = nation[fact["f_fk"]]
        cnt, total = _group(g[g >= 0], 25, fact["f_measure"][g >= 0])
        at = torch.nonzero(cnt).reshape(-1)
        return _np(at, total[at], cnt[at])
    if kind == "scan_agg":
        v = t["lineitem"]
        v = {k: x[v["l_shipdate"] <= DAY0 + DAYS - 1 - 90].to(torch.int64) for k, x in v.items()}
        disc = v["l_extendedprice"] * (100 - v["l_discount"])
        cnt, qty, price, dp, charge, d = _group(v["l_returnflag"] * 256 + v["l_linestatus"], 1 << 16, v["l_quantity"],
                                                v["l_extendedprice"], disc, disc * (100 + v["l_tax"]), v["l_discount"])
        g = torch.nonzero(cnt).reshape(-1)
        n = cnt[g]
        return _np(g // 256, g % 256, qty[g], price[g], dp[g], charge[g], qty[g] // n, price[g] // n, d[g] // n, n)
    if kind == "expand":
        return [np.array([x], dtype=np.int64) for x in _exact_expand(t)]
    if kind == "star":
        n1, n2, n3 = (len(t[k][k.replace("im", "") + "_key"]) for k in ("dim1", "dim2", "dim3"))
        ok1, ok2, ok3 = (torch.zeros(n + 1, dtype=torch.bool, device="cuda") for n in (n1, n2, n3))
        ok1[t["dim1"]["d1_key"][t["dim1"]["d1_attr"] < 50]] = True
        ok2[t["dim2"]["d2_key"][(t["dim2"]["d2_words"] < 4).any(1)]] = True
        ok3[t["dim3"]["d3_key"]] = True
        f = t["fact"]
        keep = ok1[f["f_fk1"]] & ok2[f["f_fk2"]] & ok3[f["f_fk3"]]
        key, price = f["f_fk1"][keep], f["f_price"][keep]
        cnt, total, disc = _group(key, n1 + 1, price, price * (100 - f["f_disc"][keep]))
        at = torch.arange(n1 + 1, device="cuda") * (cnt > 0)
        if not case["having"]:
            return np.stack(_np(at, total, disc, cnt))
        at = torch.nonzero(cnt > HAVING).reshape(-1)
        return [_padded(c, max(256, case["rows"] // 10_000)) for c in _np(at, total[at], disc[at], cnt[at])]
    if kind == "like_outer":
        nc = len(t["customer"]["c_custkey"])
        per = torch.bincount(t["orders"]["o_custkey"][~t["orders"]["planted"]], minlength=nc + 1)
        return torch.bincount(per[per > 0], minlength=ORDERS).cpu().numpy()
    if kind == "exists":
        return _exact_exists(t["orders"], t["lineitem"])
    if kind == "string_group":
        v = t["lineitem"]
        keep = v["l_receiptdate"] < DAY0 + DAYS // 2
        k = len(workloads.C9_INSTRUCT)
        cnt, total = _group((v["mode"] * k + v["instruct"])[keep], 28, v["l_extendedprice"][keep])
        rows = [(workloads.C9_MODES[i // k], workloads.C9_INSTRUCT[i % k], n, x)
                for i, (n, x) in enumerate(zip(cnt.tolist(), total.tolist())) if n]
        return _string_rows(sorted(rows), 28)
    if kind == "substring_anti":
        c = t["customer"]
        wanted = torch.isin(c["code"], torch.tensor([int(x) for x in workloads.C16_CODES], device="cuda"))
        balance = c["c_acctbal"]
        positive = balance[wanted & (balance > 0)]
        mean = int(positive.sum()) // max(1, len(positive))
        orders = torch.bincount(t["orders"]["o_custkey"], minlength=len(balance) + 1)
        keep = wanted & (balance > mean) & (orders[c["c_custkey"]] == 0)
        cnt, total = _group(c["code"][keep], 100, balance[keep])
        return _string_rows([(b"%02d" % i, n, x) for i, (n, x) in enumerate(zip(cnt.tolist(), total.tolist())) if n], 7)
    return _exact_excess(case, t)


def _exact_exists(orders, lines):
    """Lines per supplier: late, of an order with status F, where another
    supplier has a line of the order and no other supplier a late one."""
    no, ns = len(orders["o_orderkey"]), int(lines["l_suppkey"].max())
    key, supp = lines["l_orderkey"], lines["l_suppkey"]
    late = lines["l_receiptdate"] > lines["l_commitdate"]
    status = torch.zeros(no + 1, dtype=torch.bool, device="cuda")
    status[orders["o_orderkey"]] = orders["o_orderstatus"] == ord("F")

    def ends(keep):
        lo = torch.full((no + 1,), 1 << 40, dtype=torch.int64, device="cuda")
        lo.scatter_reduce_(0, key[keep], supp[keep], "amin")
        hi = torch.full((no + 1,), -1, dtype=torch.int64, device="cuda")
        return lo, hi.scatter_reduce_(0, key[keep], supp[keep], "amax")
    lo, hi = ends(torch.ones_like(late))
    late_lo, late_hi = ends(late)
    keep = late & status[key] & ((lo[key] != supp) | (hi[key] != supp))
    keep &= (late_lo[key] == supp) & (late_hi[key] == supp)
    return torch.bincount(supp[keep], minlength=max(16, _n(len(key), 1 / 600)) + 1).cpu().numpy()


def _exact_excess(case, t):
    s, ps, lines = t["supplier"], t["partsupp"], t["lineitem"]
    ns = len(s["s_suppkey"])
    start = DAY0 + 731
    year = (lines["l_shipdate"] >= start) & (lines["l_shipdate"] < start + 365)
    npart = len(t["part"]["p_partkey"])
    cnt, qty = _group((lines["l_partkey"] * (ns + 1) + lines["l_suppkey"])[year], (npart + 1) * (ns + 1),
                      lines["l_quantity"][year])
    pair = ps["ps_partkey"] * (ns + 1) + ps["ps_suppkey"]
    forest = t["part"]["names"][:, 0] == workloads.TPCH_COLORS.index(b"forest")
    keep = forest[ps["ps_partkey"] - 1] & (cnt[pair] > 0) & (2 * ps["ps_availqty"] > qty[pair])
    has = torch.zeros(ns + 1, dtype=torch.bool, device="cuda")
    has[ps["ps_suppkey"][keep]] = True
    chosen = torch.nonzero(has[1:] & (s["s_nationkey"] == workloads.C15_NATIONS.index(b"CANADA"))).reshape(-1)
    length, address = s["length"][chosen].tolist(), s["address"][chosen].cpu().numpy()
    rows = [(b"Supplier#%09d" % (i + 1), workloads.ALNUM[a[:n]].tobytes())
            for i, n, a in zip(chosen.tolist(), length, address)]
    return _string_rows(rows, max(256, case["rows"] // 6_000))
