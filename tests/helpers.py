"""Shared test helpers: golden fixtures and plan construction."""
import json
import os

from dogqc_b200 import workloads
from dogqc_b200.relational import RelationalAlgebra

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def golden(case):
    with open(os.path.join(GOLDEN, "ref_%s.json" % case)) as f:
        return json.load(f)


def golden_cases():
    return sorted(f[4:-5] for f in os.listdir(GOLDEN) if f.startswith("ref_") and f.endswith(".json"))


def make_case(spec):
    """Database and resolved plan (this package's front end) for a golden case spec."""
    db = workloads.GENERATORS[spec["workload"]](spec["scale"], **spec.get("gen_kw", {}))
    alg = RelationalAlgebra(db)
    plan, cfg = workloads.build(spec["workload"], alg, **spec.get("plan_kw", {}))
    plan = alg.resolveAlgebraPlan(plan, cfg)
    return db, alg, plan


def reference_rows(rows, spec):
    """Rows as a golden fixture holds them: sorted lists, and the string
    columns (``spec["str_cols"]``) as the reference's result file shows them,
    right-aligned in 10 characters and cut to 10 (oracle/mmdb.py)."""
    from mmdb import render_string
    sc = set(spec.get("str_cols", ()))
    return sorted([render_string(v) if j in sc else int(v) for j, v in enumerate(r)] for r in rows)



def result_checksum(rows, spec):
    """Checksum of result rows as the fixtures hold it: string columns as the
    reference's result file shows them."""
    from canonical import canonical_checksum
    if spec.get("str_cols"):
        return canonical_checksum(reference_rows(rows, spec))
    return canonical_checksum(rows)


def many_domains(dims, keys, groups=11, rows=20_000):
    """A filtered fact table semi-joined with ``dims`` dimensions of ``keys``
    keys each (a key bitmap a dimension), summed by ``groups`` groups."""
    import numpy as np
    import dogqc_b200.scalar as scal
    from dogqc_b200.database import Database, Table
    from dogqc_b200.relational import Reduction
    from dogqc_b200.types import Type
    r = np.random.default_rng(dims)
    fact = {"g": r.integers(0, groups, rows, dtype=np.int32), "v": r.integers(0, 1 << 30, rows).astype(np.uint64),
            "f": r.integers(0, 100, rows, dtype=np.int32)}
    tables = []
    for i in range(dims):
        k = r.permutation(keys)[:keys * 3 // 4].astype(np.int32)
        k[:2] = (0, keys - 1)
        tables.append(Table("d%d" % i, {"k%d" % i: k}, {"k%d" % i: Type.INT}))
        fact["q%d" % i] = r.integers(0, keys, rows, dtype=np.int32)
    tables.append(Table("fact", fact, {c: Type.FLOAT if c == "v" else Type.INT for c in fact}))
    db = Database(tables)
    alg = RelationalAlgebra(db)
    node = alg.selection(scal.SmallerExpr(scal.AttrExpr("f"), scal.ConstExpr("40", Type.INT)), alg.scan("fact"))
    cfg = {node.opId: {"selectivity": 0.4}}
    for i in range(dims):
        node = alg.semijoin(("k%d" % i, "q%d" % i), None, alg.scan("d%d" % i), node)
        cfg[node.opId] = {"multimatch": False, "selectivity": 0.75}
    agg = alg.aggregation(["g"], [(Reduction.SUM, "v", "s")], node)
    cfg[agg.opId] = {"numgroups": groups}
    return db, alg.resolveAlgebraPlan(agg, cfg)
