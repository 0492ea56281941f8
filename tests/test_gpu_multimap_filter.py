"""Multimaps probed through the bits of their build side's keys: key types and
domains up to the largest that has them, keys at both ends of the domain,
probes outside it, and tables whose keys leave the domain after preparation."""
import numpy as np
import pytest

from canonical import canonical_rows
from evaluator import run_plan

pytestmark = pytest.mark.gpu


def _db(lo, span, ctype, n=6000, probes=4000, seed=3):
    from dogqc_b200.database import Database, STORAGE_DTYPE, Table
    from dogqc_b200.types import Type
    r = np.random.default_rng(seed + span)
    dt = STORAGE_DTYPE[ctype]
    key = (lo + r.integers(0, span, n)).astype(dt)
    key[0], key[1] = lo, lo + span - 1
    x = r.integers(0, 1000, n, dtype=np.int32)
    x[:2] = 0
    near = np.clip(lo - 3 + r.integers(0, span + 6, probes), np.iinfo(dt).min, np.iinfo(dt).max).astype(dt)
    near[:2] = key[:2]
    return Database([Table("b", {"k": key, "x": x, "m": r.integers(0, 1 << 40, n).astype(np.uint64)},
                           {"k": ctype, "x": Type.INT, "m": Type.FLOAT}),
                     Table("p", {"q": near, "y": r.integers(0, 40, probes, dtype=np.int32)}, {"q": ctype, "y": Type.INT})])


def _plan(db, exists=False):
    import dogqc_b200.scalar as scal
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    alg = RelationalAlgebra(db)
    b = alg.selection(scal.SmallerExpr(scal.AttrExpr("x"), scal.ConstExpr("20", Type.INT)), alg.scan("b"))
    if exists:
        j = alg.semijoin(("k", "q"), scal.SmallerExpr(scal.AttrExpr("x"), scal.AttrExpr("y")), b, alg.scan("p"))
        agg = alg.aggregation(["y"], [(Reduction.COUNT, "", "n")], j)
    else:
        j = alg.join(("k", "q"), b, alg.scan("p"))
        agg = alg.aggregation([], [(Reduction.COUNT, "", "n"), (Reduction.SUM, "m", "s")], j)
    return alg.resolveAlgebraPlan(agg, {b.opId: {"selectivity": 0.02}, agg.opId: {"numgroups": 40}})


@pytest.mark.parametrize("exists", [False, True])
@pytest.mark.parametrize("kind,lo,span", [("INT", 1, 1), ("INT", -500, 1000), ("INT", -(1 << 31), 70), ("INT", (1 << 31) - 64, 64),
                                          ("INT", 5, 1 << 18), ("INT", 5, (1 << 18) + 1), ("DATE", 8035, 2557),
                                          ("DATE", (1 << 32) - 40, 40), ("CHAR", -128, 256)])
def test_domains(kind, lo, span, exists):
    from dogqc_b200.engine import Engine
    from dogqc_b200.types import Type
    db = _db(lo, span, getattr(Type, kind))
    plan = _plan(db, exists)
    e = Engine(0)
    try:
        e.register_database(db)
        p = e.prepare(plan)
        want = canonical_rows(run_plan(db, plan)[1])
        for _ in range(3):
            assert canonical_rows(p.execute().rows()) == want
        p.free()
    finally:
        e.close()


def test_keys_that_leave_the_domain():
    from dogqc_b200.database import Database, Table
    from dogqc_b200.engine import Engine
    from dogqc_b200.types import Type
    db = _db(100, 500, Type.INT)
    e = Engine(0)
    try:
        e.register_database(db)
        p = e.prepare(_plan(db))
        p.execute()
        p.execute()
        t = db.tables["b"]
        cols = dict(t.columns)
        cols["k"] = (cols["k"] * 3 - 700).astype(np.int32)
        moved = Database([Table("b", cols, t.types), db.tables["p"]])
        e.update_table(moved.tables["b"])
        want = canonical_rows(run_plan(moved, _plan(moved))[1])
        for _ in range(3):
            assert canonical_rows(p.execute().rows()) == want
        p.free()
    finally:
        e.close()
