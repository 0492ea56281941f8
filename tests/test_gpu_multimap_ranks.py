"""Multimap builds whose scatter places rows by the ranks of the count pass:
payloads of every width class, keys from unique to one hot key, row counts at
the edges of a step, filters before the sink, aggregated and temp-table
sources, and a build side whose rows outgrow the plan's estimate."""
import numpy as np
import pytest

from canonical import canonical_rows
from evaluator import run_plan

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from dogqc_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def _db(n, distinct, hot, seed):
    from dogqc_b200.database import Database, Table
    from dogqc_b200.types import Type
    r = np.random.default_rng(seed)
    key = r.integers(1, distinct + 1, n).astype(np.int32)
    key[r.random(n) < hot] = 1
    build = {"k": key, "c": r.integers(-100, 100, n).astype(np.int8), "i": r.integers(-1000, 1000, n, dtype=np.int32),
             "d": r.integers(0, 1 << 30, n).astype(np.uint32), "m": r.integers(0, 1 << 50, n).astype(np.uint64),
             "m2": r.integers(0, 1 << 50, n).astype(np.uint64)}
    probe = {"p": r.integers(0, distinct + 3, max(n // 4, 3), dtype=np.int32)}
    T = Type
    return Database([Table("b", build, {"k": T.INT, "c": T.CHAR, "i": T.INT, "d": T.DATE, "m": T.FLOAT, "m2": T.FLOAT}),
                     Table("p", probe, {"p": T.INT})])


def _check(engine, db, plan):
    engine.register_database(db, force=True)
    p = engine.prepare(plan)
    want = canonical_rows(run_plan(db, plan)[1])
    for _ in range(3):
        assert canonical_rows(p.execute().rows()) == want
    p.free()


@pytest.mark.parametrize("n,distinct,hot", [(1, 1, 0), (1023, 2000, 0), (1025, 40, 0.5), (4096, 1, 1.0), (30_001, 9000, 0.02),
                                            (30_000, 30_000, 0.9)])
@pytest.mark.parametrize("fields", ["", "c", "c i", "d m", "m m2 c", "c i d m"])
@pytest.mark.parametrize("cut", [None, 500])
def test_payloads(engine, n, distinct, hot, fields, cut):
    import dogqc_b200.scalar as scal
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    db = _db(n, distinct, hot, n + distinct)
    alg = RelationalAlgebra(db)
    build, cfg = alg.scan("b"), {}
    if cut is not None:
        build = alg.selection(scal.SmallerExpr(scal.AttrExpr("i"), scal.ConstExpr(str(cut), Type.INT)), build)
        cfg[build.opId] = {"selectivity": 0.4}
    j = alg.join(("k", "p"), build, alg.scan("p"))
    sums = [(Reduction.SUM, f, "s" + f) for f in fields.split()]
    agg = alg.aggregation([], [(Reduction.COUNT, "", "n")] + sums, j)
    _check(engine, db, alg.resolveAlgebraPlan(agg, cfg))


@pytest.mark.parametrize("groups", [16, 1, 100_000])
def test_build_side_from_an_aggregation(engine, groups):
    """The build side is an aggregation's groups, staged in a temp table whose
    estimate may be far too small."""
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    db = _db(20_000, 6000, 0, 5)
    alg = RelationalAlgebra(db)
    per = alg.aggregation(["k"], [(Reduction.SUM, "m", "t"), (Reduction.COUNT, "", "c1")], alg.scan("b"))
    j = alg.join(("k", "p"), per, alg.scan("p"))
    agg = alg.aggregation([], [(Reduction.COUNT, "", "n"), (Reduction.SUM, "t", "tt")], j)
    _check(engine, db, alg.resolveAlgebraPlan(agg, {per.opId: {"numgroups": groups}}))


@pytest.mark.parametrize("selectivity", [0.9, 0.00001])
def test_staged_build_side_outgrows_its_estimate(engine, selectivity):
    """A costly build side (its LIKE keeps it in one pass) estimated at a few
    rows: the temp table, the payload and the ranks grow, and the run repeats."""
    import dogqc_b200.scalar as scal
    from dogqc_b200 import workloads as W
    from dogqc_b200.relational import RelationalAlgebra
    from dogqc_b200.relational import Reduction
    from dogqc_b200.types import Type
    db = W.gen_tpch(0.01)
    alg = RelationalAlgebra(db)
    plan, cfg = W.plan_c17(alg, scal, Type, Reduction, numgroups=2000)
    cfg = {k: dict(v, selectivity=selectivity) if "selectivity" in v else v for k, v in cfg.items()}
    _check(engine, db, alg.resolveAlgebraPlan(plan, cfg))


def _expanding(key, first=0):
    """400 rows of x meet 500 of y (keys from ``first``; x's are 0 to 9), and
    the pairs are the build side of a join with p, grouped by ``key`` of x."""
    from dogqc_b200.database import Database, StringColumn, Table
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type as T
    r = np.random.default_rng(3)
    text = [b"name %d" % (i % 11) + b"x" * (i % 40) for i in range(400)]
    db = Database([Table("x", {"a": r.integers(0, 10, 400, dtype=np.int32), "s": StringColumn.from_list(text),
                               "t": r.integers(0, 7, 400, dtype=np.int32)}, {"a": T.INT, "s": T.STRING, "t": T.INT}),
                   Table("y", {"b": r.integers(first, first + 10, 500, dtype=np.int32),
                               "c": r.integers(0, 20, 500, dtype=np.int32)}, {"b": T.INT, "c": T.INT}),
                   Table("p", {"d": r.integers(0, 26, 60, dtype=np.int32)}, {"d": T.INT})])
    alg = RelationalAlgebra(db)
    pairs = alg.join(("a", "b"), alg.scan("x"), alg.scan("y"))
    agg = alg.aggregation([key], [(Reduction.COUNT, "", "n")], alg.join(("c", "d"), pairs, alg.scan("p")))
    return db, alg.resolveAlgebraPlan(agg, {agg.opId: {"numgroups": 400}})


@pytest.mark.parametrize("prebuilt", [False, True])
def test_expanding_build_side_outgrows_its_source(engine, prebuilt):
    """A build side that is itself a multimatch join (and, on generated kernels,
    carries a string, so that its rows are not staged) has many more rows than
    the table its pipelines scan: the run ends before a row is placed, the
    payload grows and the run repeats; alone, in a batch and served."""
    import dogqc_b200._lib as L
    from dogqc_b200.engine import Engine
    from dogqc_b200.lowering import Lowering
    from dogqc_b200.serve import Server
    db, plan = _expanding("t" if prebuilt else "s")
    if prebuilt:
        e = Engine(0, flags=L.CFG_NO_JIT)
        try:
            _check(e, db, plan)
        finally:
            e.close()
        return
    _check(engine, db, plan)
    want = canonical_rows(run_plan(db, plan)[1])
    b = engine.prepare_batch([Lowering(plan), Lowering(plan)])
    for _ in range(2):
        assert [canonical_rows(res.rows()) for res in b.execute()] == [want, want]
    b.free()
    srv = Server(engine, slots=2)
    try:
        tickets = [srv.submit(Lowering(plan)) for _ in range(4)]
        assert [canonical_rows(srv.wait(t)[0].rows()) for t in tickets] == [want] * 4
    finally:
        srv.stop()


def test_build_side_outgrows_its_source_in_a_replayed_run(engine):
    """New data makes a replayed run end for want of room; it repeats with room."""
    (few, plan), (many, _) = _expanding("s", first=9), _expanding("s")
    engine.register_database(few, force=True)
    p = engine.prepare(plan)
    for db in (few, many, few):
        engine.update_table(db["y"])
        want = canonical_rows(run_plan(db, plan)[1])
        for _ in range(4):
            assert canonical_rows(p.execute().rows()) == want
    p.free()
