"""Key bitmaps built from build sides that repeat their keys (each CTA sets bits
of its own first): domains around the word and shared-memory limits, rows below
and above the number from which that is done, semi and anti joins, and a build
side behind an expansion whose long ranges a second kernel takes."""
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


@pytest.mark.parametrize("anti", [False, True])
@pytest.mark.parametrize("keys,rows", [(1, 4), (31, 5000), (32, 127), (33, 40_000), (3000, 11_999), (3000, 12_000),
                                       (1 << 18, 1 << 20), ((1 << 18) + 1, (1 << 20) + 4)])
def test_semi_and_anti_joins(engine, anti, keys, rows):
    import dogqc_b200.scalar as scal
    from dogqc_b200.database import Database, Table
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    r = np.random.default_rng(keys + rows)
    k = (r.integers(0, keys, rows) - 7).astype(np.int32)
    k[:2] = (-7, keys - 8)
    f = r.integers(0, 10, rows, dtype=np.int32)
    q = (r.integers(0, keys + 20, 20_000) - 17).astype(np.int32)
    db = Database([Table("b", {"k": k, "f": f}, {"k": Type.INT, "f": Type.INT}),
                   Table("p", {"q": q, "g": np.arange(len(q), dtype=np.int32) % 9}, {"q": Type.INT, "g": Type.INT})])
    engine.register_database(db, force=True)
    alg = RelationalAlgebra(db)
    b = alg.selection(scal.SmallerExpr(scal.AttrExpr("f"), scal.ConstExpr("9", Type.INT)), alg.scan("b"))
    j = (alg.antijoin if anti else alg.semijoin)(("k", "q"), None, b, alg.scan("p"))
    agg = alg.aggregation(["g"], [(Reduction.COUNT, "", "n")], j)
    plan = alg.resolveAlgebraPlan(agg, {agg.opId: {"numgroups": 9}})
    p = engine.prepare(plan)
    want = canonical_rows(run_plan(db, plan)[1])
    for _ in range(2):
        assert canonical_rows(p.execute().rows()) == want
    p.free()


@pytest.mark.parametrize("anti", [False, True])
def test_keys_behind_a_deferred_expansion(engine, anti):
    """The build side is a multimatch join; the rows that meet its one long
    range hold keys no other row has."""
    from dogqc_b200.database import Database, Table
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    r = np.random.default_rng(9)
    bk = r.integers(0, 2000, 6000, dtype=np.int32)
    bk[:3000] = 7
    tq = r.integers(8, 2500, 4000, dtype=np.int32)
    tk = r.integers(0, 250, 4000, dtype=np.int32)
    tq[100:150], tk[100:150] = 7, 250 + np.arange(50) % 25
    p = r.integers(0, 300, 5000, dtype=np.int32)
    T = Type
    db = Database([Table("b", {"bk": bk}, {"bk": T.INT}), Table("t", {"tq": tq, "tk": tk}, {"tq": T.INT, "tk": T.INT}),
                   Table("p", {"q": p, "g": np.arange(len(p), dtype=np.int32) % 9}, {"q": T.INT, "g": T.INT})])
    engine.register_database(db, force=True)
    alg = RelationalAlgebra(db)
    pairs = alg.join(("bk", "tq"), alg.scan("b"), alg.scan("t"))
    j = (alg.antijoin if anti else alg.semijoin)(("tk", "q"), None, pairs, alg.scan("p"))
    agg = alg.aggregation(["g"], [(Reduction.COUNT, "", "n")], j)
    plan = alg.resolveAlgebraPlan(agg, {agg.opId: {"numgroups": 9}})
    pl = engine.prepare(plan)
    want = canonical_rows(run_plan(db, plan)[1])
    for _ in range(2):
        assert canonical_rows(pl.execute().rows()) == want
    pl.free()
