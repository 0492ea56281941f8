"""Grouped sums at the group counts where the CTA's accumulators change form:
per thread while the plan expects few groups, replicated in shared memory
beyond, global for many; groups past the expected number, the key whose packed
bits are all ones, and rows that do not fill a step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from dogqc_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("rows", [1, 1023, 40_961])
@pytest.mark.parametrize("hint,groups", [(1, 1), (6, 6), (6, 9), (6, 200), (16, 16), (17, 17), (16, 40), (3, 3000)])
def test_groups(engine, rows, hint, groups):
    import dogqc_b200.scalar as scal
    from dogqc_b200.database import Database, Table
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    r = np.random.default_rng(rows * 7919 + hint * 31 + groups)
    a = (r.integers(0, groups, rows) - 1).astype(np.int32)        # -1: all ones
    b = np.where(a == -1, -1, a % 3).astype(np.int32)
    v = r.integers(0, 1 << 62, rows).astype(np.uint64)
    w = r.integers(0, 1 << 31, rows).astype(np.int32)
    db = Database([Table("t", {"a": a, "b": b, "v": v, "w": w}, {"a": Type.INT, "b": Type.INT, "v": Type.FLOAT,
                                                                "w": Type.INT})])
    engine.register_database(db, force=True)
    alg = RelationalAlgebra(db)
    sel = alg.selection(scal.LargerEqualExpr(scal.AttrExpr("w"), scal.ConstExpr("1000", Type.INT)), alg.scan("t"))
    agg = alg.aggregation(["a", "b"], [(Reduction.SUM, "v", "s"), (Reduction.COUNT, "", "n"), (Reduction.MIN, "v", "lo"),
                                       (Reduction.MAX, "w", "hi"), (Reduction.AVG, "w", "m")], sel)
    plan = engine.prepare(alg.resolveAlgebraPlan(agg, {agg.opId: {"numgroups": hint}}))
    keep = w >= 1000
    want = {}
    for x, y, p, q in zip(a[keep].tolist(), b[keep].tolist(), v[keep].tolist(), w[keep].tolist()):
        g = want.setdefault((x, y), [0, 0, 1 << 64, 0, 0])
        g[0] = (g[0] + p) % (1 << 64)
        g[1] += 1
        g[2] = min(g[2], p)
        g[3] = max(g[3], q)
        g[4] += q
    expect = sorted((x, y, s, n, lo, hi, t // n) for (x, y), (s, n, lo, hi, t) in want.items())
    for _ in range(3):
        assert sorted(plan.execute().rows()) == expect
    plan.free()
