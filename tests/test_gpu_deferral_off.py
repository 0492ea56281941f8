"""Plans whose runs defer no range leave the deferral's launches out after two
of them, and take them up again when the data brings long ranges."""
import numpy as np
import pytest

from canonical import canonical_rows
from evaluator import run_plan

pytestmark = pytest.mark.gpu


def _db(skew, seed):
    from dogqc_b200.database import Database, Table
    from dogqc_b200.types import Type
    r = np.random.default_rng(seed)
    key = r.permutation(6000).astype(np.int32) // 3
    key[:skew] = 7
    probe = r.integers(0, 2500, 3000, dtype=np.int32)
    probe[:3] = 7
    return Database([Table("b", {"k": key, "m": r.integers(0, 1 << 40, 6000).astype(np.uint64),
                                 "x": r.integers(0, 50, 6000, dtype=np.int32)},
                           {"k": Type.INT, "m": Type.FLOAT, "x": Type.INT}),
                     Table("p", {"q": probe, "y": r.integers(0, 50, 3000, dtype=np.int32)},
                           {"q": Type.INT, "y": Type.INT})])


def _plan(db):
    import dogqc_b200.scalar as scal
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    alg = RelationalAlgebra(db)
    j = alg.join(("k", "q"), alg.scan("b"), alg.scan("p"))
    sel = alg.selection(scal.SmallerExpr(scal.AttrExpr("x"), scal.AttrExpr("y")), j)
    agg = alg.aggregation([], [(Reduction.COUNT, "", "n"), (Reduction.SUM, "m", "s")], sel)
    return alg.resolveAlgebraPlan(agg, {})


def test_long_ranges_come_and_go():
    from dogqc_b200.engine import Engine
    dbs = [_db(0, 1), _db(5000, 2)]
    plan = _plan(dbs[0])
    want = [canonical_rows(run_plan(db, plan)[1]) for db in dbs]
    e = Engine(0)
    try:
        e.register_database(dbs[0])
        p = e.prepare(plan)
        launches = []
        for turn in (0, 1, 0, 1):
            for t in dbs[turn].tables.values():
                e.update_table(t)
            for _ in range(5):
                assert canonical_rows(p.execute().rows()) == want[turn]
                launches.append(p.timing()["kernel_launches"])
        assert launches[4] == launches[0] - 4    # long after two runs that deferred nothing
        assert launches[9] == launches[0]
        assert launches[14] == launches[4] and launches[19] == launches[0]
        p.free()
    finally:
        e.close()


def test_a_very_long_range_is_not_expanded_in_place():
    """A range of more than 2^11 rows in a run without the deferral: that run
    ends and is repeated with it."""
    from dogqc_b200.engine import Engine
    dbs = [_db(0, 1), _db(2000, 2), _db(2100, 3)]
    plan = _plan(dbs[0])
    e = Engine(0)
    try:
        e.register_database(dbs[0])
        p = e.prepare(plan)
        full = None
        for turn, db in enumerate((dbs[0], dbs[1], dbs[0], dbs[2], dbs[0])):
            for t in db.tables.values():
                e.update_table(t)
            want = canonical_rows(run_plan(db, plan)[1])
            launches = []
            for _ in range(5):
                assert canonical_rows(p.execute().rows()) == want
                launches.append(p.timing()["kernel_launches"])
            full = full or launches[0]
            # the first run over changed data: in place up to 2^11 rows, else with the deferral
            assert launches[0] == (full - 4 if turn == 1 else full)
            assert launches[4] == (full - 4 if db is dbs[0] else full)
        p.free()
    finally:
        e.close()
