"""Selections above a multimatch join: those that read the build side only run
on the build rows, the others on the pairs.  Every form against the oracle,
and ranges long enough for the deferred expansion with a condition on both
sides (which stays on the pairs)."""
import numpy as np
import pytest

from canonical import canonical_rows
from evaluator import run_plan

WORDS = [b"red", b"green", b"special blue", b"blue special requests", b"black"]


CHAINS = ["b0", "b1", "b2", "b3", "t0", "b0 t1", "t0 b1", "b0 b1 b2 b3", "b0 t0 b2 t1", "p b0"]


def _run(db, plan, **config):
    from dogqc_b200.engine import Engine
    e = Engine(0, **config)
    try:
        e.register_database(db)
        p = e.prepare(plan)
        rows = [canonical_rows(p.execute().rows()) for _ in range(2)]
        p.free()
    finally:
        e.close()
    assert rows[0] == rows[1]
    return rows[0]


def _db(nb, npr, distinct, seed=1):
    from dogqc_b200.database import Database, StringColumn, Table
    from dogqc_b200.types import Type
    r = np.random.default_rng(seed)
    build = {"b_key": (r.zipf(1.5, nb) % distinct + 1).astype(np.int32), "b_x": r.integers(0, 100, nb, dtype=np.int32),
             "b_y": r.integers(-50, 50, nb, dtype=np.int32), "b_m": r.integers(1, 1 << 40, nb).astype(np.uint64),
             "b_s": StringColumn.from_list([WORDS[i] for i in r.integers(0, len(WORDS), nb)])}
    probe = {"p_key": r.integers(1, 2 * distinct, npr, dtype=np.int32), "p_x": r.integers(0, 100, npr, dtype=np.int32)}
    return Database([Table("b", build, {"b_key": Type.INT, "b_x": Type.INT, "b_y": Type.INT, "b_m": Type.FLOAT,
                                        "b_s": Type.STRING}),
                     Table("p", probe, {"p_key": Type.INT, "p_x": Type.INT})])


def _conditions(scal, Type):
    attr, const = scal.AttrExpr, lambda v: scal.ConstExpr(str(v), Type.INT)  # noqa: E731
    build = [lambda: scal.SmallerExpr(attr("b_x"), const(40)),
             lambda: scal.LargerExpr(scal.AddExpr(attr("b_x"), attr("b_y")), const(10)),
             lambda: scal.LikeExpr(attr("b_s"), scal.ConstExpr("%special%", Type.STRING)),
             lambda: scal.EqualsExpr(scal.CaseExpr([(scal.SmallerExpr(attr("b_y"), const(0)), const(1))], const(0)),
                                     const(1))]
    both = [lambda: scal.SmallerExpr(attr("b_x"), attr("p_x")),
            lambda: scal.OrExpr(scal.SmallerExpr(attr("b_x"), const(30)), scal.LargerExpr(attr("p_x"), const(70)))]
    return build, both


def _chain(kind, chain):
    import dogqc_b200.scalar as scal
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    db = _db(3000, 4000, 40)
    alg = RelationalAlgebra(db)
    keys = ("b_key", "p_key")
    node = alg.join(keys, alg.scan("b"), alg.scan("p")) if kind == "join" else \
        alg.outerjoin(keys, None, alg.scan("b"), alg.scan("p"))
    build, both = _conditions(scal, Type)
    for c in chain.split():
        cond = scal.SmallerExpr(scal.AttrExpr("p_x"), scal.ConstExpr("50", Type.INT)) if c == "p" else \
            (build if c[0] == "b" else both)[int(c[1])]()
        node = alg.selection(cond, node)
    # b_x is read above the chain as well, b_y and b_s by the chain alone
    agg = alg.aggregation(["p_x"], [(Reduction.COUNT, "", "n"), (Reduction.SUM, "b_m", "m"),
                                    (Reduction.MAX, "b_x", "x")], node)
    return db, alg.resolveAlgebraPlan(agg, {agg.opId: {"numgroups": 100}})


@pytest.mark.parametrize("kind", ["join", "outerjoin"])
@pytest.mark.parametrize("chain", CHAINS)
def test_lowered_chain_matches_oracle(kind, chain):
    """The lowered plan, evaluated on the host."""
    import cpu_eval
    db, plan = _chain(kind, chain)
    _, rows, _ = cpu_eval.Prepared(db, plan, 2).run()
    assert canonical_rows(rows) == canonical_rows(run_plan(db, plan)[1])


def test_where_selections_run():
    """Build-side selections run in both build passes, the rest after the
    expansion; profiles and lane-refill positions keep the plan's own order."""
    from dogqc_b200 import _lib as L
    from dogqc_b200.lowering import Lowering
    _, plan = _chain("join", "b0 t0 b1")

    def filters(options):
        pipes = Lowering(plan, options).pipes
        return [sum(o["kind"] == L.OP_FILTER for o in p.ops) for p in pipes[:3]]
    assert filters({}) == [2, 2, 1]
    sel = [n for n in _selections(plan)]
    assert filters({"profilers": [sel[0].opId]}) == [0, 0, 3]
    assert filters({"buffers": [sel[0].opId]}) == [1, 1, 2]


def _selections(plan):
    found, todo = [], list(plan)
    while todo:
        n = todo.pop()
        if type(n).__name__ == "Selection":
            found.append(n)
        todo += n.children()
    return found


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["join", "outerjoin"])
@pytest.mark.parametrize("chain", CHAINS)
def test_chain_matches_oracle(kind, chain):
    db, plan = _chain(kind, chain)
    assert _run(db, plan) == canonical_rows(run_plan(db, plan)[1])


@pytest.mark.gpu
@pytest.mark.parametrize("threshold", [8, 64, 1 << 20])
def test_deferred_ranges_with_a_condition_on_both_sides(threshold):
    import dogqc_b200.scalar as scal
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    db = _db(20_000, 3000, 30, seed=2)
    alg = RelationalAlgebra(db)
    node = alg.join(("b_key", "p_key"), alg.scan("b"), alg.scan("p"))
    build, both = _conditions(scal, Type)
    for cond in (both[0](), build[0](), both[1]()):
        node = alg.selection(cond, node)
    agg = alg.aggregation([], [(Reduction.COUNT, "", "n"), (Reduction.SUM, "b_m", "m")], node)
    plan = alg.resolveAlgebraPlan(agg, {})
    assert _run(db, plan, defer_threshold=threshold) == canonical_rows(run_plan(db, plan)[1])
