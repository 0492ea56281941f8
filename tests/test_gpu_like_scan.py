"""LIKE over strings the whole warp searches together: literals at the ends of
strings, across the 16-byte pieces and the 512-byte steps, beside other strings
that continue them, and empty and long strings, at row counts that leave lanes
without a string."""
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


def _strings(n, length, seed):
    r = np.random.default_rng(seed)
    out = []
    for i in range(n):
        s = bytes(r.choice(np.frombuffer(b"abs", np.uint8), int(r.integers(0, length + 1))))
        k = int(r.integers(0, 6))
        lit = (b"", b"abba", b"abba" + b"s" * int(r.integers(0, 4)) + b"sab", b"sab", b"abb", b"abbasab")[k]
        at = int(r.integers(0, len(s) + 1)) if i % 3 else (0, len(s))[i % 2]
        out.append(s[:at] + lit + s[at:])
    return out


@pytest.mark.parametrize("n", [1, 31, 33, 257, 5000])
@pytest.mark.parametrize("length", [0, 6, 40, 700])
@pytest.mark.parametrize("pattern", ["%abba%", "%abba%sab%", "%abb%", "%a%abba%", "%ab%", "%bsbsbsbsbsbsbsbsbs%", "abba%"])
def test_matches_oracle(engine, n, length, pattern):
    import dogqc_b200.scalar as scal
    from dogqc_b200.database import Database, StringColumn, Table
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    strings = _strings(n, length, n * 1000 + length) + [b"pad"]
    key = np.arange(len(strings), dtype=np.int32) % 7
    db = Database([Table("t", {"k": key, "s": StringColumn.from_list(strings)}, {"k": Type.INT, "s": Type.STRING})])
    engine.register_database(db, force=True)
    like = lambda p: scal.LikeExpr(scal.AttrExpr("s"), scal.ConstExpr(p, Type.STRING))  # noqa: E731
    alg = RelationalAlgebra(db)
    sel = alg.selection(scal.OrExpr(like(pattern), scal.NotExpr(like("%sab%"))), alg.scan("t"))
    agg = alg.aggregation(["k"], [(Reduction.COUNT, "", "n")], sel)
    plan = alg.resolveAlgebraPlan(agg, {agg.opId: {"numgroups": 8}})
    p = engine.prepare(plan)
    got = canonical_rows(p.execute().rows())
    p.free()
    assert got == canonical_rows(run_plan(db, plan)[1])
