"""A refused call leaves no error behind for the calls that follow it."""
import numpy as np
import pytest

from canonical import canonical_rows
from evaluator import run_plan

pytestmark = pytest.mark.gpu


def test_calls_after_a_refused_allocation():
    """An aggregation estimated at 2 * 10^9 groups of eight sums asks for more
    memory than the device has; the plan prepared next runs."""
    from dogqc_b200 import _lib as L
    from dogqc_b200.database import Database, Table
    from dogqc_b200.engine import Engine
    from dogqc_b200.relational import Reduction, RelationalAlgebra
    from dogqc_b200.types import Type
    n = np.arange(1000, dtype=np.int32)
    db = Database([Table("t", {"g": n % 9, "v": n}, {"g": Type.INT, "v": Type.INT})])
    e = Engine(0)
    try:
        e.register_database(db)
        for groups, sums in ((2_000_000_000, 8), (9, 1)):
            alg = RelationalAlgebra(db)
            agg = alg.aggregation(["g"], [(Reduction.SUM, "v", "s%d" % i) for i in range(sums)], alg.scan("t"))
            plan = alg.resolveAlgebraPlan(agg, {agg.opId: {"numgroups": groups}})
            if sums == 8:
                with pytest.raises(L.DqError) as err:
                    e.prepare(plan)
                assert err.value.status == L.ERR_OOM
                continue
            p = e.prepare(plan)
            assert canonical_rows(p.execute().rows()) == canonical_rows(run_plan(db, plan)[1])
            p.free()
    finally:
        e.close()
