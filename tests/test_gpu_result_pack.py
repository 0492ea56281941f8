"""Results at the sizes where their way to the host changes: up to 32 KB a
column (2,048 rows and 32 KB of text for a string column) the run's last kernel
writes them to pinned memory, larger ones are copied after the run; the first
run of a plan launches from the host, later ones replay a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _project(n, length, keep):
    import dogqc_b200.scalar as scal
    from dogqc_b200.database import Database, StringColumn, Table
    from dogqc_b200.engine import Engine
    from dogqc_b200.relational import RelationalAlgebra
    from dogqc_b200.types import Type
    r = np.random.default_rng(n * 100 + length)
    key = np.arange(n, dtype=np.int32)
    val = r.integers(0, 1 << 62, n).astype(np.uint64)
    strings = [bytes(r.integers(97, 123, int(k), dtype=np.uint8)) for k in r.integers(0, length + 1, n)]
    t = Table("t", {"k": key, "v": val, "s": StringColumn.from_list(strings)},
              {"k": Type.INT, "v": Type.FLOAT, "s": Type.STRING})
    db = Database([t])
    alg = RelationalAlgebra(db)
    sel = alg.selection(scal.SmallerExpr(scal.AttrExpr("k"), scal.ConstExpr(str(keep), Type.INT)), alg.scan("t"))
    plan = alg.resolveAlgebraPlan(alg.projection(["k", "v", "s"], sel), {})
    engine = Engine(0)
    engine.register_database(db)
    return engine, engine.prepare(plan), list(zip(key.tolist(), val.tolist(), strings))[:keep]


@pytest.mark.parametrize("n,length,keep", [
    (5000, 10, 0), (5000, 10, 1), (5000, 10, 255), (5000, 10, 257), (5000, 12, 2047), (5000, 12, 2048),
    (5000, 12, 2049), (5000, 10, 4096), (5000, 10, 4097), (9000, 10, 8193), (3000, 1, 100),
    (3000, 40, 1638), (3000, 40, 1700), (200, 3000, 20), (200, 3000, 24), (20, 40000, 3), (9000, 30, 9000)])
def test_projected_rows(n, length, keep):
    engine, plan, expect = _project(n, length, keep)
    for _ in range(3):  # launched from the host, captured, replayed
        got = plan.execute()
        assert got.nrows == len(expect)
        assert sorted(got.rows()) == expect
        for c in got.columns[:2]:
            assert c.flags.writeable
    plan.free()
    engine.close()


def test_results_outlive_their_plan_and_context():
    """Result columns are copies: a later run, the plan's end and the
    context's end leave them alone."""
    engine, plan, expect = _project(50_000, 6, 50_000)
    results = [plan.execute() for _ in range(4)]
    plan.free()
    engine.close()
    for r in results:
        assert sorted(r.rows()) == expect


def test_pinned_memory_of_large_results_is_bounded():
    """Results of a replaying plan lie in pinned blocks up to 64 MB in all, lent
    and idle; what goes past that lies in ordinary memory and is as exact."""
    import ctypes as C
    from cuda.bindings import runtime as cudart
    from dogqc_b200 import _lib as L
    from dogqc_b200.database import Database, Table
    from dogqc_b200.engine import Engine
    from dogqc_b200.relational import RelationalAlgebra
    from dogqc_b200.types import Type
    n = 3_000_000
    cols = {"k": np.arange(n, dtype=np.int32), "v": np.random.default_rng(1).integers(0, 1 << 62, n).astype(np.uint64)}
    db = Database([Table("t", cols, {"k": Type.INT, "v": Type.FLOAT})])
    alg = RelationalAlgebra(db)
    e = Engine(0)
    e.register_database(db)
    p = e.prepare(alg.resolveAlgebraPlan(alg.projection(["k", "v"], alg.scan("t")), {}))
    lib = L.lib()

    def run():
        res = C.c_void_p()
        L.check(lib.dq_plan_execute(p.handle, None, C.byref(res)), e.ctx)
        rows, ncols, view = C.c_int64(), C.c_int32(), (L.dq_result_col * L.MAX_PAY)()
        L.check(lib.dq_result_view(res, C.byref(rows), C.byref(ncols), view))
        assert rows.value == n and ncols.value == 2
        pinned = 0
        got = []
        for j, dt in enumerate((np.int32, np.uint64)):
            err, at = cudart.cudaPointerGetAttributes(view[j].data)
            pinned += view[j].bytes if at.type == cudart.cudaMemoryType.cudaMemoryTypeHost else 0
            got.append(np.frombuffer((C.c_uint8 * view[j].bytes).from_address(view[j].data), dt))
        order = np.argsort(got[0])
        assert (got[0][order] == cols["k"]).all() and (got[1][order] == cols["v"]).all()
        return res, pinned

    try:
        for _ in range(2):
            p.execute()
        for _ in range(2):  # four results held at once: 144 MB
            held = [run() for _ in range(4)]
            assert 0 < sum(b for _, b in held) <= 64 << 20
            for res, _ in held:
                lib.dq_result_free(res)
        for _ in range(3):  # one at a time: all of it pinned
            res, pinned = run()
            assert pinned == n * 12
            lib.dq_result_free(res)
    finally:
        p.free()
        e.close()
