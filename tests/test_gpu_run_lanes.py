"""Replayed runs spread their pipelines over four streams: plans with more
independent build sides than that, among them ones whose last build shares the
first stream with the pipeline that probes them all."""
import pytest

from canonical import canonical_rows
from evaluator import run_plan
from helpers import many_domains

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from dogqc_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def _check(engine, db, plan):
    engine.register_database(db, force=True)
    p = engine.prepare(plan)
    want = canonical_rows(run_plan(db, plan)[1])
    for _ in range(4):
        assert canonical_rows(p.execute().rows()) == want
    p.free()


@pytest.mark.parametrize("dims", [2, 4, 5, 6, 9])
def test_independent_builds(engine, dims):
    _check(engine, *many_domains(dims, 500))
