"""The autotuner times each configuration that differs in its work once."""
import pytest

pytestmark = pytest.mark.gpu


def test_a_tile_is_timed_once(pkg):
    plan = pkg.plan_from_shape(10_000, 32, 1184)
    with pkg.KeywordServer.synthetic(plan, seed=5) as srv:
        res = srv.autotune(32, 2)
    assert [(c["pack_cta_pair"], c["gemv_tile"]) for c in res["candidates"]] == [
        (p, t) for p in (2, 0, 1) for t in (256, 128)]
    for tile in (256, 128):
        times = {(c["ms"], c["ms_small"]) for c in res["candidates"] if c["gemv_tile"] == tile}
        assert len(times) == 1 and min(times) > (0, 0)
    assert res["chosen"]["pack_cta_pair"] == 2  # the option's default: no value of it changes the work
