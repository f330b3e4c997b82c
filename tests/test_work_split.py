"""Work splits chosen by size, at the sizes where the choice changes.

Every comparison is bit-exact against the oracle, on the first and last output of the
synthetic server (the oracle generates one output's state alone)."""
import pytest

pytestmark = pytest.mark.gpu

N, RESULT = 2048, 12288


def _plan(pkg, instances, interp=1, db_rows=2048):
    return pkg.Plan(num_items=max(db_rows, 32768), entry_size=1216, item_size_bits=9728, dim0=db_rows,
                    db_rows=db_rows, db_cols=instances * N, instances=instances, interp=interp,
                    c=instances // interp, peak_bytes=0)


def _group(resp, c, query, g):
    off = 4 + query * (4 + c * RESULT) + 4 + g * RESULT
    return resp[off:off + RESULT]


@pytest.mark.parametrize("instances", [1, 13, 14, 27, 28, 55, 56])
def test_single_payload_packing_split(pkg, orc, instances):
    """8, 4 or 2 CTAs per packing task (the count doubles until the grid is 6 CTAs per SM)"""
    plan = _plan(pkg, instances)
    with pkg.KeywordServer.synthetic(plan, seed=300 + instances) as srv:
        q = orc.synth_query(17 + instances, plan.db_rows, 2)
        got = srv.respond_to_serialized_query(q)
        assert len(got) == 4 + 2 * (4 + plan.c * RESULT) + 4
        for g in {0, instances - 1}:
            want = orc.respond(orc.SynthDB.shard_of(plan.db_rows, g, 1, 1, 1, seed=300 + instances), q)
            for query in (0, 1):
                assert _group(got, plan.c, query, g) == _group(want, 1, query, 0)
