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


@pytest.mark.parametrize("rows,per,entry,shift", [
    (2048, 2, 1216, 0),   # whole 64-row tiles, a last chunk of 192 bytes
    (64, 3, 256, 0), (72, 2, 272, 0), (8, 5, 16, 0),    # one chunk, chunk + 16 bytes, ragged row tile, smallest
    (136, 1, 6144, 0),    # the largest entry
    (36, 2, 1216, 0), (64, 2, 1218, 0),                  # rows or entry without the alignment: byte-wise form
    (64, 2, 1216, 2),     # buffers that are 2-byte aligned only
])
def test_raw_db_forms(pkg, orc, rows, per, entry, shift):
    import numpy as np
    import torch
    rng = np.random.default_rng(rows + entry)
    buckets, cols = rows * per - 1, per * (entry // 2) + 3
    entries = rng.integers(0, 256, (buckets, entry), dtype=np.uint8)
    occupied = (rng.random(buckets) < 0.6).astype(np.uint8)
    want = orc.raw_db(entries, occupied, entry, rows, cols, per)
    d_e = torch.zeros(entries.size + 16, dtype=torch.uint8, device="cuda")
    d_e[shift:shift + entries.size] = torch.from_numpy(entries.reshape(-1)).cuda()
    d_o = torch.from_numpy(occupied).cuda()
    d_raw = torch.full((rows * cols + 8,), 7, dtype=torch.int16, device="cuda")
    pkg.cuckoo_to_raw_db(d_e.data_ptr() + shift, d_o.data_ptr(), buckets, entry, rows, cols, per,
                         d_raw.data_ptr() + shift)
    got = d_raw.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[shift // 2:shift // 2 + want.size], want)
    assert (np.delete(got, np.s_[shift // 2:shift // 2 + want.size]) == 7).all()
