"""The bytes bench.py counts for a packing launch are those the kernels stream."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("instances,batch,measured", [
    (8, 64, 813.08e6), (8, 1, 806.03e6),  # dram__bytes_read.sum of one launch (profiles/)
    (352, 64, None), (352, 1, None),      # per launch of the 1M workload: read + written bytes
])
def test_packing_bytes_agree_with_the_measured_traffic(instances, batch, measured):
    """the traffic is the stream once (a few per cent more: the client operand, the outputs)"""
    bench = _bench()
    got = bench.pack_stream_bytes(instances, batch)
    traffic = measured or bench.read_traffic("k_pack_mma" if batch > 1 else "k_pack")
    assert got <= traffic <= 1.03 * got


def test_packing_bytes_follow_the_outputs():
    """every output has rows of its own: no padding to tiles of outputs"""
    bench = _bench()
    for batch in (1, 2, 64):
        one = bench.pack_stream_bytes(1, batch)
        assert [bench.pack_stream_bytes(n, batch) for n in (7, 8, 32, 33)] == [n * one for n in (7, 8, 32, 33)]
