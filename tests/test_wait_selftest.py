"""Both bounded waits of the kernels (inside a CTA, and across a cluster) run out after their limit."""
import time

import pytest

pytestmark = pytest.mark.gpu


def test_both_waits_run_out_after_their_limit(pkg):
    pkg.selftest_bounded_wait(1)  # the first launch loads the module
    t0 = time.perf_counter()
    assert pkg.selftest_bounded_wait(200_000) == -4
    took = time.perf_counter() - t0
    assert 0.4 <= took < 5.0, took  # two waits of 200 ms, one after the other
