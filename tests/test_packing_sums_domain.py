"""gpu_packing_precomp_fast (native/cuda/packing_kernel.cu:134-806) on entries that are not reduced:
the packing sums depend on the entries mod q alone."""
import numpy as np
import pytest

N = 2048
TRIES = 4096


def _largest_growth(orc):
    """2048 values below 4 q0 for which a forward transform that leaves its sums unreduced through
    seven stages (x + w y and x + 2q - w y, w y in [0, 2q)) passes 2^32, and the largest value

    The last element's x after stage s is that of stage s - 1 plus 2q - w y, and the y of
    stage s comes from the 2^s inputs whose bit s (from the top) is set and whose later bits are
    not: each of these sets is drawn until w y is close to 0."""
    q = int(orc.Q0)
    table = np.ctypeslib.as_array(orc.params().ntt).astype(np.uint64)
    w, wp = table[0, 0], table[0, 1]
    rng = np.random.default_rng(41)
    low = np.uint64(0xFFFFFFFF)

    def product(y, k):
        return (y * w[k] - ((y * wp[k]) >> np.uint64(32)) * np.uint64(q)) & low

    poly, chain = np.zeros(N, dtype=np.uint64), 4 * q - 1
    poly[0] = chain
    for s in range(7):
        idx = np.array([sum(((v >> b) & 1) << (10 - b) for b in range(s)) + (1 << (10 - s)) for v in range(1 << s)])
        x = rng.integers(0, 4 * q, (TRIES, 1 << s), dtype=np.uint64)
        y = x
        for b in range(s):  # stages 0 .. s - 1 of these inputs, down to the all-ones element
            k = (1 << (b + 1)) - 1  # twiddle of the block with b ones
            y = y[:, 0::2] + np.uint64(2 * q) - product(y[:, 1::2], k)
        best = int(np.argmin(product(y[:, 0], (1 << (s + 1)) - 1)))
        poly[idx] = x[best]
        chain += 2 * q - int(product(y[best, :1], (1 << (s + 1)) - 1)[0])
    return poly, chain


def test_unreduced_inputs_can_pass_32_bits(orc):
    """inputs below q stay below 15 q < 2^32; inputs below 4 q need not"""
    poly, largest = _largest_growth(orc)
    assert poly.max() < 4 * orc.Q0 and largest >= 1 << 32


@pytest.mark.gpu
def test_packing_sums_of_unreduced_entries(pkg, orc):
    from test_compat_offline import CC, HALF, _bind, _packing_tables
    lib, P = _bind(pkg.lib), orc.params()
    mono, idx, idxb, mod_inv = _packing_tables(orc)
    q = np.concatenate([np.full(N, orc.Q0), np.full(N, orc.Q1)]).astype(np.uint64)
    reduced = np.random.default_rng(13).integers(0, orc.Q1, (N, CC), dtype=np.uint64)
    given = reduced + np.uint64(3) * q
    poly, _ = _largest_growth(orc)
    given[:, 5], reduced[:, 5] = poly, poly % orc.Q0  # the sequence over j of slot 5, limb 0
    sums = []
    for a_ct in (reduced, given):
        a_ct = np.ascontiguousarray(a_ct)
        lib.gpu_packing_setup(mono.ctypes.data, idx.ctypes.data, idxb.ctypes.data, mod_inv.ctypes.data, HALF, N, N, 2,
                              P.q[0], P.q[1], P.barrett_cr1[0], P.barrett_cr1[1])
        r, rb = np.zeros(HALF * CC, dtype=np.uint64), np.zeros(HALF * CC, dtype=np.uint64)
        lib.gpu_packing_precomp_fast(a_ct.ctypes.data, r.ctypes.data, rb.ctypes.data)
        lib.gpu_packing_teardown()
        sums.append((r, rb))
    assert np.array_equal(sums[0][0], sums[1][0]) and np.array_equal(sums[0][1], sums[1][1])
