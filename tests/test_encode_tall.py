"""The encode of tables so tall that a quarter polynomial of columns spans more than 2^32 bytes."""
import pytest

pytestmark = pytest.mark.gpu

N = 2048


@pytest.mark.parametrize("interp,rows", [(2, (1 << 22) + 32)])
def test_encode_of_four_million_rows(pkg, orc, interp, rows):
    """rows of the first, a middle and the last (half) row tile equal the oracle's encode of those
    rows alone; all other rows are zero and stay zero"""
    import numpy as np
    import torch
    cols = interp * N
    raw = torch.zeros((cols, rows), dtype=torch.int16, device="cuda")
    out = torch.full((cols, rows), 7, dtype=torch.int16, device="cuda")
    strips = [(0, 64), (1 << 21, 64), (rows - 96, 96)]
    rng = np.random.default_rng(rows)
    want, nonzero = [], 0
    for r0, n in strips:
        v = rng.integers(0, 65536, (cols, n), dtype=np.uint16)
        raw[:, r0:r0 + n] = torch.from_numpy(v.view(np.int16)).cuda()
        want.append(orc.encode_db(v.reshape(-1), n, cols, interp).reshape(cols, n))
        nonzero += int(np.count_nonzero(want[-1]))
    pkg.encode_db(raw.data_ptr(), out.data_ptr(), rows, cols, interp)
    for (r0, n), w in zip(strips, want):
        assert np.array_equal(out[:, r0:r0 + n].cpu().numpy().view(np.uint16), w)
    assert sum(int(torch.count_nonzero(out[c:c + 64])) for c in range(0, cols, 64)) == nonzero
    del raw, out
    torch.cuda.empty_cache()
