"""ipr_offline_precompute of a DB that lies inside one of the outputs: the DB is read before the
outputs are written."""
import pytest

pytestmark = pytest.mark.gpu

N = 2048


@pytest.mark.parametrize("output", ["bold_t", "bold_t_bar"])
@pytest.mark.parametrize("offset", [0, 3069 * N])  # 64-bit words: in the first instance, in the second
def test_offline_of_a_db_inside_an_output(pkg, orc, output, offset):
    import numpy as np
    import torch
    instances = 2
    db = np.random.default_rng(offset + 1).integers(0, 65535, instances * N * N, dtype=np.uint16)
    want = orc.offline_precompute(db, N, instances)
    outs = {k: torch.full((instances * n,), 3, dtype=torch.int64, device="cuda")
            for k, n in (("a_hat", N), ("bold_t", 3069 * N), ("bold_t_bar", 3069 * N), ("bold_t_hat", 3 * N))}
    inside = outs[output][offset:offset + db.nbytes // 8]
    inside.copy_(torch.from_numpy(db.view(np.int64)))
    torch.cuda.synchronize()
    pkg.offline_precompute(inside.data_ptr(), N, instances, *[o.data_ptr() for o in outs.values()])
    for (name, o), w in zip(outs.items(), want):
        assert np.array_equal(np.asarray(w).reshape(-1), o.cpu().numpy().view(np.uint64)), name
