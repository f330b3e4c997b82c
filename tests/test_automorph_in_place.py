"""ipr_automorph_batch with an output block on the input: each polynomial is read before it is
overwritten, whatever the number of polynomials and automorphisms."""
import pytest

pytestmark = pytest.mark.gpu

N = 2048


@pytest.mark.parametrize("count,nk,block", [(1, 1, 0), (1, 64, 0), (3, 5, 0), (3, 5, 2), (3, 5, 4), (147, 2, 1),
                                            (300, 3, 0)])
def test_automorph_batch_over_its_input(pkg, orc, count, nk, block):
    import numpy as np
    import torch
    rng = np.random.default_rng(count + nk)
    polys = rng.integers(0, 249561089, (count, N), dtype=np.uint64)
    ks = (2 * rng.integers(0, N, nk) + 1).astype(np.uint32)
    d_ks = torch.from_numpy(ks.view(np.int32)).cuda()
    out = torch.full((nk, count, N), 5, dtype=torch.int64, device="cuda")
    out[block] = torch.from_numpy(polys.view(np.int64)).cuda()
    torch.cuda.synchronize()
    pkg.automorph_batch(out[block].data_ptr(), count, d_ks.data_ptr(), nk, out.data_ptr())
    got = out.cpu().numpy().view(np.uint64)
    for j, t in enumerate(ks):
        assert np.array_equal(got[j], polys[:, orc.automorph_table(int(t)).astype(np.int64)]), (j, t)
