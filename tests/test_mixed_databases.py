"""Full batches of several databases overlapping on the device: the packing GEMM of one beside the
first-dimension GEMM of another (an earlier form of the packing GEMM, on CTA pairs, did not finish
here).  Every response equals the one computed alone."""
import pytest

pytestmark = pytest.mark.gpu


def test_full_batches_of_three_databases_overlap(pkg, orc):
    import numpy as np
    import torch
    plan = pkg.Plan(num_items=32768, entry_size=1216, item_size_bits=9728, dim0=2048, db_rows=2048,
                    db_cols=32 * 2048, instances=32, interp=2, c=16, peak_bytes=0)
    n, servers = 64, []
    try:
        for k in range(3):
            srv = pkg.KeywordServer.synthetic(plan, seed=70 + k)
            srv.prepare_batch(n)
            q = torch.from_numpy(np.frombuffer(b"".join(orc.synth_query(100 * k + i, 2048, 2) for i in range(n)),
                                               dtype=np.uint8).copy()).cuda()
            out = torch.zeros((n, srv.response_bytes(2)), dtype=torch.uint8, device="cuda")
            servers.append((srv, q, out))
        alone = []
        for srv, q, out in servers:
            srv.respond_batch_device(n, q.data_ptr(), out.data_ptr())
            srv.sync()
            alone.append(out.cpu())
        for _ in range(20):
            for _, _, out in servers:
                out.zero_()
            torch.cuda.synchronize()
            for _ in range(4):
                for srv, q, out in servers:  # nothing waits between the three streams
                    srv.respond_batch_device(n, q.data_ptr(), out.data_ptr())
            for (srv, _, out), want in zip(servers, alone):
                srv.sync()
                assert torch.equal(out.cpu(), want)
    finally:
        for srv, _, _ in servers:
            srv.close()
