"""A device-side wait that ran out in an InspiRING pack reaches the caller, once, through the next
sync or pack, and the context stays usable.  The error word is set by the test: no wait runs out."""
import pytest

pytestmark = pytest.mark.gpu

N = 2048


def test_inspiring_pack_failure_is_reported_once(pkg):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(3)
    q0, q1 = 268369921, 249561089
    lwe = torch.randint(0, q0 * q1, (1, N + 1, N), dtype=torch.int64, device="cuda", generator=gen)
    keys = [torch.randint(0, q0, (3, N), dtype=torch.int64, device="cuda", generator=gen)
            | (torch.randint(0, q1, (3, N), dtype=torch.int64, device="cuda", generator=gen) << 32) for _ in range(2)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with pkg.InspiringPacker(1) as packer:
        def pack():
            out = torch.zeros((1, 2, N), dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            packer.pack(1, lwe.data_ptr(), keys[0].data_ptr(), keys[1].data_ptr(), out.data_ptr(),
                        stream.cuda_stream)
            return out

        want = pack()
        packer.sync(stream.cuda_stream)  # nothing ran out
        for report in (lambda: packer.sync(stream.cuda_stream), pack):
            pack()
            packer.debug_error(33)
            with pytest.raises(pkg.IprError) as e:
                report()
            assert e.value.status == -4 and "33" in str(pkg.lib.ipr_last_error())
            packer.sync(stream.cuda_stream)  # reported once
            again = pack()
            packer.sync(stream.cuda_stream)
            assert torch.equal(again, want)
