"""The offline precomputation and the InspiRING pack against the oracle, beyond the first instance
and with outputs of different alignments."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
SIZES = {"a_hat": N, "bold_t": 3069 * N, "bold_t_bar": 3069 * N, "bold_t_hat": 3 * N}


def _precompute(pkg, db, instances, shifts=None):
    """outputs by name, each `shifts[name]` words past a 32-byte boundary"""
    import torch
    d_db = torch.from_numpy(db.view(np.int16)).cuda()
    bufs = {k: torch.full((instances * n + 8,), 3, dtype=torch.int64, device="cuda") for k, n in SIZES.items()}
    at = {k: (shifts or {}).get(k, 0) for k in SIZES}
    outs = {k: bufs[k][at[k]:at[k] + instances * n] for k, n in SIZES.items()}
    torch.cuda.synchronize()
    pkg.offline_precompute(d_db.data_ptr(), N, instances, *[o.data_ptr() for o in outs.values()])
    for k, b in bufs.items():
        assert (b[:at[k]] == 3).all() and (b[at[k] + instances * SIZES[k]:] == 3).all(), k
    return outs


def _equal(got, want, instance):
    for (name, g), w in zip(got.items(), want):
        n = SIZES[name]
        assert np.array_equal(g[instance * n:(instance + 1) * n].cpu().numpy().view(np.uint64),
                              np.asarray(w).reshape(-1)), (name, instance)


def test_later_instances_of_one_pass_match_the_oracle(pkg, orc):
    """38 instances (four CTAs each) are more than the SMs: the general form of the collapse"""
    instances = 38
    db = np.random.default_rng(38).integers(0, 65535, instances * N * N, dtype=np.uint16)
    got = _precompute(pkg, db, instances)
    for i in (1, instances - 1):
        _equal(got, orc.offline_precompute(db[i * N * N:(i + 1) * N * N], N, 1), i)


@pytest.fixture(scope="module")
def two_instances(orc):
    db = np.random.default_rng(77).integers(0, 65535, 2 * N * N, dtype=np.uint16)
    return db, [orc.offline_precompute(db[i * N * N:(i + 1) * N * N], N, 1) for i in range(2)]


@pytest.mark.parametrize("shifts", [{"bold_t": 1}, {"bold_t": 2}, {"bold_t_bar": 1}, {"bold_t_bar": 2},
                                    {"a_hat": 1}, {"bold_t_hat": 1}, {"bold_t": 1, "bold_t_bar": 2, "bold_t_hat": 3}])
def test_outputs_of_different_alignments_match_the_oracle(pkg, two_instances, shifts):
    db, want = two_instances
    got = _precompute(pkg, db, 2, shifts)
    for i in range(2):
        _equal(got, want[i], i)


def test_later_sets_of_a_pack_match_the_oracle(pkg, orc):
    import torch
    sets, q0, q1 = 38, 268369921, 249561089
    gen = torch.Generator(device="cuda").manual_seed(9)
    lwe = torch.randint(0, q0 * q1, (sets, N + 1, N), dtype=torch.int64, device="cuda", generator=gen)
    y, z = [torch.randint(0, q0, (3, N), dtype=torch.int64, device="cuda", generator=gen)
            | (torch.randint(0, q1, (3, N), dtype=torch.int64, device="cuda", generator=gen) << 32) for _ in range(2)]
    out = torch.zeros((sets, 2, N), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    with pkg.InspiringPacker(sets) as packer:
        packer.pack(sets, lwe.data_ptr(), y.data_ptr(), z.data_ptr(), out.data_ptr())
        packer.sync()
    host = lambda t: t.cpu().numpy().view(np.uint64)  # noqa: E731
    for i in (1, sets - 1):
        assert np.array_equal(host(out[i]), orc.inspiring_pack(host(lwe[i]), host(y), host(z)).reshape(2, N)), i
