"""Work splits chosen by size, at the sizes where the choice changes.

Every comparison is bit-exact: against the oracle, on the first and last output of the synthetic
server (the oracle generates one output's state alone), or, for the alignments of the offline
precomputation and the InspiRING pack, against the aligned call (test_offline_oracle.py compares
those with the oracle)."""
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


@pytest.mark.parametrize("instances", [1, 2, 3, 13, 28, 56])
def test_single_payload_packing_split(pkg, orc, instances):
    """thirteen CTAs per packing task (one output), shares that begin and end inside tasks"""
    plan = _plan(pkg, instances)
    with pkg.KeywordServer.synthetic(plan, seed=300 + instances) as srv:
        q = orc.synth_query(17 + instances, plan.db_rows, 2)
        got = srv.respond_to_serialized_query(q)
        assert len(got) == 4 + 2 * (4 + plan.c * RESULT) + 4
        for g in {0, instances - 1}:
            want = orc.respond(orc.SynthDB.shard_of(plan.db_rows, g, 1, 1, 1, seed=300 + instances), q)
            for query in (0, 1):
                assert _group(got, plan.c, query, g) == _group(want, 1, query, 0)


@pytest.mark.parametrize("instances", [1, 3])
@pytest.mark.parametrize("payloads", [2, 4, 5, 20, 33, 64])
def test_batch_packing_tiles(pkg, orc, instances, payloads):
    """one to sixteen column groups of four clients, fewer units than SMs and more"""
    plan = _plan(pkg, instances)
    seed = 700 + instances
    with pkg.KeywordServer.synthetic(plan, seed=seed) as srv:
        qs = [orc.synth_query(900 + i, plan.db_rows, 2) for i in range(payloads)]
        got = srv.respond_batch(qs)
        sdb = orc.SynthDB(plan.db_rows, instances, 1, instances, seed=seed)
        for i in {0, payloads // 2, payloads - 1}:
            assert got[i] == orc.respond(sdb, qs[i])


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


@pytest.mark.parametrize("groups,queries", [(1, 1), (31, 4), (33, 4), (25, 6), (25, 9)])
def test_fold_form_by_chains(pkg, orc, groups, queries):
    """1 and 124 chains on clusters, 132 on two chains per SM, 150 on clusters, 225 on two per SM"""
    plan = _plan(pkg, 2 * groups, interp=2)
    with pkg.KeywordServer.synthetic(plan, seed=500 + groups) as srv:
        q = orc.synth_query(29 + queries, plan.db_rows, queries)
        got = srv.respond_to_serialized_query(q)
        for g in {0, groups - 1}:
            want = orc.respond(orc.SynthDB.shard_of(plan.db_rows, 2 * g, 2, 2, 1, seed=500 + groups), q)
            for query in range(queries):
                assert _group(got, plan.c, query, g) == _group(want, 1, query, 0)


def test_collapse_with_given_rows_matches_oracle(pkg, orc):
    """the collapse fed with W rows as arrays (the FFI's form) gives the oracle's precomputation"""
    import numpy as np
    from test_compat_offline import CC, HALF, _bind, _d2h, _dev, _free, _packing_tables
    lib, P = _bind(pkg.lib), orc.params()
    db = np.random.default_rng(6).integers(0, 65535, N * N, dtype=np.uint16)
    a_hat, bt, btb, bth = orc.offline_precompute(db, N, 1)
    tables = np.ctypeslib.as_array(P.ntt).reshape(-1).astype(np.uint64).copy()
    mono, idx, idxb, mod_inv = _packing_tables(orc)
    a_ct = np.ascontiguousarray(orc.prep_pack(db, N, 0, orc.hint_query(1)).reshape(N, CC))
    _, vm, wa, wb = orc.offline_keys()
    wa, wb, vm = (np.ascontiguousarray(x, dtype=np.uint64).reshape(-1) for x in (wa, wb, vm))
    auto = np.stack([orc.automorph_table(2 * t + 1) for t in range(N)]).astype(np.uint32)
    gen = np.array([orc.gen_pow(i) for i in range(HALF)], dtype=np.uint32)
    ptrs = d_auto, d_gen, d_act = _dev(auto), _dev(gen), _dev(a_ct)
    try:
        lib.gpu_packing_setup(mono.ctypes.data, idx.ctypes.data, idxb.ctypes.data, mod_inv.ctypes.data, HALF, N, N, 2,
                              P.q[0], P.q[1], P.barrett_cr1[0], P.barrett_cr1[1])
        lib.gpu_collapse_alloc_r(1, HALF, CC)
        lib.gpu_packing_precomp_fast_device_no_d2h(d_act)
        lib.gpu_collapse_automorph_column(lib.gpu_packing_get_s_r_out(), lib.gpu_packing_get_s_r_bar_out(), 0, HALF, CC,
                                          N, 2, d_auto, d_gen, N)
        lib.gpu_collapse_setup(wa.ctypes.data, wb.ctypes.data, vm.ctypes.data, tables.ctypes.data, 1, HALF, 3, CC)
        lib.gpu_collapse_run(1, HALF, 3, 19, P.q[0], P.q[1], P.barrett_cr1[0], P.barrett_cr1[1], P.mod0_inv_mod1,
                             P.mod1_inv_mod0, P.modulus, P.cr0_mod, P.cr1_mod)
        got_a = np.zeros(N, dtype=np.uint64)
        lib.gpu_collapse_download_a_hat(got_a.ctypes.data, 1)
        got = (got_a, _d2h(lib.gpu_collapse_get_bold_t(), 3069 * N), _d2h(lib.gpu_collapse_get_bold_t_bar(), 3069 * N),
               _d2h(lib.gpu_collapse_get_bold_t_hat(), 3 * N))
        lib.gpu_collapse_free_all()
        lib.gpu_packing_teardown()
    finally:
        for p in ptrs:
            _free(p)
    for name, w, g in zip(("a_hat", "bold_t", "bold_t_bar", "bold_t_hat"), (a_hat, bt, btb, bth), got):
        assert np.array_equal(np.asarray(w).reshape(-1), g), name


@pytest.mark.parametrize("kem,counts", [("ml-kem-512", (1, 15, 16, 17)), ("ml-kem-768", (1, 6, 7, 8, 129)),
                                        ("ml-kem-1024", (1, 3, 4, 5))])
@pytest.mark.parametrize("shift", [0, 1])
def test_dataset_tiles(pkg, orc, kem, counts, shift):
    """a CTA's records less one, all, one more; shift 1: records that are not word-aligned"""
    import torch
    gen = pkg.DatasetGenerator(kem, 1000).with_seed(11)
    for n in counts:
        d = torch.full((n * gen.record_size + 16,), 7, dtype=torch.uint8, device="cuda")
        gen.generate_device(d.data_ptr() + shift, first=3, count=n)
        got = d.cpu().numpy()
        rows = got[shift:shift + n * gen.record_size].reshape(n, -1)
        for i in {0, n // 2, n - 1}:
            rid, pk = orc.dataset_record(kem, 11, 3 + i)
            assert rows[i].tobytes() == rid + pk
        assert (got[:shift] == 7).all() and (got[shift + rows.size:] == 7).all()


@pytest.mark.parametrize("count", [1, 2, 149])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_ntt_of_any_word_alignment(pkg, orc, count, shift):
    """buffers at 0, 8 and 16 bytes past a 32-byte boundary, forward and back"""
    import numpy as np
    import torch
    rng = np.random.default_rng(count + shift)
    for limb, q in enumerate((268369921, 249561089)):
        polys = rng.integers(0, q, (count, N), dtype=np.uint64)
        polys[0, :3] = (0, q - 1, 1)
        d = torch.full((count * N + 8,), 5, dtype=torch.int64, device="cuda")
        body = d[shift:shift + count * N]
        body.copy_(torch.from_numpy(polys.reshape(-1).view(np.int64)))
        pkg.ntt_batch(body.data_ptr(), count, limb)
        got = body.cpu().numpy().view(np.uint64).reshape(count, N)
        for i in {0, count - 1}:
            both = np.zeros((2, N), dtype=np.uint64)
            both[limb] = polys[i]
            assert np.array_equal(got[i], orc.ntt_forward(both)[limb])
        pkg.ntt_batch(body.data_ptr(), count, limb, inverse=True)
        assert np.array_equal(body.cpu().numpy().view(np.uint64).reshape(count, N), polys)
        assert (d[:shift] == 5).all() and (d[shift + count * N:] == 5).all()


@pytest.mark.parametrize("interp", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("rows", [32, 64, 96])
def test_encode_row_tiles(pkg, orc, interp, rows):
    """half a 64-row tile, a whole one, one and a half; two fold groups; 65535 (zero) among the values"""
    import numpy as np
    import torch
    cols = 2 * interp * N
    raw = np.random.default_rng(interp + rows).integers(0, 65536, (cols, rows)).astype(np.uint16)
    raw[0] = raw[-1] = 65535
    d_raw = torch.from_numpy(raw.view(np.int16)).cuda()
    d_out = torch.full((cols * rows + 64,), 9, dtype=torch.int16, device="cuda")
    pkg.encode_db(d_raw.data_ptr(), d_out.data_ptr(), rows, cols, interp)
    got = d_out.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[:cols * rows], orc.encode_db(raw.reshape(-1), rows, cols, interp))
    assert (got[cols * rows:] == 9).all()


@pytest.mark.parametrize("sets", [1, 2, 38])
def test_inspiring_pack_of_any_word_alignment(pkg, sets):
    """LWE matrices 8 bytes past a 32-byte boundary pack like aligned ones, alone and beside others;
    38 sets are more chains than SMs"""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(sets)
    q0, q1 = 268369921, 249561089
    one = (N + 1) * N
    lwe = torch.randint(0, q0 * q1, (sets * one,), dtype=torch.int64, device="cuda", generator=gen)
    keys = [torch.randint(0, q0, (3, N), dtype=torch.int64, device="cuda", generator=gen)
            | (torch.randint(0, q1, (3, N), dtype=torch.int64, device="cuda", generator=gen) << 32) for _ in range(2)]
    moved = torch.empty(sets * one + 4, dtype=torch.int64, device="cuda")[1:1 + sets * one]
    moved.copy_(lwe)
    assert lwe.data_ptr() % 32 == 0 and moved.data_ptr() % 32 == 8
    outs = []
    with pkg.InspiringPacker(sets) as packer:
        for d in (lwe, moved):
            out = torch.zeros((sets, 2, N), dtype=torch.int64, device="cuda")
            packer.pack(sets, d.data_ptr(), keys[0].data_ptr(), keys[1].data_ptr(), out.data_ptr())
            outs.append(out.cpu())
        last = torch.zeros((1, 2, N), dtype=torch.int64, device="cuda")
        packer.pack(1, lwe[-one:].data_ptr(), keys[0].data_ptr(), keys[1].data_ptr(), last.data_ptr())
        assert torch.equal(outs[0], outs[1])
        assert torch.equal(last.cpu()[0], outs[0][-1])


@pytest.mark.parametrize("instances", [2, 38])
def test_offline_outputs_of_any_word_alignment(pkg, instances):
    """outputs 8 bytes past a 32-byte boundary, and several instances per pass, equal aligned ones"""
    import torch
    db = torch.randint(0, 65535, (instances * N, N), dtype=torch.int32, device="cuda",
                       generator=torch.Generator(device="cuda").manual_seed(instances)).to(torch.int16)
    sizes = [instances * N, instances * 3069 * N, instances * 3069 * N, instances * 3 * N]
    got = []
    for shift, scratch in ((0, 0), (1, 0), (2, 0), (0, 1)):
        bufs = [torch.full((n + 8,), 3, dtype=torch.int64, device="cuda") for n in sizes]
        outs = [b[shift:shift + n] for b, n in zip(bufs, sizes)]
        pkg.offline_precompute(db.data_ptr(), N, instances, *[o.data_ptr() for o in outs], scratch_bytes=scratch)
        assert all((b[:shift] == 3).all() and (b[shift + n:] == 3).all() for b, n in zip(bufs, sizes))
        got.append(outs)
        del bufs
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
