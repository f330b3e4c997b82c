"""Performance cases of the inspire-rs_b200 framework: what its users have it do, each through
the package's public entry points.

listed() names the fixed cases, draw() makes further ones of the same ranges, prepare() builds
what a program holds before the call (server, client, device buffers), run() is one pass of the
call, work() its unavoidable bytes and arithmetic, and exact() its result in plain 64-bit torch
where that is quick.  Everything is integer arithmetic: outputs are exact.
"""
import importlib.util
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N = 2048
Q = (268369921, 249561089)
QQ = Q[0] * Q[1]
INNER = 3069                 # key-switch rows per packing output
KEY = 32                     # record ID bytes
RESULT = 12288               # response bytes per fold group
VALUE = {"ml-kem-512": 800, "ml-kem-768": 1184, "ml-kem-1024": 1568}


def _package():
    """the package directory is not a Python identifier, so it is imported by path"""
    if "inspire_rs_b200" in sys.modules:
        return sys.modules["inspire_rs_b200"]
    d = os.path.join(_ROOT, "inspire-rs_b200")
    spec = importlib.util.spec_from_file_location("inspire_rs_b200", os.path.join(d, "__init__.py"),
                                                  submodule_search_locations=[d])
    m = importlib.util.module_from_spec(spec)
    sys.modules["inspire_rs_b200"] = m
    spec.loader.exec_module(m)
    return m


def _plan(case):
    return _package().plan_from_shape(case["records"], KEY, VALUE[case["kem"]])


def listed():
    return [
        # one client's lookup (two cuckoo sub-queries) on the smallest usual database, the
        # reference's default plan for 10,000 keys: latency and launches count
        {"name": "respond_10k", "kind": "respond", "records": 10_000, "kem": "ml-kem-768", "queries": 2},
        # the same lookup on a large database: the packing precomputation streams from HBM
        {"name": "respond_500k", "kind": "respond", "records": 500_000, "kem": "ml-kem-768", "queries": 2},
        # a few clients that arrived together at a small database, host bytes in and out
        {"name": "batch_7_30k", "kind": "batch", "records": 30_000, "kem": "ml-kem-512", "payloads": 7, "device": False},
        # the full batch of the serving loop on a large database, payloads resident in HBM
        {"name": "batch_64_500k", "kind": "batch", "records": 500_000, "kem": "ml-kem-768", "payloads": 64,
         "device": True},
        # a client's side of a lookup: query generation and decryption of the response
        {"name": "client_1M", "kind": "client", "records": 1_000_000, "kem": "ml-kem-768", "queries": 2},
        # batched transforms of RNS polynomials, both primes, forward ...
        {"name": "ntt_4096", "kind": "ntt", "count": 4096, "inverse": False},
        # ... and back, an odd number of them
        {"name": "intt_1501", "kind": "ntt", "count": 1501, "inverse": True},
        # Galois automorphisms of a batch of NTT-domain polynomials
        {"name": "galois_256x64", "kind": "galois", "count": 256, "exponents": 64, "limb": 0},
        # setup: bucket table -> raw column layout -> encoded database
        {"name": "encode_250k", "kind": "encode", "records": 250_000, "kem": "ml-kem-768"},
        # setup: encoded database -> packing precomputation
        {"name": "offline_250k", "kind": "offline", "records": 250_000, "kem": "ml-kem-768"},
        # InspiRING packing of 2048 LWE ciphertexts into one RLWE ciphertext
        {"name": "inspiring_1", "kind": "inspiring", "sets": 1},
        # dataset generation: seeded ML-KEM keys with their IDs, in device memory
        {"name": "dataset_20k", "kind": "dataset", "count": 20_000, "kem": "ml-kem-768"},
    ]


def _log_int(rng, lo, hi):
    """a whole number in [lo, hi], spread over its logarithm, mostly not a round one"""
    import math
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["respond", "respond", "batch", "batch", "batch", "client", "ntt", "ntt", "galois", "encode",
                       "offline", "inspiring", "dataset"])
    kem = rng.choice(sorted(VALUE))
    # at most 500,000 ML-KEM-768 keys' worth of packing outputs (ML-KEM-1024 tables are larger)
    most = {"ml-kem-512": 500_000, "ml-kem-768": 500_000, "ml-kem-1024": 250_000}[kem]
    if kind == "respond":
        return {"kind": kind, "records": _log_int(rng, 1_500, most), "kem": kem, "queries": rng.choice([1, 2, 2, 2, 3, 4])}
    if kind == "batch":
        return {"kind": kind, "records": _log_int(rng, 1_500, most), "kem": kem, "payloads": _log_int(rng, 2, 64),
                "device": rng.random() < 0.5}
    if kind == "client":
        return {"kind": kind, "records": _log_int(rng, 1_500, 1_000_000), "kem": "ml-kem-768",
                "queries": rng.choice([1, 2, 2, 3])}
    if kind == "ntt":
        return {"kind": kind, "count": _log_int(rng, 3, 4096), "inverse": rng.random() < 0.5}
    if kind == "galois":
        return {"kind": kind, "count": _log_int(rng, 5, 256), "exponents": _log_int(rng, 1, 64), "limb": rng.choice([0, 1])}
    if kind == "encode":
        return {"kind": kind, "records": _log_int(rng, 1_500, min(most, 250_000)), "kem": kem}
    if kind == "offline":
        return {"kind": kind, "records": _log_int(rng, 1_500, 250_000), "kem": rng.choice(["ml-kem-512", "ml-kem-768"])}
    if kind == "inspiring":
        return {"kind": kind, "sets": _log_int(rng, 1, 24)}
    return {"kind": kind, "count": _log_int(rng, 100, 20_000), "kem": kem}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _residues(shape, q, gen):
    return torch.randint(0, q, shape, dtype=torch.int64, device="cuda", generator=gen)


def _condensed(shape, gen):
    """a pair of residues per word: mod q0 in the low half, mod q1 in the high half"""
    return _residues(shape, Q[0], gen) | (_residues(shape, Q[1], gen) << 32)


def _payloads(n, db_rows, queries, gen):
    """n serialized query payloads on the device [n][bytes]: a count byte, then 56-bit fields of
    two residues each, as a client's uniform masks make them"""
    fields = 2 * 3 * N + queries * (db_rows + 6 * N)
    v = _residues((n, fields), Q[0], gen) | (_residues((n, fields), Q[1], gen) << 28)
    out = torch.empty((n, 1 + 7 * fields), dtype=torch.uint8, device="cuda")
    out[:, 0] = queries
    out[:, 1:] = v.view(torch.uint8).reshape(n, fields, 8)[:, :, :7].reshape(n, 7 * fields)
    return out


def prepare(case, seed):
    p = _package()
    kind, gen = case["kind"], _gen(seed)
    s = {"kind": kind, "case": case}
    if kind in ("respond", "batch"):
        plan = _plan(case)
        n = case.get("payloads", 1)
        s["server"] = p.KeywordServer.synthetic(plan, seed=seed)
        q = _payloads(n, plan.db_rows, case.get("queries", 2), gen)
        if kind == "batch":
            s["server"].prepare_batch(n)
        if case.get("device"):
            s["q"] = q.reshape(-1).contiguous()
            s["out"] = torch.empty((n, s["server"].response_bytes(2)), dtype=torch.uint8, device="cuda")
        else:
            s["q"] = [bytes(r) for r in q.cpu().numpy()]
    elif kind == "client":
        plan = _plan(case)
        s["client"] = p.KeywordClient(plan, bytes(np.random.RandomState(seed % (1 << 32)).bytes(32)))
        rng = np.random.RandomState((seed + 1) % (1 << 32))
        s["buckets"] = [int(b) for b in rng.randint(0, plan.num_items, case["queries"])]
        # a response of the server: framing, per group 2048 28-bit and 2048 20-bit fields
        groups = case["queries"] * plan.c
        lo = rng.randint(0, Q[0], (groups, N // 2, 2)).astype(np.uint64)
        hi = rng.randint(0, 1 << 20, (groups, N // 2, 2)).astype(np.uint64)
        b7 = (lo[..., 0] | (lo[..., 1] << np.uint64(28))).view(np.uint8).reshape(groups, N // 2, 8)[..., :7]
        b5 = (hi[..., 0] | (hi[..., 1] << np.uint64(20))).view(np.uint8).reshape(groups, N // 2, 8)[..., :5]
        body = np.concatenate([b7.reshape(groups, -1), b5.reshape(groups, -1)], axis=1).reshape(case["queries"], -1)
        u32 = lambda x: int(x).to_bytes(4, "little")  # noqa: E731
        s["response"] = u32(case["queries"]) + b"".join(u32(body.shape[1]) + r.tobytes() for r in body) + u32(0)
    elif kind == "ntt":
        s["polys"] = [_residues((case["count"], N), q, gen) for q in Q]
    elif kind == "galois":
        s["in"] = _residues((case["count"], N), Q[case["limb"]], gen)
        s["ks"] = (2 * torch.randint(0, N, (case["exponents"],), device="cuda", generator=gen) + 1).to(torch.int32)
        s["out"] = torch.empty((case["exponents"], case["count"], N), dtype=torch.int64, device="cuda")
    elif kind == "encode":
        plan = s["plan"] = _plan(case)
        s["entries"] = torch.randint(0, 256, (plan.num_items, plan.entry_size), dtype=torch.uint8, device="cuda",
                                     generator=gen)
        # the load of the default table: records over buckets
        s["occupied"] = (torch.rand(plan.num_items, device="cuda", generator=gen)
                         < case["records"] / plan.num_items).to(torch.uint8)
        s["raw"] = torch.empty((plan.db_cols, plan.db_rows), dtype=torch.int16, device="cuda")
        s["out"] = torch.empty_like(s["raw"])
    elif kind == "offline":
        plan = s["plan"] = _plan(case)
        s["db"] = torch.randint(0, 65535, (plan.db_cols, plan.db_rows), dtype=torch.int32, device="cuda",
                                generator=gen).to(torch.int16)
        n = plan.instances
        s["out"] = [torch.empty(sh, dtype=torch.int64, device="cuda")
                    for sh in ((n, N), (n, INNER, N), (n, INNER, N), (n, 3, N))]
    elif kind == "inspiring":
        n = case["sets"]
        s["packer"] = p.InspiringPacker(n)
        s["lwe"] = _residues((n, N + 1, N), QQ, gen)
        s["y"], s["z"] = _condensed((3, N), gen), _condensed((3, N), gen)
        s["out"] = torch.empty((n, 2, N), dtype=torch.int64, device="cuda")
    elif kind == "dataset":
        s["gen"] = p.DatasetGenerator(case["kem"], case["count"]).with_seed(seed)
        s["out"] = torch.empty((case["count"], s["gen"].record_size), dtype=torch.uint8, device="cuda")
    else:
        raise ValueError(kind)
    return s


def run(s):
    p, kind = _package(), s["kind"]
    if kind == "respond":
        return np.frombuffer(s["server"].respond_to_serialized_query(s["q"][0]), dtype=np.uint8)
    if kind == "batch":
        if "out" in s:
            s["server"].respond_batch_device(s["out"].shape[0], s["q"].data_ptr(), s["out"].data_ptr())
            return s["out"]
        return [np.frombuffer(r, dtype=np.uint8) for r in s["server"].respond_batch(s["q"])]
    if kind == "client":
        q = s["client"].query(s["buckets"])
        return [np.frombuffer(q, dtype=np.uint8), s["client"].decrypt(s["response"])]
    if kind == "ntt":
        for limb, d in enumerate(s["polys"]):
            p.ntt_batch(d.data_ptr(), d.shape[0], limb, inverse=s["case"]["inverse"])
        return s["polys"]
    if kind == "galois":
        p.automorph_batch(s["in"].data_ptr(), s["in"].shape[0], s["ks"].data_ptr(), s["ks"].shape[0],
                          s["out"].data_ptr())
        return s["out"]
    if kind == "encode":
        plan = s["plan"]
        p.cuckoo_to_raw_db(s["entries"].data_ptr(), s["occupied"].data_ptr(), plan.num_items, plan.entry_size,
                           plan.db_rows, plan.db_cols, plan.num_items // plan.db_rows, s["raw"].data_ptr())
        p.encode_db(s["raw"].data_ptr(), s["out"].data_ptr(), plan.db_rows, plan.db_cols, plan.interp)
        return s["out"]
    if kind == "offline":
        plan = s["plan"]
        p.offline_precompute(s["db"].data_ptr(), plan.db_rows, plan.instances, *[t.data_ptr() for t in s["out"]])
        return s["out"]
    if kind == "inspiring":
        s["packer"].pack(s["out"].shape[0], s["lwe"].data_ptr(), s["y"].data_ptr(), s["z"].data_ptr(),
                         s["out"].data_ptr())
        return s["out"]
    s["gen"].generate_device(s["out"].data_ptr())
    return s["out"]


# ---------------------------------------------------------------------------
# the bytes and integer operations a pass cannot do without
# ---------------------------------------------------------------------------
_NTT_OPS = 11 * (N // 2) * 2 * 3  # a butterfly is two multiplies and an addition, counted twice as for flops


def work(case):
    kind = case["kind"]
    if kind in ("respond", "batch"):
        plan, b = _plan(case), case.get("payloads", 1)
        nq = b * case.get("queries", 2)
        q = b * (1 + 7 * 6 * N) + nq * 7 * (plan.db_rows + 6 * N)
        r = nq * plan.c * RESULT
        pre = plan.instances * N * 8 * (1 + 2 * INNER + 3)
        ops = 2 * 2 * nq * plan.db_rows * plan.db_cols + 2 * 2 * 2 * b * plan.instances * INNER * N
        ops += nq * plan.instances * 16 * _NTT_OPS
        return {"bytes": plan.db_rows * plan.db_cols * 2 + pre + q + r, "flops": ops}
    if kind == "client":
        plan, n = _plan(case), case["queries"]
        polys = 2 * (6 + 6 * n) + 2 * 2 * n * plan.c
        return {"bytes": 1 + 7 * (6 * N + n * (plan.db_rows + 6 * N)) + n * plan.c * (RESULT + 2 * N),
                "flops": polys * _NTT_OPS}
    if kind == "ntt":
        return {"bytes": 2 * 2 * case["count"] * N * 8, "flops": 2 * case["count"] * _NTT_OPS}
    if kind == "galois":
        return {"bytes": (case["exponents"] + 1) * case["count"] * N * 8, "flops": 0}
    if kind == "encode":
        plan = _plan(case)
        return {"bytes": plan.num_items * (plan.entry_size + 1) + plan.db_rows * plan.db_cols * 2, "flops": 0}
    if kind == "offline":
        plan = _plan(case)
        n, polys = plan.instances, plan.db_rows // N
        ntts = n * 2 * (N * polys + N + 2 * 1023 * 4)
        return {"bytes": plan.db_rows * plan.db_cols * 2 + n * N * 8 * (1 + 2 * INNER + 3), "flops": ntts * _NTT_OPS}
    if kind == "inspiring":
        n = case["sets"]
        return {"bytes": n * (N + 1) * N * 8 + 2 * 3 * N * 8 + n * 2 * N * 8,
                "flops": n * 2 * (2 * N + 2 * 1023 * 4) * _NTT_OPS}
    k = {"ml-kem-512": 2, "ml-kem-768": 3, "ml-kem-1024": 4}[case["kem"]]
    # Keccak-f permutations: 1 + 2k noise streams, 3 SHAKE128 blocks per matrix entry, the ID
    perms = 1 + 2 * k * (2 if k == 2 else 1) + 3 * k * k + (384 * k + 60) // 136 + 1
    return {"bytes": case["count"] * (KEY + VALUE[case["kem"]]), "flops": case["count"] * perms * 24 * 25 * 2 * 3}


# ---------------------------------------------------------------------------
# 64-bit references
# ---------------------------------------------------------------------------
def _brv11(i):
    return int(format(i, "011b")[::-1], 2)


def _root(q):
    """the smallest primitive 2N-th root of unity mod q"""
    for g in range(2, 1000):
        x = pow(g, (q - 1) // (2 * N), q)
        if pow(x, N, q) == q - 1:
            return min(pow(x, k, q) for k in range(1, 2 * N, 2))
    raise ValueError("no root")


def _ntt64(x, q, inverse):
    """negacyclic transform of the rows of x: slot s holds the value at psi^(2 brv(s) + 1)"""
    psi = _root(q)
    if inverse:
        psi_i = pow(psi, q - 2, q)
        w = [pow(psi_i, _brv11(i), q) for i in range(N)]
        t = 1
        while t < N:
            h = N // (2 * t)
            v = x.view(-1, h, 2, t)
            tw = torch.tensor(w[h:2 * h], dtype=torch.int64, device=x.device).view(1, h, 1)
            a, b = v[:, :, 0], v[:, :, 1]
            x = torch.stack([(a + b) % q, (a - b) % q * tw % q], dim=2).view(-1, N)
            t *= 2
        return x * pow(N, q - 2, q) % q
    w = [pow(psi, _brv11(i), q) for i in range(N)]
    m = 1
    while m < N:
        v = x.view(-1, m, 2, N // (2 * m))
        tw = torch.tensor(w[m:2 * m], dtype=torch.int64, device=x.device).view(1, m, 1)
        a, b = v[:, :, 0], v[:, :, 1] * tw % q
        x = torch.stack([(a + b) % q, (a - b) % q], dim=2).view(-1, N)
        m *= 2
    return x


def exact(case, seed):
    kind, gen = case["kind"], _gen(seed)
    if kind == "ntt":
        polys = [_residues((case["count"], N), q, gen) for q in Q]
        return [_ntt64(x, q, case["inverse"]) for x, q in zip(polys, Q)]
    if kind == "galois":
        x = _residues((case["count"], N), Q[case["limb"]], gen)
        ks = 2 * torch.randint(0, N, (case["exponents"],), device="cuda", generator=gen) + 1
        brv = torch.tensor([_brv11(i) for i in range(N)], device="cuda")
        src = brv[(((2 * brv + 1)[None, :] * ks[:, None]) % (2 * N) - 1) // 2]  # [exponents][slot]
        return torch.stack([x[:, r] for r in src])
    return None
