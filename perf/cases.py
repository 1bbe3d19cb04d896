"""What a user of this framework has it do, as a list of measurable cases.

Every case is one call through the package's public entry points on what a
program keeps between calls: a server handle with its database loaded, its
clients registered and its scratch reserved (as ServingEngine prepares a
database), a tree, or a client handle with its secret. Three kinds:

  query   n queries answered in one batch (PirServer.make_query_batch_device
          on device buffers, make_query_batch on host buffers), over the four
          parameter sets, databases of 2^10 to 2^18 plaintexts (powers of two
          and others), batches from a lone query to 128
  tree    one tree-PIR query, every level selected (Tree.query)
  client  a client's batch work: "decrypt" responses, "pack" queries

Inputs are made from the seed: database coefficients below t, and queries and
keys uniform mod each limb, which is how ciphertexts and key rows are
distributed. All outputs are whole numbers and are the same bit for bit
whenever the inputs are.
"""
from __future__ import annotations

import numpy as np
import torch

from onionpirv2_b200 import PirParams, PirServer
from onionpirv2_b200.client import PirClient
from onionpirv2_b200.tree import Tree, make_tree_pir_params_for_scheme

K1 = "CONFIG_N2048_K1_COMP"
K1P = "CONFIG_N2048_K1"
K2MP = "CONFIG_N2048_K2_MP"
C4 = "CONFIG_N4096_K2_MP"


def _query(name, config, target, height, n, pow2=True, clients=0, host=False):
    return {"name": name, "kind": "query", "config": config, "target": target, "height": height,
            "pow2": pow2, "n": n, "clients": clients or n, "host": host}


def listed():
    return [
        # A lone query to a small database (64 MB of 13-bit coefficients in the
        # client's view): the lowest latency a lookup service can offer.
        _query("k1_2e14_one", K1, 1 << 14, 9, 1),
        # A lone query to the 2^18-plaintext database the benchmark uses: the
        # "plain" form, one client at a time.
        _query("k1_2e18_one", K1, 1 << 18, 10, 1),
        # The headline: a batch of 32 clients' queries on the 2^18 database.
        _query("k1_2e18_batch32", K1, 1 << 18, 10, 32),
        # A saturated server: 128 queries in flight, each of 32 sessions has
        # four of them.
        _query("k1_2e18_batch128", K1, 1 << 18, 10, 128, clients=32),
        # A database whose size is nobody's power of two (512 x 683 rows, the
        # reference's own layout) and an odd batch, through host buffers as a
        # C++ or numpy program without device memory of its own calls it.
        _query("k1_349526_host13", K1, 349526, 10, 13, host=True),
        # The two-RNS-limb set at N = 2048 under a medium load.
        _query("k2mp_2e16_batch8", K2MP, 1 << 16, 10, 8),
        # The reference's default parameter set (one 60-bit prime), loaded.
        _query("k1p_2e18_batch32", K1P, 1 << 18, 10, 32),
        # The wide-plaintext set (N = 4096, two 60-bit limbs), a lone query.
        _query("c4_2e15_one", C4, 1 << 15, 10, 1),
        # The same set on a large database (16 GiB in NTT form) with several
        # clients waiting.
        _query("c4_2e18_batch8", C4, 1 << 18, 11, 8),
        # A Merkle-path lookup: one tree query selects the ancestor of a leaf
        # at all 17 levels.
        {"name": "tree_L16", "kind": "tree", "config": K1, "L": 16, "a": 3},
        # A gateway that decrypts the responses of a thousand lookups, and one
        # that packs an odd number of queries for one session.
        {"name": "client_decrypt_1024", "kind": "client", "op": "decrypt", "config": K1,
         "target": 1 << 18, "height": 10, "n": 1024},
        {"name": "client_pack_777", "kind": "client", "op": "pack", "config": K1,
         "target": 1 << 18, "height": 10, "n": 777},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(float(lo) * (float(hi) / lo) ** rng.random()))


#: (weight, config, largest database, largest batch): the heaviest drawn case
#: costs no more than the heaviest listed one of its set.
_SETS = [(4, K1, 1 << 18, 128), (2, K2MP, 1 << 18, 96), (2, K1P, 1 << 18, 32), (2, C4, 1 << 17, 8)]


def draw(rng):
    kind = rng.choices(["query", "tree", "client"], [8, 1, 2])[0]
    if kind == "tree":
        L = rng.randint(13, 16)
        return {"kind": "tree", "config": K1, "L": L, "a": rng.randint(2, 3) if L > 13 else 2}
    if kind == "client":
        return {"kind": "client", "op": rng.choice(["decrypt", "pack"]), "config": rng.choice([K1, K1, C4]),
                "target": 1 << 18, "height": 10, "n": _log_uniform(rng, 1, 1024)}
    _, config, top, most = rng.choices(_SETS, [s[0] for s in _SETS])[0]
    target = _log_uniform(rng, 1 << 10, top)
    pow2 = rng.random() < 0.7
    if rng.random() < 0.5:
        target = 1 << (target.bit_length() - 1)
    # the height a deployment picks: a first dimension near the square root
    height = 8 if target < 1 << 13 else 9 if target < 1 << 16 else 10
    n = _log_uniform(rng, 1, most)
    return {"kind": "query", "config": config, "target": target, "height": height, "pow2": pow2,
            "n": n, "clients": min(n, 32), "host": rng.random() < 0.25}


_STREAM = None


def _stream():
    """The one CUDA stream this program enqueues its device-buffer calls on."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _limbs(p):
    return p.get_rns_mods()


def _uniform(rng, mods, shape):
    """Polynomials uniform mod each limb: `shape` ends in N, or (K, N)."""
    if len(mods) == 1:
        return rng.integers(0, mods[0], shape, dtype=np.uint64)
    return np.stack([rng.integers(0, m, shape[:-2] + shape[-1:], dtype=np.uint64) for m in mods],
                    axis=-2)


def _uniform_device(gen, mods, shape):
    if len(mods) == 1:
        return torch.randint(0, mods[0], shape, dtype=torch.int64, device="cuda", generator=gen)
    return torch.stack([torch.randint(0, m, shape[:-2] + shape[-1:], dtype=torch.int64,
                                      device="cuda", generator=gen) for m in mods], dim=-2)


def _generators(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return np.random.default_rng(seed), gen


def _prepare_query(case, seed):
    rng, gen = _generators(seed)
    p = PirParams(case["target"], case["height"], case["pow2"], config=case["config"])
    mods, cs, n = _limbs(p), p.ct_shape, case["n"]
    server = PirServer(p)
    server.load_data_seeded(case["target"], seed)
    for c in range(case["clients"]):
        server.set_client_keys(c, _uniform(rng, mods, (p.expansion_height, p.l_ks) + cs),
                               _uniform(rng, mods, (2 * p.l_key,) + cs))
    server.reserve(n)
    state = {"case": case, "server": server, "ids": [i % case["clients"] for i in range(n)]}
    if case["host"]:
        state["queries"] = _uniform(rng, mods, (n,) + cs)
    else:
        state["queries"] = _uniform_device(gen, mods, (n,) + cs)
        state["responses"] = torch.zeros((n, 2, p.N), dtype=torch.int64, device="cuda")
        state["stream"] = _stream()
    return state


def _prepare_tree(case, seed):
    rng, _ = _generators(seed)
    scheme = PirParams(config=case["config"])
    tree = make_tree_pir_params_for_scheme(case["L"], case["a"], scheme)
    levels = []
    for level in range(tree.L + 1):
        rows = 1 << (level - tree.r) if level >= tree.r else 1
        pts = rng.integers(0, tree.t, (rows, tree.n), dtype=np.uint64)
        pts[:, max(1, (1 << level) // rows):] = 0  # a level below r fills a plaintext in part
        levels.append(pts)
    t = Tree(scheme, tree, levels)
    mods, cs = _limbs(scheme), scheme.ct_shape
    t.set_client_keys(1, _uniform(rng, mods, (tree.h_q, scheme.l_ks) + cs),
                      _uniform(rng, mods, (2 * scheme.l_key,) + cs))
    return {"case": case, "tree": t, "query": _uniform(rng, mods, cs)}


def _prepare_client(case, seed):
    rng, gen = _generators(seed)
    p = PirParams(case["target"], case["height"], config=case["config"])
    n, N = case["n"], p.N
    state = {"case": case, "stream": _stream(),
             "client": PirClient(p, rng.integers(-1, 2, N).astype(np.int8))}
    if case["op"] == "decrypt":
        state["responses"] = torch.randint(0, p.small_q, (n, 2, N), dtype=torch.int64,
                                           device="cuda", generator=gen)
        state["plaintexts"] = torch.zeros((n, N), dtype=torch.int64, device="cuda")
        state["noise"] = torch.zeros(n, dtype=torch.int64, device="cuda")
    else:
        state["index"] = rng.integers(0, p.num_pt, n, dtype=np.uint64)
        state["a"] = _uniform_device(gen, _limbs(p), (n,) + p.ct_shape[1:])
        e = torch.randn((n, N), device="cuda", generator=gen) * 3.2
        state["e"] = e.round().to(torch.int64)
        state["queries"] = torch.zeros((n,) + p.ct_shape, dtype=torch.int64, device="cuda")
    return state


def prepare(case, seed):
    return {"query": _prepare_query, "tree": _prepare_tree, "client": _prepare_client}[case["kind"]](case, seed)


def run(state):
    case = state["case"]
    if case["kind"] == "tree":
        return state["tree"].query(1, state["query"])
    if case["kind"] == "query":
        server = state["server"]
        if case["host"]:
            return server.make_query_batch(state["ids"], state["queries"])
        server.make_query_batch_device(state["ids"], state["queries"].data_ptr(),
                                       state["responses"].data_ptr(), state["stream"].cuda_stream)
        return state["responses"]
    client, stream = state["client"], state["stream"].cuda_stream
    if case["op"] == "decrypt":
        client.decrypt_device(case["n"], state["responses"].data_ptr(), state["plaintexts"].data_ptr(),
                              state["noise"].data_ptr(), stream)
        return state["plaintexts"], state["noise"]
    client.generate_queries_device(state["index"], state["a"].data_ptr(), state["e"].data_ptr(),
                                   state["queries"].data_ptr(), stream)
    return state["queries"]


def exact(case, seed):
    """No case has a rounded output: all are whole numbers."""
    return None


def _ntt_ops(N, words):
    """Operations of one NTT: (N / 2) log2 N butterflies of one modular product
    (three multiplications) and two additions, on 32-bit words, a 64-bit one
    counted as `words` = 4 products of 32 bits."""
    return N // 2 * (N.bit_length() - 1) * (3 * words + 2)


def work(case):
    """Bytes: the database's planes (29-bit residues in 4 bytes, 60-bit ones in
    8), keys, inputs and outputs once each. Operations: the key switches, the
    external products and the scan, in multiplications and additions."""
    if case["kind"] == "client":
        p = PirParams(case["target"], case["height"], config=case["config"])
        n, N, K = case["n"], p.N, p.num_limbs
        per = 2 * N + N + 1 if case["op"] == "decrypt" else 3 * K * N + N
        return {"bytes": 8 * n * per, "flops": 2 * n * K * N * N * 2 // 3}
    if case["kind"] == "tree":
        p = PirParams(config=case["config"])
        t = make_tree_pir_params_for_scheme(case["L"], case["a"], p)
        n, first, height = 1, t.N0, t.h_q
        leaves, rows = t.w, t.b + t.r
        points = sum(1 << max(0, lv - t.r) for lv in range(t.L + 1))
        mux, outputs = points, t.L + 1
    else:
        p = PirParams(case["target"], case["height"], case["pow2"], config=case["config"])
        n, first, height = case["n"], p.fst_dim_sz, p.expansion_height
        leaves, rows = p.useful, p.num_dims - 1
        points, mux, outputs = p.num_pt, max(0, p.other_dim_sz - 1), 1
    N = p.N
    wide = case["config"] in (C4, K1P)
    planes = p.num_limbs if wide else 2     # residue planes of one polynomial
    size, words = (8, 4) if wide else (4, 1)
    ct = 2 * planes * N * size
    keys = (height * p.l_ks + 2 * p.l_key) * ct
    switches = sum(-(-leaves // (1 << (height - d))) for d in range(height))
    ntts = switches * (p.l_ks + 2) + rows * p.l_ep * (2 * p.l_key + 2) + mux * (2 * p.l_ep + 2) + 2 * first
    macs = switches * 2 * p.l_ks + rows * p.l_ep * 4 * p.l_key + mux * 4 * p.l_ep
    scan = 2 * points * 2 * planes * N * words
    flops = n * (planes * (ntts * _ntt_ops(N, words) + macs * 2 * N * words) + scan)
    nbytes = points * planes * N * size + min(n, case.get("clients", 1)) * keys
    return {"bytes": nbytes + n * (1 + outputs) * ct, "flops": flops}
