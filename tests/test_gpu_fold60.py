"""The 60-bit-prime kernels at the ends of their ranges: queries and keys whose
residues are all 0, all q - 1, alternating, or one above q / 2, where the
folding butterflies and the key products reach their bounds. Every stage
against the CPU oracle; integer work, bit-exact."""
import functools

import numpy as np
import pytest

from onionpirv2_b200 import PirParams, PirServer
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SETS = {"k1p": ("CONFIG_N2048_K1", O.k1p_params, O.Client, O.Server),
        "c4": ("CONFIG_N4096_K2_MP", O.c4_params, O.C4Client, O.C4Server)}
SHAPE = (43, 5, False)


@functools.lru_cache(maxsize=None)
def setup(name):
    config, params, client, server = SETS[name]
    op = params(*SHAPE)
    cl = client(op, 5)
    gp = PirParams(*SHAPE, config=config)
    srv, ref = PirServer(gp), server(op)
    srv.load_data_seeded(SHAPE[0], 9)
    ref.load_seeded(SHAPE[0], 9)
    return op, cl, srv, ref


def fill(pattern, q):
    k = np.arange(q.shape[-1], dtype=np.uint64)
    return np.ascontiguousarray({
        "zero": np.zeros_like(q), "top": q - np.uint64(1),
        "alternate": np.where(k & np.uint64(1), q - np.uint64(1), np.uint64(0)),
        "half": q // np.uint64(2) + np.uint64(1),
    }[pattern].astype(np.uint64))


@pytest.mark.parametrize("keys", ["client", "top", "alternate"])
@pytest.mark.parametrize("query", ["zero", "top", "alternate", "half"])
@pytest.mark.parametrize("name", ["k1p", "c4"])
def test_extreme_residues_match_oracle(name, query, keys):
    op, cl, srv, ref = setup(name)
    bv, gsw, q = cl.bv_keys(), cl.gsw_key(), cl.query(3)
    mod = np.array(list(op.q[:2]) if name == "c4" else [op.q], dtype=np.uint64)
    mod = mod[:, None] if name == "c4" else mod
    if keys != "client":
        bv, gsw = (fill(keys, np.broadcast_to(mod, x.shape)) for x in (bv, gsw))
    q = fill(query, np.broadcast_to(mod, q.shape))
    srv.set_client_keys(1, bv, gsw)
    ref.set_keys(bv, gsw)
    want = ref.expand(q)
    got = srv.expand_query(1, q)
    assert np.array_equal(got.reshape(want.shape), want)
    want_sel = ref.complete_selectors(want)
    assert np.array_equal(srv.complete_selectors(1, got).reshape(want_sel.shape), want_sel)
    assert np.array_equal(srv.make_query(1, q), ref.make_query(q))


@pytest.mark.parametrize("batch", [2, 5, 10, 19, 38, 75])
def test_k1p_batches_match_lone_queries(batch):
    """Lone queries run every level on clusters of CTAs; growing batches leave
    the 8-, 4- and 2-CTA forms one after the other for one CTA an item."""
    op, cl, srv, ref = setup("k1p")
    bv, gsw = cl.bv_keys(), cl.gsw_key()
    srv.set_client_keys(1, bv, gsw)
    ref.set_keys(bv, gsw)
    qs = [cl.query(i) for i in (0, 21, 42)]
    want = np.stack([ref.make_query(q) for q in qs])
    assert np.array_equal(np.stack([srv.make_query(1, q) for q in qs]), want)
    pick = np.arange(batch) % 3
    got = srv.make_query_batch([1] * batch, np.stack([qs[i] for i in pick]))
    assert np.array_equal(got, want[pick])
