"""The client's tensor-core product at the edges of its column tiles (16, 32
and 64 columns, the last one ragged) and on values at the ends of its
reductions: decryption against the oracle, packing against the list-form
kernel. Everything is exact, so results are compared for equality."""
import numpy as np
import pytest

from onionpirv2_b200 import PirParams
from onionpirv2_b200.client import PirClient
from oracle import oracle as O

pytestmark = pytest.mark.gpu

C4 = "CONFIG_N4096_K2_MP"


def _pair(config):
    if config == "k1":
        return PirParams(16384, 9), O.Client(O.params(16384, 9), 211), O.params(16384, 9)
    return (PirParams(16384, 9, config=C4), O.C4Client(O.c4_params(16384, 9), 213),
            O.c4_params(16384, 9))


@pytest.mark.parametrize("config,n", [("k1", 32), ("k1", 449), ("k1", 896), ("k1", 1025),
                                      ("c4", 33), ("c4", 225)])
def test_decrypt_tiles(config, n):
    gp, cl, op = _pair(config)
    rng = np.random.default_rng(n)
    resp = rng.integers(0, int(op.small_q), size=(n, 2, op.N), dtype=np.uint64)
    resp[0] = int(op.small_q) - 1           # the largest sums of both signs
    resp[1, 0], resp[1, 1] = 0, int(op.small_q) - 1
    resp[2] = 0
    pt, noise = PirClient(gp, cl.secret()).decrypt_mod_q_batch(resp, with_noise=True)
    for i in list(range(8)) + [31, n - 17, n - 2, n - 1]:
        want, want_noise = cl.decrypt_noise(resp[i])
        assert np.array_equal(pt[i], want)
        assert int(noise[i]) == want_noise


@pytest.mark.parametrize("config,n", [("k1", 32), ("k1", 449), ("k1", 897), ("c4", 33), ("c4", 225)])
def test_pack_tiles(config, n, monkeypatch):
    gp, cl, op = _pair(config)
    rng = np.random.default_rng(n)
    mods = [op.q] if config == "k1" else op.q[:2]
    a = np.stack([rng.integers(0, int(q), (n, op.N), dtype=np.uint64) for q in mods], axis=1)
    for k, q in enumerate(mods):
        a[0, k], a[1, k], a[2, k] = int(q) - 1, 0, int(q) // 2
    # words the reductions take although no client draws them
    a[3] = np.uint64((1 << 64) - 1)
    a = a.reshape((n,) + gp.ct_shape[1:])
    e = np.rint(rng.normal(0.0, 3.2, (n, op.N))).astype(np.int64)
    e[0, :2] = [np.iinfo(np.int64).min, np.iinfo(np.int64).max]
    idx = rng.integers(0, op.num_pt, n)
    got = PirClient(gp, cl.secret()).fast_generate_query_batch(idx, a, e)
    monkeypatch.setenv("OPIR_CLIENT_TC", "0")
    want = PirClient(gp, cl.secret()).fast_generate_query_batch(idx, a, e)
    assert np.array_equal(got, want)
