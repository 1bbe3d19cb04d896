"""The whole-tree call takes every level's rows through one launch when the
first dimension is at most 64 wide (N0 = 2, 16, 64 here: padded, exact and
several 16-column steps) and level by level beyond (N0 = 128); both must give
what unpack_tree_query + select_level give, which run on the tensor-core scan.
Uniform keys, query and plaintexts: the arithmetic does not depend on them."""
import numpy as np
import pytest

from onionpirv2_b200 import PirParams, PirServer
from onionpirv2_b200 import tree as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,a", [(14, 1), (16, 4), (17, 6), (18, 7)])
def test_whole_tree_equals_level_by_level(L, a):
    scheme = PirParams()
    tree = T.make_tree_pir_params_for_scheme(L, a, scheme)
    rng = np.random.default_rng(100 * L + a)
    u = lambda *shape: rng.integers(0, scheme.q, shape, dtype=np.uint64)  # noqa: E731
    pts = [rng.integers(0, tree.t, (1 << max(0, lv - tree.r), tree.n), dtype=np.uint64)
           for lv in range(L + 1)]
    pts[0][:] = tree.t - 1
    bv, gsw = u(tree.h_q, scheme.l_ks, 2, scheme.N), u(2 * scheme.l_key, 2, scheme.N)
    query = u(2, scheme.N)
    whole = T.Tree(scheme, tree, pts)
    whole.set_client_keys(4, bv, gsw)
    out = whole.query(4, query)
    with PirServer(T.tree_query_expansion_params(tree, scheme)) as srv:
        srv.set_client_keys(4, bv, gsw)
        alpha, beta, _ = T.unpack_tree_query(srv, scheme, tree, 4, query)
    for lv in [0, tree.r] + list(range(tree.r + 1, L + 1)):
        want = T.TreeLevel(scheme, tree, lv, pts[lv]).select_level(alpha, beta)
        assert np.array_equal(out[lv], want), lv
