"""A tall tree goes through a scan a level, not row by row: 1024 rows of 64
columns in the largest level took 4.3 ms row by row and 3.0 by scans. The whole
call gives what unpack_tree_query + select_level give, bit for bit."""
import numpy as np
import pytest

from onionpirv2_b200 import PirParams, PirServer
from onionpirv2_b200 import server as S
from onionpirv2_b200 import tree as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,a,scans", [(26, 6, False), (27, 6, True)])
def test_first_dimension_of_tall_trees(L, a, scans):
    scheme = PirParams()
    tree = T.make_tree_pir_params_for_scheme(L, a, scheme)
    rng = np.random.default_rng(L)
    u = lambda *shape: rng.integers(0, scheme.q, shape, dtype=np.uint64)  # noqa: E731
    block = rng.integers(0, tree.t, (1 << 10, tree.n), dtype=np.uint64)

    def level(lv):  # the block, repeated, its rows turned by the repetition
        rows = 1 << max(0, lv - tree.r)
        pts = np.empty((rows, tree.n), dtype=np.uint64)
        for k in range(0, rows, 1 << 10):
            pts[k:k + (1 << 10)] = np.roll(block, k >> 10, axis=1)[:min(1 << 10, rows - k)]
        return pts

    bv, gsw = u(tree.h_q, scheme.l_ks, 2, scheme.N), u(2 * scheme.l_key, 2, scheme.N)
    query = u(2, scheme.N)
    whole = T.Tree(scheme, tree, [level(lv) for lv in range(L + 1)])
    whole.set_client_keys(4, bv, gsw)
    before = S.launch_count()
    out = whole.query(4, query)
    # row by row: one launch for every level's first dimension; a scan a level:
    # at least the transform, the packing, the scan and its epilogue of each
    launches = S.launch_count() - before
    folds = sum(lv - tree.r - a for lv in range(tree.r + a, L + 1))
    assert (launches - folds > 4 * (L + 1)) == scans, launches
    with PirServer(T.tree_query_expansion_params(tree, scheme)) as srv:
        srv.set_client_keys(4, bv, gsw)
        alpha, beta, _ = T.unpack_tree_query(srv, scheme, tree, 4, query)
    for lv in (0, tree.r + a, L - 1, L):
        want = T.TreeLevel(scheme, tree, lv, level(lv)).select_level(alpha, beta)
        assert np.array_equal(out[lv], want), lv
