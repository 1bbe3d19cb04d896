"""The scan epilogue reads a level's rows eight at a time from any word
boundary: row counts of every remainder mod 4 with whole and partial groups of
eight, and column counts that shift the boundary from level to level, against
the CPU oracle. Integer work, bit-exact."""
import numpy as np
import pytest

from onionpirv2_b200 import PirParams, PirServer
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# database entries -> rows: 65 -> 9, 74 -> 10, 83 -> 11, 98 -> 13, 119 -> 15
@pytest.mark.parametrize("target,rows", [(65, 9), (74, 10), (83, 11), (98, 13), (119, 15)])
def test_row_counts_match_oracle(target, rows):
    op, gp = O.params(target, 5, True), PirParams(target, 5, True)
    assert gp.other_dim_sz == rows
    cl = O.Client(op, 3)
    bv, gsw = cl.bv_keys(), cl.gsw_key()
    srv, ref = PirServer(gp), O.Server(op)
    srv.load_data_seeded(target, 4)
    ref.load_seeded(target, 4)
    srv.set_client_keys(1, bv, gsw)
    ref.set_keys(bv, gsw)
    qs = [cl.query(i) for i in (0, target // 2, target - 1)]
    for q in qs:
        exp = ref.expand(q)
        want = ref.first_dim(exp[:op.fst_dim_sz])
        got = srv.evaluate_first_dim(srv.expand_query(1, q))
        assert np.array_equal(got.reshape(want.shape), want)
    want = np.stack([ref.make_query(q) for q in qs])
    # 3: less than a wave of epilogue blocks; 40 and 41: more than one
    for batch in (3, 40, 41):
        pick = np.arange(batch) % 3
        got = srv.make_query_batch([1] * batch, np.stack([qs[i] for i in pick]))
        assert np.array_equal(got, want[pick]), batch
