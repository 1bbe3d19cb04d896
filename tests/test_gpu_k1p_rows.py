"""CONFIG_N2048_K1 at row counts of every remainder mod 4, above one group of
four: 6, 10 and 14 rows read a level in 16-byte pieces from bases that are
not aligned to 32 bytes, with two rows left over; odd counts read word by
word. The batches leave the MUX levels' four- and two-CTA clusters, behind a
first level that copies its unpaired rows and one that does not. Stages and
answers against the CPU oracle. Integer work, bit-exact."""
import numpy as np
import pytest

from onionpirv2_b200 import PirParams, PirServer
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("target,height,pow2,rows", [
    (65, 5, True, 5), (81, 5, True, 6), (97, 5, True, 7), (113, 5, True, 8),
    (257, 6, True, 9), (289, 6, True, 10), (321, 6, True, 11), (157, 5, False, 14),
    (181, 5, False, 16)])
def test_row_counts_match_oracle(target, height, pow2, rows):
    op = O.k1p_params(target, height, pow2)
    gp = PirParams(target, height, pow2, config="CONFIG_N2048_K1")
    assert gp.other_dim_sz == rows
    cl = O.Client(op, 3)
    bv, gsw = cl.bv_keys(), cl.gsw_key()
    srv, ref = PirServer(gp), O.Server(op)
    srv.load_data_seeded(target, 4)
    ref.load_seeded(target, 4)
    srv.set_client_keys(1, bv, gsw)
    ref.set_keys(bv, gsw)
    qs = [cl.query(i) for i in (0, target // 2, target - 1)]
    exp = ref.expand(qs[1])
    mid = ref.first_dim(exp[:op.fst_dim_sz])
    assert np.array_equal(srv.evaluate_first_dim(exp).reshape(mid.shape), mid)
    want = np.stack([ref.make_query(q) for q in qs])
    # pairs of a level x batch: 4 CTAs a pair up to 74, 2 up to 148, then one
    for batch in (1, 3, 19, 38, 75):
        pick = np.arange(batch) % 3
        got = srv.make_query_batch([1] * batch, np.stack([qs[i] for i in pick]))
        assert np.array_equal(got, want[pick]), batch
