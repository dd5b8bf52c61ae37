"""Pair sums share one inversion among hundreds of sums, of several items of a
batch: a sum without an inverse (a point with y = 0, twice: not on the curve,
but no caller's bases are checked) must leave the others alone."""
import numpy as np
import pytest

from _loader import load
from oracle import oracle as O

mzk = load()
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [2, 4, 600])
def test_a_sum_without_an_inverse_stays_alone(copies):
    ctx = mzk.Context(0)
    n = 1 << 20
    ds, db = ctx.gen_rand_fr(67, n), ctx.gen_bases(71, n + copies)
    b = db.download((n + copies, 12))
    b[n:] = b[0]
    b[n:, 6:] = 0
    db.upload(b)
    ones = ctx.alloc(copies * 32)
    ones.upload(np.repeat(O.fr_const(0).reshape(1, 4), copies, axis=0))
    ctx.set_msm_window(13)
    want = ctx.msm_device(ds, db, n)
    got = ctx.msm_batch_device(db, n + copies, [(ds, 0, n), (ones, n, copies)])
    assert np.array_equal(got[0], want)
    assert not got[1].any()  # an even number of them: the identity
    ctx.close()
