"""MSMs whose entries lie in few buckets, far apart (one scalar, few different
ones, small ones): the walks over empty buckets of every accumulation, against
the oracle, and their time against scalars that fill the buckets."""
import time

import numpy as np
import pytest

from _loader import load
from oracle import oracle as O

mzk = load()
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mzk.Context(0)
    yield c
    c.close()


def few(n, values):
    """n scalars of `values` different ones, so at most that many buckets per window."""
    return O.rand_fr(83, values)[np.random.default_rng(values).integers(0, values, n)]


# quads (60000 entries), lanes (1.2 M); 4096 and 131072 buckets per window; gaps of one bucket to whole windows
@pytest.mark.parametrize("n,c", [(3000, 13), (3000, 18), (60000, 13), (60000, 18)])
@pytest.mark.parametrize("values", [1, 3, 40, 1000])
def test_few_buckets(ctx, n, c, values):
    s, b = few(n, values), O.gen_bases(89, n)
    ctx.set_msm_window(c)
    try:
        got = ctx.msm_best(s, b)
    finally:
        ctx.set_msm_window(0)
    assert np.array_equal(mzk.affine(got), O.msm_best(s, b))


# three rounds of pair sums: 21 M entries
@pytest.mark.parametrize("values", [1, 3, 40, 1000])
def test_few_buckets_in_pairs(ctx, values):
    n, m = 1 << 20, 1 << 16
    ds, db = ctx.alloc(n * 32), ctx.gen_bases(97, n)
    ds.upload(few(n, values))
    ctx.set_msm_window(13)
    try:
        paired = ctx.msm_device(ds, db, n)
        assert ctx.msm_last_pair_sums()[0] == 3
    finally:
        ctx.set_msm_window(0)
    parts = [ctx.msm_device(ds.ptr + i * 32, db.ptr + i * 96, m) for i in range(0, n, m)]
    assert np.array_equal(paired, mzk.g1_sum(np.stack(parts)))


def test_few_buckets_cost_no_more(ctx):
    """2^22 points: one scalar has as many additions as uniform ones and 15 gaps of 2^17 buckets (an MSM that walks
    them bucket by bucket took four times as long)."""
    n = 1 << 22
    uniform, db, one = ctx.gen_rand_fr(101, n), ctx.gen_bases(103, n), ctx.alloc(n * 32)
    one.upload(np.repeat(O.rand_fr(107, 1), n, axis=0))

    def best(ds):
        times = []
        for _ in range(5):
            t = time.perf_counter()
            ctx.msm_device(ds, db, n)
            times.append(time.perf_counter() - t)
        return min(times)

    assert best(one) < 1.5 * best(uniform)


def test_empty_buckets_are_cheap_to_reduce(ctx):
    """2^22 scalars of 8 bits fill 255 of 1.9 M buckets; reducing them took as long as reducing full ones."""
    n = 1 << 22
    uniform, db, small = ctx.gen_rand_fr(109, n), ctx.gen_bases(113, n), ctx.alloc(n * 32)
    values = np.stack([O.fr_op("from_canonical", np.array([v, 0, 0, 0], np.uint64)) for v in range(256)])
    small.upload(values[np.random.default_rng(5).integers(0, 256, n)])

    def reduce_ms(ds):
        ctx.msm_device(ds, db, n)
        ctx.set_profiling(True)
        for _ in range(3):
            ctx.msm_device(ds, db, n)
        ms, calls = ctx.phase_stats()["reduce"]
        ctx.set_profiling(False)
        return ms / calls

    assert reduce_ms(small) < 0.5 * reduce_ms(uniform)
