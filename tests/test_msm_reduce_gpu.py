"""The bucket reduction of an MSM (partial sums of cut buckets, the tree over a
window's buckets, running sums over groups of them where buckets are many)
against the oracle's plain double-and-add sum, bit-exact.

The inputs drive every additions' special cases: buckets that hold the same
point (doublings all the way up the tree), opposite points (the tree meets
infinity), empty buckets, and buckets cut into few and into many chunks.
"""
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


def small_scalars(values):
    """Montgomery forms of small whole numbers, by repeated doubling and adding."""
    one = O.fr_const(0)
    out = np.zeros((len(values), 4), np.uint64)
    for i, v in enumerate(values):
        acc = np.zeros(4, np.uint64)
        for bit in bin(int(v))[2:]:
            acc = O.fr_op("add", acc, acc)
            if bit == "1":
                acc = O.fr_op("add", acc, one)
        out[i] = acc
    return out


def negated(p):
    q = p.copy()
    q[6:] = O.fp_op("sub", np.zeros(6, np.uint64), p[6:])
    return q


def inputs(kind):
    g = O.gen_bases(11, 400)
    if kind == "one point":              # every bucket the same point
        s, b = small_scalars(range(1, 301)), np.repeat(g[:1], 300, axis=0)
    elif kind == "opposite points":      # neighbouring buckets cancel pairwise
        s = small_scalars([1 + i // 2 for i in range(300)])
        b = np.stack([g[0] if i % 4 in (0, 3) else negated(g[0]) for i in range(300)])
    elif kind == "cut buckets":          # spans of 1 .. 300 chunks, both sides of the short-span limit
        runs = [1, 2, 3, 11, 12, 13, 14, 15, 63, 64, 65, 66, 129, 300]
        s = small_scalars([7 * (i + 1) for i, r in enumerate(runs) for _ in range(r)])
        b = np.concatenate([g[:r] for r in runs])
    else:
        s, b = O.rand_fr(13, 400), g
    return s, np.ascontiguousarray(b)


# 5: the narrowest window; 8 and 9: one block of the tree and two; 13, 16, 18: several launches; 20: groups first
@pytest.mark.parametrize("c", [5, 8, 9, 13, 16, 18, 20])
@pytest.mark.parametrize("kind", ["one point", "opposite points", "cut buckets", "uniform"])
def test_reduction_matches_the_plain_sum(ctx, c, kind):
    s, b = inputs(kind)
    ctx.set_msm_window(c)
    try:
        got = ctx.msm_best(s, b)
    finally:
        ctx.set_msm_window(0)
    assert np.array_equal(mzk.affine(got), O.msm_naive(s, b))


# 29 windows of width 9: 149988 and 150017 digits, either side of the line between quads and lanes per chunk
@pytest.mark.parametrize("n", [5172, 5173])
@pytest.mark.parametrize("sparse", [False, True])
def test_accumulation_by_quads_and_by_lanes(ctx, n, sparse):
    s, b = O.rand_fr(17, n), O.gen_bases(19, n)
    if sparse:  # heavy buckets and an identity base
        s[:n // 2] = O.fr_const(0)
        s[n // 2:2 * n // 3] = 0
        b[5] = 0
    ctx.set_msm_window(9)
    try:
        got = ctx.msm_best(s, b)
    finally:
        ctx.set_msm_window(0)
    assert np.array_equal(mzk.affine(got), O.msm_best(s, b))


# 2^20 points of width 13: 20 M digits over 81920 buckets, three rounds of pair sums before the mixed additions
@pytest.mark.parametrize("kind", ["uniform", "pairs"])
def test_pair_sums(ctx, kind):
    n = 1 << 20
    ds, db = ctx.gen_rand_fr(23, n), ctx.gen_bases(29, n)
    if kind == "pairs":  # neighbours in a bucket: equal (doublings), opposite (infinity), and identity points
        s, b = ds.download((n, 4)), db.download((n, 12))
        s[1::4], s[3::4] = s[0::4], s[2::4]
        b[1::4] = b[0::4]
        b[3::4, :6], b[3::4, 6:] = b[2::4, :6], b[2::4, 6:]
        b[7::64] = np.stack([negated(p) for p in b[6::64]])
        b[8::64] = 0
        ds.upload(s)
        db.upload(b)
    ctx.set_msm_window(13)
    try:
        paired = ctx.msm_device(ds, db, n)
    finally:
        ctx.set_msm_window(0)
    # the same MSM in slices too short for pair sums
    m = 1 << 16
    parts = [ctx.msm_device(ds.ptr + i * 32, db.ptr + i * 96, m) for i in range(0, n, m)]
    assert np.array_equal(paired, mzk.g1_sum(np.stack(parts)))
