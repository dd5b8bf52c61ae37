"""Linear recurrences (eval_polynomial, kate_division) and batch inversion at the
edges of their blocks, against Python integers, bit-exact."""
import numpy as np
import pytest

from _loader import load

mzk = load()
pytestmark = pytest.mark.gpu

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
MONT = (1 << 256) % R
MONT_INV = pow(MONT, -1, R)


@pytest.fixture(scope="module")
def ctx():
    c = mzk.Context(0)
    yield c
    c.close()


def ints(a):
    """Stored (Montgomery) values as integers."""
    return [int.from_bytes(row.tobytes(), "little") for row in np.ascontiguousarray(a, np.uint64)]


def limbs(v):
    return np.frombuffer(int(v).to_bytes(32, "little"), np.uint64)


# 1024, 2048 and 4096 elements per block (4, 8 and 16 per thread from 1.2 and 2.4 million elements on)
@pytest.mark.parametrize("n", [1, 2, 3, 5, 1023, 1024, 1025, 1026, 4097, 1048577, 1212415, 1212417, 2424833])
def test_recurrences(ctx, n):
    buf, b = ctx.gen_rand_fr(n, n), limbs(0x1234567890ABCDEF1234567890ABCDEF % R)
    point = ints(b.reshape(1, 4))[0] * MONT_INV % R  # the factor that multiplies stored values
    a = ints(buf.download((n, 4)))
    acc, y = 0, [0] * n
    for i in range(n - 1, -1, -1):
        acc = (a[i] + point * acc) % R
        y[i] = acc
    assert np.array_equal(ctx.eval_polynomial_device(buf, n, b), limbs(y[0]))
    if n > 1:  # the quotient of a(X) by X - b: q_i = y_{i+1}
        q = ctx.alloc(n * 32)
        ctx.kate_division_device(buf, n, b, q)
        assert ints(q.download((n - 1, 4))) == y[1:]


# 128 threads with 1, 2, 4, 8 and 16 elements each: 18944, 37888, 75776 and 303104 are the lines on 148 SMs
@pytest.mark.parametrize("n", [1, 127, 128, 129, 18944, 18945, 37888, 37889, 75777, 303104, 303105])
def test_batch_inversion(ctx, n):
    buf = ctx.gen_rand_fr(7 * n, n)
    a = buf.download((n, 4))
    a[::5] = 0
    buf.upload(a)
    ctx.batch_invert_device(buf, n)
    got = buf.download((n, 4))
    assert not got[::5].any()
    one = MONT * MONT % R  # x R times x^-1 R
    for x, z in zip(ints(a)[1::7], ints(got)[1::7]):
        assert (x * z) % R == (one if x else 0)
