"""Every element of batch inversions at the sizes where a launch gains a block
or a row of elements (test_column_scans_gpu.py samples them): x times its
inverse is one, zeros stay zero, and nothing past the end is written."""
import numpy as np
import pytest

from _loader import load

mzk = load()
pytestmark = pytest.mark.gpu

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
ONE = pow(1 << 256, 2, R)  # x 2^256 times x^-1 2^256


@pytest.fixture(scope="module")
def ctx():
    c = mzk.Context(0)
    yield c
    c.close()


def ints(a):
    raw = np.ascontiguousarray(a, np.uint64).tobytes()
    return [int.from_bytes(raw[i:i + 32], "little") for i in range(0, len(raw), 32)]


# 128 threads with 1, 2, 4, 8 and 16 elements each; on 148 SMs a row is 18944 elements
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 18944, 18945, 37888, 37889, 75776, 75777, 303104, 303105])
@pytest.mark.parametrize("last_zero", [False, True])
def test_every_element(ctx, n, last_zero):
    buf = ctx.gen_rand_fr(11 * n, n + 1)
    a = buf.download((n + 1, 4))
    a[3:n:5] = 0
    if last_zero:
        a[n - 1] = 0
    elif not a[n - 1].any():
        a[n - 1] = a[n]
    buf.upload(a)
    ctx.batch_invert_device(buf, n)
    got = buf.download((n + 1, 4))
    assert np.array_equal(got[n], a[n])
    wrong = [i for i, (x, z) in enumerate(zip(ints(a[:n]), ints(got[:n]))) if x * z % R != (ONE if x else 0) or (not x and z)]
    assert not wrong, wrong[:10]
