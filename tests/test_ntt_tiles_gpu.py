"""The transforms either side of the line between small and large tiles (2^18
elements in one launch): single transforms against the oracle, batches against
single transforms, in place as well, bit-exact."""
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


# one tile and two (8, 9); the last small transform and the first large one (18, 19)
@pytest.mark.parametrize("k", [7, 8, 9, 15, 17, 18, 19])
@pytest.mark.parametrize("op", ["coeff_to_lagrange", "lagrange_to_coeff"])
def test_single_transforms(ctx, k, op):
    d, o = mzk.EvaluationDomain(ctx, 2, k), O.Domain(2, k)
    a = O.rand_fr(31 * k, 1 << k)
    assert np.array_equal(getattr(d, op)(a), getattr(o, op)(a))
    d.close()


@pytest.mark.parametrize("count", [1, 4, 5])  # 2^16, 2^18 and 5 x 2^16 extended elements
@pytest.mark.parametrize("op", ["coeff_to_extended", "extended_to_coeff"])
def test_batches(ctx, count, op):
    d = mzk.EvaluationDomain(ctx, 5, 14)
    n_in = d.n if op == "coeff_to_extended" else d.extended_len
    ins = [ctx.gen_rand_fr(100 + i, n_in) for i in range(count)]
    want = [getattr(d, op)(b.download((n_in, 4))) for b in ins]
    outs = [ctx.alloc(d.extended_len * 32) for _ in range(count)]
    d.op_batch_device(op, ins, outs)
    assert all(np.array_equal(b.download((d.extended_len, 4)), w) for b, w in zip(outs, want))
    if op == "extended_to_coeff":  # in place
        d.op_batch_device(op, ins, ins)
        assert all(np.array_equal(b.download((n_in, 4)), w) for b, w in zip(ins, want))
    d.close()
