"""The memory of the pair sums: a context holds no more than its limit whatever
the MSM, the parts that its keys are cut into give the sum that the same MSM
gives without pair sums (which the other tests hold against the oracle), and
without room or memory the MSM runs unpaired."""
import numpy as np
import pytest
import torch

from _loader import load

mzk = load()
pytestmark = pytest.mark.gpu
GIB = 1 << 30


@pytest.fixture
def ctx():
    c = mzk.Context(0)
    yield c
    c.close()


def scratch_bytes():
    """What the kernel's 256 sums per thread take before any array of sums."""
    return torch.cuda.get_device_properties(0).multi_processor_count * 2 * 128 * 256 * 56


# 2^20 + 3 points of width 13: 20 windows, 21 M digits, 81920 buckets.  Room for every part: none, less than a
# bucket, one to a few hundred buckets (a bucket of 2^19 equal scalars exceeds it), a few windows, everything.
@pytest.mark.parametrize("room", [0, 256, 4096, 1 << 20, 1 << 23, 1 << 27, 1 << 31])
@pytest.mark.parametrize("kind", ["uniform", "heavy"])
def test_parts_give_the_same_sum(ctx, room, kind):
    n = (1 << 20) + 3
    ds, db = ctx.gen_rand_fr(31, n), ctx.gen_bases(37, n)
    if kind == "heavy":  # one bucket of every window holds half of the points
        s = ds.download((n, 4))
        s[::2] = s[0]
        ds.upload(s)
    ctx.set_msm_window(13)
    ctx.set_msm_pair_memory(0)
    want = ctx.msm_device(ds, db, n)
    assert ctx.msm_last_pair_sums() == (0, 0)
    ctx.set_msm_pair_memory(scratch_bytes() + room)
    assert np.array_equal(ctx.msm_device(ds, db, n), want)
    rounds, parts = ctx.msm_last_pair_sums()
    if room == 0:
        assert (rounds, parts) == (0, 0)
    if room >= 1 << 20:
        assert rounds == 3 and (parts > 1) == (room < 1 << 31)


def test_one_bucket_set_is_cut_to_the_limit(ctx):
    """An item over a window table keeps every entry in one bucket set: 2^22 points of width 20 are 54.5 M entries
    over 2^19 buckets, whose sums in one part would take 4.5 GB."""
    n, c = 1 << 22, 20
    rows = mzk.Context.msm_table_rows(c)
    ds, db = ctx.gen_rand_fr(41, n), ctx.gen_bases(43, n)
    table = ctx.alloc(rows * n * 96)
    table.upload(db.download((n, 12)))
    ctx.msm_window_table(table, n, c, rows)
    items = [(ds, 0, n)]
    free0 = torch.cuda.mem_get_info(0)[0]
    got = ctx.msm_batch_table_device(table, n, c, rows, 1, items)
    taken = free0 - torch.cuda.mem_get_info(0)[0]
    # beside the pair sums: digits and sorted entries, 4 bytes each, the buckets (192 bytes a key) and under 0.1 GB
    assert taken <= 25 * GIB / 8 + 8 * 13 * n + 192 * (1 << 19) + 10**8
    assert ctx.msm_last_pair_sums() == (3, 2)
    ctx.set_msm_pair_memory(0)
    assert np.array_equal(ctx.msm_batch_table_device(table, n, c, rows, 1, items), got)


def test_the_limit_frees_what_is_held(ctx):
    n = 1 << 20
    ds, db = ctx.gen_rand_fr(47, n), ctx.gen_bases(53, n)
    ctx.msm_device(ds, db, n)
    assert ctx.msm_last_pair_sums()[0] > 0
    free0 = torch.cuda.mem_get_info(0)[0]
    ctx.set_msm_pair_memory(0)
    assert torch.cuda.mem_get_info(0)[0] - free0 >= scratch_bytes()


def test_little_free_memory(ctx):
    """What is needed gets the pair sums' memory back, and they take no more than a quarter of what is free."""
    n = 1 << 20
    ds, db = ctx.gen_rand_fr(59, n), ctx.gen_bases(61, n)
    ctx.set_msm_window(13)
    want = ctx.msm_device(ds, db, n)
    rounds, _ = ctx.msm_last_pair_sums()
    assert rounds > 0  # 1.9 GiB held: 10.5 and 5.3 M sums and the kernel's scratch
    most = ctx.alloc(torch.cuda.mem_get_info(0)[0] - GIB)
    need = ctx.alloc(2 * GIB)  # more than the 1 GiB left
    assert np.array_equal(ctx.msm_device(ds, db, n), want)
    assert ctx.msm_last_pair_sums() == (0, 0)
    need.free()
    assert torch.cuda.mem_get_info(0)[0] >= 2 * GIB  # enough for the sums, which leave it alone
    assert np.array_equal(ctx.msm_device(ds, db, n), want)
    assert ctx.msm_last_pair_sums() == (0, 0)
    most.free()
    assert np.array_equal(ctx.msm_device(ds, db, n), want)
    assert ctx.msm_last_pair_sums()[0] == rounds
