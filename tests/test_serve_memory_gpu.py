"""What a lane of the proving service holds stays within its memory budget, the
pair sums of its MSMs included."""
import pytest
import torch

from _plonk_setup import Circuit, mzk

pytestmark = pytest.mark.gpu


def test_a_lane_stays_within_its_budget():
    ctx = mzk.Context(0)
    # 2^12 rows: 8 MB of polynomials a proof, but a wave's quotient limbs are MSMs of 8 M digits: pair sums of any
    # size make it 1.9 GB
    c = Circuit(ctx, 12, seed=71, oracle=False)
    budget = 10**9
    free0 = torch.cuda.mem_get_info(0)[0]
    srv = mzk.ProvingServer(ctx, max_batch=20, lanes=1, mem_budget_bytes=budget)
    blinds = [c.blinds(300 + i) for i in range(24)]
    tickets = [srv.submit(c.key, c.advice, b) for b in blinds]
    proofs = [srv.wait(t)[0] for t in tickets]
    taken = free0 - torch.cuda.mem_get_info(0)[0]
    stats = srv.stats()
    srv.close()
    for i in (0, 23):
        assert proofs[i] == mzk.create_proofs(ctx, [(c.key, c.advice, blinds[i])])[0]
    assert stats["waves"] < 24  # waves of many proofs
    assert taken <= budget
    ctx.close()
