"""The pullback of a batch that was used again and failed in between: a block
without a factor gets a zero gradient, the others theirs."""
import numpy as np
import pytest
import torch

from test_batched_gpu import _spd_blocks
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 4])
def test_pullback_after_a_failed_block(mf, ref, rng, N):
    sizes = np.array([33, 7, 70, 20])
    blocks = _spd_blocks(ref, rng, N, sizes)
    rhs = [syn.randn_mf(rng, N, int(n), 1)[:, :, 0] for n in sizes]
    batch = mf.batched.SPDBatch(N, sizes)

    def fill(bad):
        for i, (S, b) in enumerate(zip(blocks, rhs)):
            S = S.copy()
            if i in bad:
                S[0, 3, 3] = -1e6
            batch.set_block(i, S)
            batch.set_rhs(i, b)
    fill(())
    x, pullback = mf.batched.solve_spd_batched_rrule(batch)
    w = torch.ones_like(x)
    want, _ = pullback(w)
    fill((1, 2))
    info = mf.batched.potrf_potrs_batched_(batch, check=False)
    assert np.array_equal(info != 0, [False, True, True, False])
    stale = [torch.full_like(batch.S, float("nan")) for _ in range(4)]
    del stale  # what an uninitialised gradient would be taken from
    got, bbar = pullback(w)
    for i in range(len(sizes)):
        have = batch.block(i, got)
        assert np.array_equal(have, batch.block(i, want) if i in (0, 3) else np.zeros_like(have))
    assert np.array_equal(batch.rhs(1, bbar), np.ones_like(rhs[1]))
