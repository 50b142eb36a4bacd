"""LDL^T's cluster kernel at its size edges (one CTA, sixteen CTAs, ragged row
groups, 2x2 blocks on a panel's last column, long panels) and the interchange
of the solves, bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_ldlt_gpu import _run, _sym
from test_oracle import syn

pytestmark = pytest.mark.gpu


def _saddle(rng, N, n):
    S = _sym(rng, N, n)
    c = n - n // 3
    S[:, c:, c:] = 0.0
    S[:, np.arange(n), np.arange(n)] *= 2.0 ** -8  # 2x2 blocks almost everywhere
    return S


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("make", [_sym, _saddle], ids=["random", "saddle"])
@pytest.mark.parametrize("n,blocked,block", [(32, False, 1), (65, False, 1), (260, False, 1),
                                             (31, True, 2), (33, True, 3), (130, True, 64),
                                             (300, True, 12)], ids=str)
def test_ldlt_cluster_matches_oracle(mf, ref, rng, N, make, n, blocked, block):
    S = make(rng, N, n)
    F, Sd, cfg = _run(mf, S, blocked, block)
    Fr, dsr, pvr, blr, info = ref.sytrf(S, blocked=blocked, block=block)
    assert mf.factor_status(F) == info == 0
    assert np.array_equal(mf.factor_pivots(F), pvr)
    assert np.array_equal(mf.factor_blocks(F), blr)
    assert_bitwise(F.dsub.cpu().numpy(), dsr, "dsub")
    assert_bitwise(Sd.to_numpy(), Fr, "factor")
    B = syn.randn_mf(rng, N, n, 2)
    Xr, rc = ref.sytrs(Fr, dsr, pvr, blr, B)
    assert rc == 0
    assert_bitwise(mf.solve(F, mf.MFMatrix.from_numpy(B), config=cfg).to_numpy(), Xr, "solve")


@pytest.mark.parametrize("N", [2, 4])
@pytest.mark.parametrize("blocked", [False, True], ids=["unblocked", "blocked"])
@pytest.mark.parametrize("at", [0, 37, 79])
def test_ldlt_singular_column(mf, ref, rng, N, blocked, at):
    """a zero row and column: both routes stop with the oracle's status"""
    S = _sym(rng, N, 80)
    S[:, at, :] = 0.0
    S[:, :, at] = 0.0
    F, _, _ = _run(mf, S, blocked, 8)
    assert mf.factor_status(F) == ref.sytrf(S, blocked=blocked, block=8)[4] > 0
