"""The LU panel's cluster kernel and the block-row kernel at their size edges
(one to sixteen CTAs, rows beyond them, panel widths 1 to 17, wide and tall
matrices, ties, a zero pivot), bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("m,n,block", [(2, 2, 16), (16, 40, 16), (33, 17, 16), (64, 64, 1),
                                       (130, 50, 7), (300, 290, 15), (600, 20, 17),
                                       (513, 70, 16), (4097, 18, 16)], ids=str)
def test_lu_panel_sizes(mf, ref, rng, N, m, n, block):
    A = syn.randn_mf(rng, N, m, n)
    Ad = mf.MFMatrix.from_numpy(A)
    F = mf.lu_(Ad, config=mf.KernelConfig(lu_block=block))
    LU, piv, info = ref.getrf(A, block=block)
    assert mf.factor_status(F) == info == 0
    assert np.array_equal(mf.factor_pivots(F), piv)
    assert_bitwise(Ad.to_numpy(), LU, "lu factor")


@pytest.mark.parametrize("N", [2, 4])
def test_lu_panel_ties_and_sorted_rows(mf, ref, rng, N):
    """equal magnitudes take the first row; a reversed column moves every row"""
    A = syn.randn_mf(rng, N, 90, 90)
    A[:, :, 0] = 0.0
    A[0, :, 0] = np.where(np.arange(90) % 2, 1.0, -1.0)
    A[0, :, 1] += np.arange(90) * 8.0
    Ad = mf.MFMatrix.from_numpy(A)
    F = mf.lu_(Ad)
    LU, piv, info = ref.getrf(A)
    assert mf.factor_status(F) == info == 0
    assert np.array_equal(mf.factor_pivots(F), piv)
    assert_bitwise(Ad.to_numpy(), LU, "lu factor")


@pytest.mark.parametrize("N", [2, 4])
@pytest.mark.parametrize("at", [0, 5, 15, 16, 39])
def test_lu_zero_column(mf, ref, rng, N, at):
    A = syn.randn_mf(rng, N, 40, 40)
    A[:, :, at] = 0.0
    Ad = mf.MFMatrix.from_numpy(A)
    F = mf.lu_(Ad, check=False)
    LU, piv, info = ref.getrf(A)
    assert mf.factor_status(F) == info == at + 1
    assert np.array_equal(mf.factor_pivots(F)[:at + 1], piv[:at + 1])
