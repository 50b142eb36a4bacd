"""The LU factor after a zero pivot: the whole matrix as the oracle leaves it (the
steps before it on every column, nothing after), in the first and in later
panels, on square, wide and tall matrices."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("m,n,at,block", [(40, 40, 0, 16), (40, 40, 5, 16), (40, 40, 15, 16),
                                          (40, 90, 16, 16), (40, 90, 37, 16), (300, 60, 33, 16),
                                          (70, 70, 69, 16), (50, 50, 23, 7), (60, 80, 30, 24),
                                          (4100, 40, 18, 16)], ids=str)
def test_lu_state_after_zero_pivot(mf, ref, rng, N, m, n, at, block):
    A = syn.randn_mf(rng, N, m, n)
    A[:, :, at] = 0.0
    Ad = mf.MFMatrix.from_numpy(A)
    F = mf.lu_(Ad, check=False, config=mf.KernelConfig(lu_block=block))
    LU, piv, info = ref.getrf(A, block=block)
    assert mf.factor_status(F) == info == at + 1
    assert np.array_equal(mf.factor_pivots(F)[:at + 1], piv[:at + 1])
    assert_bitwise(Ad.to_numpy(), LU, "factor")
