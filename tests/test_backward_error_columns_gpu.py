"""The normwise backward error on both sides of the lines between its CTA sizes:
every column as a call with that column alone gives it."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nrhs", [(2, 148), (2, 149), (2, 296), (2, 297), (3, 149), (3, 592),
                                    (3, 593), (4, 149), (4, 296), (4, 297)], ids=str)
@pytest.mark.parametrize("m,k", [(3, 5), (300, 130)], ids=str)
def test_columns(mf, rng, N, nrhs, m, k):
    A, X = syn.randn_mf(rng, N, m, k), syn.randn_mf(rng, N, k, nrhs)
    B, R = syn.randn_mf(rng, N, m, nrhs), syn.randn_mf(rng, N, m, nrhs)
    X[0, k - 1, 2] = np.nan
    R[0, m - 1, nrhs - 1] = np.inf
    Ad = mf.MFMatrix.from_numpy(A)
    anorm = mf.OpNormInf(Ad)

    def run(c):
        return mf.normwise_backward_error(Ad, *(mf.MFMatrix.from_numpy(np.ascontiguousarray(M[:, :, c]))
                                                for M in (X, B, R)), anorm=anorm)
    got = run(slice(0, nrhs))
    assert np.isnan(got[2][0]) and np.isnan(got[nrhs - 1][0])
    for j in (0, 1, nrhs // 2, nrhs - 2):
        assert_bitwise(got[j], run(slice(j, j + 1))[0], f"column {j}")
