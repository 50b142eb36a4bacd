"""Left triangular solves at the edges of their kernels (16 / 32 / 64 rows over
a warp's lanes, 256-term slabs of the backward chain, the column-count rules),
bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_blas_gpu import _tri
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("uplo,trans", [("lower", "N"), ("upper", "T"), ("lower", "T"),
                                        ("upper", "N")])
@pytest.mark.parametrize("m,n", [(1, 3), (2, 5), (16, 9), (17, 3), (32, 7), (33, 4), (64, 5),
                                 (65, 2), (257, 2), (258, 1), (5, 593), (3, 297)], ids=str)
@pytest.mark.parametrize("diag", ["nonunit", "unit"])
def test_left_solve_edges(mf, ref, rng, N, uplo, trans, m, n, diag):
    big = syn.randn_mf(rng, N, m + 3, m + 2)
    T = _tri(rng, N, m, uplo == "lower")
    if diag == "unit":
        T[:, np.arange(m), np.arange(m)] = np.nan  # never read
        T *= 0.125
    big[:, 2:2 + m, 1:1 + m] = T
    B = syn.randn_mf(rng, N, m, n)
    Bd = mf.MFMatrix.from_numpy(B)
    mf.trsm_(Bd, mf.MFMatrix.from_numpy(big).view(slice(2, 2 + m), slice(1, 1 + m)), 1.0, "left",
             uplo, trans, diag)
    assert_bitwise(Bd.to_numpy(), ref.trsm(B, T, 1.0, "left", uplo, trans, diag), "trsm")
