"""Products with few rows and more column tiles than a grid's y dimension
holds, bit for bit against the oracle, and the column limit."""
import pytest

from conftest import assert_bitwise
from test_oracle import syn

pytestmark = pytest.mark.gpu

GRID = 65535


@pytest.mark.parametrize("N,m,n", [(2, 8, GRID * 8), (2, 8, GRID * 8 + 9), (2, 33, GRID * 16 + 5),
                                   (3, 5, GRID * 16 + 17), (4, 3, GRID * 16 + 1)], ids=str)
def test_gemm_many_columns(mf, ref, rng, N, m, n):
    A, B, C0 = syn.randn_mf(rng, N, m, 2), syn.randn_mf(rng, N, 2, n), syn.randn_mf(rng, N, m, n)
    Cd = mf.MFMatrix.from_numpy(C0)
    mf.gemm_(Cd, mf.MFMatrix.from_numpy(A), mf.MFMatrix.from_numpy(B), -1.0, 1.0)
    assert_bitwise(Cd.to_numpy(), ref.gemm(A, B, C0, -1.0, 1.0), "gemm")


@pytest.mark.parametrize("N,n", [(2, GRID * 8 + 9), (4, GRID * 16 + 1)], ids=str)
def test_trmm_many_columns(mf, ref, rng, N, n):
    A, B = syn.randn_mf(rng, N, 4, 4), syn.randn_mf(rng, N, 4, n)
    Bd = mf.MFMatrix.from_numpy(B)
    mf.trmm_(Bd, mf.MFMatrix.from_numpy(A))
    assert_bitwise(Bd.to_numpy(), ref.trmm(B, A), "trmm")


def test_gemm_column_limit(mf):
    n = GRID * 32 + 1
    A, B = mf.MFMatrix.zeros(4, 1, 1), mf.MFMatrix.zeros(4, 1, n)
    with pytest.raises(mf.ArgumentError):
        mf.gemm_(mf.MFMatrix.empty(4, 1, n), A, B)
