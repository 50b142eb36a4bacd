"""Left triangular solves of many columns, on both sides of the lines between
their kernels, bit for bit against the oracle."""
import pytest

from conftest import assert_bitwise
from test_blas_gpu import _tri
from test_oracle import syn

pytestmark = pytest.mark.gpu


def _check(mf, ref, rng, N, m, n, uplo, trans, diag="nonunit"):
    T = _tri(rng, N, m, uplo == "lower")
    if diag == "unit":
        T *= 2.0 ** -8  # bounded growth
    B = syn.randn_mf(rng, N, m, n)
    Bd = mf.MFMatrix.from_numpy(B)
    mf.trsm_(Bd, mf.MFMatrix.from_numpy(T), 1.0, "left", uplo, trans, diag)
    assert_bitwise(Bd.to_numpy(), ref.trsm(B, T, 1.0, "left", uplo, trans, diag), "trsm")


@pytest.mark.parametrize("uplo,trans", [("lower", "N"), ("upper", "T")])
@pytest.mark.parametrize("N,m,line", [(2, 4, 2560), (3, 17, 2465), (4, 16, 3200), (4, 33, 1980)],
                         ids=str)
@pytest.mark.parametrize("past", [0, 1])
def test_forward_short_triangle(mf, ref, rng, N, m, line, uplo, trans, past):
    _check(mf, ref, rng, N, m, line + past, uplo, trans)


@pytest.mark.parametrize("uplo,trans,diag", [("lower", "N", "nonunit"), ("upper", "T", "unit")])
@pytest.mark.parametrize("N,m,n", [(2, 65, 296), (2, 65, 297), (2, 300, 445), (2, 65, 593),
                                   (3, 70, 148), (3, 70, 149), (4, 66, 148), (4, 257, 149),
                                   (2, 2049, 149), (4, 2049, 2)], ids=str)
def test_forward_wavefront(mf, ref, rng, N, m, n, uplo, trans, diag):
    _check(mf, ref, rng, N, m, n, uplo, trans, diag)


@pytest.mark.parametrize("uplo,trans,diag", [("upper", "N", "nonunit"), ("lower", "T", "unit")])
@pytest.mark.parametrize("N,m,n", [(2, 65, 296), (2, 65, 297), (2, 257, 149), (2, 5, 592),
                                   (2, 5, 593), (3, 64, 149), (3, 1, 400), (4, 2, 444), (4, 2, 445),
                                   (4, 67, 149), (4, 65, 4096)], ids=str)
def test_backward(mf, ref, rng, N, m, n, uplo, trans, diag):
    _check(mf, ref, rng, N, m, n, uplo, trans, diag)
