"""The matched product's tile shapes and the matrix-vector kernel at the edges
of their ranges, bit for bit against the oracle (every shape runs the same
chain per output)."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("m,k,n", [(15, 17, 9), (16, 16, 8), (17, 33, 7), (300, 31, 257),
                                   (513, 9, 301), (1024, 3, 2368), (1184, 5, 1024)], ids=str)
def test_gemm_tile_shapes(mf, ref, rng, N, m, k, n):
    A, B, C0 = syn.randn_mf(rng, N, m, k), syn.randn_mf(rng, N, k, n), syn.randn_mf(rng, N, m, n)
    Cd = mf.MFMatrix.from_numpy(C0)
    mf.gemm_(Cd, mf.MFMatrix.from_numpy(A), mf.MFMatrix.from_numpy(B), -1.0, 1.0)
    assert_bitwise(Cd.to_numpy(), ref.gemm(A, B, C0, -1.0, 1.0), "gemm")


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("m,k", [(1, 200), (31, 32), (32, 31), (33, 33), (97, 64), (5000, 3),
                                 (70, 0)], ids=str)
def test_gemv_slab_and_row_edges(mf, ref, rng, N, trans, m, k):
    big = syn.randn_mf(rng, N, *((m + 5, k + 3) if trans == "N" else (k + 5, m + 3)))
    rows, cols = (m, k) if trans == "N" else (k, m)
    A = np.ascontiguousarray(big[:, 2:2 + rows, 1:1 + cols])
    x, y0 = syn.randn_mf(rng, N, k, 1), syn.randn_mf(rng, N, m, 1)
    Ad = mf.MFMatrix.from_numpy(big).view(slice(2, 2 + rows), slice(1, 1 + cols))
    yd = mf.MFMatrix.from_numpy(y0[:, :, 0])
    mf.gemv_(yd, Ad, mf.MFMatrix.from_numpy(x[:, :, 0]), 1.0, -1.0, trans=trans)
    op = A if trans == "N" else np.ascontiguousarray(A.transpose(0, 2, 1))
    want = ref.gemm(op, x, y0.copy(), 1.0, -1.0, x3_fused=False)[:, :, 0]
    assert_bitwise(yd.to_numpy(), want, "gemv")


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("uplo", ["lower", "upper"])
@pytest.mark.parametrize("n", [1, 32, 33, 97])
def test_symv_diagonal_blocks(mf, ref, rng, N, uplo, n):
    S = syn.randn_mf(rng, N, n, n)
    lower = np.tril(S) if uplo == "lower" else np.triu(S).transpose(0, 2, 1)
    full = lower + np.tril(lower, -1).transpose(0, 2, 1)
    x = syn.randn_mf(rng, N, n, 1)
    yd = mf.MFMatrix.zeros(N, n)
    mf.symv_(yd, mf.MFMatrix.from_numpy(S), mf.MFMatrix.from_numpy(x[:, :, 0]), uplo=uplo)
    assert_bitwise(yd.to_numpy(), ref.gemm(full, x, x3_fused=False)[:, :, 0], "symv")
