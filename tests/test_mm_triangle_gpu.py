"""x2 products into a triangle on both sides of the line between their tile
shapes, and a lone row transposed, bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1856, 2), (1920, 3), (2000, 2)], ids=str)
def test_triangle_tiles(mf, ref, rng, n, k):
    Q, P, P2 = syn.randn_mf(rng, 2, k, n), syn.randn_mf(rng, 2, n, k), syn.randn_mf(rng, 2, n, k)
    C0 = syn.randn_mf(rng, 2, n, n)
    Cd = mf.MFMatrix.from_numpy(C0)
    mf.gemmt_(Cd, mf.MFMatrix.from_numpy(P), mf.MFMatrix.from_numpy(P2), -1.0, 1.0)
    assert_bitwise(Cd.to_numpy(), ref.gemmt_lower(P, P2, C0.copy(), -1.0, 1.0), "gemmt")
    Cd = mf.MFMatrix.from_numpy(C0)
    mf.syrk_(Cd, mf.MFMatrix.from_numpy(Q), -1.0, 1.0)
    want = ref.gemmt_lower(Q.transpose(0, 2, 1).copy(), Q.transpose(0, 2, 1).copy(), C0.copy(), -1.0,
                           1.0)
    assert_bitwise(Cd.to_numpy(), want, "syrk")


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("view", [False, True])
def test_lone_row_transposed(mf, ref, rng, N, view):
    n = 1000
    big = syn.randn_mf(rng, N, 3 if view else 1, n)
    A = np.ascontiguousarray(big[:, 1:2] if view else big)
    Ad = mf.MFMatrix.from_numpy(big)
    Ad = Ad.view(slice(1, 2), slice(0, n)) if view else Ad
    x, y0 = syn.randn_mf(rng, N, 1, 1), syn.randn_mf(rng, N, n, 1)
    yd = mf.MFMatrix.from_numpy(y0[:, :, 0])
    mf.gemv_(yd, Ad, mf.MFMatrix.from_numpy(x[:, :, 0]), 1.0, -1.0, trans="T")
    want = ref.gemm(np.ascontiguousarray(A.transpose(0, 2, 1)), x, y0.copy(), 1.0, -1.0,
                    x3_fused=False)[:, :, 0]
    assert_bitwise(yd.to_numpy(), want, "gemv")
