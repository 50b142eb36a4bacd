"""QR's column norms over several tiles of rows (zeros, new maxima within and
across tiles) and apply_q! on both sides of its kernel rule, bit for bit."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_oracle import syn

pytestmark = pytest.mark.gpu


def _panel(rng, N, m, n):
    """columns that rise, fall, start with zeros, hold zeros in between or only
    one nonzero entry"""
    A = syn.randn_mf(rng, N, m, n)
    rise = np.exp2(np.linspace(-30, 30, m))
    A[:, :, 0] *= np.exp2(np.round(np.log2(rise)))
    A[:, :, 1] *= np.exp2(np.round(np.log2(rise[::-1])))
    A[:, :min(m - 1, 300), 2] = 0.0
    A[:, rng.random(m) < 0.5, 3] = 0.0
    A[:, :m - 1, 4] = 0.0
    return A


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("pivoted", [False, True], ids=["qr", "rrqr"])
@pytest.mark.parametrize("m,n", [(255, 6), (256, 9), (257, 6), (640, 40)], ids=str)
def test_norm_tiles(mf, ref, rng, N, pivoted, m, n):
    A = _panel(rng, N, m, n)
    F = (mf.rrqr_ if pivoted else mf.qr_)(mf.MFMatrix.from_numpy(A))
    want, wtau, wperm, _ = (ref.rrqr if pivoted else ref.qr)(A)
    assert np.array_equal(mf.factor_permutation(F), wperm)
    assert_bitwise(F.tau.cpu().numpy(), wtau, "tau")
    assert_bitwise(F.factors.to_numpy(), want, "factors")


@pytest.mark.parametrize("N", [2, 4])
@pytest.mark.parametrize("nd", [1, 296, 297])
def test_apply_q_column_counts(mf, ref, rng, N, nd):
    A, D = syn.randn_mf(rng, N, 270, 3), syn.randn_mf(rng, N, 270, nd)
    F = mf.qr_(mf.MFMatrix.from_numpy(A))
    Dd = mf.MFMatrix.from_numpy(D)
    mf.apply_q_(Dd, F, trans="T")
    assert_bitwise(Dd.to_numpy(), ref.apply_q(F.factors.to_numpy(), F.tau.cpu().numpy(), D, "T"))


@pytest.mark.parametrize("N,m,n", [(2, 128, 296), (2, 129, 297), (2, 127, 20), (3, 130, 148),
                                   (4, 128, 148), (4, 130, 149)])
def test_initial_norms_at_the_rule(mf, ref, rng, N, m, n):
    """a CTA or a warp per column for the first norms of a pivoted QR"""
    A = _panel(rng, N, m, n)
    F = mf.rrqr_(mf.MFMatrix.from_numpy(A))
    want, wtau, wperm, _ = ref.rrqr(A)
    assert np.array_equal(mf.factor_permutation(F), wperm)
    assert_bitwise(F.tau.cpu().numpy(), wtau, "tau")
    assert_bitwise(F.factors.to_numpy(), want, "factors")
