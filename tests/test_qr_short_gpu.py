"""QR on both sides of the line between the reflector's two norms (a warp for
short columns, nine warps for tall ones), bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_qr_chains_gpu import _panel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("pivoted", [False, True], ids=["qr", "rrqr"])
@pytest.mark.parametrize("m,n", [(5, 5), (33, 7), (87, 5), (88, 6), (92, 9), (100, 170)], ids=str)
def test_reflector_norms(mf, ref, rng, N, pivoted, m, n):
    A = _panel(rng, N, m, n)
    F = (mf.rrqr_ if pivoted else mf.qr_)(mf.MFMatrix.from_numpy(A))
    want, wtau, wperm, _ = (ref.rrqr if pivoted else ref.qr)(A)
    assert np.array_equal(mf.factor_permutation(F), wperm)
    assert_bitwise(F.tau.cpu().numpy(), wtau, "tau")
    assert_bitwise(F.factors.to_numpy(), want, "factors")
