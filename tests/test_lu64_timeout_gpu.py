"""The one-launch binary64 solve when its waits run out (a limit of one poll):
every CTA returns, the status word says so, solve_mixed_lu raises, and the next
solve on the same handle is right."""
import numpy as np
import pytest
import torch

from conftest import assert_bitwise
from test_lu64_gpu import _factor
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.fixture
def one_poll(mf):
    lib, h = mf._native.load(), mf._handle(0)

    def limit(polls):
        assert lib.mflab_set_tc_debug(h, polls, 0) == 0
    yield limit
    limit(0)
    mf.device_status()


@pytest.mark.parametrize("n,nrhs", [(1000, 3), (4096, 32)])
def test_solve_reports_and_recovers(mf, one_poll, n, nrhs):
    rng = np.random.default_rng(n)
    A, B = rng.standard_normal((n, n)) + 3 * np.eye(n), rng.standard_normal((n, nrhs))
    LU, ipiv, work = _factor(mf, A)
    lib, h, s = mf._native.load(), mf._handle(0), torch.cuda.current_stream().cuda_stream

    def run():
        X = mf.MFMatrix.from_numpy(B[None])
        assert lib.mflab_lu64_solve(h, s, n, nrhs, LU.ptr(), LU.ld, work.data_ptr(), X.ptr(),
                                    X.ld) == 0
        return X.to_numpy()
    want = run()
    assert mf.device_status() == 0
    one_poll(1)
    run()
    assert mf.device_status() == 6
    one_poll(0)
    assert_bitwise(run(), want, "after the timeout")
    assert mf.device_status() == 0


def test_solve_mixed_lu_raises(mf, rng, one_poll):
    A = mf.MFMatrix.from_numpy(syn.randn_mf(rng, 2, 600, 600))
    B = mf.MFMatrix.from_numpy(syn.randn_mf(rng, 2, 600, 2))
    want, _ = mf.solve_mixed_lu(A, B, residual="matched")
    one_poll(1)
    with pytest.raises(mf.MFLABError, match="status 6"):
        mf.solve_mixed_lu(A, B, residual="matched", maxiter=3)
    one_poll(0)
    got, report = mf.solve_mixed_lu(A, B, residual="matched")
    assert report["converged"]
    assert_bitwise(got.to_numpy(), want.to_numpy(), "after the timeout")
