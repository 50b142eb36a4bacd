"""The narrow residue products (at most 32 columns) against the library int8
engine bit for bit at the edges of their tiles, through both entry points, and
their timeout path; the one-launch binary64 solves against the block kernel."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import assert_bitwise
from test_lu64_gpu import _factor
from test_oracle import syn

pytestmark = pytest.mark.gpu


def _config(mf, engine, moduli=0):
    return mf.KernelConfig(gemm_strategy="ozaki", ozaki_scheme="modular", ozaki_engine=engine,
                           ozaki_moduli=moduli)


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (128, 128, 16), (129, 127, 17), (300, 513, 32),
                                   (1111, 257, 5), (130, 300, 33)], ids=str)
def test_narrow_products_match_library(mf, rng, N, m, k, n):
    A, B = syn.randn_mf(rng, N, m, k, spread=8), syn.randn_mf(rng, N, k, n, spread=8)
    C0 = syn.randn_mf(rng, N, m, n)
    got = []
    for engine in ("tcgen05", "library"):
        Cd = mf.MFMatrix.from_numpy(C0)
        mf.gemm_(Cd, mf.MFMatrix.from_numpy(A), mf.MFMatrix.from_numpy(B), -1.0, 1.0,
                 config=_config(mf, engine))
        got.append((Cd.to_numpy(), mf.ozaki_last_moduli()))
    assert got[0][1] == got[1][1] and mf.device_status() == 0
    assert_bitwise(got[0][0], got[1][0], "narrow product")
    P = mf.PreparedInt8Operand(mf.MFMatrix.from_numpy(A), got[0][1])
    out = []
    for engine in ("tcgen05", "library"):
        Cd = mf.MFMatrix.from_numpy(C0)
        mf.gemm_prepared_(Cd, P, mf.MFMatrix.from_numpy(B), -1.0, 1.0,
                          config=_config(mf, engine, got[0][1]))
        out.append(Cd.to_numpy())
    assert_bitwise(out[0], out[1], "prepared narrow product")


def test_narrow_timeout_is_reported(mf, rng):
    N = 2
    A, B = syn.randn_mf(rng, N, 500, 300), syn.randn_mf(rng, N, 300, 9)
    lib, h = mf._native.load(), mf._handle(0)
    run = lambda: mf.gemm_(mf.MFMatrix.zeros(N, 500, 9), mf.MFMatrix.from_numpy(A),  # noqa: E731
                           mf.MFMatrix.from_numpy(B), config=_config(mf, "tcgen05", 30)).to_numpy()
    want = run()
    assert mf.device_status() == 0
    assert lib.mflab_set_tc_debug(h, 1 << 20, 1) == 0
    try:
        run()
        assert mf.device_status() == 2
    finally:
        lib.mflab_set_tc_debug(h, 0, 0)
    assert_bitwise(run(), want, "after the timeout")
    assert mf.device_status() == 0


@pytest.mark.parametrize("n,nrhs", [(n, r) for n in (1, 31, 32, 33, 127, 128, 129, 160, 1000)
                                    for r in (1, 16, 17, 32)] + [(4096, 17)])
def test_one_launch_solve_matches_block_kernel(mf, n, nrhs):
    """33 columns take the block kernel; its first columns are the same sums"""
    rng = np.random.default_rng(n + nrhs)
    A = rng.standard_normal((n, n)) + 3 * np.eye(n)
    B = rng.standard_normal((n, 33))
    LU, ipiv, work = _factor(mf, A)
    lib, h, s = mf._native.load(), mf._handle(0), torch.cuda.current_stream().cuda_stream
    outs = []
    for cols in (nrhs, 33):
        X = mf.MFMatrix.from_numpy(np.ascontiguousarray(B[None, :, :cols]))
        assert lib.mflab_lu64_solve(h, s, n, cols, LU.ptr(), LU.ld, work.data_ptr(), X.ptr(),
                                    X.ld) == 0
        outs.append(X.to_numpy()[0][:, :nrhs])
    assert mf.device_status() == 0
    assert_bitwise(outs[0], outs[1], "solve")
