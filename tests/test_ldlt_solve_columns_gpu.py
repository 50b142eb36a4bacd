"""LDL^T solves on both sides of the line between the two interchange kernels
(a CTA or a thread per right-hand-side column), bit for bit against the
oracle."""
import pytest

from conftest import assert_bitwise
from test_ldlt_cluster_gpu import _saddle
from test_ldlt_gpu import _run
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n,nrhs", [(2, 2, 1), (2, 8, 700), (3, 9, 700), (2, 32, 3000), (2, 32, 3001),
                                      (4, 9, 3001), (3, 33, 3001), (2, 34, 20000), (2, 34, 20001)],
                         ids=str)
def test_ldlt_solve_columns(mf, ref, rng, N, n, nrhs):
    S = _saddle(rng, N, n)
    F, _, cfg = _run(mf, S, False, 1)
    Fr, dsr, pvr, blr, info = ref.sytrf(S, blocked=False, block=1)
    assert info == 0
    B = syn.randn_mf(rng, N, n, nrhs)
    Xr, rc = ref.sytrs(Fr, dsr, pvr, blr, B)
    assert rc == 0
    assert_bitwise(mf.solve(F, mf.MFMatrix.from_numpy(B), config=cfg).to_numpy(), Xr, "solve")
