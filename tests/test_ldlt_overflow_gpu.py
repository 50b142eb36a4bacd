"""LDL^T of finite matrices whose elimination overflows: the pivot scans meet
infinities and NaN, and every thread of the cluster takes the same branch, the
one of the oracle's folds (max(x, y) is y where x is NaN)."""
import numpy as np
import pytest

from test_ldlt_gpu import _run

pytestmark = pytest.mark.gpu


def _fill(N, n):
    """after step 0 entry (32, 2) is NaN; the row scan of step 1 meets it"""
    S = np.zeros((N, n, n))
    for i, j, v in [(0, 0, 1e308), (2, 0, 1e308), (32, 0, 1e308), (32, 2, -1e308),
                    (2, 2, 1e308 + 1e300), (2, 1, 1e299)]:
        S[0, i, j] = S[0, j, i] = v
    return S


def _sparse(N, n, density, scale):
    rng = np.random.default_rng(3)
    M = rng.choice([-1.0, 1.0], (n, n)) * rng.uniform(0.5, 1.0, (n, n)) * scale
    M = np.tril(M * (rng.random((n, n)) < density))
    d = np.arange(n)
    M[d, d] += np.where(M[d, d] == 0.0, 1e300, 0.0)
    S = np.zeros((N, n, n))
    S[0] = M + np.tril(M, -1).T
    return S


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("blocked", [False, True], ids=["unblocked", "blocked"])
@pytest.mark.parametrize("S", [lambda N: _fill(N, 34), lambda N: _fill(N, 300),
                               lambda N: _sparse(N, 40, 0.2, 1e308),
                               lambda N: _sparse(N, 100, 0.05, 1.7e308),
                               lambda N: _sparse(N, 300, 0.02, 1e308),
                               lambda N: _sparse(N, 300, 0.2, 1.7e308)],
                         ids=["fill-34", "fill-300", "40", "100", "300", "300-dense"])
def test_ldlt_overflow_follows_oracle(mf, ref, N, blocked, S):
    S = S(N)
    F, _, _ = _run(mf, S, blocked, 8)
    _, _, pivots, blocks, info = ref.sytrf(S, blocked=blocked, block=8)
    assert info > 0 and mf.factor_status(F) == info
    assert np.array_equal(mf.factor_pivots(F)[:info - 1], pivots[:info - 1])
    assert np.array_equal(mf.factor_blocks(F)[:info - 1], blocks[:info - 1])
