"""Operands that are no MFMatrix are refused as such, in the first place too."""
import numpy as np
import pytest
import torch


@pytest.mark.parametrize("x", [np.zeros((2, 3, 3)), [1.0, 2.0], torch.zeros(2, 3, 3), None, 1.0],
                         ids=lambda x: type(x).__name__)
@pytest.mark.parametrize("call", [lambda mf, x: mf.gemm_(x, x, x), lambda mf, x: mf.cholesky_(x),
                                  lambda mf, x: mf.mfdot(x, x)], ids=["gemm", "cholesky", "dot"])
def test_operand_type(mf, x, call):
    with pytest.raises(mf.ArgumentError, match="expected MFMatrix operands"):
        call(mf, x)
