"""Batches on both sides of the line between the factor's CTA sizes, and panels
too wide to stage, bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_batched_gpu import _spd_blocks
from test_oracle import syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("most,block", [(1, 16), (48, 16), (49, 16), (48, 17), (49, 64)], ids=str)
@pytest.mark.parametrize("threads", [64, 512])
def test_factor_shapes(mf, ref, rng, N, most, block, threads):
    sizes = np.concatenate([[most], rng.integers(0, most + 1, 20)])
    blocks = _spd_blocks(ref, rng, N, sizes)
    rhs = [syn.randn_mf(rng, N, int(n), 1)[:, :, 0] for n in sizes]
    batch = mf.batched.SPDBatch(N, sizes)
    for i, (S, b) in enumerate(zip(blocks, rhs)):
        batch.set_block(i, S)
        batch.set_rhs(i, b)
    info = mf.batched.potrf_potrs_batched_(batch, block=block,
                                           tuning={"threads": threads, "grid": 0})
    assert not np.any(info)
    for i, n in enumerate(sizes):
        if n:
            L, _ = ref.potrf(blocks[i], block=block)
            assert_bitwise(np.tril(batch.block(i)), np.tril(L), f"factor {i}")
            assert_bitwise(batch.rhs(i), ref.potrs(L, rhs[i][:, :, None])[:, :, 0], f"solve {i}")
