"""The batched SPD kernels at their edges: sizes around the 16-column panel, the
32-term slabs and the lanes' row groups, blocks of very different sizes sharing
a warp, failed and empty blocks among them, batches on both sides of the
forward kernel's rule, panels too large to stage; bit for bit against the
oracle."""
import numpy as np
import pytest
import torch

from conftest import assert_bitwise
from test_batched_gpu import _spd_blocks
from test_oracle import syn

pytestmark = pytest.mark.gpu


def _run(mf, ref, rng, N, sizes, bad=(), block=16, check=None):
    sizes = np.asarray(sizes)
    blocks = _spd_blocks(ref, rng, N, sizes)
    for i in bad:
        blocks[i][0, sizes[i] // 2, sizes[i] // 2] = -1e6
    rhs = [syn.randn_mf(rng, N, int(n), 1)[:, :, 0] for n in sizes]
    batch = mf.batched.SPDBatch(N, sizes)
    for i, (S, b) in enumerate(zip(blocks, rhs)):
        batch.set_block(i, S)
        batch.set_rhs(i, b)
    info = mf.batched.potrf_potrs_batched_(batch, block=block, check=False)
    for i in check if check is not None else range(len(sizes)):
        L, want = ref.potrf(blocks[i], block=block)
        assert info[i] == want and (want != 0) == (i in bad)
        if want == 0 and sizes[i]:
            assert_bitwise(np.tril(batch.block(i)), np.tril(L), f"factor {i}")
            assert_bitwise(batch.rhs(i), ref.potrs(L, rhs[i][:, :, None])[:, :, 0], f"solve {i}")


@pytest.mark.parametrize("N", [2, 3, 4])
def test_sizes_and_failures_side_by_side(mf, ref, rng, N):
    _run(mf, ref, rng, N, [1, 2, 15, 16, 17, 31, 32, 33, 34, 48, 63, 64, 65, 66, 97, 129, 0, 5],
         bad=(4, 11))


@pytest.mark.parametrize("N,n", [(2, 449), (3, 297), (4, 225)])
def test_panel_too_large_to_stage(mf, ref, rng, N, n):
    _run(mf, ref, rng, N, [n, 20])


@pytest.mark.parametrize("block", [5, 16, 20])
def test_block_widths(mf, ref, rng, block):
    _run(mf, ref, rng, 2, [3, 40, 61], block=block)


def test_many_small_blocks(mf, ref, rng):
    sizes = rng.integers(1, 12, 2400)
    _run(mf, ref, rng, 2, sizes, check=range(0, 2400, 97))


@pytest.mark.parametrize("N", [2, 4])
def test_adjoint_of_uneven_blocks(mf, ref, rng, N):
    sizes = np.array([1, 33, 7, 70])
    blocks = _spd_blocks(ref, rng, N, sizes)
    batch = mf.batched.SPDBatch(N, sizes)
    for i, S in enumerate(blocks):
        batch.set_block(i, S)
        batch.set_rhs(i, syn.randn_mf(rng, N, int(sizes[i]), 1)[:, :, 0])
    x, pullback = mf.batched.solve_spd_batched_rrule(batch)
    w = np.zeros((N, int(sizes.sum())))
    w[0] = rng.standard_normal(w.shape[1])
    sb, xb = pullback(torch.from_numpy(w).cuda())
    for i, S in enumerate(blocks):
        n, o = int(sizes[i]), int(batch.boffsets_host[i])
        L, _ = ref.potrf(S)
        bbar = ref.potrs(L, np.ascontiguousarray(w[:, o:o + n, None]))[:, :, 0]
        assert_bitwise(xb[:, o:o + n].cpu().numpy(), bbar, f"bbar {i}")
        xi, got = x[:, o:o + n].cpu().numpy(), batch.block(i, sb)
        outer = lambda a, b: ref.gemm(a[:, :, None], b[:, None, :], x3_fused=False)  # noqa: E731
        want = -0.5 * ref.to_double(outer(bbar, xi) + outer(xi, bbar))
        assert np.max(np.abs(ref.to_double(got) - want)) <= 2.0 ** -50 * np.max(np.abs(want))
