"""Split-K partial tiles of the split-precision H_eff*psi (needs a GPU).

A slot holds column pairs over the tile's valid rows only, so the cases are odd row and
column counts, 64-row and compact column tails and slot counts around multiples of four.
Operands are integers of magnitude 2 at most: every sum stays an integer below 2^24 (2 x 2
x 130 after stage 1, x 2 x 130 x 9 after stage 2), which TF32 hi + lo, FP32 and FP64 sums all
hold exactly, so that results equal the oracle's.
"""
import numpy as np
import pytest

from tests.test_gpu_fp64_tensor import bond, dev

pytestmark = pytest.mark.gpu


def integers(rng, shape):
    return rng.integers(-2, 3, shape).astype(float)


@pytest.mark.parametrize("target", [1, 152 * 4, 1 << 20])
@pytest.mark.parametrize("db", [[1, 2, 31, 33], [63, 65, 15, 17], [127, 129, 128, 130]])
@pytest.mark.parametrize("nw", [3, 5])
def test_odd_tiles_in_slots(db, target, nw):
    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core
    from oracle import dmrg as od
    from oracle import qsd as oq

    ctx = core.Context(0)
    L, R, P = bond([65, 1, 129, 64], db, integers, seed=nw, nw=nw)
    ref = oq.QSDArray()
    od.compute_sigma_vector(L, R, P, ref)
    core.set_precision(ctx, core.SPLIT_TF32)
    ctx.set_sigma_schedule(0, target, False)
    p = dev(ctx, P)
    s = p.like()
    core.compute_sigma_vector(ctx, dev(ctx, L), dev(ctx, R), p, s)
    for t, b in s.to_blocks().items():
        assert np.array_equal(b, ref.blocks[t])
