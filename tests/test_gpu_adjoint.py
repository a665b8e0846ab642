"""dE/dW at the edges of the adjoint kernel's work split, against the oracle (needs a GPU).

E is linear in each MPO entry, so dE/dW_e is E with that entry 1 and the side's others 0.
Tolerance: both are FP64 sums whose terms pass through at most some 4000 additions in a row:
4000 x 2^-53 < 1e-12 of the same sum over magnitudes.
"""
import numpy as np
import pytest

from tests.test_gpu_merge_diag import dev, environment

pytestmark = pytest.mark.gpu


# blocks below and above a warp, the eight warps' 256 elements and four loads of each, ragged
# against 32 columns; one to some twenty entries meet a sub-block
@pytest.mark.parametrize("dl,dr", [([1, 2, 3, 5], [5, 1, 4, 2]), ([33, 1, 31, 4], [2, 17, 1, 9]),
                                   ([7, 64, 3, 40], [3, 2, 65, 1])])
def test_gradient_entries(dl, dr):
    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core
    from oracle import dmrg as od
    from oracle import qsd as oq

    ctx = core.Context(0)
    lm, le = environment(dl, True, 3)
    rm, re = environment(dr, False, 4)
    mL, mR = od.compute_merged_operator(True, lm, le), od.compute_merged_operator(False, rm, re)
    rng = np.random.default_rng(5)
    psi = oq.QSDArray((4, 0), [mL.qshape[0], mR.qshape[0]], [mL.dshape[0], mR.dshape[0]])
    psi.allocate(0.0)
    for t in psi.blocks:
        psi.blocks[t] = rng.standard_normal(psi.blocks[t].shape)
    norm = np.sqrt(sum(np.sum(b * b) for b in psi.blocks.values()))
    for t in psi.blocks:
        psi.blocks[t] /= norm
    assert len(psi.blocks) > 2

    def magnitudes(a):
        a = a.copy()
        for t in a.blocks:
            a.blocks[t] = np.abs(a.blocks[t])
        return a

    def energy(x, y, p):
        s = oq.QSDArray()
        od.compute_sigma_vector(x, y, p, s)
        return sum(np.sum(s.blocks[t] * p.blocks[t]) for t in p.blocks if t in s.blocks)

    def single(mpo, tag):
        one = mpo.copy()
        one.blocks = {tag: np.ones((1, 1, 1, 1))}
        return one

    grads = core.mpo_gradient(ctx, *[dev(ctx, x) for x in (lm, rm, le, re, psi)])
    for left, mpo, env, got in ((True, lm, le, grads[0]), (False, rm, re, grads[1])):
        for tag, g in zip(sorted(mpo.blocks), got):
            m = od.compute_merged_operator(left, single(mpo, tag), env)
            ops = (m, mR) if left else (mL, m)
            top = energy(*[magnitudes(x) for x in ops], magnitudes(psi))
            assert abs(g - energy(*ops, psi)) <= 1e-12 * top
