"""Merged operators and diagonals at the edges of their kernels' tiles, against the oracle
(needs a GPU).  A merged element is a sum of at most 16 products and a diagonal one of at most
40: FP64 sums in another order agree to 40 x 2^-53 of the sum of magnitudes, below 1e-14 of
the products of the largest magnitudes times the number of terms."""
import numpy as np
import pytest

from tests.bondcase import to_dict

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core

    return core.Context(0)


def dev(ctx, a):
    from mpsxx_gb300 import core

    return core.Tensor.from_dict(ctx, to_dict(a))


def environment(dims, left, seed):
    """An environment with bond sectors of the given dimensions and a site MPO with some of the
    allowed entries, coefficients of 1 and -1 among them."""
    from oracle import qsd as oq

    rng = np.random.default_rng(seed)
    site = [(0, 0), (1, 1), (1, -1), (2, 0)]
    neg = lambda q: [(-x, -y) for x, y in q]  # noqa: E731
    q = [(i, i % 2) for i in range(len(dims))]
    w = [(0, 0), (0, 0), (1, 1), (-1, -1), (1, -1), (-1, 1)]
    v = w + [(2, 0), (-2, 0)]
    a, b = (w, v) if left else (v, w)
    mpo = oq.QSDArray((0, 0), [a, site, neg(site), neg(b)], [[1] * len(a), [1] * 4, [1] * 4, [1] * len(b)])
    mpo.allocate(0.0)
    for t in list(mpo.blocks):
        if rng.random() < 0.4:
            del mpo.blocks[t]
        else:
            mpo.blocks[t] = np.full((1, 1, 1, 1), rng.choice([1.0, -1.0, rng.standard_normal()]))
    mid = neg(a) if left else b
    env = oq.QSDArray((0, 0), [q, mid, neg(q)], [dims, [1] * len(mid), dims])
    env.allocate(0.0)
    for t in list(env.blocks):
        if rng.random() < 0.2:
            del env.blocks[t]  # sub-blocks without a source
        else:
            env.blocks[t] = rng.standard_normal(env.blocks[t].shape)
    return mpo, env


@pytest.mark.parametrize("left", [True, False])
@pytest.mark.parametrize("dims", [[1, 2, 3, 5], [4, 31, 1, 33], [32, 128, 7, 12], [130, 3, 64, 1]])
def test_merged_operator_edges(ctx, dims, left):
    from oracle import dmrg as od
    from mpsxx_gb300 import core

    mpo, env = environment(dims, left, len(dims) + dims[1])
    ref = od.compute_merged_operator(left, mpo, env)
    for _ in range(2):  # the second result reuses the first one's memory
        got = core.compute_merged_operator(ctx, left, dev(ctx, mpo), dev(ctx, env))
        tags, _ = got.blocks()
        assert list(tags) == sorted(ref.blocks)
        top = 16 * max(np.abs(b).max() for b in env.blocks.values()) * max(np.abs(b).max() for b in mpo.blocks.values())
        for t, b in got.to_blocks().items():
            assert np.max(np.abs(b - ref.blocks[t])) <= 1e-14 * top
        junk = got.like()
        junk.upload(np.full(got.nnz, 7.0))
        del got, junk


@pytest.mark.parametrize("da,db", [([1, 2, 3], [1, 5, 4]), ([31, 64, 65], [33, 1, 2]), ([1, 7, 130], [3, 130, 1]),
                                   ([9, 257, 8], [17, 16, 32])])
def test_diagonal_edges(ctx, da, db):
    from oracle import dmrg as od
    from oracle import qsd as oq
    from mpsxx_gb300 import core

    rng = np.random.default_rng(da[1])
    n = len(da)
    qa, qb = [(i, 0) for i in range(n)], [(n - i, 0) for i in range(n)]
    neg = lambda q: [(-x, -y) for x, y in q]  # noqa: E731
    w = [(0, 0)] * 37 + [(1, 0), (-1, 0)]  # two stages of pairs
    L = oq.QSDArray((0, 0), [qa, w, neg(qa)], [da, [1] * len(w), da])
    R = oq.QSDArray((0, 0), [qb, neg(w), neg(qb)], [db, [1] * len(w), db])
    P = oq.QSDArray((n, 0), [qa, qb], [da, db])
    for a in (L, R, P):
        a.allocate(0.0)
        for t in a.blocks:
            a.blocks[t] = rng.standard_normal(a.blocks[t].shape)
    D = dev(ctx, P)
    D.upload(np.zeros(D.nnz))
    core.compute_diagonal_elements(ctx, dev(ctx, L), dev(ctx, R), D)
    ref = P.empty_like()
    od.compute_diagonal_elements(L, R, ref)
    top = 40 * 25.0
    for t, b in D.to_blocks().items():
        assert np.max(np.abs(b - ref.blocks.get(t, np.zeros_like(b)))) <= 1e-14 * top
