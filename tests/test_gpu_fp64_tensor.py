"""FP64 products on the tensor cores (error-free slicing) against the oracle (needs a GPU).

Tolerance: an operand element is kept to 2^-56 of its row's power-of-two scale, which is at
most twice the row's largest magnitude, and dropped digit products are below that; FP64
sums of K terms (the oracle's) are off by at most K 2^-53 of the sum of magnitudes.  Both
stay below 4 K 2^-53 of (row maximum x column maximum) summed over the K terms, with
K <= 1200 here: 6e-13 of the product of the largest magnitudes.
"""
import numpy as np
import pytest

from tests.bondcase import to_dict

pytestmark = pytest.mark.gpu

# edges of the 128/64-row and 32/16-column tiles, of the 16-wide K slices and of the
# 160-long exact groups
EDGES = [1, 15, 16, 17, 33, 63, 64, 65, 127, 128, 129, 160, 161, 200]


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core

    c = core.Context(0)
    c.set_fp64_route(0.0)
    return c


def dev(ctx, a):
    from mpsxx_gb300 import core

    return core.Tensor.from_dict(ctx, to_dict(a))


def bond(da, db, fill, seed=0, nw=3):
    """Merged operators and wavefunction with row sectors of dimensions da, db."""
    from oracle import qsd as oq

    rng = np.random.default_rng(seed)
    n = len(da)
    qa, qb = [(i, 0) for i in range(n)], [(n - i, 0) for i in range(n)]
    qw = [(0, 0)] + [(s * k, 0) for k in range(1, nw) for s in (1, -1)]
    neg = lambda q: [(-x, -y) for x, y in q]  # noqa: E731
    one = [1] * len(qw)
    L = oq.QSDArray((0, 0), [qa, qw, neg(qa)], [da, one, da])
    R = oq.QSDArray((0, 0), [qb, neg(qw), neg(qb)], [db, one, db])
    P = oq.QSDArray((n, 0), [qa, qb], [da, db])
    for a in (L, R, P):
        a.allocate(0.0)
        for t in a.blocks:
            a.blocks[t] = fill(rng, a.blocks[t].shape)
    return L, R, P


def gauss(rng, shape):
    return rng.standard_normal(shape)


def decaying(rng, shape):
    """Rows and columns over eight decades, some rows zero, a constant block now and then."""
    x = rng.standard_normal(shape)
    for ax in (0, len(shape) - 1):
        s = [1] * len(shape)
        s[ax] = shape[ax]
        x = x * (10.0 ** (-8 * rng.random(shape[ax]))).reshape(s)
    x[rng.random(shape[0]) < 0.1] = 0.0
    return np.full(shape, 1.0 / 3.0) if rng.random() < 0.2 else x


def constant(rng, shape):
    """The largest digits everywhere: the longest exact sums."""
    return np.full(shape, np.nextafter(1.0, 0.0) * rng.choice([1.0, -1.0]))


def scaled(rng, shape):
    """Magnitudes far from 1 in every row."""
    x = rng.standard_normal(shape)
    e = rng.integers(-140, 140, shape[0])
    return np.ldexp(x, e.reshape([-1] + [1] * (len(shape) - 1)))


FILLS = {f.__name__: f for f in (gauss, decaying, constant, scaled)}


@pytest.mark.parametrize("fill", sorted(FILLS))
@pytest.mark.parametrize("dims", [(EDGES, EDGES[::-1]), ([3], [170]), ([321], [5]), ([1, 1, 2], [1, 3, 1])],
                         ids=["edges", "wide", "tall", "tiny"])
def test_sigma_matches_oracle(ctx, dims, fill):
    from oracle import dmrg as od
    from oracle import qsd as oq
    from mpsxx_gb300 import core

    L, R, P = bond(list(dims[0]), list(dims[1]), FILLS[fill], seed=len(fill))
    d = [dev(ctx, x) for x in (L, R, P)]
    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    ref = oq.QSDArray()
    od.compute_sigma_vector(L, R, P, ref)
    got = S.to_blocks()
    if fill == "scaled":
        # rows of very different scale meet in one sum: compare with the sum of magnitudes
        mag = oq.QSDArray()
        ab = [x.copy() for x in (L, R, P)]
        for x in ab:
            for t in x.blocks:
                x.blocks[t] = np.abs(x.blocks[t])
        od.compute_sigma_vector(*ab, mag)
        K = 3 * max(map(max, dims))
        for t, b in got.items():
            # (a column scale is the column's largest magnitude, met by every row)
            top = mag.blocks[t].max()
            assert np.max(np.abs(b - ref.blocks[t])) <= 4 * K * 2.0 ** -53 * top
    else:
        top = max(np.abs(b).max() for b in ref.blocks.values())
        assert max(np.max(np.abs(b - ref.blocks[t])) for t, b in got.items()) <= 6e-13 * top
    core.compute_sigma_vector(ctx, *d, S)  # accumulates
    for t, b in S.to_blocks().items():
        assert np.allclose(b, 2 * got[t], rtol=1e-15, atol=0.0)


def test_sum_that_rounds_up_to_a_power_of_two(ctx):
    """1 - 2^-53 + 0.75 2^-53 is 1 - 2^-55, whose nearest double is 1; twice the terms, 2."""
    from mpsxx_gb300 import core

    L, R, P = bond([4], [1], lambda rng, shape: np.zeros(shape), nw=1)
    a, b = np.nextafter(1.0, 0.0), 0.75 * 2.0 ** -53
    (tl,), (tr,), (tp,) = L.blocks, R.blocks, P.blocks
    L.blocks[tl][:, 0, :] = [[a, b, 0, 0], [0, 0, b, a], [a, b, a, b], [-a, -b, 0, 0]]
    R.blocks[tr][...] = 1.0
    P.blocks[tp][...] = 1.0
    d = [dev(ctx, x) for x in (L, R, P)]
    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    assert S.download().tolist() == [1.0, 1.0, 2.0, -1.0]


@pytest.mark.parametrize("forward", [True, False])
@pytest.mark.parametrize("fill", ["gauss", "decaying"])
def test_renormalize_matches_oracle(ctx, forward, fill):
    from oracle import dmrg as od
    from oracle import qsd as oq
    from mpsxx_gb300 import core

    L, R, _ = bond(EDGES, EDGES[::-1], FILLS[fill], seed=3)
    opr = L if forward else R
    q, d = opr.qshape[0], opr.dshape[0]
    rng = np.random.default_rng(9)
    k = [max(1, x // 3) for x in d]
    site = []
    for _ in range(2):  # a ket distinct from the bra
        if forward:
            u = oq.QSDArray((0, 0), [q, [(-a, -b) for a, b in q]], [d, k])
        else:
            u = oq.QSDArray((0, 0), [[(-a, -b) for a, b in q], q], [k, d])
        u.allocate(0.0)
        for t in u.blocks:
            u.blocks[t] = FILLS[fill](rng, u.blocks[t].shape)
        site.append(u)
    got = core.renormalize(ctx, forward, dev(ctx, opr), dev(ctx, site[0]), dev(ctx, site[1]))
    ref = od.renormalize_merged(forward, opr, *site)
    tags, _ = got.blocks()
    assert list(tags) == sorted(ref.blocks)
    top = max(np.abs(b).max() for b in ref.blocks.values())
    assert max(np.max(np.abs(b - ref.blocks[t])) for t, b in got.to_blocks().items()) <= 6e-13 * top


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 2.0 ** 500])
def test_values_without_digits(ctx, bad):
    """Operands that cannot be sliced give what FP64 arithmetic gives."""
    from mpsxx_gb300 import core

    L, R, P = bond([5, 40], [33, 7], gauss, seed=1)
    for x, t in ((L, 1), (R, 2), (P, 0)):
        y = x.copy()
        tag = sorted(y.blocks)[t]
        y.blocks[tag].reshape(-1)[3] = bad
        ops = [y if z is x else z for z in (L, R, P)]
        res = []
        for route in (float("inf"), 0.0):
            ctx.set_fp64_route(route)
            d = [dev(ctx, z) for z in ops]
            S = d[2].like()
            core.compute_sigma_vector(ctx, *d, S)
            res.append(S.download())
        fin = np.isfinite(res[0])
        assert np.array_equal(fin, np.isfinite(res[1]))
        assert np.array_equal(np.isnan(res[0]), np.isnan(res[1]))
        if fin.any():
            s = np.abs(res[0][fin]).max()
            assert np.max(np.abs(res[0][fin] - res[1][fin])) <= 1e-12 * s


def test_operand_written_through_its_pointer(ctx):
    """A product reads the operands' current data, also what a caller wrote there itself."""
    import torch
    from mpsxx_gb300 import core

    L, R, P = bond([20, 40], [33, 17], gauss, seed=2)
    d = [dev(ctx, z) for z in (L, R, P)]

    class Array:
        def __init__(self, t):
            self.__cuda_array_interface__ = {"shape": (t.nnz,), "typestr": "<f8", "data": (t.device_ptr(), False),
                                             "version": 2}

    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    first = S.download()
    for t in d[:2]:
        torch.as_tensor(Array(t), device="cuda").mul_(2.0)
    torch.cuda.synchronize()
    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    assert np.array_equal(S.download(), 4.0 * first)
    core.accumulate(ctx, 1.0, d[0], d[0].like())
    acc = d[0].like()
    core.accumulate(ctx, 3.0, d[0], acc)
    S = d[2].like()
    core.compute_sigma_vector(ctx, acc, d[1], d[2], S)
    core.accumulate(ctx, -2.0, d[0], acc)  # the operand changes again: 1 x L
    S2 = d[2].like()
    core.compute_sigma_vector(ctx, acc, d[1], d[2], S2)
    assert np.max(np.abs(S.download() - 3.0 * S2.download())) <= 1e-12 * np.abs(S.download()).max()


def test_wait_limit(ctx):
    """Waits that run out give DEVICE_TIMEOUT; the context computes correctly afterwards."""
    from mpsxx_gb300 import core
    from mpsxx_gb300._lib import MpsxxError

    L, R, P = bond([100, 200], [50, 90], gauss, seed=4)
    d = [dev(ctx, z) for z in (L, R, P)]
    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    ref = S.download()
    ctx.set_device_timeout(1)
    with pytest.raises(MpsxxError) as e:
        core.compute_sigma_vector(ctx, *d, d[2].like())
    assert e.value.code == 4
    ctx.set_device_timeout()
    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    assert np.array_equal(S.download(), ref)
