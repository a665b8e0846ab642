"""FP64 products over the layouts that the calls accept, on either route, against the oracle
(needs a GPU): row sectors that repeat a quantum number, sectors without states.

Tolerance: Gaussian operands, sums of at most 3 x 241 products per contraction and two
contractions; either route keeps every sum to 2 K 2^-53 of (row maximum x column maximum) summed
over its K terms, and the largest results are above that sum divided by K: 1e-11 of the
largest element is far above it, one product left out or counted twice far beyond it.
"""
import numpy as np
import pytest

from tests.bondcase import to_dict

pytestmark = pytest.mark.gpu

FORMS = {
    "repeated": ([70, 3, 130, 41], [33, 64, 17, 20], [(0, 0), (0, 0), (1, 0), (0, 0)]),
    "repeated-columns": ([5, 9, 16], [40, 2, 7], [(1, 0), (0, 0), (1, 0)]),
    "plain": ([5, 9, 16], [40, 2, 7], [(0, 0), (1, 0), (2, 0)]),
    "empty": ([70, 0, 41], [33, 17, 0], [(0, 0), (1, 0), (2, 0)]),
    "one": ([1, 1], [1, 1], [(0, 0), (0, 0)]),
}


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core

    return core.Context(0)


def neg(q):
    return [(-a, -b) for a, b in q]


def bond(form, seed=0):
    """L, R, psi; sectors of psi's rows (columns) as given, empty blocks stored as well."""
    from oracle import qsd as oq

    da, db, qa = FORMS[form]
    n = len(da)
    qb = [(n - a, 0) for a, _ in qa]
    qw = [(0, 0), (1, 0), (-1, 0)]
    rng = np.random.default_rng(seed)
    out = []
    for q, qs, ds in (((0, 0), [qa, qw, neg(qa)], [da, [1] * 3, da]), ((0, 0), [qb, neg(qw), neg(qb)], [db, [1] * 3, db]),
                      ((n, 0), [qa, qb], [da, db])):
        a = oq.QSDArray(q, qs, ds)
        for i in np.ndindex(*[len(x) for x in qs]):
            if all(sum(x[k][c] for x, k in zip(qs, i)) == q[c] for c in range(2)):
                a.blocks[a.tag(i)] = rng.standard_normal([d[k] for d, k in zip(ds, i)])
        out.append(a)
    return out


def check(got, ref):
    top = max(np.abs(b).max() for b in ref.blocks.values() if b.size)
    assert {t for t, b in ref.blocks.items() if b.size and np.abs(b).max()} <= set(got)
    for t, b in got.items():
        assert np.all(np.abs(b - ref.blocks.get(t, 0.0)) <= 1e-11 * top), t


@pytest.mark.parametrize("route", [0.0, float("inf")], ids=["sliced", "pipe"])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_products(ctx, form, route):
    from oracle import dmrg as od
    from oracle import qsd as oq
    from mpsxx_gb300 import core

    ctx.set_fp64_route(route)
    L, R, P = bond(form)
    d = [core.Tensor.from_dict(ctx, to_dict(x)) for x in (L, R, P)]
    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    full = lambda x: oq.QSDArray(x.q, x.qshape, x.dshape)  # noqa: E731
    ref = oq.QSDArray()
    strip = []
    for x in (L, R, P):  # the oracle holds no empty blocks
        y = full(x)
        y.blocks = {t: b for t, b in x.blocks.items() if b.size}
        strip.append(y)
    od.compute_sigma_vector(*strip, ref)
    check(S.to_blocks(), ref)
    for forward, opr in ((True, 0), (False, 1)):
        q, dims = strip[opr].qshape[0], strip[opr].dshape[0]
        k = [(x + 2) // 3 for x in dims]
        u = full(strip[opr])
        u = oq.QSDArray((0, 0), [q, neg(q)], [dims, k]) if forward else oq.QSDArray((0, 0), [neg(q), q], [k, dims])
        u.allocate(0.0)
        rng = np.random.default_rng(5)
        u.blocks = {t: rng.standard_normal(b.shape) for t, b in u.blocks.items() if b.size}
        du = core.Tensor.from_dict(ctx, to_dict(u))
        got = core.renormalize(ctx, forward, d[opr], du, du)
        check(got.to_blocks(), od.renormalize_merged(forward, strip[opr], u, u))


@pytest.mark.parametrize("small, big", [(-470, 400), (-500, 400), (-560, 460), (-1000, 470), (-1060, 470)])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_rows_of_small_numbers(ctx, which, small, big):
    """Rows below the range of the digits (2^-480), down to subnormal numbers, are computed like any
    others: the FP64 pipe's result up to the rounding of sums of at most 16 and 3 x 40 terms, whose
    magnitudes are at most 16 times the largest result's."""
    from mpsxx_gb300 import core

    x = bond("plain", seed=3)
    rng = np.random.default_rng(which)
    for i, a in enumerate(x):
        e = {which: small, (which + 1) % 3: big}.get(i, 0)
        for t, b in a.blocks.items():
            row = np.ones(b.shape[0])
            if i == which:
                row[rng.random(b.shape[0]) < 0.3] = 0.0  # rows of zeros among them
            a.blocks[t] = np.ldexp(b, e) * row.reshape([-1] + [1] * (b.ndim - 1))
    res = []
    for route in (float("inf"), 0.0):
        ctx.set_fp64_route(route)
        d = [core.Tensor.from_dict(ctx, to_dict(a)) for a in x]
        S = d[2].like()
        core.compute_sigma_vector(ctx, *d, S)
        res.append(S.download())
    top = np.abs(res[0]).max()
    assert top > 0.0
    assert np.max(np.abs(res[1] - res[0])) <= 1e-13 * top
