"""Errors of the sliced FP64 products element by element (needs a GPU), against sums in extended
precision.

An operand row is kept to half a unit of 2^-55 of a power of two above its largest magnitude,
and a group of products is rounded to half a unit of 2^-55 of the product of those powers of
two, so that a sum of K products is off by at most K 2^-53 of (row maximum x column maximum).
The maxima are those of the balanced operands: a contraction's elements are multiplied by powers
of two that bring the rows of the wavefunction (its columns, the rows of a renormalisation's
site tensors) to the same magnitude.
"""
import numpy as np
import pytest

from tests.bondcase import to_dict
from tests.test_gpu_fp64_forms import neg

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
DA, DB = [24, 40], [33, 17]
QA, QB, QW = [(0, 0), (1, 0)], [(2, 0), (1, 0)], [(0, 0), (1, 0), (-1, 0)]


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core

    c = core.Context(0)
    c.set_fp64_route(0.0)
    return c


def array(q, qs, ds, fill):
    from oracle import qsd as oq

    a = oq.QSDArray(q, qs, ds)
    a.allocate(0.0)
    for t in a.blocks:
        a.blocks[t] = fill(a.index(t), a.blocks[t].shape)
    return a


def operator(qs, ds, fill):
    return array((0, 0), [qs, QW if qs is QA else neg(QW), neg(qs)], [ds, [1] * 3, ds], fill)


def even(rng):
    """Magnitudes in [1/2, 1) of either sign."""
    return lambda i, shape: (0.5 + 0.5 * rng.random(shape)) * rng.choice([-1.0, 1.0], shape)


def ramp(n, decades):
    return 10.0 ** (-decades * np.arange(n) / max(1, n - 1))


def product(ctx, L, R, P):
    from mpsxx_gb300 import core

    d = [core.Tensor.from_dict(ctx, to_dict(x)) for x in (L, R, P)]
    S = d[2].like()
    core.compute_sigma_vector(ctx, *d, S)
    return S.to_blocks()


def exact(a, b):
    """a @ b in extended precision."""
    return (a.astype(np.longdouble)[:, :, None] * b.astype(np.longdouble)[None]).sum(1)


def power(x):
    """Exponent e with max |x| in [2^(e-1), 2^e) along the last axis; -127 for zeros."""
    m = np.abs(x).max(-1)
    return np.where(m > 0, np.clip(np.frexp(m)[1], -127, 127), -127)


def maxima(a, b, e):
    """(row maximum x column maximum) of a 2^e and 2^-e b."""
    return np.outer(np.abs(np.ldexp(a, e[None, :])).max(1), np.abs(np.ldexp(b, -e[:, None])).max(0))


def reference(L, R, P):
    """{tag: (result, sum of magnitudes, bound on the error)}."""
    out = {}
    by_row = {P.index(t)[0]: (P.index(t)[1], b) for t, b in P.blocks.items()}
    for tl, l in L.blocks.items():
        i, w, i2 = L.index(tl)
        j, (j2, p) = by_row[i][0], by_row[i2]
        r = R.blocks.get(R.tag((j, w, j2)))
        if r is None:
            continue
        l, r = l[:, 0, :], r[:, 0, :].T
        t = exact(l, p)
        tf = t.astype(np.float64)
        e1, e2 = power(p), power(p.T)
        err = l.shape[1] * U * maxima(l, p, e1) @ np.abs(r) + r.shape[0] * U * maxima(tf, r, -e2)
        x = out.setdefault(P.tag((i, j)), [0, 0, 0])
        x[0] = x[0] + exact(t, r)
        x[1] = x[1] + np.abs(l) @ np.abs(p) @ np.abs(r)
        x[2] = x[2] + 1.01 * err
    return out


@pytest.mark.parametrize("decades", [4, 8, 16])
@pytest.mark.parametrize("where", ["left", "right", "both"])
@pytest.mark.parametrize("falling", ["operator", "wavefunction", "wavefunction alone"])
def test_opposite_gradings(ctx, where, falling, decades):
    """Operator and wavefunction graded in opposite directions along a contraction: errors as
    without the gradings.  All balanced magnitudes are within 1/4 .. 1, so that (row maximum x
    column maximum) is at most 16/K of the sum of magnitudes: 16 U of it for each of the two
    contractions and 6 roundings of sums, below 40 U."""
    rng = np.random.default_rng(decades)
    L, R = operator(QA, DA, even(rng)), operator(QB, DB, even(rng))
    P = array((2, 0), [QA, QB], [DA, DB], even(rng))
    up = {"operator": -1.0, "wavefunction": 1.0, "wavefunction alone": 1.0}[falling]
    alone = falling.endswith("alone")
    if where != "right":
        for t, b in P.blocks.items():
            P.blocks[t] = b * ramp(b.shape[0], up * decades)[:, None]
        for t, b in L.blocks.items():
            L.blocks[t] = b if alone else b * ramp(b.shape[2], -up * decades)
    if where != "left":
        for t, b in P.blocks.items():
            P.blocks[t] = b * ramp(b.shape[1], up * decades)[None, :]
        for t, b in R.blocks.items():
            R.blocks[t] = b if alone else b * ramp(b.shape[2], -up * decades)
    ref = reference(L, R, P)
    got = product(ctx, L, R, P)
    for t, (x, mag, _) in ref.items():
        err = np.abs(got[t] - x).astype(np.float64)
        if alone:  # (the sums hold the gradings: their largest terms are a few)
            assert np.all(err <= 40 * 64 * U * mag)
        else:
            assert np.all(err <= 40 * U * mag)


def spread(rng):
    """Every element at its own magnitude over 30 decades, a third of them zero."""
    return lambda i, s: rng.standard_normal(s) * 10.0 ** (-30 * rng.random(s)) * (rng.random(s) < 0.67)


def unit(rng):
    """Identity blocks with noise."""

    def fill(i, s):
        x = 1e-17 * rng.standard_normal(s)
        if i[0] == i[-1]:
            x[:, 0, :] += np.eye(s[0])
        return x

    return fill


def graded(rng):
    """Rows and columns over eight decades in any order."""
    return lambda i, s: rng.standard_normal(s) * 10.0 ** (-8 * rng.random((s[0],) + (1,) * (len(s) - 1))) * 10.0 ** (
        -8 * rng.random(s[-1]))


@pytest.mark.parametrize("wave", [even, graded, spread])
@pytest.mark.parametrize("op", [even, graded, spread, unit])
def test_error_bound(ctx, op, wave):
    """The bound of this file's head, element by element, and 6 roundings of sums."""
    rng = np.random.default_rng(7)
    L, R = operator(QA, DA, op(rng)), operator(QB, DB, op(rng))
    P = array((2, 0), [QA, QB], [DA, DB], wave(rng))
    got = product(ctx, L, R, P)
    for t, (x, mag, bound) in reference(L, R, P).items():
        err = np.abs(got[t] - x).astype(np.float64)
        assert np.all(err <= bound + 6 * U * mag)


def test_small_element_met_by_a_zero(ctx):
    """[1, 2^-60] . [0, 1] is 2^-60."""
    one = lambda i, s: np.ones(s)  # noqa: E731
    L, R = operator(QA, [2, 1], one), operator(QB, [1, 1], one)
    P = array((2, 0), [QA, QB], [[2, 1], [1, 1]], lambda i, s: np.zeros(s))
    L.blocks[L.tag((0, 0, 0))][:, 0, :] = [1.0, 2.0 ** -60]
    P.blocks[P.tag((0, 0))][:, 0] = [0.0, 1.0]
    got = product(ctx, L, R, P)
    assert got[P.tag((0, 0))].ravel().tolist() == [2.0 ** -60] * 2


@pytest.mark.parametrize("decades", [4, 8, 16])
@pytest.mark.parametrize("falling", [1.0, -1.0])
@pytest.mark.parametrize("forward", [True, False])
def test_renormalisation_with_opposite_gradings(ctx, forward, falling, decades):
    """As test_opposite_gradings, for the two contractions with the site tensors."""
    from mpsxx_gb300 import core

    rng = np.random.default_rng(decades)
    q, d = (QA, DA) if forward else (QB, DB)
    O = operator(q, d, even(rng))
    k = [max(1, x // 3) for x in d]
    site = []
    for _ in range(2):
        u = (array((0, 0), [q, neg(q)], [d, k], even(rng)) if forward
             else array((0, 0), [neg(q), q], [k, d], even(rng)))
        for t, b in u.blocks.items():
            g = ramp(b.shape[0 if forward else 1], falling * decades)
            u.blocks[t] = b * (g[:, None] if forward else g[None, :])
        site.append(u)
    for t, b in O.blocks.items():
        O.blocks[t] = b * ramp(b.shape[0], -falling * decades)[:, None, None] * ramp(b.shape[2], -falling * decades)
    got = core.renormalize(ctx, forward, *[core.Tensor.from_dict(ctx, to_dict(x)) for x in (O, *site)])
    res = got.to_blocks()
    bra, ket = [{u.index(t)[0]: (b if forward else b.T) for t, b in u.blocks.items()} for u in site]
    n = 0
    for t, b in O.blocks.items():
        i, w, j = O.index(t)
        x = exact(exact(bra[i].T, b[:, 0, :]), ket[j])
        mag = np.abs(bra[i].T) @ np.abs(b[:, 0, :]) @ np.abs(ket[j])
        y = res[O.tag((i, w, j))][:, 0, :]
        assert np.all(np.abs(y - x).astype(np.float64) <= 40 * U * mag)
        n += 1
    assert n == len(res)
