"""Split-precision products after writes through the operands' device pointers (needs a GPU).

The operators' packed copies are kept between products; what a caller writes through a
pointer that it got earlier has to be seen by the next product.  The result is compared with
that of new tensors that hold the same data: the same kernels on the same values, equal bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Array:
    def __init__(self, t):
        self.__cuda_array_interface__ = {"shape": (t.nnz,), "typestr": "<f8", "data": (t.device_ptr(), False),
                                         "version": 2}


def one_bit(x, i):
    x.view(dtype=__import__("torch").int64)[i] ^= 1 << 44


def swapped(x, i):
    a = x[i].clone()
    x[i] = x[i - 1]
    x[i - 1] = a


def negated(x, i):
    x[i] = -x[i]


@pytest.mark.parametrize("dims", [[1, 2], [40, 24, 33], [300, 200]], ids=["tiny", "small", "large"])
@pytest.mark.parametrize("op", [0, 1])
def test_writes_are_seen(dims, op):
    import torch

    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core
    from tests.fakecuda import operands

    ctx = core.Context(0)
    core.set_precision(ctx, core.SPLIT_TF32)
    ctx.set_sigma_schedule(0)
    rng = np.random.default_rng(len(dims))
    t = operands(core, ctx, dims)
    for x in t:
        x.upload(rng.standard_normal(x.nnz))

    def product(L, R, P):
        S = P.like()
        core.compute_sigma_vector(ctx, L, R, P, S)
        return S.download()

    held = torch.as_tensor(Array(t[op]), device="cuda")
    n = t[op].nnz
    last = product(*t)
    assert np.array_equal(product(*t), last)
    for write, i in ((one_bit, 0), (one_bit, n - 1), (negated, n // 2), (swapped, n - 1), (swapped, 1),
                     (lambda x, i: x.mul_(2.0), 0)):
        write(held, i)
        torch.cuda.synchronize()
        got = product(*t)
        new = operands(core, ctx, dims)
        for x, y in zip(new, t):
            x.upload(y.download())
        assert np.array_equal(got, product(*new))
        assert not np.array_equal(got, last)
        last = got
