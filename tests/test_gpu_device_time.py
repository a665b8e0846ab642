"""Device times of H_eff*psi (needs a GPU)."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "SPLIT_TF32"])
def test_no_time_of_a_product_that_gave_up(precision):
    """Kernels whose wait limit runs out return early: DEVICE_TIMEOUT, not a time."""
    import __graft_entry__

    __graft_entry__.build()
    from mpsxx_gb300 import core
    from mpsxx_gb300._lib import MpsxxError, check, lib
    from tests.fakecuda import operands

    ctx = core.Context(0)
    ctx.set_fp64_route(0.0)
    ctx.set_sigma_schedule(0)
    core.set_precision(ctx, getattr(core, precision))
    L, R, P = operands(core, ctx, (200, 100))
    S = P.like()
    sec = C.c_double(-1.0)
    time = lambda: check(lib().mpsxx_sigma_device_time(ctx.h, L.h, R.h, P.h, S.h, 2, C.byref(sec)))  # noqa: E731
    ctx.set_device_timeout(1)
    with pytest.raises(MpsxxError) as e:
        time()
    assert e.value.code == 4 and sec.value == -1.0
    ctx.set_device_timeout()
    time()
    assert sec.value > 0.0
