"""Which kernels a call runs, and what it does when a step of it fails, without a device
(tests/fake_cuda.cpp)."""
import pytest

from tests.fakecuda import run


@pytest.mark.parametrize("dims, cols, qrow", [([5, 3, 4], [2, 6, 7], [(0, 0), (0, 0), (1, 0)]), ([5, 0, 4], [2, 6, 7], None)],
                         ids=["repeated", "empty"])
def test_wavefunctions_that_do_not_stack_take_the_general_path(dims, cols, qrow):
    """Row sectors that repeat a quantum number give an L psi block several pairs, an empty
    one leaves L psi blocks without any."""
    out = run(f"""
    ctx = core.Context(0)
    ctx.set_fp64_route(0.0)
    L, R, P = operands(core, ctx, {dims}, cols={cols}, qrow={qrow})
    launches()
    out = [error(core.compute_sigma_vector, ctx, L, R, P, P.like()), len(launches("gemm_f64"))]
    """)
    assert out == [0, 2]
