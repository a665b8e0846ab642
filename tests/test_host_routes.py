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


def test_products_on_a_second_device():
    """Limits of shared memory that are raised for a kernel hold on one device only."""
    out = run("""
    fake.fake_devices(2)
    out = []
    for dev in (0, 1):
        ctx = core.Context(dev)
        ctx.set_fp64_route(0.0)
        L, R, P = operands(core, ctx)
        launches()
        for prec in (core.FP64, core.SPLIT_TF32):
            core.set_precision(ctx, prec)
            core.compute_sigma_vector(ctx, L, R, P, P.like())
        out.append(sorted({x.split()[1] for x in launches("%d " % dev)}))
    """)
    assert out[0] == out[1]
    assert any("gemm_oz_kernel" in x for x in out[1]) and any("gemm_pk_kernel" in x for x in out[1])


@pytest.mark.parametrize("kernel", ["gemm_oz", "oz_pack", "gemm_f64", "gemm_pk_kernel", "pack_kernel", "diag_kernel"])
def test_a_launch_that_fails_is_an_error(kernel):
    """Once the kernel can be launched the same calls succeed."""
    out = run(f"""
    ctx = core.Context(0)
    L, R, P = operands(core, ctx)
    def calls():
        bad = []
        for prec, route in ((core.FP64, 0.0), (core.FP64, float("inf")), (core.SPLIT_TF32, 0.0)):
            core.set_precision(ctx, prec)
            ctx.set_fp64_route(route)
            bad.append(error(core.compute_sigma_vector, ctx, L, R, P, P.like()))
        bad.append(error(core.compute_diagonal_elements, ctx, L, R, P.like()))
        return bad
    fake.fake_fail_launch({kernel!r}.encode())
    out = [calls()]
    fake.fake_fail_launch(b"")
    out.append(calls())
    """)
    assert 6 in out[0] and set(out[0]) <= {0, 6}
    assert out[1] == [0, 0, 0, 0]


def test_a_launch_that_fails_while_a_graph_is_captured():
    """The capture ends with the call; the next call captures again."""
    out = run("""
    ctx = core.Context(0)
    core.set_precision(ctx, core.SPLIT_TF32)
    ctx.set_sigma_schedule(1)
    L, R, P = operands(core, ctx, dims=(40, 24, 30))
    fake.fake_fail_launch(b"gemm_pk_kernel")
    out = [error(core.compute_sigma_vector, ctx, L, R, P, P.like())]
    fake.fake_fail_launch(b"")
    out.append(error(core.compute_sigma_vector, ctx, L, R, P, P.like()))
    out.append(len(launches("gemm_pk_kernel")))
    """)
    assert out[:2] == [6, 0] and out[2] > 2  # a pair of products for each group of w


def test_products_after_an_allocation_that_failed():
    """Whichever allocation of a sliced product fails, the call gives a result on the FP64 pipe or
    an allocation error, and the next one cuts all digits."""
    out = run("""
    out = []
    for k in range(40):
        L = R = P = S = ctx = None
        ctx = core.Context(0)
        ctx.set_fp64_route(0.0)
        empty_cache(ctx)
        L, R, P = operands(core, ctx, (300, 200), cols=(40, 300))
        S = P.like()
        launches()
        fake.fake_fail_alloc(k, 2)  # (an allocation is tried again after the cache is emptied)
        code = error(core.compute_sigma_vector, ctx, L, R, P, S)
        fake.fake_fail_alloc(0, 0)
        a = [x.split(None, 1)[1] for x in launches()]
        code2 = error(core.compute_sigma_vector, ctx, L, R, P, S)
        b = [x.split(None, 1)[1] for x in launches()]
        digits = lambda x: [int(y.split()[1]) for y in x if "oz_pack" in y]
        pipe = sum("gemm_f64" in y for y in a)
        out.append([code, pipe, digits(a), code2, digits(b)])
    """)
    failed = [x for x in out if x[0] or x[1]]
    assert len(failed) > 4 and any(x[1] for x in failed) and out[-1][:2] == [0, 0]
    for code, pipe, first, code2, second in out:
        assert code in (0, 2) and code2 == 0
        if code == 0:
            assert (pipe, first) in ((2, []), (0, [3, 1]))
        assert second == [3, 1]  # L, R and psi, then L psi


@pytest.mark.parametrize("precision, kernel", [("FP64", "oz_pack_kernel"), ("SPLIT_TF32", "pack_kernelEPKNS_5DPack")])
def test_operators_are_packed_anew_where_a_caller_may_have_written_them(precision, kernel):
    """Digits are cut in every call.  Packed split operators are kept; of a tensor whose device
    pointer was handed out the data may be other data in every call: it is packed anew where
    its fingerprint is another one (or none was taken of the packed data)."""
    out = run(f"""
    ctx = core.Context(0)
    core.set_precision(ctx, core.{precision})
    ctx.set_fp64_route(0.0)
    ctx.set_sigma_schedule(0)
    L, R, P = operands(core, ctx)
    S = P.like()
    packed = lambda: sum(int((x.split() + [1])[2]) for x in launches("{kernel}"))
    out = []
    for t, contents in ((None, 1), (None, 2), (L, 2), (None, 2), (None, 3), (R, 3), (None, 3), (None, 4)):
        if t:
            t.device_ptr()
        fake.fake_contents(contents)
        packed()
        core.compute_sigma_vector(ctx, L, R, P, S)
        out.append(packed())
    """)
    if precision == "FP64":
        assert [x - 1 for x in out] == 8 * [3]  # (and the packing of L psi)
    else:
        assert out == [3, 1, 2, 1, 2, 2, 1, 3]


def test_memory_of_the_digits():
    """One bond's digits at most are held, and only until memory is short; a product without
    memory for them runs on the FP64 pipe."""
    out = run("""
    ctx = core.Context(0)
    ctx.set_fp64_route(0.0)
    empty_cache(ctx)
    bonds = [operands(core, ctx, (400 - 30 * k, 60 * k + 20)) for k in range(5)]
    small = operands(core, ctx, (9, 30))
    def product(b):
        launches()
        code = error(core.compute_sigma_vector, ctx, *b, b[2].like())
        ran = launches()
        return [code] + [sum(k in x for x in ran) for k in ("gemm_oz", "gemm_f64")]
    bonds.sort(key=lambda b: -b[0].nnz - b[1].nnz)
    product(small)
    used = [fake.fake_used()]
    runs = [product(bonds[0])]
    used.append(fake.fake_used())
    runs += [product(b) for b in bonds + bonds[::-1]]
    used.append(fake.fake_used())
    # a tensor for which there is room only where the digits were
    fake.fake_limit(fake.fake_used())
    n = 14 * (bonds[0][0].nnz + bonds[0][1].nnz)  # L's and R's digits
    t = core.Tensor.create(ctx, (0, 0), [[(0, 0)]], [[n // 8]])
    short = product(bonds[0])
    fake.fake_limit(0)
    out = [runs, used, short, product(bonds[0])]
    """)
    runs, used, short, after = out
    assert runs == 11 * [[0, 2, 0]]
    assert used[2] - used[1] < (used[1] - used[0]) // 4  # the other nine products add no digits
    assert short == [0, 0, 2] and after == [0, 2, 0]
