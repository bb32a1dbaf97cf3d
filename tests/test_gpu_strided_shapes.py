"""Reductions and element-wise products around the edges of their thread layouts: a handful of kept elements
under a long range and the other way round, short inner runs, unit stride on either side, several
slices, misaligned and odd rows.

Sums: any order of n terms is off by at most n - 1 roundings of the sum of magnitudes (one more for
alpha).  Max and Min are exact, products take one rounding (four of |x||y| for a complex one)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def eps(dtype):
    return np.finfo(np.dtype(dtype)).eps / 2


@pytest.mark.parametrize("shape,kept", [
    ((1,), []), ((257,), []), ((100003,), []), ((5, 70001), [0]), ((70001, 5), [0]), ((3, 4099, 7), [0, 2]),
    ((25, 8, 513), [1, 2]), ((27, 38, 1191), [1]), ((12, 56, 881, 17), [0, 3]), ((9, 40, 33), [0, 2]),
    ((63, 300), [1]), ((64, 2049), [1]), ((2048, 65), [1]), ((129, 2, 130), [0, 2]), ((600, 700), [0]),
])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("turned", [False, True])
def test_reduce_layouts(tb, oracle, shape, kept, dtype, turned):
    x = oracle.normal(3, shape, dtype)
    t = tb.Tensor.from_numpy(x)
    if turned:  # reversed index order: the unit stride changes sides
        order = list(range(len(shape)))[::-1]
        t, x = t.permute(order), x.transpose(order)
        kept = [len(shape) - 1 - k for k in kept][::-1]
    axes = tuple(i for i in range(x.ndim) if i not in kept)
    out_shape = tuple(x.shape[i] for i in kept)
    ops = ["Sum"] if np.dtype(dtype).kind == "c" else ["Sum", "Max", "Min"]
    if not axes:
        return
    for op in ops:
        c = oracle.normal(4, out_shape or (1,), dtype).reshape(out_shape)
        out = tb.Tensor.from_numpy(c)
        plan = tb.CudaBackend.plan(tb.PrimDescriptor.Reduce(list(range(x.ndim)), kept, tb.ReduceOp[op]), [x.shape, out_shape], dtype)
        beta = 0.5 if op == "Sum" else 0.0
        tb.CudaBackend.execute(plan, 1.0, [t], beta, out)
        got = out.to_numpy()
        if op == "Sum":
            wide = np.complex128 if np.dtype(dtype).kind == "c" else np.float64
            n = x.size // max(1, got.size)
            bound = 2 * (n + 2) * eps(dtype) * (abs(x).astype(np.float64).sum(axis=axes) + 0.5 * abs(c))
            assert (abs(got - (x.astype(wide).sum(axis=axes) + 0.5 * c.astype(wide))) <= bound).all()
        else:
            assert np.array_equal(got, x.max(axis=axes) if op == "Max" else x.min(axis=axes))


@pytest.mark.parametrize("special", [-np.inf, np.nan, np.finfo(np.float64).min])
def test_max_of_special_values(tb, special):
    x = np.full((300, 41), special)
    x[7, 5] = np.finfo(np.float64).min if special == -np.inf else special
    out = tb.Tensor.from_numpy(np.zeros(41))
    plan = tb.CudaBackend.plan(tb.PrimDescriptor.Reduce([0, 1], [1], tb.ReduceOp.Max), [x.shape, (41,)], np.float64)
    tb.CudaBackend.execute(plan, 1.0, [tb.Tensor.from_numpy(x)], 0.0, out)
    assert np.array_equal(out.to_numpy(), x.max(axis=0), equal_nan=True)


@pytest.mark.parametrize("special", [-np.inf, np.inf, np.nan, np.finfo(np.float64).min])
@pytest.mark.parametrize("shape,kept", [((300001, 3), 1), ((3, 300001), 0)])
@pytest.mark.parametrize("op", ["Max", "Min"])
def test_special_values_in_slices(tb, special, shape, kept, op):
    """Few kept elements under a long range: several slices and the launch that combines them."""
    x = np.full(shape, special)
    rows = x if kept == 1 else x.T
    rows[:, 1] = np.arange(300001.0)
    rows[150000, 1] = special  # one special value among ordinary ones, somewhere in the middle
    rows[299999, 2] = 1.0  # and the other way round, in the last slice
    out = tb.Tensor.from_numpy(np.zeros(3))
    plan = tb.CudaBackend.plan(tb.PrimDescriptor.Reduce([0, 1], [kept], tb.ReduceOp[op]), [x.shape, (3,)], np.float64)
    plan.ctx.profile_begin()
    tb.CudaBackend.execute(plan, 1.0, [tb.Tensor.from_numpy(x)], 0.0, out)
    plan.ctx.synchronize()
    assert plan.ctx.profile_read("reduce_finish")[0] == 1
    plan.ctx.profile_end()
    want = (np.max if op == "Max" else np.min)(rows, axis=0)
    assert np.array_equal(out.to_numpy(), want, equal_nan=True)


@pytest.mark.parametrize("notation", ["asb,b->asb", "a,asb->asb", "asb,asb->asb", "asb,a->asb", "asb,bsa->asb", "asb,s->asb"])
@pytest.mark.parametrize("size", [(1, 1, 1), (4, 2, 8), (33, 3, 65), (64, 2, 130), (1025, 4, 31)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("beta,offset", [(0.0, 0), (0.5, 1)])
def test_elementwise_layouts(tb, oracle, notation, size, dtype, beta, offset):
    ext = dict(zip("asb", size))
    ins, out_labels = notation.split("->")
    arrays = [oracle.normal(5 + i, [ext[c] for c in t], dtype) for i, t in enumerate(ins.split(","))]
    c = oracle.normal(8, [ext[l] for l in out_labels], dtype)

    def put(x):  # `offset` elements into a buffer: rows lose their 16-byte alignment
        flat = np.concatenate([np.zeros(offset, x.dtype), x.reshape(-1, order="F"), np.zeros(3, x.dtype)])
        whole = tb.Tensor.from_numpy(flat)
        strides, acc = [], 1
        for d in x.shape:
            strides.append(acc)
            acc *= d
        return tb.Tensor(whole._block, x.shape, strides, offset, x.dtype, whole.logical_memory_space())

    ops = [put(x) for x in arrays]
    out = put(c)
    if np.dtype(dtype).kind == "c":
        ops[1], arrays[1] = ops[1].into_conj(), arrays[1].conj()
    tb.einsum_into(notation, ops, 1.0, beta, out)
    wide = np.complex128 if np.dtype(dtype).kind == "c" else np.float64
    prod = np.einsum(notation, *[x.astype(wide) for x in arrays])
    bound = 8 * eps(dtype) * (np.einsum(notation, *[abs(x).astype(np.float64) for x in arrays]) + abs(beta) * abs(c))
    assert (abs(out.to_numpy() - (prod + beta * c.astype(wide))) <= bound).all()


@pytest.mark.parametrize("shape,perm", [
    ((5, 7), (1, 0)), ((3, 5, 7, 2, 9), (4, 3, 2, 1, 0)), ((14, 9, 15, 10, 11), (4, 2, 3, 1, 0)), ((33, 65, 7), (2, 0, 1)),
    ((11, 13, 9, 7, 5), (0, 4, 1, 2, 3)), ((2, 300, 3, 70), (0, 3, 2, 1)), ((2, 129, 257), (0, 2, 1)), ((257, 2), (1, 0)),
    ((1000, 3, 2), (2, 1, 0)), ((64, 64, 3), (1, 2, 0)), ((68, 132), (1, 0)), ((3, 6, 30, 33, 2, 3), (1, 2, 4, 3, 5, 0)),
    ((1, 513, 1, 70), (3, 2, 1, 0)), ((70, 71, 72), (0, 2, 1)), ((600, 601), (1, 0)),
])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("padded", [False, True])
def test_permute_orders(tb, oracle, shape, perm, dtype, padded):
    x = oracle.normal(6, shape, dtype)
    dims = [shape[i] for i in perm]
    if padded:  # gaps between the columns on both sides, last index of the output reversed
        big = np.zeros([d + 1 for d in shape], x.dtype)
        big[tuple(slice(0, d) for d in shape)] = x
        base = tb.Tensor.from_numpy(big)
        t = tb.Tensor(base._block, shape, base.strides(), 0, x.dtype, base.logical_memory_space())
        hold = tb.Tensor.from_numpy(np.full([d + 2 for d in dims], 7, x.dtype))
        strides = list(hold.strides())
        strides[-1] = -strides[-1]
        out = tb.Tensor(hold._block, dims, strides, (dims[-1] - 1) * -strides[-1], x.dtype, hold.logical_memory_space())
    else:
        t, out = tb.Tensor.from_numpy(x), tb.Tensor.from_numpy(np.zeros(dims, x.dtype))
    for alpha, beta in ((1.0, 0.0), (2.0, -1.0)):
        plan = tb.CudaBackend.plan(tb.PrimDescriptor.Permute(list(range(len(shape))), list(perm)), [shape, dims], dtype)
        tb.CudaBackend.execute(plan, alpha, [t], beta, out)
    # 2 x - x is exact
    want = x.transpose(perm)
    if padded:
        got = hold.to_numpy()
        inside = tuple(slice(0, d) for d in dims)
        assert np.array_equal(got[inside][..., ::-1], want)
        got[inside] = 7
        assert (got == 7).all()  # nothing between the columns was written
    else:
        assert np.array_equal(out.to_numpy(), want)


# Large enough for tiles of grouped modes, and what other paths take: (shape, order, types on tiles)
EVERY = (np.float32, np.float64, np.complex64, np.complex128)


@pytest.mark.parametrize("shape,perm,on_tiles", [
    ((14, 89, 15, 10, 3), (4, 2, 3, 1, 0), EVERY), ((27, 9, 68, 24, 2), (4, 1, 3, 0, 2), EVERY), ((5, 70001, 2), (1, 2, 0), EVERY),
    ((1000, 3, 6, 40), (2, 1, 3, 0), EVERY), ((3, 5, 7, 11, 13, 31), (5, 4, 3, 2, 1, 0), EVERY),
    ((3, 40, 1200, 9), (0, 3, 2, 1), EVERY[1:]),  # short rows far apart
    ((3, 9, 1200, 40), (0, 2, 1, 3), ()), ((701, 803), (1, 0), ()),
])
@pytest.mark.parametrize("dtype", EVERY)
@pytest.mark.parametrize("padded", [False, True])
def test_permute_tiles(tb, oracle, shape, perm, on_tiles, dtype, padded):
    ctx = tb.Context.get(0)
    ctx.profile_begin()
    test_permute_orders(tb, oracle, shape, perm, dtype, padded)
    ran = ctx.profile_read("permute_tile")[0]
    ctx.profile_end()
    assert ran == (2 if dtype in on_tiles else 0)


@pytest.mark.parametrize("shape,kept", [((20, 29, 13, 32), [0, 1]), ((119, 62, 465), [1]), ((31, 2003, 23), [0, 2]), ((5000, 40), [1]), ((200, 200), [])])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex128])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_slices_combined_by_the_last_block(tb, oracle, shape, kept, dtype, beta):
    """Sums over whole numbers, exact in every type and order, three times over the same counters."""
    x = oracle.normal(5, shape, np.float64).round().astype(dtype)
    gone = tuple(i for i in range(len(shape)) if i not in kept)
    c = np.arange(np.prod([shape[i] for i in kept], dtype=int), dtype=dtype).reshape([shape[i] for i in kept])
    plan = tb.CudaBackend.plan(tb.PrimDescriptor.Reduce(list(range(len(shape))), kept, tb.ReduceOp.Sum), [shape, c.shape], dtype)
    held = tb.Tensor.from_numpy(x)
    for _ in range(3):
        out = tb.Tensor.from_numpy(c)
        tb.CudaBackend.execute(plan, 2.0, [held], beta, out)
        assert np.array_equal(out.to_numpy(), 2 * x.sum(axis=gone) + dtype(beta) * c)
