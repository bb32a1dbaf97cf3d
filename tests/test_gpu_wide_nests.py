"""Strided kernels over more than 2^31 elements, where offsets and walks are kept in 64 bits.  Inputs are broadcast
views of small buffers.

Sums are exact whatever their order: the terms are integers and every partial sum is below 2^53 (f64) or 2^24 (f32).
Max and Min are exact."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def broadcast_view(tb, rng, dims, strides, dtype):
    """A buffer of small integers (f32: a few ones) under the given strides: (tensor, its part without the
    broadcast modes as an array, the number of times each of its elements is read)."""
    live = [d if s else 1 for d, s in zip(dims, strides)]
    first = sum((d - 1) * -s for d, s in zip(dims, strides) if s < 0)
    n = first + 1 + sum((d - 1) * s for d, s in zip(dims, strides) if s > 0)
    buf = rng.integers(0, 1000, n).astype(dtype)
    if dtype == np.float32:
        buf = np.zeros(n, dtype)
        buf[rng.choice(n, 5)] = 1
    whole = tb.Tensor.from_numpy(buf)
    view = tb.Tensor(whole._block, dims, strides, first, dtype, whole.logical_memory_space())
    it = buf.itemsize
    host = np.lib.stride_tricks.as_strided(buf[first:], live, [s * it for s in strides])
    return view, host, math.prod(d for d, s in zip(dims, strides) if not s)


@pytest.mark.parametrize("dims,strides,kept", [
    ([70001, 40000], [1, 0], []),
    ([46341, 46400], [-1, 0], []),
    ([1001, 1500, 1500], [1, 1002, 0], []),
    ([300, 300, 200, 120], [1, 301, 0, 90601], []),
    ([7, 1000, 320000], [1, 8, 0], []),
    ([3, 5, 7, 11, 13, 150000], [1, 4, 24, 200, 2400, 0], []),
    ([2, 33000, 66000], [1, 3, 0], [0]),
    ([1300, 1300, 1300, 2], [1, 1301, 0, 1692601], [3]),
])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_reduce(tb, dims, strides, kept, dtype):
    assert math.prod(d for i, d in enumerate(dims) if i not in kept) >= 2**31 or kept == [3]
    x, host, times = broadcast_view(tb, np.random.default_rng(5), dims, strides, dtype)
    out_dims = [dims[i] for i in kept]
    axes = tuple(i for i in range(len(dims)) if i not in kept)
    for op in ("Sum", "Max", "Min"):
        out = tb.Tensor.from_numpy(np.full(out_dims or (1,), 7, dtype).reshape(out_dims))
        plan = tb.CudaBackend.plan(tb.PrimDescriptor.Reduce(list(range(len(dims))), kept, tb.ReduceOp[op]), [dims, out_dims], dtype)
        tb.CudaBackend.execute(plan, 1.0, [x], 0.0, out)
        if op == "Sum":
            want = host.astype(np.float64).sum(axis=axes) * times
            assert want.max() < (2**24 if dtype == np.float32 else 2**53)
        else:
            want = host.max(axis=axes) if op == "Max" else host.min(axis=axes)
        assert np.array_equal(out.to_numpy(), want)
