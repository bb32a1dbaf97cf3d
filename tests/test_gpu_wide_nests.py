"""Strided kernels over more than 2^31 elements, where offsets and walks are kept in 64 bits.  Inputs are broadcast
views of small buffers.

Sums are exact whatever their order: the terms are integers and every partial sum is below 2^53 (f64) or 2^24 (f32).
Max and Min are exact."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def broadcast_view(tb, rng, dims, strides, dtype):
    """A buffer of small integers (f32: mostly zeros) under the given strides: (tensor, its part without the
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


def same_as_rows(flat, want_block, times):
    """Whether a flat device tensor is `times` repetitions of a host block."""
    import torch

    want = torch.from_numpy(want_block).cuda()
    return bool((flat.view(times, want.numel()) == want).all())


def device_output(tb, dims, dtype):
    import torch

    flat = torch.zeros(math.prod(dims), device="cuda", dtype={np.float32: torch.float32, np.float64: torch.float64}[dtype])
    torch.cuda.synchronize()
    return flat, tb.Tensor.from_device_pointer(flat.data_ptr(), flat.numel() * flat.element_size(), dims, dtype,
                                               tb.LogicalMemorySpace.GpuMemory(0), flat)


def kernels(ctx, fn, names):
    ctx.profile_begin()
    fn()
    ctx.synchronize()
    ran = [n for n in names if ctx.profile_read(n)[0]]
    ctx.profile_end()
    return ran


# (dims and strides of the input, order of the output, kernel): a patch of the first and the last index, the middle
# one broadcast
@pytest.mark.parametrize("dims,strides,perm,kernel", [
    ([8, 2**25 + 3, 8], [1, 0, 8], [2, 0, 1], "permute_generic"),
    ([15, 9600003, 17], [1, 0, 15], [2, 0, 1], "permute_generic"),  # fewer than 256 elements in a tile
    ([16, 8400003, 16], [1, 0, 16], [2, 0, 1], "permute_tiled"),  # 16-byte accesses
    ([17, 7500003, 17], [1, 0, 17], [2, 0, 1], "permute_tiled"),
    ([8, 1000003, 300], [1, 0, 9], [2, 0, 1], "permute_tiled"),
    ([4099, 524003, 1], [1, 0, 1], [0, 2, 1], "permute_rows"),
    ([4096, 524291, 1], [1, 0, 1], [0, 2, 1], "permute_rows"),  # 16-byte accesses
])
def test_permute(tb, dims, strides, perm, kernel):
    assert math.prod(dims) >= 2**31
    x, host, times = broadcast_view(tb, np.random.default_rng(6), dims, strides, np.float32)
    assert host.any()
    out_dims = [dims[i] for i in perm]
    flat, out = device_output(tb, out_dims, np.float32)
    plan = tb.CudaBackend.plan(tb.PrimDescriptor.Permute(list(range(3)), perm), [dims, out_dims], np.float32)
    ran = kernels(plan.ctx, lambda: tb.CudaBackend.execute(plan, 1.0, [x], 0.0, out),
                  ["permute_generic", "permute_tiled", "permute_rows", "permute_tile"])
    assert ran == [kernel]
    assert same_as_rows(flat, host.transpose(perm).reshape(-1, order="F"), times)


@pytest.mark.parametrize("rows", [4099, 4100])  # element by element and in 16-byte accesses
def test_elementwise(tb, rows):
    cols = 2**31 // rows + 5
    a = np.random.default_rng(7).integers(-9, 9, rows).astype(np.float32)
    b = np.arange(rows, dtype=np.float32) % 7
    views = []
    for v in (a, b):
        t = tb.Tensor.from_numpy(v)
        views.append(tb.Tensor(t._block, [rows, cols], [1, 0], 0, np.float32, t.logical_memory_space()))
    flat, out = device_output(tb, [rows, cols], np.float32)
    plan = tb.CudaBackend.plan(tb.PrimDescriptor.ElementwiseMul(), [[rows, cols]] * 3, np.float32)
    tb.CudaBackend.execute(plan, 1.0, views, 0.0, out)
    plan.ctx.synchronize()
    assert same_as_rows(flat, a * b, cols)
