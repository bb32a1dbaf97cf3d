"""Grouped products inside a capture, for the three kernels that stand behind them: a captured one-shot call
keeps the table it was given however often other tables are laid out afterwards, a plan made while capturing
works inside and outside the graph, and a plan given up while capturing does not disturb it.

Expected values are the products formed on the host in double precision, to the relative Frobenius error that
every contraction of the library keeps."""
import ctypes as C

import numpy as np
import pytest

from conftest import TOL

pytestmark = pytest.mark.gpu

# all multiples of 16: the mma.sync kernel; 16-byte aligned columns: tcgen05; odd columns: the general kernel
TABLES = {"grouped_tf32x3": [(16, 32, 48), (64, 16, 16)] * 20, "grouped_tcgen05": [(20, 36, 12), (68, 8, 44)] * 20,
          "grouped_simt": [(7, 9, 5), (33, 3, 21)] * 20, "grouped_dmma": [(7, 9, 5), (33, 3, 21)] * 20}


class Batch:
    """Operands of a table on the device, back to back, C zeroed."""

    def __init__(self, tb, oracle, table, dtype, seed):
        self.tb, self.dtype, self.table = tb, np.dtype(dtype), table
        self.a = [oracle.uniform(seed + 3 * p, (m, k), dtype) for p, (m, n, k) in enumerate(table)]
        self.b = [oracle.uniform(seed + 3 * p + 1, (k, n), dtype) for p, (m, n, k) in enumerate(table)]
        flat = [np.concatenate([x.ravel(order="F") for x in xs]) for xs in (self.a, self.b)]
        self.dev = [tb.Tensor.from_numpy(x) for x in flat]
        self.dev.append(tb.Tensor.from_numpy(np.zeros(sum(m * n for m, n, k in table), dtype)))
        self.rows, at = [], [0, 0, 0]
        for m, n, k in table:
            row = [m, n, k]
            for t, (r, c) in enumerate(((m, k), (k, n), (m, n))):
                row += [self.dev[t]._block.ptr + at[t] * self.dtype.itemsize, 1, r]
                at[t] += r * c
            self.rows.append(tuple(row))

    def clear(self):
        block = self.dev[2]._block
        block.ctx.memset(block.ptr, 0, block.nbytes)

    def set_a(self, factor):
        x = factor * self.a_flat()
        block = self.dev[0]._block
        block.ctx.h2d(block.ptr, x.ctypes.data_as(C.c_void_p), x.nbytes)
        block.ctx.synchronize()

    def a_flat(self):
        return np.concatenate([x.ravel(order="F") for x in self.a])

    def check(self, factor=1.0):
        want = [factor * (a.astype(np.float64) @ b.astype(np.float64)) for a, b in zip(self.a, self.b)]
        want = np.concatenate([x.ravel(order="F") for x in want])
        assert np.linalg.norm(self.dev[2].to_numpy() - want) <= TOL[self.dtype] * np.linalg.norm(want)


@pytest.mark.parametrize("kernel", list(TABLES))
def test_grouped_calls_in_a_capture(tb, oracle, kernel):
    dtype = np.float64 if kernel == "grouped_dmma" else np.float32
    ctx = tb.Context.get(0)
    one, planned, other = (Batch(tb, oracle, TABLES[kernel], dtype, 1000 * s) for s in (1, 2, 3))
    ctx.profile_begin()
    tb.grouped_gemm(one.rows, dtype)  # first use: kernel attributes
    ctx.synchronize()
    assert ctx.profile_read(kernel)[0] == 1
    ctx.profile_end()
    one.check()
    one.clear()
    earlier = tb.PreparedGroupedGemm(other.rows, dtype)
    ctx.synchronize()

    ctx.capture_begin()
    tb.grouped_gemm(one.rows, dtype)
    plan = tb.PreparedGroupedGemm(planned.rows, dtype)
    plan.run()
    del earlier  # given up while capturing
    graph = ctx.capture_end()
    ctx.synchronize()
    assert not one.dev[2].to_numpy().any() and not planned.dev[2].to_numpy().any()  # capturing ran nothing

    plan.run()  # outside the graph, before its first replay
    planned.check()
    planned.clear()
    for factor in (1.0, 2.0):
        # other tables through the same host buffers and through the pool
        for _ in range(3):
            tb.grouped_gemm(other.rows[::-1], dtype)
            tb.PreparedGroupedGemm(other.rows, dtype).run()
        ctx.synchronize()
        other.check()
        one.set_a(factor)
        planned.set_a(factor)
        graph.launch()
        ctx.synchronize()
        one.check(factor)
        planned.check(factor)
        one.clear()
        planned.clear()
    del graph
    plan.run()
    planned.check(2.0)
