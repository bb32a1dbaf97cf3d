"""The grouped product's general kernel (double precision, complex, and every f32 table the two
tensor-core kernels decline): sizes around the edges of its output tiles (64 real, 32 complex),
stage depth (32) and MMA steps (8), stored column- or row-major, back to back or aligned, against
the host product in double precision.

The bound is the standard one of a dot product, component by component: K + 4 roundings of
|A| |B|, twice that for the two real sums in each part of a complex product, at the unit roundoff of
the type."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (m, n, k): tiles' edges, fragment edges (16 rows, 8 columns), stage edges, no k at all
SIZES = [(1, 1, 1), (16, 8, 16), (17, 9, 15), (31, 33, 32), (64, 64, 48), (65, 63, 17), (129, 20, 7), (5, 130, 200), (40, 24, 0)]


def place(layouts, arrays, pad):
    """Back to back in one flat buffer (`pad` elements between blocks): (buffer, [(offset, rs, cs)])."""
    parts, where, at = [], [], 0
    for order, x in zip(layouts, arrays):
        rs, cs = (1, x.shape[0]) if order == "F" else (x.shape[1], 1)
        where.append((at, rs, cs))
        flat = np.concatenate([x.ravel(order=order), np.full(pad, np.nan, x.dtype)])
        parts.append(flat)
        at += flat.size
    return np.concatenate(parts), where


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("layout", ["FFF", "CCC", "CFF", "FCC"])
@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_grouped_units(tb, oracle, dtype, layout, pad, beta):
    dtype = np.dtype(dtype)
    # f32: one problem without alignment keeps the whole table on this kernel
    table = SIZES + [(8, 8, 4)] * 40
    if layout == "FFF":  # longer than the window of records a CTA holds: about 20 units each
        table = table + [(m, n, 4) for m in range(1, 97) for n in range(1, 97)]
    mats = [[oracle.normal(11 * p + 100 * t, s, dtype) for p, s in enumerate(shapes)]
            for t, shapes in enumerate(([(m, k) for m, n, k in table], [(k, n) for m, n, k in table], [(m, n) for m, n, k in table]))]
    bufs, wheres = zip(*(place([layout[t]] * len(table), mats[t], pad) for t in range(3)))
    dev = [tb.Tensor.from_numpy(b) for b in bufs]
    es = dtype.itemsize
    probs = []
    for p, (m, n, k) in enumerate(table):
        row = [m, n, k]
        for t in range(3):
            off, rs, cs = wheres[t][p]
            row += [dev[t]._block.ptr + off * es, rs, cs]
        probs.append(tuple(row))
    alpha = 1.5 - 0.5j if dtype.kind == "c" else 1.5
    plan = tb.PreparedGroupedGemm(probs, dtype, alpha, beta)
    ctx = plan.ctx
    ctx.profile_begin()
    plan.run()
    ctx.synchronize()
    name = "grouped_simt" if es == 4 or dtype == np.complex64 else "grouped_dmma"
    assert ctx.profile_read(name)[0] == 1
    ctx.profile_end()
    out = dev[2].to_numpy()
    u = np.finfo(dtype).eps / 2
    wide = np.complex128 if dtype.kind == "c" else np.float64
    live = np.zeros(out.size, bool)
    for p, (m, n, k) in enumerate(table):
        off, rs, cs = wheres[2][p]
        at = off + np.arange(m)[:, None] * rs + np.arange(n)[None, :] * cs
        live[at] = True
        a, b, c0 = (mats[t][p].astype(wide) for t in range(3))
        want = alpha * (a @ b) + beta * c0
        terms = (2 if dtype.kind == "c" else 1) * k + 4
        bound = 2 * terms * u * (abs(alpha) * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(c0)) + 1e-300
        assert (np.abs(out[at] - want) <= bound).all(), (p, m, n, k)
    assert np.isnan(out[~live]).all()  # nothing outside the blocks was written


# (m, n, k) and the strides of A, B and C: broadcast rows, columns or everything, reversed directions, both strides alike
# (overlapping diagonals), a transposed and reversed C
STRIDES = [((33, 20, 17), (0, 1), (1, 17), (1, 33)), ((33, 20, 17), (1, 0), (0, 1), (1, 33)), ((65, 9, 40), (0, 0), (1, 0), (1, 65)),
           ((40, 66, 18), (-1, 40), (18, -1), (1, 40)), ((40, 66, 18), (18, 1), (-66, 1), (1, 40)),
           ((31, 34, 19), (-1, -31), (1, 1), (1, 31)), ((17, 65, 16), (1, 1), (1, 16), (-65, 1)),
           ((64, 64, 16), (2, 1), (1, 3), (-1, -64)), ((1, 1, 33), (5, 1), (1, 7), (3, 3)), ((70, 1, 9), (1, 70), (1, 1), (1, 1)),
           ((1, 70, 9), (1, 1), (70, 1), (9, 1))]


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_strides(tb, oracle, dtype, beta):
    dtype = np.dtype(dtype)
    wide = np.complex128 if dtype.kind == "c" else np.float64
    rows, mats = [], []
    for p, ((m, n, k), *strides) in enumerate(STRIDES):
        row, part = [m, n, k], []
        for t, (shape, (rs, cs)) in enumerate(zip(((m, k), (k, n), (m, n)), strides)):
            first = -min(0, (shape[0] - 1) * rs) - min(0, (shape[1] - 1) * cs)
            size = first + max(0, (shape[0] - 1) * rs) + max(0, (shape[1] - 1) * cs) + 1
            flat = oracle.normal(50 * p + t, (size + 3,), dtype)
            dev = tb.Tensor.from_numpy(flat)
            at = first + np.arange(shape[0])[:, None] * rs + np.arange(shape[1])[None, :] * cs
            row += [dev._block.ptr + first * dtype.itemsize, rs, cs]
            part.append((flat, at, dev))
        rows.append(tuple(row))
        mats.append(part)
    plan = tb.PreparedGroupedGemm(rows, dtype, 1.0, beta)
    plan.run()
    plan.ctx.synchronize()
    u = np.finfo(dtype).eps / 2
    for ((m, n, k), *_), part in zip(STRIDES, mats):
        (fa, ia, _), (fb, ib, _), (fc, ic, dev) = part
        a, b, c0 = fa[ia].astype(wide), fb[ib].astype(wide), fc[ic].astype(wide)
        out = dev.to_numpy()
        terms = (2 if dtype.kind == "c" else 1) * k + 4
        bound = 2 * terms * u * (np.abs(a) @ np.abs(b) + beta * np.abs(c0)) + 1e-300
        assert (np.abs(out[ic] - (a @ b + beta * c0)) <= bound).all(), (m, n, k)
        rest = np.ones(out.size, bool)
        rest[ic] = False
        assert np.array_equal(out[rest], fc[rest])


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("layout", ["CCF", "FFC"])
def test_edges_of_deeper_stages(tb, oracle, dtype, layout, monkeypatch):
    """K around one, two and three stages of 32, with sides that leave warps and lanes without a part."""
    sizes = [(20, 20, 31), (20, 21, 33), (64, 64, 63), (65, 30, 64), (33, 65, 65), (16, 16, 95), (9, 70, 96), (70, 9, 97), (1, 64, 32), (64, 1, 34)]
    monkeypatch.setitem(globals(), "SIZES", sizes)
    test_grouped_units(tb, oracle, dtype, layout, 3, 0.5)
