"""Double-precision contractions whose extents no short run divides: the four-product complex form on
one load per run, and products on copies of operands that no tensor map can describe.  Sizes lie around
the edges of the tiles (32, 64, 128), of a k-iteration (16) and of a run (8, 4).

The bound is that of a dot product, part by part: K + 4 roundings of |A| |B| (twice the terms in each
part of a complex product) at the unit roundoff, doubled for the split of K over several blocks."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = np.finfo(np.float64).eps / 2


def product(notation, a, b):
    """The product in double precision on the host, batch by batch through BLAS."""
    import torch

    wide = np.complex128 if np.iscomplexobj(a) else np.float64
    return torch.einsum(notation, torch.from_numpy(a.astype(wide)), torch.from_numpy(b.astype(wide))).numpy()


def run(tb, oracle, notation, shapes, dtype, conj, beta):
    a, b = (oracle.normal(7 + t, s, dtype) for t, s in enumerate(shapes))
    want_shape = np.einsum(notation, np.zeros(shapes[0], np.int8), np.zeros(shapes[1], np.int8)).shape
    c = oracle.normal(9, want_shape, dtype)
    ta, tc = tb.Tensor.from_numpy(a), tb.Tensor.from_numpy(b)
    out = tb.Tensor.from_numpy(c)
    if conj:
        tc, b = tc.into_conj(), b.conj()
    tb.einsum_into(notation, [ta, tc], 1.0, beta, out)
    got = out.to_numpy()

    def parts(x):
        return (x.real, x.imag) if np.iscomplexobj(x) else (x,)

    mag = sum(np.einsum(notation, abs(p), abs(q), optimize=True) for p in parts(a) for q in parts(b))
    want = np.einsum(notation, a, b, optimize=True) + beta * c
    terms = a.size * b.size // max(1, want.size)
    k = max(8, int(np.sqrt(terms))) + 4
    bound = 2 * k * (2 if len(parts(a)) == 2 else 1) * U * (mag + abs(beta) * abs(c))
    for x, y in zip(parts(got), parts(want)):
        assert (abs(x - y) <= bound).all()


@pytest.mark.parametrize("notation", ["ij,jk->ik", "ji,jk->ik", "ij,kj->ik", "bij,bjk->bik"])
@pytest.mark.parametrize("mnk", [(33, 31, 15), (1, 63, 17), (65, 64, 9), (97, 194, 97), (130, 71, 33), (257, 259, 40)])
@pytest.mark.parametrize("conj", [False, True])
def test_complex_extents(tb, oracle, notation, mnk, conj):
    m, n, k = mnk
    size = {"i": m, "k": n, "j": k, "b": 3}
    shapes = [tuple(size[c] for c in t) for t in notation.split("->")[0].split(",")]
    run(tb, oracle, notation, shapes, np.complex128, conj, 0.5)


@pytest.mark.parametrize("notation,sizes", [
    ("ij,jk->ik", dict(i=331, j=1021, k=333)),  # odd leading extents
    ("ji,jk->ik", dict(i=129, j=6001, k=131)),
    ("ijk,kjl->il", dict(i=131, j=57, k=103, l=137)),  # contracted modes in different orders
    ("bij,bjk->bik", dict(b=21, i=67, j=1025, k=71)),  # the batch index innermost
    ("ijab,abk->kij", dict(i=9, j=31, a=65, b=17, k=331)),
])
@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
def test_operands_without_a_map(tb, oracle, notation, sizes, dtype):
    assert 2 * np.prod([float(v) for v in sizes.values()]) >= 2e8  # from here on operands are copied
    shapes = [tuple(sizes[c] for c in t) for t in notation.split("->")[0].split(",")]
    run(tb, oracle, notation, shapes, dtype, False, 0.5)


COPIES = ("permute_rows", "permute_tiled", "permute_tile", "permute_generic")


def launches(ctx, fn, names):
    ctx.profile_begin()
    fn()
    ctx.synchronize()
    got = [ctx.profile_read(name)[0] for name in names]
    ctx.profile_end()
    return got


# (notation, sizes, pairs of the tree, operands copied): one operand keeps its map, two batch modes that do not fuse, a
# multiplier fused into the product
@pytest.mark.parametrize("notation,sizes,pairs,copies", [
    ("ij,jk->ik", dict(i=331, j=1024, k=512), [(0, 1)], {"f": 1, "c": 0}),
    ("ij,jk->ik", dict(i=332, j=1021, k=511), [(0, 1)], {"f": 1, "c": 0}),
    ("ijl,jk->ilk", dict(i=33, j=640, l=17, k=514), [(0, 1)], {"f": 1, "c": 1}),
    ("kj,ijl->kil", dict(i=33, j=640, l=17, k=516), [(0, 1)], {"f": 1, "c": 1}),
    ("bijc,bjkc->bikc", dict(b=5, i=67, j=1201, c=4, k=70), [(0, 1)], {"f": 2, "c": 2}),
    ("ijl,ljk,ik->ik", dict(i=255, j=51, l=33, k=257), [(0, 1), (2, 3)], {"f": 2, "c": 2}),
])
@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("conj", [False, True])
def test_copied_operands(tb, oracle, notation, sizes, pairs, copies, dtype, conj):
    ins, out_labels = notation.split("->")
    ins = ins.split(",")
    assert 2 * np.prod([float(sizes[c]) for c in set(ins[0] + ins[1])]) >= 2e8
    arrays = [oracle.normal(17 + t, [sizes[c] for c in term], dtype) for t, term in enumerate(ins)]
    c0 = oracle.normal(29, [sizes[c] for c in out_labels], dtype)
    ops, out = [tb.Tensor.from_numpy(x) for x in arrays], tb.Tensor.from_numpy(c0)
    if conj:
        ops, arrays = [x.into_conj() for x in ops], [x.conj() for x in arrays]
    tree = tb.ContractionTree.from_pairs(tb.Subscripts.parse(notation), [x.shape for x in arrays], pairs)
    ctx = tb.Context.get(0)
    ran = launches(ctx, lambda: tb.einsum_with_plan_into(tree, ops, 1.0, 0.5, out), COPIES + ("contract_dmma", "contract_dmma_fixup"))
    kind = np.dtype(dtype).kind
    assert sum(ran[:4]) == copies[kind] and ran[4] == 1 and ran[5] == 0
    parts = lambda x: (x.real, x.imag) if kind == "c" else (x,)
    # products of magnitudes, part by part; the multiplier's parts on top
    mag = sum(np.einsum(notation, *[abs(q) for q in pick], optimize=True)
              for pick in itertools.product(*[parts(x) for x in arrays]))
    want = np.einsum(notation, *arrays, optimize=True) + 0.5 * c0
    k = np.prod([sizes[c] for c in set(ins[0] + ins[1]) - set(out_labels)]) + 8
    bound = 2 * k * (2 if kind == "c" else 1) * U * (mag + 0.5 * abs(c0))
    for x, y in zip(parts(out.to_numpy()), parts(want)):
        assert (abs(x - y) <= bound).all()


def device_product(tb, m, n, k):
    """i j, j k -> i k on small integers (sums are exact in any order): (call, output, expected, whatever holds the operands)."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(3)
    a, b = (torch.randint(0, 4, s, device="cuda", generator=gen, dtype=torch.int8).double() for s in ((k, m), (n, k)))
    out = torch.zeros((n, m), device="cuda", dtype=torch.float64)
    want = b @ a
    space = tb.LogicalMemorySpace.GpuMemory(0)
    views = [tb.Tensor.from_device_pointer(t.data_ptr(), t.numel() * 8, dims, np.float64, space, t)
             for t, dims in ((a, (m, k)), (b, (k, n)), (out, (m, n)))]
    tree = tb.ContractionTree.optimize(tb.Subscripts.parse("ij,jk->ik"), [(m, k), (k, n)])
    torch.cuda.synchronize()
    return lambda: tb.einsum_with_plan_into(tree, views[:2], 1.0, 0.0, views[2]), out, want


@pytest.mark.parametrize("m,n,k,copies", [
    (65, 64, 262140, 1),  # B's rows just below 2 MiB apart
    (65, 64, 262144, 0),
    (65, 67, 6000001, 0),  # 6.9 GB of copies: more than the pool may keep
])
def test_when_operands_are_not_copied(tb, m, n, k, copies):
    import torch

    call, out, want = device_product(tb, m, n, k)
    ctx = tb.Context.get(0)
    kept = ctx.pool_stats()[0]
    assert sum(launches(ctx, call, COPIES)) == copies
    assert torch.equal(out, want)
    if not copies:
        assert ctx.pool_stats()[0] - kept < 1 << 30


@pytest.mark.parametrize("notation,sizes", [
    ("ibj,jbk->bik", dict(b=7, i=200, j=48, k=100)),  # K that 32-deep iterations would pad by a third
    ("ij,jk->ik", dict(i=128, j=40000, k=128)),  # few outputs and a K that fills the chip: large tiles
    ("ij,jk->ik", dict(i=97, j=20001, k=97)),  # ... in the four-product form
    ("ij,jk->ik", dict(i=129, j=40000, k=65)),  # ... where they would be padding: small tiles
    ("ij,ij->", dict(i=275, j=301)),  # one tile with a long K: by gather
    ("ij,jk->ik", dict(i=20, j=70001, k=33)),
    ("ji,kj->ki", dict(i=344, j=280, k=312)),  # tiles in equal ranges rather than three pieces each
])
@pytest.mark.parametrize("conj", [False, True])
def test_complex_tiles(tb, oracle, notation, sizes, conj):
    shapes = [tuple(sizes[c] for c in t) for t in notation.split("->")[0].split(",")]
    run(tb, oracle, notation, shapes, np.complex128, conj, 0.5)


@pytest.mark.parametrize("cluster", ["0", "1"])
@pytest.mark.parametrize("dtype,mnk", [
    (np.float64, (64, 64, 4096)),  # pieces that meet in shared memory, or in a second launch
    (np.float64, (32, 36, 128)),   # one iteration per CTA
    (np.float64, (228, 252, 260)),
    (np.float64, (448, 452, 1028)),  # ranges that cut tiles
    (np.float64, (24, 1044, 992)),   # four pieces of 15 or 16 iterations
    (np.float64, (128, 128, 5004)),
    (np.float64, (60, 60, 260)),     # four pieces of 17 iterations
    (np.complex128, (16, 12, 5128)),
    (np.complex128, (30, 66, 1000)),
    (np.complex128, (64, 128, 64)),
    (np.complex128, (98, 196, 100)),
    (np.complex128, (258, 322, 324)),
])
@pytest.mark.parametrize("conj", [False, True])
def test_split_of_k(tb, oracle, monkeypatch, dtype, mnk, cluster, conj):
    monkeypatch.setenv("TFB_DMMA_CLUSTER", cluster)
    m, n, k = mnk
    run(tb, oracle, "ij,jk->ik", [(m, k), (k, n)], dtype, conj, 0.5)
    # the order of the sums does not depend on which block comes last
    x, y = (tb.Tensor.from_numpy(oracle.normal(3 + t, s, dtype)) for t, s in enumerate([(m, k), (k, n)]))
    first = tb.einsum("ij,jk->ik", [x, y]).to_numpy()
    for _ in range(3):
        assert np.array_equal(tb.einsum("ij,jk->ik", [x, y]).to_numpy(), first)


@pytest.mark.parametrize("notation,sizes", [
    ("bij,bjk->bik", dict(b=37, i=67, j=1025, k=71)),
    ("bij,bjk->bik", dict(b=16, i=260, j=515, k=301)),
    ("bij,bkj->bki", dict(b=33, i=129, j=517, k=131)),      # operands change places
    ("bij,jkb->bik", dict(b=40, i=129, j=261, k=259)),      # one operand with the batch outermost
    ("bijx,bjxk->bki", dict(b=32, i=128, j=33, k=129, x=31)),  # two contracted modes
    ("bijx,bkj->bkix", dict(b=33, i=17, j=515, k=129, x=9)),   # two free modes
])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
def test_batch_innermost(tb, oracle, monkeypatch, notation, sizes, dtype):
    """On copies with the batch outermost and as the operands lie, both against the host product.  Frobenius: 1e-5 for a
    3xTF32 product, 1e-13 for double (K + 4 roundings at 1.1e-16, K up to 1025); single elements ten times that of the largest."""
    a, b = (oracle.normal(7 + t, tuple(sizes[c] for c in s), dtype) for t, s in enumerate(notation.split("->")[0].split(",")))
    c = oracle.normal(9, tuple(sizes[x] for x in notation.split("->")[1]), dtype)
    ta, tc = tb.Tensor.from_numpy(a), tb.Tensor.from_numpy(b).into_conj()
    got = []
    for on in "10":
        monkeypatch.setenv("TFB_BATCH_OUTERMOST", on)
        out = tb.Tensor.from_numpy(c)
        tb.einsum_into(notation, [ta, tc], 0.75, 0.5, out)
        got.append(out.to_numpy())
    wide = np.complex128 if np.dtype(dtype).kind == "c" else np.float64
    want = 0.75 * np.einsum(notation, a.astype(wide), np.conj(b).astype(wide), optimize=True) + 0.5 * c
    tol = 1e-13 if dtype in (np.float64, np.complex128) else 1e-5
    for x in got:
        assert np.linalg.norm(x - want) <= tol * np.linalg.norm(want)
    assert np.abs(got[0] - got[1]).max() <= 10 * tol * np.abs(want).max()


@pytest.mark.parametrize("notation,sizes", [
    # twelve free modes and the batch lie one by one in the output: no single pass puts it back
    ("bacegikx,bxdfhjlm->badcfehgjilkm", dict(b=64, x=512)),
    # ... and in an operand: no single pass copies it
    ("bavcwexgyizks,bvwxyzsd->bacegikd", dict(b=64, d=400)),
])
def test_batch_innermost_in_more_modes_than_a_pass_takes(tb, oracle, notation, sizes):
    shapes = [tuple(sizes.get(c, 2) for c in t) for t in notation.split("->")[0].split(",")]
    run(tb, oracle, notation, shapes, np.float64, False, 0.5)


@pytest.mark.parametrize("notation,sizes", [
    ("bij,bjk->bik", dict(b=1000, i=100, j=100, k=100)),
    ("bij,bkj->bki", dict(b=8, i=600, j=600, k=600)),
    ("bij,jkb->bik", dict(b=33, i=257, j=700, k=120)),
])
def test_small_f32_products_stay_exact(tb, oracle, monkeypatch, notation, sizes):
    """Products too small for their operands to be copied for 3xTF32 (1e9 operations each) keep the exact kernel's error,
    which the cut of K moves by a few per cent at most; that of 3xTF32 is three to five times as large."""
    assert 2 * np.prod([float(v) for v in sizes.values()]) >= 1e9 > 2.0 * sizes["i"] * sizes["j"] * sizes["k"]
    a, b = (oracle.normal(7 + t, tuple(sizes[c] for c in s), np.float32) for t, s in enumerate(notation.split("->")[0].split(",")))
    ta, tc = tb.Tensor.from_numpy(a), tb.Tensor.from_numpy(b)
    want = product(notation, a, b)
    err = []
    for kernel in ("0", "1"):  # chosen by the library; the exact one
        monkeypatch.setenv("TFB_FORCE_KERNEL", kernel)
        err.append(oracle.rel_frobenius(tb.einsum(notation, [ta, tc]).to_numpy(), want))
    assert err[0] <= 1.1 * err[1]


# every type on its side of the route's thresholds; chunks of 32 and a last one of 1, 8 and 31 products; outputs that L2 does
# not hold where an operand stays in place
@pytest.mark.parametrize("notation,sizes", [
    ("bij,bjk->bik", dict(b=65, i=169, j=321, k=300)),
    ("bij,bkj->bki", dict(b=72, i=331, j=260, k=129)),
    ("bij,jkb->bik", dict(b=95, i=340, j=105, k=383)),  # the second operand is not copied
    ("ijb,bjk->bik", dict(b=95, i=383, j=105, k=340)),
    ("ijb,jkb->bik", dict(b=129, i=300, j=320, k=304)),  # ... nor the first
    ("bijx,bjxk->bki", dict(b=65, i=301, j=13, k=300, x=16)),
])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64])
@pytest.mark.parametrize("chunk", ["32", "0"])
def test_batch_innermost_in_chunks(tb, oracle, monkeypatch, notation, sizes, dtype, chunk):
    """The passes of each chunk are counted: both operands' copies where they lie so, and the output's.  Bounds as above."""
    work = (8 if dtype is np.complex64 else 2) * np.prod([float(v) for v in sizes.values()])
    assert work >= (2e8 if dtype is np.float64 else 1e9)
    monkeypatch.setenv("TFB_BATCH_CHUNK", chunk)
    terms = notation.split("->")[0].split(",")
    a, b = (oracle.normal(7 + t, tuple(sizes[c] for c in s), dtype) for t, s in enumerate(terms))
    c = oracle.normal(9, tuple(sizes[x] for x in notation.split("->")[1]), dtype)
    ta, tc, out = tb.Tensor.from_numpy(a), tb.Tensor.from_numpy(b).into_conj(), tb.Tensor.from_numpy(c)
    ctx = tb.Context.get(0)
    ctx.profile_begin()
    tb.einsum_into(notation, [ta, tc], 0.75, 0.5, out)
    ctx.synchronize()
    passes = sum(ctx.profile_read(k)[0] for k in ("permute_tile", "permute_tiled", "permute_rows", "permute_generic"))
    ctx.profile_end()
    chunks = -(-sizes["b"] // 32) if chunk == "32" else 1
    if dtype is np.float64 and sum(t[0] == "b" for t in terms) < 2:  # one double precision operand in place may be copied besides
        assert passes >= chunks * (1 + sum(t[0] == "b" for t in terms))
    else:
        assert passes == chunks * (1 + sum(t[0] == "b" for t in terms))
    want = 0.75 * product(notation, a, np.conj(b)) + 0.5 * c
    tol = 1e-13 if dtype is np.float64 else 1e-5
    got = out.to_numpy()
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
    assert np.abs(got - want).max() <= 10 * tol * np.abs(want).max()


@pytest.mark.parametrize("n,scratch", [(1000, 1.1e9), (2304, 1.1e9)])
def test_batch_innermost_memory(tb, n, scratch):
    """Copies of a gigabyte at most, or of eight products where those take more: the pool holds no more afterwards."""
    ctx = tb.Context(0)
    plan = tb.CudaBackend.plan(tb.PrimDescriptor.Contract([0, 1, 2], [0, 2, 3], [0, 1, 3]), [(40, n, n), (40, n, n), (40, n, n)], np.float64, ctx)
    a, b, c = (tb.Tensor.zeros((40, n, n)) for _ in range(3))
    tb.Context.get(0).synchronize()
    tb.CudaBackend.execute(plan, 1.0, [a, b], 0.0, c)
    ctx.synchronize()
    assert ctx.pool_stats()[0] <= scratch
