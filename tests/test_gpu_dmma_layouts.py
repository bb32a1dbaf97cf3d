"""Double-precision contractions whose extents no short run divides: the four-product complex form on
one load per run, and products on copies of operands that no tensor map can describe.  Sizes lie around
the edges of the tiles (32, 64, 128), of a k-iteration (16) and of a run (8, 4).

The bound is that of a dot product, part by part: K + 4 roundings of |A| |B| (twice the terms in each
part of a complex product) at the unit roundoff, doubled for the split of K over several blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = np.finfo(np.float64).eps / 2


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
