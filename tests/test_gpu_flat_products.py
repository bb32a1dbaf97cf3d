"""Element-wise products whose output lies without a gap and has runs of an odd number of elements: sixteen bytes at a time
along the whole tensor, the other operand element by element; remainders, broadcasts, conjugation, beta and updates in place."""
import numpy as np
import pytest

from conftest import random_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("notation", ["asb,b->asb", "a,asb->asb", "asb,asb->asb", "asb,s->asb", "ab,asb->asb", "asb,bsa->asb"])
@pytest.mark.parametrize("dims", [(333, 3, 101), (3, 2, 17001), (1, 3, 34567), (100003, 1, 1), (2, 5, 10007), (341, 2, 151)])
def test_products_over_runs_of_any_length(tb, oracle, dtype, notation, dims):
    ext = dict(zip("asb", dims))
    rng = np.random.default_rng(sum(dims))
    ins, out = notation.split("->")
    ops = [random_array(rng, tuple(ext[c] for c in t), dtype) for t in ins.split(",")]
    c0 = random_array(rng, dims, dtype)
    ulp = np.finfo(dtype).eps  # a product and a sum of two roundings each, four for complex parts
    for alpha, beta, conj in ((1.0, 0.0, False), (-0.5, 0.75, True)):
        held = [tb.Tensor.from_numpy(x) for x in ops]
        if conj and np.dtype(dtype).kind == "c":
            held[0] = held[0].into_conj()
            want = np.conj(ops[0])
        else:
            want = ops[0]
        want = alpha * oracle.np_einsum(notation, [want, ops[1]]) + beta * c0
        got = tb.Tensor.from_numpy(c0.copy())
        tb.einsum_into(notation, held, alpha, beta, got)
        assert oracle.rel_frobenius(got.to_numpy(), want) <= 4 * ulp


def test_in_place(tb, oracle):
    rng = np.random.default_rng(1)
    a, w = random_array(rng, (1001, 3, 77), np.float32), random_array(rng, (77,), np.float32)
    t = tb.Tensor.from_numpy(a)
    tb.einsum_into("asb,b->asb", [t, tb.Tensor.from_numpy(w)], 1.0, 0.0, t)
    assert np.array_equal(t.to_numpy(), a * w)
