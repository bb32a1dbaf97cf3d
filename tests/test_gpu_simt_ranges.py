"""The exact-arithmetic contraction kernel around its tile (64), its k slice (16; 8 for 16-byte elements) and
its ranges over K, forced for every type and run over the tropical semirings.

The bound is that of a dot product at the unit roundoff, four products per complex term; Max and Min of
sums of two are exact up to the one rounding of the sum, which the host makes alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = [(1, 1, 1), (3, 65, 15), (64, 64, 16), (63, 2, 129), (65, 31, 1000), (5, 130, 257), (129, 66, 300)]


def plan_for(tb, shapes, dtype, algebra=None):
    desc = tb.PrimDescriptor.Contract([0, 2], [2, 1], [0, 1])
    return tb.CudaBackend.plan(desc, shapes, dtype, algebra=algebra or tb.Algebra.Standard)


@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_simt(tb, oracle, m, n, k, dtype, beta):
    a, b, c = (oracle.normal(20 + i, s, dtype) for i, s in enumerate([(m, k), (k, n), (m, n)]))
    plan = plan_for(tb, [a.shape, b.shape, c.shape], dtype)
    plan.force_kernel(tb.ContractKernel.Simt)
    out = tb.Tensor.from_numpy(c)
    tb.CudaBackend.execute(plan, 1.0, [tb.Tensor.from_numpy(a), tb.Tensor.from_numpy(b)], beta, out)
    wide = np.complex128 if np.dtype(dtype).kind == "c" else np.float64
    want = a.astype(wide) @ b.astype(wide) + beta * c.astype(wide)
    terms = (4 if np.dtype(dtype).kind == "c" else 1) * k + 4
    bound = 2 * terms * np.finfo(dtype).eps / 2 * (abs(a).astype(np.float64) @ abs(b) + beta * abs(c))
    assert (abs(out.to_numpy() - want) <= bound).all()


@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("algebra", ["MaxPlus", "MinPlus"])
def test_semirings(tb, oracle, m, n, k, dtype, algebra):
    a, b = (oracle.normal(30 + i, s, dtype) for i, s in enumerate([(m, k), (k, n)]))
    best = np.max if algebra == "MaxPlus" else np.min
    zero = -np.inf if algebra == "MaxPlus" else np.inf
    out = tb.Tensor.from_numpy(np.zeros((m, n), dtype))
    plan = plan_for(tb, [a.shape, b.shape, (m, n)], dtype, tb.Algebra[algebra])
    tb.CudaBackend.execute(plan, 0.0, [tb.Tensor.from_numpy(a), tb.Tensor.from_numpy(b)], zero, out)
    want = np.stack([best(a[i][:, None] + b, axis=0) for i in range(m)])
    assert np.array_equal(out.to_numpy(), want)
