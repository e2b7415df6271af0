"""Ozaki DGEMM across the wide tile's ring and the INT32 chunk limit, and the
slicing of subnormal and widely scaled entries.

The 128-column tile runs K twice (diagonals 5-8, then 2-4) through a ring of
four slots: K slab counts that are odd, even and past one chunk (148 slabs of
64) are checked at sampled entries against the double-double oracle, 4e-15
component-wise as in the other Ozaki tests.  Products that are exact in fp64
must come back exactly.
"""
import numpy as np
import pytest
import torch

import coral_b200 as cb
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def ozaki_mode():
    cb.set_gemm_mode(cb.GemmMode.OZAKI_INT8)
    yield
    cb.set_gemm_mode(cb.GemmMode.NATIVE)


@pytest.mark.parametrize("m,n,k", [(2048, 2048, 1200), (2048, 2048, 1280), (2047, 2017, 9600), (130, 70, 9600)])
def test_slabs_and_chunks(cuda, m, n, k):
    rng = np.random.default_rng(k)
    a, b, c = (rng.uniform(-1, 1, s) for s in (m * k, k * n, m * n))
    C = torch.from_numpy(c).cuda()
    cb.dgemm(0, 0, m, n, k, 1.5, torch.from_numpy(a).cuda(), m, torch.from_numpy(b).cuda(), k, 0.5, C, m)
    ii, jj = rng.integers(0, m, 512), rng.integers(0, n, 512)
    want, bound = oracle.gemm_sample(0, 0, m, n, k, 1.5, a, m, b, k, 0.5, c, m, ii, jj)
    got = C.cpu().numpy().reshape(n, m).T[ii, jj]
    assert (np.abs(got - want) <= 4e-15 * bound).all()


@pytest.mark.parametrize("op", [0, 1])
def test_exact_products(cuda, op):
    """A holds 40-bit integers at exponents down to the smallest subnormal, B a
    power of two on its diagonal: every entry of the product is exact."""
    m, k = 40, 140
    rng = np.random.default_rng(op)
    scale = np.ldexp(1.0, rng.choice([-1074, -1070, -1022, -300, 0, 500], m))[:, None]
    ints = rng.integers(-(2 ** 40), 2 ** 40, (m, k)).astype(np.float64)
    ints[3] = 0.0
    ints[:, 7] = 0.0
    A = ints * scale
    B = np.diag(np.full(k, 2.0 ** 60))
    a = A.T if op == 0 else A  # column-major A, or its transpose
    C = torch.full((m * k,), float("nan"), dtype=torch.float64, device="cuda")
    cb.dgemm(op, 0, m, k, k, 1.0, torch.from_numpy(np.ascontiguousarray(a).ravel()).cuda(), m if op == 0 else k,
             torch.from_numpy(B.ravel()).cuda(), k, 0.0, C, m)
    np.testing.assert_array_equal(C.cpu().numpy().reshape(k, m).T, A * 2.0 ** 60)
