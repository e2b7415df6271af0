"""Native-precision GEMM at the edges of its tiles and K parts.

Every type and operation pair on sizes that straddle the 64 x 64 tile, the K
slab and the parts K is split into (one part empty, one part short, one part
per CTA of a cluster of 8), and on the 128 x 128 tile of large fp32.  Each
result is checked against the double-double oracle, |C - C_oracle| <= tol *
(|alpha| |op(A)||op(B)| + |beta||C|) with tol 1e-5 (fp32 kinds: k * 2^-24
with k <= 130 plus margin, sequential sums) and 1e-13 (fp64 kinds), and the
same operands shifted one element off the 16-byte boundary must give the same
bits: alignment changes the copies, not the order of summation.
"""
import numpy as np
import pytest
import torch

import coral_b200 as cb
import oracle

pytestmark = pytest.mark.gpu

FN = {np.float32: cb.sgemm, np.float64: cb.dgemm, np.complex64: cb.cgemm, np.complex128: cb.zgemm}
SHAPES = [(1, 1, 1), (63, 65, 15), (64, 64, 16), (65, 63, 17), (70, 5, 130), (3, 66, 1000), (200, 130, 33)]
OPS = [(0, 0), (1, 0), (0, 2), (2, 1)]


def rnd(rng, n, dtype):
    x = rng.uniform(-1, 1, n)
    return (x + 1j * rng.uniform(-1, 1, n)).astype(dtype) if np.issubdtype(dtype, np.complexfloating) else x.astype(dtype)


def check(dtype, op_a, op_b, m, n, k, seed):
    rng = np.random.default_rng(seed)
    even = lambda rows: -(-(rows + 1) // 4) * 4  # 16-byte multiple for every type
    lda, ldb, ldc = even(m if op_a == 0 else k), even(k if op_b == 0 else n), m + 1
    a = rnd(rng, lda * (k if op_a == 0 else m), dtype)
    b = rnd(rng, ldb * (n if op_b == 0 else k), dtype)
    c = rnd(rng, ldc * n, dtype)
    alpha, beta = (1.5 - 0.25j, 0.5 + 0.125j) if np.issubdtype(dtype, np.complexfloating) else (1.5, 0.5)
    outs = []
    for shift in (0, 1):
        at = [torch.from_numpy(np.concatenate([np.zeros(shift, dtype), v])).cuda()[shift:] for v in (a, b)]
        C = torch.from_numpy(c).cuda()
        FN[dtype](op_a, op_b, m, n, k, alpha, at[0], lda, at[1], ldb, beta, C, ldc)
        outs.append(C.cpu().numpy())
    np.testing.assert_array_equal(outs[0], outs[1])
    got = outs[0].reshape(n, ldc).T
    np.testing.assert_array_equal(got[m:], c.reshape(n, ldc).T[m:])
    if m * n <= 20000:
        ii, jj = (g.ravel() for g in np.meshgrid(np.arange(m), np.arange(n), indexing="ij"))
    else:
        ii, jj = rng.integers(0, m, 2048), rng.integers(0, n, 2048)
    want, bound = oracle.gemm_sample(op_a, op_b, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, ii, jj)
    tol = 1e-5 if dtype in (np.float32, np.complex64) else 1e-13
    assert (np.abs(got[ii, jj] - want) <= tol * np.maximum(bound, 1e-300)).all()


@pytest.mark.parametrize("dtype", list(FN), ids=lambda d: d.__name__)
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_native_gemm_edges(cuda, dtype, shape):
    for i, ops in enumerate(OPS):
        check(dtype, *ops, *shape, seed=i + sum(shape))


@pytest.mark.parametrize("ops", OPS, ids=str)
def test_native_sgemm_large_tile_edges(cuda, ops):
    check(np.float32, *ops, 1665, 1663, 47, seed=7)
