"""Batched STRSV at the edges of its 64-row blocks and of the size ordering.

Every uplo / trans / diag form on sizes around one, two and sixteen blocks and
past what stays in shared memory, strided right-hand sides and padded leading
dimensions, in a batch large enough to be started in size order (with empty
instances in it); results against the STRSV oracle with the tolerance of the
batched test, |x - x_ref| <= 1e-4 max(|x|, |x_ref|) + 1e-6.  A zero on the
diagonal and an infinite right-hand side must leave what a division leaves.
"""
import numpy as np
import pytest
import torch

import coral_b200 as cb
import oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 192, 193, 1023, 1024, 1025, 1100]


def system(rng, n, lda, diag):
    a = rng.uniform(-1, 1, max(1, lda * n)).astype(np.float32)
    d = np.arange(n)
    if n:
        a.reshape(n, lda)[d, d] = np.float32(n) + rng.uniform(0, 1, n).astype(np.float32)
        if diag == 0:
            a /= np.float32(n)
    return a


def solve(cases):
    rec = np.zeros(len(cases), dtype=cb.strsv_problem_dtype())
    keep = []
    for i, (uplo, trans, diag, n, a, lda, x, incx) in enumerate(cases):
        keep.append((torch.from_numpy(a).cuda(), torch.from_numpy(x).cuda()))
        rec[i] = (uplo, trans, diag, n, keep[i][0].data_ptr(), keep[i][1].data_ptr(), lda, incx)
    cb.strsv_batched(len(cases), torch.from_numpy(rec.view(np.uint8)).cuda())
    return [k[1].cpu().numpy() for k in keep]


@pytest.mark.parametrize("filler", [0, 400], ids=["input order", "size order"])
def test_forms_and_sizes(cuda, filler):
    rng = np.random.default_rng(5)
    cases = []
    for q, n in enumerate(SIZES):
        for uplo in (0, 1):
            for trans in (0, 1, 2):
                diag, incx = (q + uplo + trans) % 2, 1 + (q + trans) % 3
                lda = n + q % 3
                cases.append((uplo, trans, diag, n, system(rng, n, lda, diag), lda,
                              rng.uniform(-1, 1, (n - 1) * incx + 1).astype(np.float32), incx))
    for i in range(filler):
        n = int(rng.integers(0, 40))
        cases.append((1, 0, 1, n, system(rng, n, max(n, 1), 1), max(n, 1),
                      rng.uniform(-1, 1, max(n, 1)).astype(np.float32), 1))
    for case, got in zip(cases, solve(cases)):
        uplo, trans, diag, n, a, lda, x, incx = case
        if n == 0:
            np.testing.assert_array_equal(got, x)
            continue
        want = np.asarray(oracle.strsv(uplo, trans, diag, n, a, lda, x, incx))
        err = np.abs(got[::incx][:n] - want)
        tol = 1e-4 * np.maximum(np.abs(got[::incx][:n]), np.abs(want)) + 1e-6
        assert (err <= tol).all(), (case[:4], float(err.max()))
        mask = np.ones(x.size, bool)
        mask[::incx] = False
        np.testing.assert_array_equal(got[mask], x[mask])  # between the strides


@pytest.mark.parametrize("row", [0, 5, 63, 64, 100])
def test_infinite_rows_follow_the_division(cuda, row):
    n = 130
    rng = np.random.default_rng(row)
    a, x = system(rng, n, n, 1), rng.uniform(0.5, 1, n).astype(np.float32)
    zero = a.copy()
    zero[row * n + row] = 0.0
    inf = x.copy()
    inf[row] = np.inf
    plain = np.asarray(oracle.strsv(1, 0, 1, n, a, n, x, 1))
    for got in solve([(1, 0, 1, n, zero, n, x, 1), (1, 0, 1, n, a, n, inf, 1)]):
        np.testing.assert_allclose(got[:row], plain[:row], rtol=1e-4, atol=1e-6)
        assert np.isinf(got[row])
        assert not np.isfinite(got[row + 1:]).any()
