"""Batched STRSV where systems of up to 32 rows take a warp each: sizes around that line
in every form, batches of one window (1024 instances) and of several, and tickets that
are back at zero for the next call.  Oracle and tolerance of the batched test,
|x - x_ref| <= 1e-4 max(|x|, |x_ref|) + 1e-6."""
import numpy as np
import pytest

import oracle
from test_batched_trsv_gpu import solve, system

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 3, 7, 8, 9, 16, 17, 31, 32, 33, 40, 64, 65]


def _cases(count, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        n = int(rng.choice(SIZES)) if i % 97 else 200
        uplo, trans, diag, incx = (int(v) for v in (i % 2, i // 2 % 3, i // 6 % 2, 1 + i // 12 % 3))
        lda = max(1, n + i % 3)
        out.append((uplo, trans, diag, n, system(rng, n, lda, diag), lda,
                    rng.uniform(-1, 1, max(0, (n - 1) * incx) + 1).astype(np.float32), incx))
    return out


def _check(cases, results):
    for case, got in zip(cases, results):
        uplo, trans, diag, n, a, lda, x, incx = case
        if n == 0:
            np.testing.assert_array_equal(got, x)
            continue
        want = np.asarray(oracle.strsv(uplo, trans, diag, n, a, lda, x, incx))
        err, mag = np.abs(got[::incx][:n] - want), np.maximum(np.abs(got[::incx][:n]), np.abs(want))
        assert (err <= 1e-4 * mag + 1e-6).all(), (case[:4], float(err.max()))


@pytest.mark.parametrize("count", [297, 1023, 1024, 1025, 2500])
def test_small_systems(cuda, count):
    for seed in (1, 2):     # the second call finds the tickets as the first did
        cases = _cases(count, seed)
        _check(cases, solve(cases))


@pytest.mark.parametrize("n,row", [(1, 0), (5, 4), (32, 0), (32, 31), (31, 7)])
def test_small_rows_that_need_the_division(cuda, n, row):
    """A zero, a tiny and a huge diagonal entry, and an infinite right-hand side."""
    rng = np.random.default_rng(n + row)
    a, x = system(rng, n, n, 1), rng.uniform(0.5, 1, n).astype(np.float32)
    filler = [(1, 0, 1, 4, system(rng, 4, 4, 1), 4, np.ones(4, np.float32), 1)] * 300
    plain = np.asarray(oracle.strsv(1, 0, 1, n, a, n, x, 1))
    zero, tiny, huge, inf = a.copy(), a.copy(), a.copy(), x.copy()
    zero[row * n + row], tiny[row * n + row], huge[row * n + row] = 0.0, 1e-30, 1e30
    inf[row] = np.inf
    got = solve([(1, 0, 1, n, m, n, b, 1) for m, b in ((zero, x), (a, inf), (tiny, x), (huge, x))] + filler)
    for g in got[:2]:
        np.testing.assert_allclose(g[:row], plain[:row], rtol=1e-4, atol=1e-6)
        assert np.isinf(g[row]) and not np.isfinite(g[row + 1:]).any()
    for g, m in zip(got[2:4], (tiny, huge)):
        want = np.asarray(oracle.strsv(1, 0, 1, n, m, n, x, 1))
        np.testing.assert_allclose(g, want, rtol=1e-4, atol=1e-6)
