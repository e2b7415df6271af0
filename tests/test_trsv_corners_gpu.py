"""DTRSV / CTRSV / ZTRSV: the corner substitution and the panel staging at block
and cluster edges (blocks of 64 rows, corners of 8 or 4, clusters of 16 blocks)."""
import numpy as np
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu

TYPES = {"d": (torch.float64, np.float64, np.longdouble, "dtrsv"),
         "c": (torch.complex64, np.complex64, np.complex128, "ctrsv"),
         "z": (torch.complex128, np.complex128, np.clongdouble, "ztrsv")}


def _system(t, n, seed):
    rng = np.random.default_rng(seed)
    dt = TYPES[t][1]
    a = rng.standard_normal((n, n)) / np.sqrt(n)
    b = rng.standard_normal(n)
    if t != "d":
        a = a + 1j * rng.standard_normal((n, n)) / np.sqrt(n)
        b = b + 1j * rng.standard_normal(n)
    a[np.arange(n), np.arange(n)] += 2.0
    return a.astype(dt), b.astype(dt)


def _solve(t, uplo, trans, unit, a, b, pad=0, incx=1):
    n = len(b)
    dt = TYPES[t][0]
    am = torch.full((n, n + pad), float("nan"), dtype=dt, device="cuda")   # column j at row j
    am[:, :n] = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    x = torch.zeros(n * incx, dtype=dt, device="cuda")
    x[::incx] = torch.from_numpy(b).cuda()
    getattr(cb, TYPES[t][3])(uplo, trans, 0 if unit else 1, n, am, n + pad, x, incx)
    return x[::incx].cpu().numpy()


def _op(a, uplo, trans, unit):
    m = np.tril(a) if uplo == 1 else np.triu(a)
    if unit:
        m = m.copy()
        np.fill_diagonal(m, 1)
    return m if trans == 0 else (m.T if trans == 1 else m.conj().T)


@pytest.mark.parametrize("unit", [False, True])
@pytest.mark.parametrize("trans", [0, 1, 2])
@pytest.mark.parametrize("uplo", [0, 1])
@pytest.mark.parametrize("t", ["d", "c", "z"])
def test_block_and_cluster_edges(t, uplo, trans, unit):
    eps = np.finfo(TYPES[t][1]).eps
    for n, pad, incx in ((1, 0, 1), (7, 3, 2), (63, 0, 1), (65, 1, 3), (127, 5, 1), (200, 0, 1), (1025, 7, 1)):
        a, b = _system(t, n, n)
        x = _solve(t, uplo, trans, unit, a, b, pad, incx)
        w = TYPES[t][2]
        m = _op(a, uplo, trans, unit).astype(w)
        resid = np.abs(b.astype(w) - m @ x.astype(w))
        # row-wise backward error of substitution: n + 2 roundings of the sums, the
        # scaled row's two and the reciprocal's one; complex products take 2 sqrt 2
        bound = (n + 6) * eps * (1 if t == "d" else 3) * (np.abs(m) @ np.abs(x.astype(w)) + np.abs(b))
        assert np.all(resid <= bound), (n, float(np.max(resid / bound)))


@pytest.mark.parametrize("k", [0, 3, 12, 40, 63, 70])
@pytest.mark.parametrize("uplo", [0, 1])
@pytest.mark.parametrize("t", ["d", "c", "z"])
def test_zero_pivot_reaches_later_rows_only(t, uplo, k):
    n = 150
    a, b = _system(t, n, 5)
    clean = _solve(t, uplo, 0, False, a, b)
    row = k if uplo == 1 else n - 1 - k
    a[row, row] = 0
    x = _solve(t, uplo, 0, False, a, b)
    before, after = (slice(0, row), slice(row, n)) if uplo == 1 else (slice(row + 1, n), slice(0, row + 1))
    assert np.array_equal(x[before], clean[before])
    assert not np.isfinite(x[after]).any()
