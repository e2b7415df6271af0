"""SYMV / HEMV / TRMV: the diagonal blocks at their edges.  The unstored triangle
holds NaN and one entry of x is infinite: only outputs whose stored elements meet
that entry may be affected, and they are infinite, not NaN (real types)."""
import numpy as np
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu

DT = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}


def _stored(t, n, uplo, seed):
    g = torch.Generator().manual_seed(seed)
    a = torch.rand(n, n, generator=g, dtype=torch.float64) + 0.5
    a = a.to(DT[t])
    i = torch.arange(n)
    keep = i[:, None] >= i[None, :] if uplo == 1 else i[:, None] <= i[None, :]
    return torch.where(keep, a, torch.full_like(a, float("nan"))), keep


@pytest.mark.parametrize("uplo", [0, 1])
@pytest.mark.parametrize("n,pad", [(1, 0), (17, 3), (64, 0), (65, 1), (130, 2), (200, 0)])
@pytest.mark.parametrize("t", ["s", "d", "c", "z"])
def test_infinite_entry(t, n, pad, uplo):
    a, keep = _stored(t, n, uplo, n)
    am = torch.full((n, n + pad), float("nan"), dtype=DT[t])
    am[:, :n] = a.T
    am = am.cuda()
    for k in sorted({0, n // 3, min(63, n - 1), n - 1}):
        x = torch.zeros(n, dtype=DT[t])
        x[k] = float("inf")
        y = torch.zeros(n, dtype=DT[t], device="cuda")
        {"s": cb.ssymv, "d": cb.dsymv, "c": cb.chemv, "z": cb.zhemv}[t](uplo, n, 1.0, am, n + pad, x.cuda(), 1,
                                                                        0.0, y, 1)
        if t in "sd":
            assert torch.isinf(y).all() and (y > 0).all(), k
        else:
            assert not torch.isfinite(torch.view_as_real(y)).all(1).any(), k
        for trans in (0, 1, 2):
            z = x.cuda()
            {"s": cb.strmv, "d": cb.dtrmv, "c": cb.ctrmv, "z": cb.ztrmv}[t](uplo, trans, 1, n, am, n + pad, z, 1)
            hit = (keep[:, k] if trans == 0 else keep[k, :]).numpy()
            got = z.cpu().numpy()
            assert np.array_equal(~np.isfinite(got), hit), (trans, k)
            if t in "sd":
                assert np.all(np.isposinf(got[hit])) and np.all(got[~hit] == 0), (trans, k)
