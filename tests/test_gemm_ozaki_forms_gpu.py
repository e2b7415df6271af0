"""Ozaki DGEMM / ZGEMM at the lines between its forms: single tiles (one per CTA, one
chunk of K) and several per CTA, 64 and 128 columns wide, slices of 32 and of 128 K
values per CTA, with ragged sides.  Against the 64-bit product with the tolerance of
the Ozaki tests, 1e-13 of |alpha| |op(A)||op(B)| + |beta||C|."""
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (127, 65, 31), (129, 63, 33), (300, 130, 127), (17, 1000, 129), (640, 1850, 40),
          (4000, 510, 70), (4700, 33, 129), (128, 64, 9472), (128, 64, 9473)]


@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128], ids=["d", "z"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_forms(cuda, shape, dtype):
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a, b, c0 = (torch.randn(s, dtype=dtype, device="cuda", generator=g) for s in ((k, m), (n, k), (n, m)))
    ab = b @ a
    mag = b.abs() @ a.abs()
    fn, alpha = (cb.dgemm, -1.25) if dtype == torch.float64 else (cb.zgemm, 1.5 - 0.5j)
    for beta in (0.0, 1.0, 0.5 if dtype == torch.float64 else 0.25 + 1j):
        c = c0.clone()
        if beta == 0.0:
            c.fill_(float("nan"))      # not read
        cb.set_gemm_mode(cb.GemmMode.OZAKI_INT8)
        try:
            fn(0, 0, m, n, k, alpha, a, m, b, k, beta, c, m)
        finally:
            cb.set_gemm_mode(cb.GemmMode.NATIVE)
        want = alpha * ab + (beta * c0 if beta != 0.0 else 0.0)
        scale = abs(alpha) * mag + abs(beta) * c0.abs()
        assert ((c - want).abs() <= 1e-13 * scale).all(), beta
