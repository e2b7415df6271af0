"""Split-BF16 GEMM with 256-column tiles whose second box of B lies past the last row and
is not loaded: what an earlier call left in its place (infinities here) may not show.
Bound as in the half tiles' test: 3 * 2^-18 of the terms for the dropped pieces, 2^-23
for each of the 3 k tensor-core additions and the epilogue's, and one per K part."""
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [1, 4])
@pytest.mark.parametrize("m,n,k", [(130, 1, 300), (300, 100, 513), (128, 128, 64), (200, 129, 100), (129, 300, 260)])
def test_narrow_products(cuda, m, n, k, splits):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    h = cb.handle()
    inf = torch.full((512, 512), float("inf"), device="cuda")

    def gemm(a, b, c, m, n, k):
        cb.set_gemm_mode(cb.GemmMode.SPLIT_BF16X3)
        h.set_gemm_tile(128, 256, splits)
        try:
            cb.sgemm(0, 0, m, n, k, 1.5, a, m, b, k, 0.5, c, m)
        finally:
            h.set_gemm_tile(0, 0, 0)
            cb.set_gemm_mode(cb.GemmMode.NATIVE)

    a, b, c0 = (torch.randn(s, device="cuda", generator=g) for s in ((k, m), (n, k), (n, m)))
    gemm(inf, inf, torch.zeros_like(inf), 512, 512, 512)
    c = c0.clone()
    gemm(a, b, c, m, n, k)
    ref = 1.5 * (b.double() @ a.double()) + 0.5 * c0.double()
    scale = 1.5 * (b.double().abs() @ a.double().abs()) + 0.5 * c0.double().abs()
    assert ((c.double() - ref).abs() <= (3 * 2 ** -18 + (3 * k + 4 + splits) * 2 ** -23) * scale).all()
