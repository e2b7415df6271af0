"""Split-BF16 GEMM: last waves that go as half tiles, against the 64-bit product and
against calls of whole tiles only."""
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu


def _gemm(op_a, op_b, a, b, c, m, n, k, beta):
    h = cb.handle()
    cb.set_gemm_mode(cb.GemmMode.SPLIT_BF16X3)
    h.set_gemm_tile(128, 256, 1)
    try:
        cb.sgemm(op_a, op_b, m, n, k, 1.5, a, a.shape[1], b, b.shape[1], beta, c, m)
    finally:
        h.set_gemm_tile(0, 0, 0)
        cb.set_gemm_mode(cb.GemmMode.NATIVE)
    return c


# tiles of 128 x 256 on 148 SMs: one more than a wave, 74 more (the most that are
# halved), 75 more (not halved), ragged sides, and two waves and a bit
@pytest.mark.parametrize("m,n,k", [(128 * 149, 256, 96), (128 * 111, 512, 40), (128 * 223, 256, 64),
                                   (2001, 3003, 77), (2050, 3203, 33), (128 * 100 - 5, 3 * 256 + 130, 50)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_halves_equal_whole_tiles(m, n, k, beta):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(k, m, device="cuda", generator=g)      # column-major m x k
    b = torch.randn(n, k, device="cuda", generator=g)      # column-major k x n
    c0 = torch.randn(n, m, device="cuda", generator=g)
    got = _gemm(0, 0, a, b, c0.clone(), m, n, k, beta)
    # the same columns in calls of at most one wave of whole tiles
    want = c0.clone()
    step = 256 * max(1, 148 // ((m + 127) // 128))
    if (m + 127) // 128 <= 148:
        for j in range(0, n, step):
            w = min(step, n - j)
            want[j:j + w] = _gemm(0, 0, a, b[j:j + w].contiguous(), c0[j:j + w].clone(), m, w, k, beta)
    else:
        half = 128 * 100
        for i, rows in ((0, half), (half, m - half)):
            part = _gemm(0, 0, a[:, i:i + rows].contiguous(), b, c0[:, i:i + rows].contiguous(), rows, n, k, beta)
            want[:, i:i + rows] = part
    # two bf16 pieces hold a value to 2^-18 of it and the product a1 b1 left out is
    # 2^-18 of a term: 3 * 2^-18; each of the 3 k tensor-core additions and the
    # epilogue's adds a 2^-23
    ref = 1.5 * (b.double() @ a.double()) + beta * c0.double()
    scale = 1.5 * (b.double().abs() @ a.double().abs()) + abs(beta) * c0.double().abs()
    assert ((got.double() - ref).abs() <= (3 * 2 ** -18 + (3 * k + 4) * 2 ** -23) * scale).all()
    assert ((got.double() - want.double()).abs() <= 2 * (3 * k + 4) * 2 ** -23 * scale).all()
