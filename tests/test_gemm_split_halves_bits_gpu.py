"""Split-BF16 GEMM: tiles that go as two halves give the bits of whole tiles.  K is one
slab (32), so the direction a wave walks its slabs in plays no part."""
import pytest
import torch

from test_gemm_split_halves_gpu import _gemm

pytestmark = pytest.mark.gpu


# 128 x 256 tiles on 148 SMs: 2001 x 3003 has 192 of them, 44 in the last wave; 149 tiles
@pytest.mark.parametrize("m,n", [(2001, 3003), (128 * 111, 512), (128 * 100 - 5, 3 * 256 + 130)])
@pytest.mark.parametrize("k", [1, 19, 32])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_halves_give_the_bits_of_whole_tiles(m, n, k, beta):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(k, m, device="cuda", generator=g)      # column-major m x k
    b = torch.randn(n, k, device="cuda", generator=g)      # column-major k x n
    c0 = torch.randn(n, m, device="cuda", generator=g)
    got = _gemm(0, 0, a, b, c0.clone(), m, n, k, beta)
    want = torch.empty_like(c0)
    step = 256 * max(1, 148 // ((m + 127) // 128))         # at most one wave: whole tiles only
    for j in range(0, n, step):
        w = min(step, n - j)
        want[j:j + w] = _gemm(0, 0, a, b[j:j + w].contiguous(), c0[j:j + w].clone(), m, w, k, beta)
    assert torch.equal(got, want)
