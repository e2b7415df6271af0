"""The split GEMM's default rule has one place, the library: what tuning.default_choice
calls the default is what a call without a selector runs."""
import pytest

from coral_b200 import tuning


@pytest.mark.parametrize("shape,tile", [
    ((4096, 4096, 256, 0, 0), (128, 128, 1)),     # K of 5 slabs or fewer: 128 columns, not pairs
    ((4096, 4096, 321, 0, 0), (256, 256, 1)),
    ((1500, 1500, 700, 0, 0), (128, 128, 1)),     # one wave of 128 x 128
    ((4096, 4096, 256, 0, 0, 6), (256, 256, 1)),  # the short-K line is for three products
    ((700, 700, 1000, 0, 0), (128, 256, 8)),      # few tiles, deep K
    ((64, 64, 1 << 20, 0, 0), (128, 256, 16)),
    ((0, 64, 4096, 0, 0), (128, 128, 1)),         # no tiles at all
])
def test_default_choice_is_the_librarys(shape, tile):
    assert tuning.CANDIDATES[tuning.default_choice(shape)] == tile


@pytest.mark.gpu
def test_default_choice_is_what_a_call_runs(cuda):
    import torch

    import coral_b200 as cb
    h = cb.Handle()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for s in tuning.generate_shapes(400, seed=17):
        products = tuning.shape_products(s)
        want = tuning.CANDIDATES[tuning.default_choice(s, sms)]
        assert h.gemm_tile(products, int(s[3]), int(s[4]), *(int(v) for v in s[:3])) == want, s
