"""Waits that run out: with a limit of some nanoseconds a tensor-core call either still
finishes (the wait instruction itself may outlast the limit) or winds down and reports
a timeout; the next call on the handle is right either way."""
import numpy as np
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu


def _gemm(mode, dtype, tile=(0, 0, 0)):
    g = torch.Generator(device="cuda").manual_seed(3)
    m, n, k = 700, 900, 1100
    a, b = (torch.empty(s, dtype=dtype, device="cuda").uniform_(-1, 1, generator=g) for s in ((k, m), (n, k)))
    c = torch.empty(n, m, dtype=dtype, device="cuda")
    fn = cb.sgemm if dtype == torch.float32 else cb.dgemm
    h = cb.handle()

    def call():
        c.fill_(float("nan"))
        cb.set_gemm_mode(mode)
        h.set_gemm_tile(*tile)
        fn(0, 0, m, n, k, 1.0, a, m, b, k, 0.0, c, m)
        h.set_gemm_tile(0, 0, 0)
        cb.set_gemm_mode(cb.GemmMode.NATIVE)
        return c
    return call


def _grouped(bf16):
    g = torch.Generator(device="cuda").manual_seed(4)
    count, n = 600, 100
    a = torch.empty(count, n, n, device="cuda").uniform_(-1, 1, generator=g)
    if bf16:
        a = a.bfloat16()
    c = torch.empty(count, n, n, device="cuda")
    rec = np.zeros(count, dtype=cb.sgemm_problem_dtype())
    rec["m"] = rec["n"] = rec["k"] = rec["lda"] = rec["ldb"] = rec["ldc"] = n
    rec["op_a"], rec["alpha"] = np.arange(count) % 2, 1.0
    i = np.arange(count) * n * n
    rec["a"], rec["b"], rec["c"] = (t.data_ptr() + t.element_size() * i for t in (a, a, c))
    probs = torch.from_numpy(rec.view(np.uint8)).cuda()

    def call():
        c.fill_(float("nan"))
        cb.set_gemm_mode(cb.GemmMode.SPLIT_BF16X3)
        cb.sgemm_grouped(1 if bf16 else 0, count, probs)
        cb.set_gemm_mode(cb.GemmMode.NATIVE)
        return c
    call.keep = (a, probs)
    return call


@pytest.mark.parametrize("make", [
    lambda: _gemm(cb.GemmMode.SPLIT_BF16X3, torch.float32, (128, 256, 1)),
    lambda: _gemm(cb.GemmMode.SPLIT_BF16X3, torch.float32, (128, 128, 4)),
    lambda: _gemm(cb.GemmMode.SPLIT_BF16X6, torch.float32, (128, 128, 1)),
    lambda: _gemm(cb.GemmMode.OZAKI_INT8, torch.float64),
    lambda: _grouped(False), lambda: _grouped(True)], ids=["x3", "x3 split K", "x6", "ozaki", "grouped", "grouped bf16"])
def test_a_short_limit_ends_and_leaves_the_handle_usable(cuda, make):
    call, h = make(), cb.handle()
    want = call().clone()
    h.sync()
    for _ in range(3):
        h.set_wait_limit(1)
        try:
            got = call()
            h.sync()
            assert torch.equal(got, want)
        except cb.CoralError as e:
            assert e.status == 3
        finally:
            h.set_wait_limit(0)
        assert torch.equal(call(), want)
        h.sync()
