"""Scalar results of the reductions at the edges of one block (2048 and 4096
elements), delivered to the host and to device memory; whole-number data, so every
sum is exact."""
import ctypes as C

import numpy as np
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu

N = (1, 2, 2047, 2048, 2049, 4095, 4096, 4097, 9000)


def _vector(rng, n, dtype):
    v = rng.integers(-40, 41, n).astype(dtype)
    return v + 1j * rng.integers(-40, 41, n) if np.iscomplexobj(v) else v


@pytest.mark.parametrize("inc", [1, 2])
@pytest.mark.parametrize("t,dtype", [("s", np.float32), ("d", np.float64), ("c", np.complex64),
                                     ("z", np.complex128)])
def test_results_exact_in_both_pointer_modes(t, dtype, inc):
    rng = np.random.default_rng(7)
    h = cb.blas.handle()
    for n in N:
        x, y = (_vector(rng, n, dtype).astype(dtype) for _ in range(2))
        x[n // 2] = 100
        X, Y = (torch.zeros(n * inc, dtype=torch.from_numpy(x).dtype, device="cuda") for _ in range(2))
        X[::inc], Y[::inc] = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        dot, asum, amax = {"s": ("sdot", "sasum", "isamax"), "d": ("ddot", "dasum", "idamax"),
                           "c": ("cdotu", "scasum", "icamax"), "z": ("zdotu", "dzasum", "izamax")}[t]
        want = (np.dot(x, y), np.sum(np.abs(x.real) + np.abs(x.imag)), n // 2)
        got = (getattr(cb, dot)(n, X, inc, Y, inc), getattr(cb, asum)(n, X, inc), getattr(cb, amax)(n, X, inc))
        assert got == want, n
        out = torch.zeros(3, 2, dtype=torch.float64, device="cuda")   # 16 bytes a result
        h.set_pointer_mode(1)
        try:
            px, py = C.c_void_p(X.data_ptr()), C.c_void_p(Y.data_ptr())
            at = [C.c_void_p(out.data_ptr() + 16 * i) for i in range(3)]
            h.call("coral_" + dot, n, px, inc, py, inc, at[0])
            h.call("coral_" + asum, n, px, inc, at[1])
            h.call("coral_" + amax, n, px, inc, at[2])
        finally:
            h.set_pointer_mode(0)
        raw = out.cpu().numpy()
        real = np.float32 if t in "sc" else np.float64
        assert raw[0].view(dtype)[0] == want[0] and raw[1].view(real)[0] == want[1], n
        assert raw[2].view(np.uint64)[0] == want[2], n
