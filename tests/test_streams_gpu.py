"""One thread's calls on several torch streams share the handle's scratch, arrival
counters and TRSV slots: a call waits for the call before it, whichever streams they
are on, and results are those of one stream.  The first call is long (some
milliseconds), so that an unordered second one would run into it."""
import ctypes

import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu


def _uniform(shape, seed, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.empty(shape, dtype=dtype, device="cuda").uniform_(-1, 1, generator=g)


def _work():
    """(long call, short call) pairs on shared state, each filling its own output."""
    n, k = 3072, 1024
    a, b = _uniform((n, n), 1), _uniform((n, n), 2)
    d = [_uniform((k, k), 3 + i, torch.float64) for i in range(2)]
    tri = _uniform((n, n), 5, torch.float64)
    tri.diagonal().add_(n)

    def split(x, y, c, m):
        cb.set_gemm_mode(cb.GemmMode.SPLIT_BF16X6)
        cb.sgemm(0, 0, m, m, m, 1.0, x, n, y, n, 0.0, c, m)
        cb.set_gemm_mode(cb.GemmMode.NATIVE)

    def ozaki(x, y, c, m):
        cb.set_gemm_mode(cb.GemmMode.OZAKI_INT8)
        cb.dgemm(0, 0, m, m, m, 1.0, x, k, y, k, 0.0, c, m)
        cb.set_gemm_mode(cb.GemmMode.NATIVE)

    return [
        (lambda: [split(a, b, c := torch.empty(n, n, device="cuda"), n), c][1],
         lambda: [split(b, a, c := torch.empty(512, 512, device="cuda"), 512), c][1]),
        (lambda: [ozaki(d[0], d[1], c := torch.empty(k, k, dtype=torch.float64, device="cuda"), k), c][1],
         lambda: [ozaki(d[1], d[0], c := torch.empty(300, 300, dtype=torch.float64, device="cuda"), 300), c][1]),
        (lambda: [cb.dtrsv(1, 0, 1, n, tri, n, x := tri[7].clone(), 1), x][1],
         lambda: [cb.dtrsv(1, 1, 1, n, tri, n, x := tri[9].clone(), 1), x][1]),
        (lambda: [cb.ssymv(0, n, 1.0, a, n, a[3].contiguous(), 1, 0.0, y := torch.zeros(n, device="cuda"), 1), y][1],
         lambda: [cb.sgemv(0, n, n, 1.0, b, n, b[4].contiguous(), 1, 0.0, y := torch.zeros(n, device="cuda"), 1), y][1]),
    ]


def _streams(external):
    own = [torch.cuda.Stream() for _ in range(2)]
    return own, [torch.cuda.ExternalStream(s.cuda_stream) for s in own] if external else own


@pytest.mark.parametrize("external", [False, True])
def test_calls_on_two_streams(cuda, external):
    work = _work()
    want = [(f(), g()) for f, g in work]      # (also sizes the scratch)
    torch.cuda.synchronize()
    keep, (s, t) = _streams(external)
    for rep in range(5):
        for i, (f, g) in enumerate(work):
            with torch.cuda.stream(s):
                x = f()
            with torch.cuda.stream(t):
                y = g()
            with torch.cuda.stream(s):
                z = g()
            torch.cuda.synchronize()
            assert torch.equal(x, want[i][0]) and torch.equal(y, want[i][1]) and torch.equal(z, want[i][1]), (rep, i)


def test_stream_set_by_hand_between_calls(cuda):
    """A direct coral_set_stream is the caller's to order, and does not outlast the next call."""
    work = _work()
    want = [(f(), g()) for f, g in work]
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    h = cb.handle()
    for i, (f, g) in enumerate(work):
        h.lib.coral_set_stream(h.h, ctypes.c_void_p(s.cuda_stream))
        x = f()
        bound = ctypes.c_void_p()
        h.lib.coral_get_stream(h.h, ctypes.byref(bound))
        assert (bound.value or 0) == torch.cuda.current_stream().cuda_stream
        with torch.cuda.stream(s):
            y = g()
        torch.cuda.synchronize()
        assert torch.equal(x, want[i][0]) and torch.equal(y, want[i][1]), i


def test_capture_after_work_on_another_stream(cuda):
    """A capture takes no dependency on work outside of it, inside it the streams are ordered."""
    work = _work()
    want = [(f(), g()) for f, g in work]
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    for i, (f, g) in enumerate(work):
        with torch.cuda.stream(other):
            f()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            x = f()
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                y = g()
            torch.cuda.current_stream().wait_stream(side)
        with torch.cuda.stream(other):
            z = g()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, want[i][0]) and torch.equal(y, want[i][1]) and torch.equal(z, want[i][1]), i
