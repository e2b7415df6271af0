"""Batched STRSV calls of one handle that run at the same time: two captured calls replayed on
two streams, and calls on streams that are set by hand.  Each has its own tickets, so each
solves what it solves alone, bit for bit, and so does the call after."""
import ctypes

import numpy as np
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu


class Batch:
    """`count` unit lower systems of 32 to 300 rows; run() solves copies of the right-hand sides."""

    def __init__(self, count, seed):
        rng = np.random.default_rng(seed)
        n = np.exp(rng.uniform(np.log(32), np.log(300), count)).astype(np.int64)
        at = lambda s: np.concatenate([[0], np.cumsum(s)[:-1]])
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.a = torch.empty(int((n * n).sum()), device="cuda").uniform_(-1, 1, generator=g) / 300
        self.b = torch.empty(int(n.sum()), device="cuda").uniform_(-1, 1, generator=g)
        self.x = torch.empty_like(self.b)
        rec = np.zeros(count, dtype=cb.strsv_problem_dtype())
        rec["uplo"], rec["trans"], rec["diag"], rec["n"] = 1, 0, 0, n
        rec["a"], rec["x"] = self.a.data_ptr() + 4 * at(n * n), self.x.data_ptr() + 4 * at(n)
        rec["lda"], rec["incx"] = n, 1
        self.count, self.desc = count, torch.from_numpy(rec.view(np.uint8)).cuda()

    def run(self):
        self.x.copy_(self.b)
        cb.strsv_batched(self.count, self.desc)

    def wanted(self):
        self.run()
        torch.cuda.synchronize()
        self.want = self.x.clone()
        self.x.zero_()
        return self


@pytest.mark.parametrize("counts", [(700, 1000), (1500, 2500), (500, 3000)])
def test_captured_calls_side_by_side(cuda, counts):
    batches = [Batch(c, i).wanted() for i, c in enumerate(counts)]
    graphs = []
    for b in batches:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            b.run()
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in batches]
    torch.cuda.synchronize()
    for rep in range(20):
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
        torch.cuda.synchronize()
        for b in batches:
            assert torch.equal(b.x, b.want), (rep, b.count)
    for b in batches:
        b.x.zero_()
        b.run()
        torch.cuda.synchronize()
        assert torch.equal(b.x, b.want), b.count


def test_calls_on_streams_set_by_hand(cuda):
    batches = [Batch(c, 10 + c).wanted() for c in (700, 1500)]
    streams = [torch.cuda.Stream() for _ in batches]
    h = cb.handle()
    for rep in range(20):
        for b in batches:
            b.x.copy_(b.b)
        torch.cuda.synchronize()
        for b, s in zip(batches, streams):
            h.lib.coral_set_stream(h.h, ctypes.c_void_p(s.cuda_stream))
            h.check(h.lib.coral_strsv_batched(h.h, b.count, ctypes.c_void_p(b.desc.data_ptr())), "coral_strsv_batched")
        torch.cuda.synchronize()
        for b in batches:
            assert torch.equal(b.x, b.want), (rep, b.count)
