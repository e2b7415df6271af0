"""Grouped SGEMM over batches that leave the plan's and the scheduler's usual
range: more instances than the plan keeps in registers, descriptors off the
16-byte boundary, fewer tiles than SMs, empty instances among them, and tiles
whose rows, columns and K end inside a 32-row block or a 32-deep slab, in all
four operation pairs.  Component-wise tolerance 4e-5 against float64, as in the
other grouped tests (split-BF16x3: 2^-16 per product plus fp32 accumulation).
"""
import numpy as np
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu


def run(shapes, bf16, desc_offset=0, seed=0):
    rng = np.random.default_rng(seed)
    dt = torch.bfloat16 if bf16 else torch.float32
    rec = np.zeros(len(shapes), dtype=cb.sgemm_problem_dtype())
    sizes = np.array([(m * k, k * n, m * n) for _, _, m, n, k in shapes])
    at = np.concatenate([np.zeros((1, 3), np.int64), np.cumsum(sizes, axis=0)])
    a, b, c = (torch.from_numpy(rng.uniform(-1, 1, max(1, int(at[-1][i]))).astype(np.float32)).cuda() for i in range(3))
    a, b, c0 = a.to(dt), b.to(dt), c.clone()
    for i, (op_a, op_b, m, n, k) in enumerate(shapes):
        rec[i] = (op_a, op_b, m, n, k, 1.5, 0.5, 0, a.data_ptr() + int(at[i][0]) * a.element_size(),
                  b.data_ptr() + int(at[i][1]) * b.element_size(), c.data_ptr() + int(at[i][2]) * 4,
                  max(1, k if op_a else m), max(1, n if op_b else k), max(1, m))
    raw = np.zeros(desc_offset + rec.nbytes, np.uint8)
    raw[desc_offset:] = rec.view(np.uint8)
    desc = torch.from_numpy(raw).cuda()[desc_offset:]
    h = cb.handle()
    h.set_gemm_mode(cb.GemmMode.SPLIT_BF16X3)
    try:
        cb.sgemm_grouped(1 if bf16 else 0, len(shapes), desc)
    finally:
        h.set_gemm_mode(cb.GemmMode.NATIVE)
    got, c0 = c.double(), c0.double()
    for i, (op_a, op_b, m, n, k) in enumerate(shapes):
        av, bv = a[at[i][0]:at[i][0] + m * k].double(), b[at[i][1]:at[i][1] + k * n].double()
        av = av.view(m, k) if op_a else av.view(k, m).T
        bv = bv.view(k, n) if op_b else bv.view(n, k).T
        cv = c0[at[i][2]:at[i][2] + m * n].view(n, m).T
        want, bound = 1.5 * (av @ bv) + 0.5 * cv, 1.5 * (av.abs() @ bv.abs()) + 0.5 * cv.abs()
        err = (got[at[i][2]:at[i][2] + m * n].view(n, m).T - want).abs()
        assert (err <= 4e-5 * bound + 1e-30).all(), (i, shapes[i])


@pytest.mark.parametrize("bf16", [False, True])
def test_block_and_slab_edges(cuda, bf16):
    edges = [1, 7, 31, 32, 33, 65, 127, 129]
    shapes = [(i & 1, (i >> 1) & 1, edges[i % 8], edges[(i // 3) % 8], edges[(i // 5) % 8]) for i in range(120)]
    run(shapes + [(0, 0, 130, 300, 70), (1, 1, 257, 64, 1), (1, 0, 40, 513, 95)], bf16)


@pytest.mark.parametrize("count,offset", [(4097, 8), (9000, 0), (3, 8)])
def test_counts_and_descriptor_alignment(cuda, count, offset):
    rng = np.random.default_rng(count)
    m, n, k = rng.integers(0, 40, (3, count))
    ops = rng.integers(0, 2, (2, count))
    m[0], n[0], k[0] = 200, 30, 20
    run([tuple(int(v) for v in s) for s in zip(*ops, m, n, k)], False, offset, seed=count)
