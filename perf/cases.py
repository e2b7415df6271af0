"""The timed cases: what a program that uses this BLAS engine has it do.

Every case goes through the public entry points of ``coral_b200`` on CUDA
tensors.  The sizes are the ones the repository's benchmark and tests quote
(8192 SGEMM / GEMV / SYMV, 4096 DGEMM and triangular solves, 512 plain SGEMM,
the 4096-instance grouped GEMM, the 1024-instance batched solve, vectors of
2^26), plus small, odd and unaligned ones.  Matrices are column-major; a
tensor ``view(cols, ld)`` of one is its transpose.
"""
import math

import numpy as np
import torch

import coral_b200 as cb

DTYPE = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
SIZE = {"s": 4, "d": 8, "c": 8, "z": 16}
MODE = {"native": cb.GemmMode.NATIVE, "split3": cb.GemmMode.SPLIT_BF16X3,
        "split6": cb.GemmMode.SPLIT_BF16X6, "ozaki": cb.GemmMode.OZAKI_INT8}


def listed():
    return [
        # Vector steps of an iterative solver on a small system: three calls,
        # two of which hand a scalar back to the host; latency is all there is.
        {"name": "vectors_1000", "kind": "vectors", "dtype": "s", "n": 1000, "inc": 1},
        # The same steps on vectors that fill HBM pages rather than caches.
        {"name": "vectors_2e26", "kind": "vectors", "dtype": "s", "n": 1 << 26, "inc": 1},
        # A dense matrix applied both ways and updated by rank one (bidiagonalisation,
        # quasi-Newton): GEMV N, GEMV T, GER.
        {"name": "gemv_ger_8192", "kind": "gemv_ger", "dtype": "s", "m": 8192, "n": 8192, "pad": 0},
        # A symmetric operator from its upper triangle (Krylov iterations).
        {"name": "symv_8192", "kind": "symv", "dtype": "s", "n": 8192, "uplo": 0, "pad": 0},
        # Triangular solve with one right-hand side in double precision, the
        # back half of a direct solver.
        {"name": "dtrsv_4096", "kind": "trsv", "dtype": "d", "n": 4096, "uplo": 1, "trans": 0, "pad": 0},
        # The plain FP32 GEMM of ordinary size.
        {"name": "sgemm_512", "kind": "gemm", "dtype": "s", "mode": "native", "op_a": 0, "op_b": 0,
         "m": 512, "n": 512, "k": 512, "pad": 0},
        # Plain FP64 with odd sides and leading dimensions off the vector
        # boundary, one operand transposed (normal equations).
        {"name": "dgemm_ragged_tn", "kind": "gemm", "dtype": "d", "mode": "native", "op_a": 1, "op_b": 0,
         "m": 777, "n": 1001, "k": 1501, "pad": 0},
        # The large FP32 GEMM on the tensor cores.
        {"name": "sgemm_split3_8192", "kind": "gemm", "dtype": "s", "mode": "split3", "op_a": 0, "op_b": 0,
         "m": 8192, "n": 8192, "k": 8192, "pad": 0},
        # A mid-sized one with odd sides and a transposed operand.
        {"name": "sgemm_split3_ragged_tn", "kind": "gemm", "dtype": "s", "mode": "split3", "op_a": 1,
         "op_b": 0, "m": 2001, "n": 3003, "k": 1027, "pad": 0},
        # The large FP64 GEMM by INT8 slices.
        {"name": "dgemm_ozaki_4096", "kind": "gemm", "dtype": "d", "mode": "ozaki", "op_a": 0, "op_b": 0,
         "m": 4096, "n": 4096, "k": 4096, "pad": 0},
        # Thousands of uneven products in one call, fp32 inputs.
        {"name": "grouped_4096", "kind": "grouped", "dtype": "s", "count": 4096, "lo": 16, "hi": 512,
         "sizes": 2024},
        # Thousands of uneven triangular systems in one call.
        {"name": "trsv_batched_1024", "kind": "trsv_batched", "dtype": "s", "count": 1024, "lo": 32,
         "hi": 1024, "sizes": 2024},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges.  Odd leading dimensions come with odd
    sides; `pad` adds rows that are not part of the matrix."""
    kind = rng.choice(["vectors", "gemv_ger", "symv", "trsv", "gemm", "gemm", "gemm", "grouped",
                       "trsv_batched"])
    dt = rng.choice("sdcz")
    pad = rng.choice([0, 0, 3, 8])
    if kind == "vectors":
        return {"kind": kind, "dtype": dt, "n": _log_int(rng, 1000, 1 << (26 if dt == "s" else 24)),
                "inc": rng.choice([1, 1, 1, 2])}
    if kind == "gemv_ger":
        return {"kind": kind, "dtype": dt, "m": _log_int(rng, 256, 8192), "n": _log_int(rng, 256, 8192),
                "pad": pad}
    if kind == "symv":
        return {"kind": kind, "dtype": dt, "n": _log_int(rng, 256, 8192), "uplo": rng.choice([0, 1]),
                "pad": pad}
    if kind == "trsv":
        return {"kind": kind, "dtype": dt, "n": _log_int(rng, 128, 4096), "uplo": rng.choice([0, 1]),
                "trans": rng.choice([0, 1, 2]), "pad": pad}
    if kind == "gemm":
        mode = rng.choice({"s": ["native", "split3", "split3", "split6"], "d": ["native", "ozaki"],
                           "c": ["native", "split3"], "z": ["native", "ozaki"]}[dt])
        hi = {"native": 1024 if dt == "z" else 2048, "split3": 8192 if dt == "s" else 4096,
              "split6": 4096, "ozaki": 4096 if dt == "d" else 2048}[mode]
        return {"kind": kind, "dtype": dt, "mode": mode, "op_a": rng.choice([0, 1, 2]),
                "op_b": rng.choice([0, 1, 2]), "m": _log_int(rng, 64, hi), "n": _log_int(rng, 64, hi),
                "k": _log_int(rng, 64, hi), "pad": pad}
    if kind == "grouped":
        return {"kind": kind, "dtype": rng.choice(["s", "bf16"]), "count": _log_int(rng, 256, 4096),
                "lo": 16, "hi": _log_int(rng, 64, 512), "sizes": rng.randrange(1 << 30)}
    return {"kind": kind, "dtype": "s", "count": _log_int(rng, 64, 1024), "lo": 32,
            "hi": _log_int(rng, 128, 1024), "sizes": rng.randrange(1 << 30)}


# ------------------------------------------------------------------ inputs ----
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, count, dtype):
    """`count` entries uniform in [-1, 1) (both parts, where complex)."""
    t = torch.empty(count, dtype=dtype, device="cuda")
    (torch.view_as_real(t) if dtype.is_complex else t).uniform_(-1, 1, generator=g)
    return t


def _gemm_dims(case):
    """Rows and columns of A, B and C as stored."""
    m, n, k = case["m"], case["n"], case["k"]
    a = (m, k) if case["op_a"] == 0 else (k, m)
    b = (k, n) if case["op_b"] == 0 else (n, k)
    return a, b, (m, n)


def _batch_dims(case, per):
    """Sizes of a batch's instances (one seed's worth per case) and their op(A)."""
    rng = np.random.default_rng(case["sizes"])
    dims = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), (case["count"], per)))
    return np.maximum(1, dims.astype(np.int64)), np.where(rng.uniform(size=case["count"]) < 0.5, 0, 1)


def _starts(sizes):
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind == "vectors":
        dt = DTYPE[case["dtype"]]
        for name in "xy":
            st[name] = _uniform(g, case["n"] * case["inc"], dt)
    elif kind == "gemv_ger":
        dt, m, n = DTYPE[case["dtype"]], case["m"], case["n"]
        st["a"] = _uniform(g, (m + case["pad"]) * n, dt)
        for name, length in (("x", n), ("y", m), ("z", m), ("w", n)):
            st[name] = _uniform(g, length, dt)
    elif kind == "symv":
        dt, n = DTYPE[case["dtype"]], case["n"]
        st["a"] = _uniform(g, (n + case["pad"]) * n, dt)
        st["x"], st["y"] = _uniform(g, n, dt), _uniform(g, n, dt)
    elif kind == "trsv":
        dt, n = DTYPE[case["dtype"]], case["n"]
        st["a"] = _uniform(g, (n + case["pad"]) * n, dt)
        diag = st["a"].view(n, n + case["pad"]).diagonal()
        diag.add_(n)  # n + U[-1, 1): well conditioned
        st["b"], st["x"] = _uniform(g, n, dt), torch.empty(n, dtype=dt, device="cuda")
    elif kind == "gemm":
        dt = DTYPE[case["dtype"]]
        for name, (rows, cols) in zip("abc", _gemm_dims(case)):
            st[name] = _uniform(g, (rows + case["pad"]) * cols, dt)
    elif kind == "grouped":
        bf16 = case["dtype"] == "bf16"
        dims, ops = _batch_dims(case, 3)
        m, n, k = dims[:, 0], dims[:, 1], dims[:, 2]
        oa, ob, oc = _starts(m * k), _starts(k * n), _starts(m * n)
        st["a"], st["b"] = _uniform(g, int(oa[-1]), torch.float32), _uniform(g, int(ob[-1]), torch.float32)
        if bf16:
            st["a"], st["b"] = st["a"].bfloat16(), st["b"].bfloat16()
        st["c"] = _uniform(g, int(oc[-1]), torch.float32)
        rec = np.zeros(case["count"], dtype=cb.sgemm_problem_dtype())
        rec["op_a"], rec["m"], rec["n"], rec["k"] = ops, m, n, k
        rec["alpha"], rec["beta"] = 1.5, 0.5
        es = st["a"].element_size()
        for name, start, size in (("a", oa, es), ("b", ob, es), ("c", oc, 4)):
            rec[name] = st[name].data_ptr() + size * start[:-1]
        rec["lda"], rec["ldb"], rec["ldc"] = np.where(ops == 0, m, k), k, m
        st["problems"] = torch.from_numpy(rec.view(np.uint8)).cuda()
    else:
        n = _batch_dims(case, 1)[0][:, 0]
        oa, ox = _starts(n * n), _starts(n)
        st["a"] = _uniform(g, int(oa[-1]), torch.float32)
        st["b"] = _uniform(g, int(ox[-1]), torch.float32)
        st["x"] = torch.empty_like(st["b"])
        at = np.concatenate([oa[i] + np.arange(s) * (s + 1) for i, s in enumerate(n)])
        st["a"][torch.from_numpy(at).cuda()] += torch.from_numpy(np.repeat(n, n).astype(np.float32)).cuda()
        rec = np.zeros(case["count"], dtype=cb.strsv_problem_dtype())
        rec["uplo"], rec["diag"], rec["n"] = int(cb.CoralTriangular.LowerTriangular), \
            int(cb.CoralDiagonal.NonUnitDiagonal), n
        rec["a"], rec["x"] = st["a"].data_ptr() + 4 * oa[:-1], st["x"].data_ptr() + 4 * ox[:-1]
        rec["lda"], rec["incx"] = n, 1
        st["problems"] = torch.from_numpy(rec.view(np.uint8)).cuda()
    return st


# -------------------------------------------------------------------- pass ----
ALPHA, BETA, STEP = 1.5, 0.5, 1.0 / 1024


def run(st):
    case = st["case"]
    kind, t = case["kind"], case["dtype"]
    if kind == "vectors":
        n, inc, x, y = case["n"], case["inc"], st["x"], st["y"]
        dot = {"s": cb.sdot, "d": cb.ddot, "c": cb.cdotc, "z": cb.zdotc}[t](n, x, inc, y, inc)
        {"s": cb.saxpy, "d": cb.daxpy, "c": cb.caxpy, "z": cb.zaxpy}[t](n, STEP, x, inc, y, inc)
        peak = {"s": cb.isamax, "d": cb.idamax, "c": cb.icamax, "z": cb.izamax}[t](n, x, inc)
        return (dot.real, dot.imag, y, peak) if t in "cz" else (dot, y, peak)
    if kind == "gemv_ger":
        m, n, ld = case["m"], case["n"], case["m"] + case["pad"]
        gemv = {"s": cb.sgemv, "d": cb.dgemv, "c": cb.cgemv, "z": cb.zgemv}[t]
        ger = {"s": cb.sger, "d": cb.dger, "c": cb.cgerc, "z": cb.zgerc}[t]
        gemv(0, m, n, ALPHA, st["a"], ld, st["x"], 1, BETA, st["y"], 1)
        gemv(2, m, n, ALPHA, st["a"], ld, st["z"], 1, BETA, st["w"], 1)
        ger(m, n, STEP, st["z"], 1, st["x"], 1, st["a"], ld)
        return st["y"], st["w"], st["a"]
    if kind == "symv":
        n, ld = case["n"], case["n"] + case["pad"]
        symv = {"s": cb.ssymv, "d": cb.dsymv, "c": cb.chemv, "z": cb.zhemv}[t]
        symv(case["uplo"], n, ALPHA, st["a"], ld, st["x"], 1, BETA, st["y"], 1)
        return st["y"]
    if kind == "trsv":
        n, ld = case["n"], case["n"] + case["pad"]
        {"s": cb.scopy, "d": cb.dcopy, "c": cb.ccopy, "z": cb.zcopy}[t](n, st["b"], 1, st["x"], 1)
        trsv = {"s": cb.strsv, "d": cb.dtrsv, "c": cb.ctrsv, "z": cb.ztrsv}[t]
        trsv(case["uplo"], case["trans"], cb.CoralDiagonal.NonUnitDiagonal, n, st["a"], ld, st["x"], 1)
        return st["x"]
    if kind == "gemm":
        cb.set_gemm_mode(MODE[case["mode"]])
        gemm = {"s": cb.sgemm, "d": cb.dgemm, "c": cb.cgemm, "z": cb.zgemm}[t]
        lda, ldb, ldc = (rows + case["pad"] for rows, _ in _gemm_dims(case))
        gemm(case["op_a"], case["op_b"], case["m"], case["n"], case["k"], ALPHA, st["a"], lda, st["b"], ldb,
             BETA, st["c"], ldc)
        return st["c"]
    if kind == "grouped":
        cb.set_gemm_mode(cb.GemmMode.SPLIT_BF16X3)
        cb.sgemm_grouped(1 if t == "bf16" else 0, case["count"], st["problems"])
        return st["c"]
    cb.scopy(st["b"].numel(), st["b"], 1, st["x"], 1)
    cb.strsv_batched(case["count"], st["problems"])
    return st["x"]


# -------------------------------------------------------------------- work ----
def work(case):
    """Bytes and useful operations of one pass; every call of a pass reads its
    own operands once and writes its results once.  The emulated GEMMs count
    the product they stand for, not the tensor-core products behind it."""
    kind, t = case["kind"], case["dtype"]
    if kind == "grouped":
        m, n, k = (col.astype(float) for col in _batch_dims(case, 3)[0].T)
        es = 2 if t == "bf16" else 4
        return {"bytes": float((es * (m * k + k * n) + 8 * m * n).sum()), "flops": float((2 * m * n * k).sum())}
    if kind == "trsv_batched":
        n = _batch_dims(case, 1)[0][:, 0].astype(float)
        return {"bytes": float((4 * (n * (n + 1) / 2 + 4 * n)).sum()), "flops": float((n * n).sum())}
    es, mul = SIZE[t], 4 if t in "cz" else 1
    n = case["n"]
    if kind == "vectors":
        return {"bytes": 6 * n * es, "flops": 5 * n * mul}
    if kind == "gemv_ger":
        m = case["m"]
        return {"bytes": es * (4 * m * n + 5 * (m + n)), "flops": 6 * mul * m * n}
    if kind == "symv":
        return {"bytes": es * (n * (n + 1) // 2 + 3 * n), "flops": 2 * mul * n * n}
    if kind == "trsv":
        return {"bytes": es * (n * (n + 1) // 2 + 4 * n), "flops": mul * n * n}
    m, k = case["m"], case["k"]
    return {"bytes": es * (m * k + k * n + 2 * m * n), "flops": 2 * mul * m * n * k}


# ------------------------------------------------------------------- exact ----
def _op(view, op, rows, cols):
    """op(M) as a rows x cols tensor, from the `view(cols, ld)` of stored M."""
    if op == 0:
        return view[:, :rows].T
    out = view[:, :cols]
    return out.conj() if op == 2 and out.is_complex() else out


def _product(a, b):
    """a @ b, in blocks of 16 K values summed with compensation: the rounding
    of a long 64-bit sum would otherwise be as large as what is measured."""
    total = torch.zeros(a.shape[0], b.shape[1], dtype=a.dtype, device=a.device)
    lost = torch.zeros_like(total)
    for k0 in range(0, a.shape[1], 16):
        part = a[:, k0:k0 + 16] @ b[k0:k0 + 16] - lost
        new = total + part
        lost = (new - total) - part
        total = new
    return total


def _solve(a, b, upper):
    """Triangular solve by substitution, the sums in numpy's extended precision."""
    wide = np.clongdouble if a.is_complex() else np.longdouble
    cols = np.ascontiguousarray(a.T.cpu().numpy())  # one row per column of a
    x = b.cpu().numpy().astype(wide)
    n = x.size
    for j in (range(n - 1, -1, -1) if upper else range(n)):
        x[j] /= wide(cols[j, j])
        rest = slice(0, j) if upper else slice(j + 1, n)
        x[rest] -= cols[j, rest] * x[j]
    return torch.from_numpy(x.astype(np.complex128 if a.is_complex() else np.float64)).cuda()


def exact(case, seed):
    st = prepare(case, seed)
    kind, t = case["kind"], case["dtype"]
    wide = torch.complex128 if t in ("c", "z") else torch.float64
    up = {k: v.to(wide) for k, v in st.items() if k not in ("case", "problems")}
    if kind == "vectors":
        n, inc = case["n"], case["inc"]
        x, y = up["x"][::inc], up["y"][::inc]
        dot = torch.vdot(x, y).item()
        y.add_(x, alpha=STEP)
        # |re| + |im| is rounded in the element type: no 64-bit index for it
        peak = None if t in "cz" else int((x.abs() == x.abs().max()).nonzero()[0])
        return (dot.real, dot.imag, up["y"], peak) if t in "cz" else (dot, up["y"], peak)
    if kind == "gemv_ger":
        m, n = case["m"], case["n"]
        av = up["a"].view(n, m + case["pad"])[:, :m]
        y = ALPHA * (av.T @ up["x"]) + BETA * up["y"]
        w = ALPHA * (av.conj() @ up["z"]) + BETA * up["w"]
        av.add_(torch.outer(up["x"].conj(), up["z"]), alpha=STEP)
        return y, w, up["a"]
    if kind == "symv":
        n = case["n"]
        a = up["a"].view(n, n + case["pad"])[:, :n].T
        tri = a.triu(1) if case["uplo"] == 0 else a.tril(-1)
        diag = a.diagonal().real if wide.is_complex else a.diagonal()
        return ALPHA * (tri @ up["x"] + tri.conj().T @ up["x"] + diag * up["x"]) + BETA * up["y"]
    if kind == "trsv":
        n = case["n"]
        a = _op(up["a"].view(n, n + case["pad"]), case["trans"], n, n)
        upper = (case["uplo"] == 0) == (case["trans"] == 0)
        return _solve(a, up["b"], upper)
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        (_, ac), (_, bc), _ = _gemm_dims(case)
        a = _op(up["a"].view(ac, -1), case["op_a"], m, k)
        b = _op(up["b"].view(bc, -1), case["op_b"], k, n)
        c = up["c"].view(n, -1)[:, :m].T
        c.copy_(ALPHA * _product(a, b) + BETA * c)
        return up["c"]
    if kind == "grouped":
        dims, ops = _batch_dims(case, 3)
        oa = ob = oc = 0
        for (m, n, k), op in zip(dims.tolist(), ops.tolist()):
            a = _op(up["a"][oa:oa + m * k].view(k if op == 0 else m, -1), op, m, k)
            b = up["b"][ob:ob + k * n].view(n, k).T
            c = up["c"][oc:oc + m * n].view(n, m).T
            c.copy_(ALPHA * (a @ b) + BETA * c)
            oa, ob, oc = oa + m * k, ob + k * n, oc + m * n
        return up["c"]
    out, oa, ox = up["b"], 0, 0
    for n in _batch_dims(case, 1)[0][:, 0].tolist():
        a = up["a"][oa:oa + n * n].view(n, n).T
        out[ox:ox + n] = torch.linalg.solve_triangular(a, out[ox:ox + n, None], upper=False)[:, 0]
        oa, ox = oa + n * n, ox + n
    return out
