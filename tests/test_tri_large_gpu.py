"""SYMV / TRMV past 32768 rows off the 16-byte boundary, where a column block has
more than 1024 strips of 32 rows, checked on sampled rows.

The matrix (4.4 GB) repeats a short random vector, so a row of the triangle is
known without a copy of it in 64 bits.  Bound of an output: a term goes through
at most 64 additions inside its column block, a tree of 16 partials, 5 rounds of
it, 8 groups and the diagonal block's and column part's few: fewer than 128
roundings of 2^-24, each at most the sum of |a| |x|.
"""
import pytest
import torch

import coral_b200 as cb

pytestmark = pytest.mark.gpu

N, P = 33001, 4099   # P: period of the matrix's entries


@pytest.mark.parametrize("uplo", [0, 1])
def test_rows_past_1024_strips(cuda, uplo):
    g = torch.Generator(device="cuda").manual_seed(5)
    v = torch.rand(P, device="cuda", generator=g) - 0.5
    x = torch.rand(N, device="cuda", generator=g) - 0.5
    a = v.repeat(N * N // P + 1)[:N * N]      # stored element (r, c) at r + c N: N is odd, so no 16-byte rows
    i = torch.arange(N, device="cuda")
    rows = [0, 1, 31, 32, 16500, 32767, 32768, 32799, 32800, 32900, N - 1]

    def element(r, c):
        return v.double()[(r + c * N) % P]

    def check(got, want, bound, what):
        assert abs(got.item() - want.item()) <= 128 * 2.0 ** -24 * bound.item(), what

    y = torch.zeros(N, device="cuda")
    cb.ssymv(uplo, N, 1.0, a, N, x, 1, 0.0, y, 1)
    tn, tt = x.clone(), x.clone()
    cb.strmv(uplo, 0, 1, N, a, N, tn, 1)
    cb.strmv(uplo, 1, 1, N, a, N, tt, 1)
    xd = x.double()
    for r in rows:
        row, col = element(r, i), element(i, r)            # A(r, :) and A(:, r) as stored
        in_row = i >= r if uplo == 0 else i <= r            # stored part of the row, of the column
        in_col = i <= r if uplo == 0 else i >= r
        n_row, t_row = torch.where(in_row, row, 0.0), torch.where(in_col, col, 0.0)
        s_row = n_row + t_row
        s_row[r] = row[r]
        for got, w, what in ((y, s_row, "symv"), (tn, n_row, "trmv N"), (tt, t_row, "trmv T")):
            check(got[r], w @ xd, w.abs() @ xd.abs(), (what, r))
