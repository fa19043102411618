"""The value tables of the mixed-precision products (csrc/sellq.cuh): slices
whose rows share their values read them from a table once the iteration's
vectors and values outgrow the near half of the L2.  The same system with an
explicit zero in every 16th row has no uniform slice and streams every entry:
the iterates are bit for bit the same."""
import numpy as np
import pytest

from ofeli_b200 import ofeli as F

pytestmark = pytest.mark.gpu


def padded(rp, ci, a, n):
    """One explicit zero (column n, or 1 in rows that have it) in every 16th row."""
    rows = np.arange(0, n, 16)
    has = ci[rp[rows + 1] - 1] == n
    col = np.where(has, 1, n)
    keep = ~(has & (ci[rp[rows]] == 1))
    rows, col = rows[keep], col[keep]
    at = np.where(col == n, rp[rows + 1], rp[rows])
    order = np.argsort(at, kind="stable")
    ci2 = np.insert(ci, at[order], col[order])
    a2 = np.insert(a, at[order], 0.0)
    add = np.zeros(n + 1, np.int64)
    add[rows + 1] = 1
    return rp + np.cumsum(add), ci2, a2


@pytest.mark.parametrize("nx,ny", [(1203, 1201), (1100, 1180), (700, 650)])
@pytest.mark.parametrize("bits", [0, 32])
def test_shared_values_give_the_streamed_iteration(cuda, nx, ny, bits):
    """1203 x 1201 is above the line for BF16 and FP32 values alike, 700 x 650
    below it; nx != ny makes the values inexact in BF16."""
    mesh = F.Mesh(0.0, 1.0, 0.0, 1.0, nx, ny, 1, 1, 1, 1)
    eq = F.Laplace2DT3(mesh)
    eq.setSource(np.sin(np.arange(mesh.nn) * 0.37))
    eq.setDirichlet(np.zeros(mesh.nn))
    eq.build()
    A, b = eq.getMatrix(), eq.getRHS()
    rp, ci = A.pattern()
    B = F.SpMatrix(*padded(rp, ci, A.values(), A.n))
    out = []
    for M in (A, B):
        x = np.zeros(M.n)
        res = F.solve_mixed(M, b, x, inner_bits=bits, toler=1e-10, max_inner=150)
        out.append((x, res))
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0]) and np.abs(out[0][0]).max() > 0
