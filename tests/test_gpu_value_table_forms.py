"""The value tables of the mixed-precision products (csrc/sellq.cuh) in the
forms that a constant coefficient on a large square meets: BF16 values of A,
and the learned factors G and G^T.  The streamed bytes that the library counts
say whether tables were read."""
import numpy as np
import pytest

from ofeli_b200 import capi
from ofeli_b200 import ofeli as F
from test_gpu_value_tables import padded

pytestmark = pytest.mark.gpu


def poisson(nx, ny):
    mesh = F.Mesh(0.0, 1.0, 0.0, 1.0, nx, ny, 1, 1, 1, 1)
    eq = F.Laplace2DT3(mesh)
    eq.setSource(np.sin(np.arange(mesh.nn) * 0.37))
    eq.setDirichlet(np.zeros(mesh.nn))
    eq.build()
    return eq.getMatrix(), eq.getRHS()


def counted(family, f):
    """f()'s result and the bytes counted per launch of a kernel family."""
    capi.profile_enable(1)
    try:
        out = f()
        n, _, total = capi.profile_read(family)
    finally:
        capi.profile_enable(0)
    assert n > 0
    return out, total / n


@pytest.mark.parametrize("nx,ny,bits,tables", [(2048, 1024, 16, True), (1300, 1203, 32, True),
                                               (1024, 512, 16, False), (700, 650, 32, False)])
def test_tables_of_a(cuda, nx, ny, bits, tables):
    """With powers of two the values are exact in BF16, and the automatic format
    takes it.  The same system with explicit zeros streams every entry and gives
    the same iterates, bit for bit."""
    A, b = poisson(nx, ny)
    rp, ci = A.pattern()
    B = F.SpMatrix(*padded(rp, ci, A.values(), A.n))
    out = []
    for M in (A, B):
        x = np.zeros(M.n)
        res, each = counted("spmv%d" % bits, lambda: F.solve_mixed(M, b, x, inner_bits=0, toler=1e-10,
                                                                   max_inner=150))
        out.append((x, res))
        streamed = bits // 8 * M.nnz + 12.0 * M.n
        assert (each < streamed) == (tables and M is A)
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0]) and np.abs(out[0][0]).max() > 0


def test_tables_of_the_learned_factors(cuda):
    """Three copies of a grid side by side are above the line, one is below it:
    the iterates of a copy are those of the grid alone.  The sums of the three
    round differently (FP64); 30 FP32 iterations carry that to some 30 2^-24,
    times a growth of 100: 2e-4; a wrong table value is of the order of G's."""
    A, b = poisson(800, 800)
    rp, ci = A.pattern()
    a, n = A.values(), A.n
    three = F.SpMatrix(np.concatenate([rp, rp[1:] + rp[-1], rp[1:] + 2 * rp[-1]]),
                       np.concatenate([ci, ci + n, ci + 2 * n]), np.concatenate([a, a, a]))
    net = F.LearnedNet(7)
    out = []
    for M, rhs in ((A, b), (three, np.concatenate([b, b, b]))):
        P = F.Prec(M, F.LEARNED_PREC, net=net)
        x = np.zeros(M.n)
        res, each = counted("learned_apply", lambda: F.fcg_learned(
            P, rhs, x, inner_bits=0, toler=1e-12, max_outer=1, max_inner=30))
        # two products a direction: values of G and G^T, gathered vectors
        streamed = (M.nnz + M.n) + 10.0 * M.n
        assert (each < streamed) == (M is three)
        out.append((x, res))
    assert out[0][1][1] == out[1][1][1] and not out[0][1][3] and not out[1][1][3]
    x, y = out[0][0], out[1][0]
    assert np.abs(x).max() > 0
    for part in (y[:n], y[n:2 * n], y[2 * n:]):
        assert np.abs(part - x).max() <= 2e-4 * np.abs(x).max()
