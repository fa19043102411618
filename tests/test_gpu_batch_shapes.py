"""The batched solver's launch shape chosen from the problems' sizes: problems
of one unknown, around a block's rows, one problem far larger than the rest
(clusters), many small ones (one block each), and columns too far from the row
for 16-bit offsets.  Checked as the tuned
shapes are: assembled values bit-exact, solutions to 1e-9, iterations +-2."""
import numpy as np
import pytest

from ofeli_b200 import fields
from ofeli_b200 import ofeli as F
from oracle import oracle as O
from test_gpu_batch import check_against_oracle, small_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("sizes", [[2], [2, 3, 6, 7], [33, 2, 34], [5, 120, 9], [40, 90, 41, 42],
                                   [8 + i % 5 for i in range(200)]],
                         ids=["one", "tiny", "rows", "large", "mixed", "many"])
def test_chosen_shape(cuda, sizes, bits):
    B, ref, _ = small_batch(sizes, bc=True)
    B.set_precision(bits)
    for _ in range(2):
        B.solve(100000, 1e-10)
        if bits == 64:
            check_against_oracle(B, ref)
        else:
            u, it, res = B.results()
            assert (res <= 1e-10).all() and (it >= 0).all()
            want = np.concatenate([r["u"] for r in ref])
            assert np.linalg.norm(u - want) <= 1e-8 * np.linalg.norm(want)


@pytest.mark.parametrize("nx,ny", [(40000, 3), (3, 40000)])
def test_far_columns(cuda, nx, ny):
    xy, elem, code = O.mesh2d(nx, ny)
    xy = (xy.reshape(-1, 2) * np.array([nx, ny])).ravel()  # unit cells
    f = fields.uniform_pm1(3, code.size)
    m = F.Mesh(0.0, 1.0, 0.0, 1.0, nx, ny, 1, 1, 1, 1)
    m.setCoords(xy)
    dof, n = O.number_equations(code)
    rp, ci = O.node_graph(elem, 3, dof, n)
    a, b = O.assemble(2, xy, elem, dof, code, n, rp, ci, k=None, f=f, bc=None)
    x, it = O.cg(rp, ci, a, b, O.DIAG, 100000, 1e-10)
    ref = [{"a": a, "b": b, "x": x, "it": it, "u": O.insert_bc(code, x, np.zeros(code.size)),
            "nnz": int(rp[-1]), "n": n}]
    B = F.Batch([m])
    B.set_inputs(None, f, None)
    for bits in (64, 32):
        B.set_precision(bits)
        B.solve(100000, 1e-10)
        if bits == 64:
            check_against_oracle(B, ref)
        else:
            u, _, res = B.results()
            assert res[0] <= 1e-10
            assert np.linalg.norm(u - ref[0]["u"]) <= 1e-8 * np.linalg.norm(u)
