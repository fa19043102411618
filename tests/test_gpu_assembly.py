"""The row-gather assembly over incidence records (csrc/assembly.cu) against
the oracle, bit for bit: slices with nodes of unequal degree, rows too long
for the records (the general kernel), and coordinates whose quotients leave
the range of the shared reciprocal."""
import numpy as np
import pytest

from ofeli_b200 import ofeli as F
from ofeli_b200 import problems
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def fan(k, rings):
    """k * rings triangles around one node: its row has k + 1 entries."""
    t = 2 * np.pi * np.arange(k) / k
    xy = [np.zeros((1, 2))] + [(r + 1.0) / rings * np.stack([np.cos(t), np.sin(t)], 1)
                               for r in range(rings)]
    el = [[0, 1 + j, 1 + (j + 1) % k] for j in range(k)]
    for r in range(rings - 1):
        a, b = 1 + r * k, 1 + (r + 1) * k
        for j in range(k):
            n = (j + 1) % k
            el += [[a + j, b + j, b + n], [a + j, b + n, a + n]]
    code = np.zeros(1 + k * rings, np.int32)
    code[-k:] = 2
    return 2, np.concatenate(xy).reshape(-1), np.array(el, np.int32).reshape(-1), code


def ring(seed):
    xy, elem, code, _, _ = problems.ring_mesh(9, 37, seed=seed)
    return 2, xy.reshape(-1), elem.reshape(-1), code


def square():
    xy, elem, code = O.mesh2d(33, 17)
    return 2, xy, elem, code


def cube():
    xyz, elem, code = O.mesh3d(7)
    return 3, xyz, elem, code


CASES = {"square": square, "ring": lambda: ring(1), "cube": cube,
         "row_of_16": lambda: fan(15, 3), "row_of_17": lambda: fan(16, 3),
         "row_of_40": lambda: fan(39, 2)}


@pytest.mark.parametrize("scale", [1.0, 1e-100, 3e80])
@pytest.mark.parametrize("name", sorted(CASES))
def test_assembly_is_the_oracles_bit_for_bit(cuda, name, scale):
    dim, xy, elem, code = CASES[name]()
    if dim == 3 and scale != 1.0:
        scale = 1.0 + 1e-3 * (scale > 1.0)   # volumes of 1e-300 would underflow
    xy = np.asarray(xy) * scale
    rng = np.random.default_rng(5)
    k = rng.uniform(0.5, 2.0, elem.size // (dim + 1))
    f, bc = rng.uniform(-1, 1, code.size), rng.uniform(-1, 1, code.size)
    dof, n = O.number_equations(code)
    rp, ci = O.node_graph(elem, dim + 1, dof, n)
    a, b = O.assemble(dim, xy, elem, dof, code, n, rp, ci, k=k, f=f, bc=bc)
    eq = (F.Laplace2DT3 if dim == 2 else F.DC3DT4)(F.Mesh.from_arrays(dim, xy, elem, code))
    eq.setElementCoefficient(k)
    eq.setSource(f)
    eq.setDirichlet(bc)
    eq.build()
    assert np.array_equal(eq.getMatrix().values(), a)
    assert np.array_equal(eq.getRHS(), b)
