"""The wavefront sweeps (csrc/wave.cu): D-ILU pivots and Prec applications
against the oracle at the edges of their groups (32 and 31 lines), tiles (32 steps)
and chunks (8 steps), on shapes that take the wavefront's masked form (lines
of unequal length, two steps apart) and on shapes that must be left to the
general sweeps, with right-hand sides that are not finite."""
import numpy as np
import pytest

from ofeli_b200 import ofeli as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def square(nx, ny, codes=(1, 1, 1, 1)):
    xy, elem, code = O.mesh2d(nx, ny, codes)
    return 2, xy, elem, code


def flipped(nx, ny, every=1):
    """The square with the other diagonal in every `every`-th cell."""
    xy, elem, code = O.mesh2d(nx, ny)
    e = elem.reshape(-1, 6).copy()
    a, b, c, d = e[:, 0], e[:, 1], e[:, 2], e[:, 4]   # corners, a-c the diagonal
    f = np.stack([a, b, d, b, c, d], 1)
    pick = np.arange(e.shape[0]) % every == 0
    e[pick] = f[pick]
    return 2, xy, e.reshape(elem.shape).astype(elem.dtype), code


def staircase(nx, ny, step):
    """Dirichlet nodes in one corner: lines of unequal length."""
    xy, elem, code = O.mesh2d(nx, ny)
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), indexing="ij")
    code = code.copy().reshape(nx + 1, ny + 1)
    code[j > ny - step * (nx - i) // nx] = 1
    return 2, xy, elem, code.reshape(-1)


def cube(M):
    xyz, elem, code = O.mesh3d(M)
    return 3, xyz, elem, code


SHAPES = {
    "one_group": lambda: square(32, 9),          # 31 lines of 8
    "full_group": lambda: square(33, 40),        # 32 lines
    "two_groups": lambda: square(34, 40),        # 32 + 1 lines
    "tiles": lambda: square(95, 258),            # 32 + 31 + 31 lines of 257
    "ragged": lambda: square(64, 171),
    "neumann": lambda: square(40, 33, (0, 1, 1, 0)),
    "wide": lambda: square(4, 700),              # few lanes: the general sweeps
    "flipped": lambda: flipped(70, 61),          # lines two steps apart
    "mixed": lambda: flipped(40, 41, every=3),   # no such order: the general sweeps
    "staircase": lambda: staircase(70, 66, 30),
    "stair_long": lambda: staircase(64, 200, 150),
    "cube_10": lambda: cube(10),
    "cube_32": lambda: cube(32),                 # planes of 31 lines
    "cube_37": lambda: cube(37),                 # planes of 32 + 4 lines
    # more groups than blocks: a block goes on from group to group
    "cube_70": lambda: cube(70),                 # planes of 32 + 31 + 6 lines
    "cube_64": lambda: cube(64),                 # planes of 32 + 31 lines
    "tall": lambda: square(4710, 27),
}


def system(name, seed=3):
    dim, xy, elem, code = SHAPES[name]()
    dof, n = O.number_equations(code)
    rp, ci = O.node_graph(elem, dim + 1, dof, n)
    rng = np.random.default_rng(seed)
    k = rng.uniform(0.3, 3.0, elem.size // (dim + 1))
    a, _ = O.assemble(dim, xy, elem, dof, code, n, rp, ci, k=k, f=np.ones(code.size),
                      bc=np.zeros(code.size))
    return rp, ci, a, n, rng.uniform(-1, 1, n)


@pytest.mark.parametrize("name", sorted(SHAPES))
@pytest.mark.parametrize("ptype", [F.ILU_PREC, F.SSOR_PREC])
def test_apply_matches_oracle(cuda, name, ptype):
    """A row's result carries a handful of roundings of its own and those of
    the rows before, damped by the diagonally dominant triangle: 1e-13."""
    rp, ci, a, n, b = system(name)
    A = F.SpMatrix(rp, ci, a)
    P = F.Prec(A, ptype)
    idv, piv = O.prec_setup(ptype, rp, ci, a)
    if ptype == F.ILU_PREC:
        assert np.array_equal(P.getPivot(), piv)
    z0 = O.prec_apply(ptype, rp, ci, a, idv, piv, b)
    z = P.solve(b)
    assert np.abs(z - z0).max() <= 1e-13 * np.abs(z0).max()
    assert np.array_equal(P.solve(b), z)         # a second sweep finds its buffers clean
    x = b.copy()
    P.solve(x, x)                                # in place
    assert np.array_equal(x, z)
    # new values through the same plan
    A.set_values(2.0 * a)
    P.setMatrix()
    assert np.abs(2.0 * P.solve(b) - z0).max() <= 1e-13 * np.abs(z0).max()


@pytest.mark.parametrize("name", ["two_groups", "ragged", "flipped", "staircase", "stair_long",
                                  "cube_32"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_values_that_are_not_finite_stay_where_they_belong(cuda, name, value):
    """The rows that come out finite are the oracle's, and have its values."""
    rp, ci, a, n, b = system(name)
    A = F.SpMatrix(rp, ci, a)
    P = F.Prec(A, F.ILU_PREC)
    pv = O.prec_setup(F.ILU_PREC, rp, ci, a)
    for where in (0, n // 3, n // 2, n - 1):
        c = b.copy()
        c[where] = value
        z0 = O.prec_apply(F.ILU_PREC, rp, ci, a, *pv, c)
        z = P.solve(c)
        assert np.array_equal(np.isfinite(z), np.isfinite(z0))
        f = np.isfinite(z0)
        if f.any():
            assert np.abs(z[f] - z0[f]).max() <= 1e-13 * np.abs(z0[f]).max()
    assert np.isfinite(P.solve(b)).all()
