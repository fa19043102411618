"""What the two plans of the wavefront sweeps (csrc/wave.cu) have to agree on
and leave alone: patterns that are not symmetric, blocks that go on from group
to group, values written through the device pointer, right-hand sides that
hold the sweeps' own marker.  Checked against the oracle; a row's result
carries a handful of roundings of its own and those of the rows before, damped
by the diagonally dominant triangle: 1e-13."""
import ctypes

import numpy as np
import pytest
import torch

from ofeli_b200 import capi
from ofeli_b200 import ofeli as F
from oracle import oracle as O
from test_gpu_wave import cube, square

pytestmark = pytest.mark.gpu


def assembled(mesh, seed=3):
    dim, xy, elem, code = mesh
    dof, n = O.number_equations(code)
    rp, ci = O.node_graph(elem, dim + 1, dof, n)
    rng = np.random.default_rng(seed)
    k = rng.uniform(0.3, 3.0, elem.size // (dim + 1))
    a, _ = O.assemble(dim, xy, elem, dof, code, n, rp, ci, k=k, f=np.ones(code.size),
                      bc=np.zeros(code.size))
    return rp, ci, a, n


def rows_of(rp):
    return np.repeat(np.arange(1, rp.size), np.diff(rp))


def from_triplets(row, col, val, n):
    order = np.lexsort((col, row))
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(row - 1, minlength=n))
    return rp, col[order], val[order]


def one_more(mesh, at):
    """The mesh's matrix and one entry far from the diagonal."""
    rp, ci, a, n = assembled(mesh)
    i, j = at(n)
    return from_triplets(np.append(rows_of(rp), i), np.append(ci, j), np.append(a, 0.5), n) + (n,)


def one_sided(mesh, far, upper):
    """Without the couplings of `far` columns or more to one side."""
    rp, ci, a, n = assembled(mesh)
    r = rows_of(rp)
    keep = ci - r < far if upper else r - ci < far
    return from_triplets(r[keep], ci[keep], a[keep], n) + (n,)


def check(P, ptype, rp, ci, a, b):
    idv, piv = O.prec_setup(ptype, rp, ci, a)
    if ptype == F.ILU_PREC:
        assert np.array_equal(P.getPivot(), piv)
    z0 = O.prec_apply(ptype, rp, ci, a, idv, piv, b)
    z = P.solve(b)
    assert np.abs(z - z0).max() <= 1e-13 * np.abs(z0).max()
    return z


UNSYMMETRIC = {
    "far_upper": lambda: one_more(square(64, 64), lambda n: (5, n - 1)),
    "far_lower": lambda: one_more(square(64, 64), lambda n: (n - 1, 5)),
    "planes_lower": lambda: one_sided(cube(12), 11 * 11, True),
    "planes_upper": lambda: one_sided(cube(12), 11 * 11, False),
}


@pytest.mark.parametrize("ptype", [F.ILU_PREC, F.SSOR_PREC])
@pytest.mark.parametrize("name", sorted(UNSYMMETRIC))
def test_unsymmetric_patterns(cuda, name, ptype):
    rp, ci, a, n = UNSYMMETRIC[name]()
    b = np.random.default_rng(4).uniform(-1, 1, n)
    P = F.Prec(F.SpMatrix(rp, ci, a), ptype)
    z = check(P, ptype, rp, ci, a, b)
    assert np.array_equal(P.solve(b), z)
    x = b.copy()
    P.solve(x, x)
    assert np.array_equal(x, z)


def blocks(count):
    """Grids of 40 lines of 9 to 71 rows side by side, uncoupled."""
    parts = [assembled(square(41, 10 + 61 * q // (count - 1)), seed=q) for q in range(count)]
    off = np.cumsum([0] + [p[3] for p in parts])
    nz = np.cumsum([0] + [p[1].size for p in parts])
    rp = np.concatenate([[0]] + [p[0][1:] + z for p, z in zip(parts, nz)])
    return rp, np.concatenate([p[1] + o for p, o in zip(parts, off)]), np.concatenate(
        [p[2] for p in parts]), int(off[-1])


# more groups than a GPU has SMs, so that blocks go on from group to group; the
# first group's steps end inside a tile (with 9, 17 and 29 chunks of eight)
TALL = {
    "tall_36": lambda: assembled(square(4710, 36)),
    "tall_100": lambda: assembled(square(4710, 100)),
    "tall_200": lambda: assembled(square(4700, 200)),
    "blocks": lambda: blocks(110),
}


@pytest.mark.parametrize("ptype", [F.ILU_PREC, F.SSOR_PREC])
@pytest.mark.parametrize("name", sorted(TALL))
def test_blocks_go_on_from_group_to_group(cuda, name, ptype):
    rp, ci, a, n = TALL[name]()
    b = np.random.default_rng(4).uniform(-1, 1, n)
    A = F.SpMatrix(rp, ci, a)
    P = F.Prec(A, ptype)
    z = check(P, ptype, rp, ci, a, b)
    piv = P.getPivot()
    x = np.empty(n)
    for q in range(200):
        if q % 10 == 0:
            P.setMatrix()
            assert np.array_equal(P.getPivot(), piv)
        P.solve(b, x)
        assert np.array_equal(x, z)


class Values:
    """The matrix's device value array as a tensor's source."""

    def __init__(self, A):
        p = ctypes.c_void_p()
        capi.call("ofg_matrix_device_arrays", A._h, None, None, ctypes.byref(p))
        self.__cuda_array_interface__ = dict(shape=(A.nnz,), typestr="<f8",
                                             data=(p.value, False), version=3)


@pytest.mark.parametrize("ptype", [F.ILU_PREC, F.SSOR_PREC])
@pytest.mark.parametrize("mesh", [square(64, 64), cube(12)], ids=["square", "cube"])
def test_values_written_through_the_device_pointer(cuda, mesh, ptype):
    """setMatrix(), and a new Prec, take the values that are there, whenever
    they were written, with copies of earlier ones made in between."""
    rp, ci, a, n = assembled(mesh)
    rng = np.random.default_rng(6)
    b = rng.uniform(-1, 1, n)
    A = F.SpMatrix(rp, ci, a)
    values = torch.as_tensor(Values(A), device="cuda:0")
    P = F.Prec(A, ptype)
    check(P, ptype, rp, ci, a, b)
    for _ in range(3):
        A.Mult(b)
        a = a * rng.uniform(0.95, 1.0, a.size)
        values.copy_(torch.from_numpy(a))
        torch.cuda.synchronize()
        P.setMatrix()
        z = check(P, ptype, rp, ci, a, b)
        assert np.array_equal(F.Prec(A, ptype).solve(b), z)


MARKER = np.array([0x7FF4DEADBEEF0001], np.uint64).view(np.float64)[0]


@pytest.mark.parametrize("ptype", [F.ILU_PREC, F.SSOR_PREC])
@pytest.mark.parametrize("mesh", [square(64, 64), cube(12)], ids=["square", "cube"])
def test_the_sweeps_own_marker_is_a_nan_like_any_other(cuda, mesh, ptype):
    """In the right-hand side or in the matrix: the results are those of a
    NaN in its place."""
    rp, ci, a, n = assembled(mesh)
    b = np.random.default_rng(6).uniform(-1, 1, n)
    A = F.SpMatrix(rp, ci, a)
    P = F.Prec(A, ptype)
    for at in ([0], [n // 2, n // 2 + 1], [n - 1], list(range(n))):
        c, d = b.copy(), b.copy()
        c[at], d[at] = MARKER, np.nan
        z, z0 = P.solve(c), P.solve(d)
        assert np.isnan(z[at]).all()
        assert np.array_equal(z, z0, equal_nan=True)
    r = n // 2
    row = np.arange(rp[r], rp[r + 1])          # a lower, the diagonal and an upper entry
    for k in (row[0], row[ci[row] == r + 1][0], row[-1]):
        z = []
        for v in (MARKER, np.nan):
            c = a.copy()
            c[k] = v
            A.set_values(c)
            P.setMatrix()
            z.append(P.solve(b))
        assert np.isnan(z[0]).any()
        assert np.array_equal(z[0], z[1], equal_nan=True)


def box(rows, lines, planes, seed=5):
    """A box of unknowns coupled as the Kuhn cube's: 14 neighbours."""
    dims, st = (rows, lines, planes), (1, rows, rows * lines)
    idx = np.arange(rows * lines * planes)
    at = [idx // s % d for s, d in zip(st, dims)]
    r, c = [idx], [idx]
    for q in range(1, 8):
        step = [(q >> k) & 1 for k in range(3)]
        ok = np.all([a + s < d for a, s, d in zip(at, step, dims)], axis=0)
        to = idx[ok] + sum(s * t for s, t in zip(step, st))
        r += [idx[ok], to]
        c += [to, idx[ok]]
    r, c = np.concatenate(r), np.concatenate(c)
    a = np.where(r == c, 16.0, -np.random.default_rng(seed).uniform(0.5, 1.0, r.size))
    return from_triplets(r + 1, c + 1, a, idx.size) + (idx.size,)


@pytest.mark.parametrize("ptype", [F.ILU_PREC, F.SSOR_PREC])
@pytest.mark.parametrize("dims", [(80, 8, 8), (81, 8, 8), (40, 12, 6), (33, 34, 5), (500, 6, 3),
                                  (9, 40, 7)], ids=str)
def test_boxes_on_both_sides_of_the_line(cuda, dims, ptype):
    """Boxes of short lines take the wavefront, those of long ones the strands
    (80 and 81 rows are next to it for 8 lines and 8 planes)."""
    rp, ci, a, n = box(*dims)
    b = np.random.default_rng(4).uniform(-1, 1, n)
    P = F.Prec(F.SpMatrix(rp, ci, a), ptype)
    z = check(P, ptype, rp, ci, a, b)
    assert np.array_equal(P.solve(b), z)
