"""The measured cases: the work a user of ofeli_b200 has it do, through its
public entry points, from the smallest calls to the benchmark's own sizes.

Families (the sizes are those of the tests and of bench.py):

* ``mult``      SpMatrix::Mult, the product a user's own iteration calls.
* ``assemble``  Equation::build() of an unstructured (randomly numbered) or a
                structured P1 problem with a coefficient per element and
                Dirichlet data.
* ``prec``      Prec::setMatrix + Prec::solve: the factorisation of new values
                and one application (what a user's own Krylov loop pays).
* ``cg``        OFELI's own method: build(), Prec, CG, insertBC in FP64.
* ``mixed``     the benchmark's chosen form: build(), FP64 refinement around
                the FP32 CG (Jacobi or learned preconditioner), insertBC.
* ``step``      one time step of the convection-diffusion problem: build(),
                GMRes + ILU (OFELI's method) or the mixed flexible GMRES,
                insertBC; the state advances from call to call.
* ``batch``     many independent uneven problems in one launch.
* ``train``     Adam steps of the learned preconditioner's network (forward
                and backward pass).

Inputs are made on the GPU from the seed; vectors are device tensors, as in a
program that keeps its data there.
"""
import ctypes
import math

import numpy as np
import torch

from ofeli_b200 import capi, learned
from ofeli_b200 import ofeli as F

DEV = "cuda:0"
TOL = 1e-10
EPS, DT = 1e-3, 1e-3   # the transient benchmark's diffusion and time step


# ----------------------------------------------------------------- the cases
def listed():
    return [
        # one product on the smallest grid of the tests: launch and call cost
        dict(name="mult_65", family="mult", mesh="square", nx=64, ny=64),
        # a user's unstructured mesh: random numbering, two-sided Dirichlet data
        dict(name="assemble_ring", family="assemble", mesh="ring", nx=256, ny=1024),
        # D-ILU of new values and one application at the headline grid
        dict(name="ilu_2049", family="prec", mesh="square", nx=2048, ny=2048, prec="ILU"),
        # symmetric Gauss-Seidel on the 3-D benchmark grid
        dict(name="ssor_kuhn_129", family="prec", mesh="kuhn", nx=128, ny=128, prec="SSOR"),
        # OFELI's CG + ILU: a small, an ordinary and a 3-D problem
        dict(name="cg_ilu_65", family="cg", mesh="square", nx=64, ny=64, prec="ILU"),
        dict(name="cg_ilu_513", family="cg", mesh="square", nx=512, ny=512, prec="ILU"),
        dict(name="cg_ilu_kuhn_65", family="cg", mesh="kuhn", nx=64, ny=64, prec="ILU"),
        # the benchmark's headline problem and its 3-D problem, chosen form
        dict(name="learned_2049", family="mixed", mesh="square", nx=2048, ny=2048,
             prec="LEARNED"),
        dict(name="jacobi_kuhn_129", family="mixed", mesh="kuhn", nx=128, ny=128, prec="DIAG"),
        # the transient benchmark: the chosen form and OFELI's method
        dict(name="step_fgmres_1025", family="step", mesh="square", nx=1024, ny=1024,
             prec="DIAG"),
        dict(name="step_ilu_1025", family="step", mesh="square", nx=1024, ny=1024, prec="ILU"),
        # uneven problems solved in one launch
        dict(name="batch_192", family="batch", mesh="square", count=192, nmin=1000, nmax=32000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["mult", "assemble", "prec", "prec", "cg", "cg", "mixed", "step", "step",
                         "batch", "train"])
    if family == "batch":
        return dict(family="batch", mesh="square", count=rng.randrange(24, 200),
                    nmin=1000, nmax=_log_int(rng, 4000, 32000))
    if family == "train":
        return dict(family="train", mesh="square", nx=_log_int(rng, 63, 512),
                    ny=_log_int(rng, 63, 512), batch=rng.choice([8, 16, 32]))
    if family == "step":
        n = _log_int(rng, 64, 1024)
        return dict(family="step", mesh="square", nx=n, ny=max(48, int(n * rng.uniform(0.5, 1.0))),
                    prec=rng.choice(["DIAG", "ILU"]))
    kinds = {"mult": ["square", "kuhn", "ring"], "assemble": ["square", "kuhn", "ring"],
             "prec": ["square", "kuhn"], "cg": ["square", "kuhn"],
             "mixed": ["square", "kuhn"]}[family]
    mesh = rng.choice(kinds)
    if mesh == "kuhn":
        # whole solves from 34 cells a side: below, one costs more than any
        # listed case; single applications cover the smaller cubes
        n = _log_int(rng, 34, 64) if family == "cg" else _log_int(rng, 12, 128)
        c = dict(family=family, mesh=mesh, nx=n, ny=n)
    elif mesh == "ring":
        c = dict(family=family, mesh=mesh, nx=_log_int(rng, 16, 256), ny=_log_int(rng, 64, 1024))
    else:
        hi = {"mult": 2048, "assemble": 1536, "prec": 2048, "cg": 512, "mixed": 1536}[family]
        n = _log_int(rng, 48, hi)
        # rectangles, a little wider or higher than square
        c = dict(family=family, mesh=mesh, nx=n, ny=max(40, int(n * rng.uniform(0.6, 1.0))))
    if family in ("prec", "cg"):
        c["prec"] = rng.choice(["ILU", "SSOR"])
    if family == "mixed":
        c["prec"] = "LEARNED" if mesh == "square" else "DIAG"
    return c


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, n):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 2.0 - 1.0


def _lognormal(g, pts, sigma, corr=0.1, modes=48):
    """exp(sigma g), g a smooth random field of unit variance."""
    k = torch.randn(modes, pts.shape[1], generator=g, device=DEV, dtype=torch.float64) / corr
    ph = torch.rand(modes, generator=g, device=DEV, dtype=torch.float64) * (2 * math.pi)
    s = torch.zeros(pts.shape[0], device=DEV, dtype=torch.float64)
    for m in range(modes):
        s += torch.cos(pts @ k[m] + ph[m])
    return torch.exp(s.mul_(sigma * math.sqrt(2.0 / modes)))


def _square(nx, ny):
    """OFELI's structured triangulation of the unit square: nodes with y
    fastest, two triangles per cell.  (coords, elem, code) on the GPU."""
    i = torch.arange(nx + 1, device=DEV)
    j = torch.arange(ny + 1, device=DEV)
    I, J = torch.meshgrid(i, j, indexing="ij")
    xy = torch.stack([I.double() / nx, J.double() / ny], -1).reshape(-1, 2)
    code = ((I == 0) | (J == 0) | (I == nx) | (J == ny)).int().reshape(-1)
    I, J = torch.meshgrid(i[1:], j[1:], indexing="ij")
    n = (I * (ny + 1) + J + 1).reshape(-1)
    e = torch.stack([n - ny - 3, n - 2, n - 1, n - 1, n - ny - 2, n - ny - 3], 1)
    return xy, e.reshape(-1, 3), code


def _kuhn(M):
    P = M + 1
    k, j, i = torch.meshgrid(*[torch.arange(P, device=DEV)] * 3, indexing="ij")
    xyz = torch.stack([i, j, k], -1).reshape(-1, 3).double() / M
    code = ((i == 0) | (j == 0) | (k == 0) | (i == M) | (j == M) | (k == M)).int().reshape(-1)
    k, j, i = torch.meshgrid(*[torch.arange(M, device=DEV)] * 3, indexing="ij")
    o = (i + P * (j + P * k)).reshape(-1)
    step = [1, P, P * P]
    tets = []
    for perm, odd in (((0, 1, 2), 0), ((0, 2, 1), 1), ((1, 0, 2), 1), ((1, 2, 0), 0),
                      ((2, 0, 1), 0), ((2, 1, 0), 1)):
        a = o + step[perm[0]]
        b = a + step[perm[1]]
        c = b + step[perm[2]]
        tets.append(torch.stack([o, b, a, c] if odd else [o, a, b, c], 1))
    return xyz, torch.stack(tets, 1).reshape(-1, 4), code


def _ring(nr, nt, g):
    """A jittered annulus with random diagonals and a random node numbering:
    the shape of a user's mesh file; codes on both circles."""
    i, j = torch.meshgrid(torch.arange(nr + 1, device=DEV), torch.arange(nt, device=DEV),
                          indexing="ij")
    inner = ((i > 0) & (i < nr)).double()
    jr, jt = (_uniform(g, i.numel()).reshape(i.shape) * 0.2 * inner for _ in range(2))
    r = 0.5 + 0.5 * (i + jr) / nr
    t = 2 * math.pi * (j + jt) / nt
    xy = torch.stack([r * torch.cos(t), r * torch.sin(t)], -1).reshape(-1, 2)
    code = ((i == 0).int() + 2 * (i == nr).int()).reshape(-1)
    a, b = torch.meshgrid(torch.arange(nr, device=DEV), torch.arange(nt, device=DEV),
                          indexing="ij")
    a, b = a.reshape(-1), b.reshape(-1)
    c = (b + 1) % nt
    p00, p10, p11, p01 = a * nt + b, (a + 1) * nt + b, (a + 1) * nt + c, a * nt + c
    flip = (torch.rand(a.numel(), generator=g, device=DEV) < 0.5)[:, None]
    t1 = torch.where(flip, torch.stack([p00, p10, p01], 1), torch.stack([p00, p10, p11], 1))
    t2 = torch.where(flip, torch.stack([p10, p11, p01], 1), torch.stack([p00, p11, p01], 1))
    elem = torch.stack([t1, t2], 1).reshape(-1, 3)
    perm = torch.randperm(xy.shape[0], generator=g, device=DEV)
    new_xy, new_code = torch.empty_like(xy), torch.empty_like(code)
    new_xy[perm], new_code[perm] = xy, code
    return new_xy, perm[elem], new_code


def _geometry(case, g):
    if case["mesh"] == "kuhn":
        return _kuhn(case["nx"])
    if case["mesh"] == "ring":
        return _ring(case["nx"], case["ny"], g)
    return _square(case["nx"], case["ny"])


def _inputs(case, seed):
    """Everything a case's problem is made of, as torch tensors."""
    g = _gen(seed)
    fam = case["family"]
    xy, elem, code = _geometry(case, g)
    d = dict(xy=xy, elem=elem, code=code, k=None, bc=None)
    d["f"] = _uniform(g, code.numel())
    # a constant coefficient on the square (the headline problem), a
    # log-normal one on the cube (the 3-D benchmark) and where it is the point
    if case["mesh"] == "kuhn" or fam in ("assemble", "mult"):
        pts = xy[elem].mean(1)
        d["k"] = _lognormal(g, pts, 1.5 if case["mesh"] == "kuhn" else 1.0)
    if fam == "assemble":
        d["bc"] = torch.where(code > 0, _uniform(g, code.numel()), 0.0)
    if fam == "step":
        c = torch.rand(2, generator=g, device=DEV, dtype=torch.float64) * 0.2 + 0.4
        d["v"] = torch.stack([-(xy[:, 1] - c[1]), xy[:, 0] - c[0]], 1).reshape(-1).contiguous()
        p = torch.rand(2, generator=g, device=DEV, dtype=torch.float64) * 0.4 + 0.3
        u = torch.exp(-((xy - p) ** 2).sum(1) / (2 * 0.05 ** 2))
        d["u"] = torch.where(code > 0, 0.0, u)
    return d


def _batch_sizes(case, seed):
    r = np.random.default_rng(int(seed))
    nodes = np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["count"]))
    return [int(round(math.sqrt(v))) - 1 for v in nodes]


def _batch_inputs(case, seed):
    """Per problem (xy, elem, code, k, f): jittered squares of uneven size.
    The sizes depend on the case alone, the fields on the seed."""
    g = _gen(seed)
    out = []
    for n in _batch_sizes(case, case["count"]):
        xy, elem, code = _square(n, n)
        j = _uniform(g, 2 * code.numel()).reshape(-1, 2) * (0.2 / n)
        xy = xy + torch.where(code[:, None] > 0, 0.0, j)
        k = _lognormal(g, xy[elem].mean(1), 1.0, modes=16)
        out.append((xy, elem, code, k, _uniform(g, code.numel())))
    return out


# ------------------------------------------------------------ what a user has
_NET = []


def _network():
    """The learned preconditioner's trained weights (the same in every case;
    one training per process, as a program that loads its weights once)."""
    if not _NET:
        net = F.LearnedNet(7)
        data = []
        for s in range(4):
            A, _, mesh = learned.square_problem(128, 100 + s, None if s % 2 == 0 else 1.0)
            data.append((A, mesh) + F.LearnedNet.make_pairs_operator(A, 32, seed=1000 + s))
        for _ in range(6):
            for A, _, R, E in data:
                net.train(A, R, E, steps=10, batch=16)
        _NET.append(net)
    return _NET[0]


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


class _Raw:
    """Device memory of the library as a tensor's source; keeps its owner."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False),
                                             version=3)


def _values(A):
    """The matrix's device value array as a tensor (no copy)."""
    rp, col, val = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    capi.call("ofg_matrix_device_arrays", A._h, ctypes.byref(rp), ctypes.byref(col),
              ctypes.byref(val))
    return torch.as_tensor(_Raw(A, val.value, A.nnz), device=DEV)


def _mesh(case, d):
    if case["mesh"] == "kuhn":
        return F.Mesh.kuhn(case["nx"])
    if case["mesh"] == "ring":
        return F.Mesh.from_arrays(2, d["xy"].cpu().numpy(), d["elem"].int().cpu().numpy(),
                                  d["code"].cpu().numpy())
    return F.Mesh(0.0, 1.0, 0.0, 1.0, case["nx"], case["ny"], 1, 1, 1, 1)


def _assemble(s):
    capi.call("ofg_assemble_p1", s["mesh"]._h, s["A"]._h, _ptr(s["k"]), _ptr(s["f"]),
              _ptr(s["bc"]), _ptr(s["b"]))


def prepare(case, seed):
    fam = case["family"]
    s = dict(case=case)
    if fam == "batch":
        meshes, ks, fs = [], [], []
        for (xy, elem, code, k, f), n in zip(_batch_inputs(case, seed),
                                             _batch_sizes(case, case["count"])):
            m = F.Mesh(0.0, 1.0, 0.0, 1.0, n, n, 1, 1, 1, 1)
            m.setCoords(xy.reshape(-1).contiguous())
            meshes.append(m)
            ks.append(k)
            fs.append(f)
        B = F.Batch(meshes)
        s.update(meshes=meshes, B=B, k=torch.cat(ks), f=torch.cat(fs))
        s["u"] = torch.zeros(B.nodes, dtype=torch.float64, device=DEV)
        s["it"] = torch.zeros(B.nprob, dtype=torch.int32, device=DEV)
        s["res"] = torch.zeros(B.nprob, dtype=torch.float64, device=DEV)
        return s
    d = _inputs(case, seed)
    mesh = _mesh(case, d)
    A = F.SpMatrix(mesh)
    z = lambda n: torch.zeros(n, dtype=torch.float64, device=DEV)  # noqa: E731
    s.update(mesh=mesh, A=A, k=d["k"], f=d["f"], bc=d["bc"], b=z(A.n), x=z(A.n), u=z(mesh.nn))
    torch.cuda.synchronize()
    if fam == "step":
        s.update(v=d["v"], u=d["u"].clone())
        torch.cuda.synchronize()
        _step_assemble(s)
        s["P"] = F.Prec(A, F.ILU_PREC if case["prec"] == "ILU" else F.DIAG_PREC)
        return s
    _assemble(s)
    if fam == "mult":
        s["r"] = _uniform(_gen(seed + 7), A.n)
    elif fam == "prec":
        s["r"] = _uniform(_gen(seed + 7), A.n)
        s["P"] = F.Prec(A, F.ILU_PREC if case["prec"] == "ILU" else F.SSOR_PREC)
    elif fam == "cg":
        s["P"] = F.Prec(A, F.ILU_PREC if case["prec"] == "ILU" else F.SSOR_PREC)
    elif fam == "mixed" and case["prec"] == "LEARNED":
        s["P"] = F.Prec(A, F.LEARNED_PREC, net=_network())
    elif fam == "train":
        s["net"] = F.LearnedNet(5)
        E = torch.randn(case["batch"], A.n, generator=_gen(seed + 7), device=DEV,
                        dtype=torch.float64)
        R = torch.zeros_like(E)
        torch.cuda.synchronize()
        for p in range(case["batch"]):
            A.Mult(E[p], R[p])
        s["E"], s["R"] = E.float().contiguous(), R.float().contiguous()
    return s


def _step_assemble(s):
    capi.call("ofg_assemble_cd2d", s["mesh"]._h, s["A"]._h, EPS, _ptr(s["v"]), DT, _ptr(s["u"]),
              None, _ptr(s["b"]))


def run(s):
    case = s["case"]
    fam = case["family"]
    A = s.get("A")
    if fam == "mult":
        return A.Mult(s["r"], s["x"])
    if fam == "assemble":
        _assemble(s)
        return dict(values=_values(A), b=s["b"])
    if fam == "prec":
        s["P"].setMatrix()
        return s["P"].solve(s["r"], s["x"])
    if fam == "batch":
        B = s["B"]
        B.set_inputs(s["k"], s["f"])
        B.solve(100000, TOL)
        capi.call("ofg_batch_get_results", B._h, _ptr(s["u"]), _ptr(s["it"]), _ptr(s["res"]))
        return dict(u=s["u"])
    if fam == "train":
        hist = s["net"].train(A, s["R"], s["E"], steps=4, batch=case["batch"])
        params, m, v, _ = s["net"].get_params()
        return dict(loss=hist, params=params, m=m, v=v)
    if fam == "step":
        _step_assemble(s)
        if case["prec"] == "DIAG":
            F.fgmres_mixed(s["P"], s["b"], s["x"], m=30, toler=TOL)
        else:
            F.GMRes(A, s["P"], s["b"], s["x"], 30, 1000, TOL)
        capi.call("ofg_insert_bc", s["mesh"]._h, _ptr(s["x"]), None, _ptr(s["u"]))
        return dict(u=s["u"], x=s["x"])
    # cg, mixed: a whole solve from a zero starting guess
    _assemble(s)
    s["x"].zero_()
    torch.cuda.current_stream().synchronize()  # the library works on its own stream
    if fam == "cg":
        s["P"].setMatrix()
        it = F.CG(A, s["P"], s["b"], s["x"], 100000, TOL)
    elif case["prec"] == "LEARNED":
        it = F.fcg_learned(s["P"], s["b"], s["x"], inner_bits=0, toler=TOL)[1]
    else:
        it = F.solve_mixed(A, s["b"], s["x"], prec=F.DIAG_PREC, inner_bits=0, toler=TOL)[1]
    capi.call("ofg_insert_bc", s["mesh"]._h, _ptr(s["x"]), None, _ptr(s["u"]))
    return dict(iterations=it, x=s["x"], u=s["u"])


# ------------------------------------------------------- work of one pass
def _counts(case):
    """(nodes, elements, unknowns, nonzeros) of a case's mesh."""
    if case["mesh"] == "kuhn":
        M, m = case["nx"], case["nx"] - 1
        nnz = m ** 3 + 6 * m * m * (m - 1) + 6 * m * (m - 1) ** 2 + 2 * (m - 1) ** 3
        return (M + 1) ** 3, 6 * M ** 3, m ** 3, nnz
    nx, ny = case["nx"], case["ny"]
    if case["mesh"] == "ring":
        n = (nx - 1) * ny
        return (nx + 1) * ny, 2 * nx * ny, n, 7 * n - 4 * ny
    n = (nx - 1) * (ny - 1)
    return (nx + 1) * (ny + 1), 2 * nx * ny, n, 7 * n - 4 * (nx + ny - 2) + 2


def work(case):
    fam = case["family"]
    if fam == "batch":
        by = fl = 0.0
        for n in _batch_sizes(case, case["count"]):
            w = work(dict(family="cg", mesh="square", nx=n, ny=n, prec="DIAG"))
            by, fl = by + w["bytes"], fl + w["flops"]
        return dict(bytes=by, flops=fl)
    nn, ne, n, nnz = _counts(case)
    dim = 3 if case["mesh"] == "kuhn" else 2
    spmv = 12.0 * nnz + 20.0 * n
    # coordinates, connectivity, codes, coefficients in; values and b out
    build = 8.0 * dim * nn + 4.0 * (dim + 1) * ne + 16.0 * nn + 8.0 * ne + 12.0 * nnz + 8.0 * n
    build_fl = 60.0 * ne
    sweeps = 12.0 * (nnz - n) + 16.0 * n + 16.0 * n     # both triangles, pivots, r, z
    if fam == "mult":
        return dict(bytes=spmv, flops=2.0 * nnz)
    if fam == "assemble":
        return dict(bytes=build, flops=build_fl)
    if fam == "prec":
        return dict(bytes=(12.0 * nnz + 8.0 * n) + sweeps, flops=5.0 * nnz)
    if fam == "train":
        # 4 steps: per layer and row the activations forward and back, and
        # the three 128 x 64 products
        return dict(bytes=4 * (4 * 6 * 128.0 * n + 8.0 * nnz + case["batch"] * 8.0 * n),
                    flops=4 * 4 * 3 * 2.0 * 128 * 64 * n)
    if fam == "step":
        its = 6 if case["prec"] == "DIAG" else 4
        return dict(bytes=build + 24.0 * nn + its * (spmv + 24.0 * n + (
            sweeps if case["prec"] == "ILU" else 0)), flops=build_fl + its * 8.0 * nnz)
    side = max(case["nx"], case["ny"])
    # iterations to 1e-10 on these meshes (measured: 2030 with ILU and about
    # 3990 with the learned factor at 2049^2, 257 and 847 on the 129^3 cube)
    its = {"ILU": 1.0, "SSOR": 1.0, "LEARNED": 2.0, "DIAG": 3.5}[case["prec"]] * side
    if case["mesh"] == "kuhn":
        its *= 2.0
    if fam == "cg":
        vec = 88.0 * n + (sweeps if case["prec"] in ("ILU", "SSOR") else 0.0)
        return dict(bytes=build + its * (spmv + vec), flops=its * 6.0 * nnz)
    # FP32 iteration: BF16 or FP32 values, FP32 vectors; G and G^T in BF16
    it_bytes = (2.0 if case["mesh"] == "square" else 6.0) * nnz + 36.0 * n
    if case["prec"] == "LEARNED":
        it_bytes += 2.0 * (nnz + n) + 12.0 * n
    return dict(bytes=build + its * it_bytes, flops=its * 4.0 * nnz)


# ----------------------------------------------------------- 64-bit answers
def _assembled(xy, elem, code, k, f, bc, extra=None):
    """(A as torch CSR with sorted columns, b): P1 stiffness (times k) with
    the lumped source and the Dirichlet lift, in 64 bits.  extra(grad, area,
    elem) replaces the element matrices and right-hand sides."""
    dim = xy.shape[1]
    p = xy[elem]
    if dim == 2:
        d1, d2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        det = d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0]
        size = det / 2
    else:
        det = torch.linalg.det(p[:, 1:] - p[:, :1])
        size = det / 6
    J = (p[:, 1:] - p[:, :1])
    gi = torch.linalg.inv(J).transpose(1, 2)        # rows: gradients of phi_1 ..
    grad = torch.cat([-gi.sum(1, keepdim=True), gi], 1)
    del p, J, gi, det
    if extra is None:
        em = torch.einsum("eia,eja->eij", grad, grad) * (size * (1.0 if k is None else k))[:, None,
                                                                                          None]
        er = (f[elem] * (size / (dim + 1))[:, None]) if f is not None else None
    else:
        em, er = extra(grad, size, elem)
    del grad
    free = code == 0
    n = int(free.sum())
    eq = torch.where(free, torch.cumsum(free.long(), 0) - 1, -1)
    le = eq[elem]
    b = torch.zeros(n, dtype=torch.float64, device=xy.device)
    if bc is not None:
        ub = torch.where(free, 0.0, bc)[elem]
        er = er - torch.einsum("eij,ej->ei", em, ub)
    m = le >= 0
    b.index_add_(0, le[m], er[m])
    m = (le[:, :, None] >= 0) & (le[:, None, :] >= 0)
    key = (le[:, :, None] * n + le[:, None, :])[m]
    key, inv = torch.unique(key, return_inverse=True)
    val = torch.zeros(key.numel(), dtype=torch.float64, device=xy.device)
    val.index_add_(0, inv, em[m])
    rows, cols = key // n, key % n
    rp = torch.zeros(n + 1, dtype=torch.int64, device=xy.device)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return torch.sparse_csr_tensor(rp, cols, val, size=(n, n)), b, rows


def _tight_cg(A, b, dinv, group=None, tol=1e-14, most=40000):
    """Jacobi-CG in 64 bits to the rounding level; group: the problem every
    row belongs to (independent problems side by side)."""
    if group is None:
        ng = 1
        dot = lambda a, c: torch.dot(a, c)[None]  # noqa: E731
        ext = lambda s: s  # noqa: E731
    else:
        ng = int(group.max()) + 1
        dot = lambda a, c: torch.zeros(ng, dtype=a.dtype, device=a.device).index_add_(0, group, a * c)  # noqa: E731,E501
        ext = lambda s: s[group]  # noqa: E731
    x = torch.zeros_like(b)
    r = b.clone()
    z = dinv * r
    p = z.clone()
    rz = dot(r, z)
    bb = dot(b, b)
    for it in range(1, most + 1):
        q = A @ p
        pq = dot(p, q)
        a = torch.where(pq > 0, rz / pq, 0.0)
        x += ext(a) * p
        r -= ext(a) * q
        z = dinv * r
        new = dot(r, z)
        p = z + ext(torch.where(rz > 0, new / rz, 0.0)) * p
        rz = new
        if it % 100 == 0 and bool((dot(r, r) <= tol * tol * bb).all()):
            break
    return x


def _tight_bicgstab(A, b, x, dinv, tol=1e-15, most=400):
    r = b - A @ x
    rh = r.clone()
    rho = a = w = torch.ones((), dtype=b.dtype, device=b.device)
    v = p = torch.zeros_like(b)
    nb = float(b.norm())
    for _ in range(most):
        if float(r.norm()) <= tol * nb:
            break
        new = torch.dot(rh, r)
        p = r + (new / rho) * (a / w) * (p - w * v)
        rho = new
        ph = dinv * p
        v = A @ ph
        a = rho / torch.dot(rh, v)
        s = r - a * v
        sh = dinv * s
        t = A @ sh
        w = torch.dot(t, s) / torch.dot(t, t)
        x = x + a * ph + w * sh
        r = s - w * t
    return x


def _diag(A, rows):
    cols = A.col_indices()
    m = rows == cols
    d = torch.zeros(A.shape[0], dtype=torch.float64, device=cols.device)
    d[rows[m]] = A.values()[m]
    return d


def _nodal(code, x):
    u = torch.zeros(code.numel(), dtype=torch.float64, device=x.device)
    u[code == 0] = x
    return u


def _cd_element(u, v):
    def f(grad, area, elem):
        dev = area.device
        m1 = (torch.full((3, 3), 1.0 / 12, dtype=torch.float64, device=dev)
              + torch.eye(3, dtype=torch.float64, device=dev) * (1.0 / 12 + 1.0 / 3))
        m1 = m1[None] * (area / DT)[:, None, None]
        a0 = EPS * area[:, None, None] * torch.einsum("eia,eja->eij", grad, grad)
        v3 = v.reshape(-1, 2)[elem].sum(1)
        a0 = a0 + (area / 9)[:, None, None] * torch.einsum("ea,eja->ej", v3, grad)[:, None, :]
        return m1 + a0, torch.einsum("eij,ej->ei", m1, u[elem])
    return f


def _sweeps(A, rows, r, nx, ny, prec):
    """D-ILU or symmetric Gauss-Seidel on the structured square, a diagonal
    of the grid at a time (rows of one diagonal do not depend on each other)."""
    H, W = nx - 1, ny - 1
    n = H * W
    cols, val = A.col_indices(), A.values()

    def band(off):
        t = torch.zeros(n, dtype=torch.float64, device=val.device)
        m = cols - rows == off
        t[rows[m]] = val[m]
        return t.reshape(H, W)

    offs = [-W - 1, -W, -1]

    def skew(t):
        """Row (i, j) at [i + j, i]: a diagonal of the grid is a row here."""
        s = torch.zeros(H + W - 1, H, dtype=t.dtype, device=t.device)
        i = torch.arange(H, device=t.device)[:, None]
        j = torch.arange(W, device=t.device)[None, :]
        s[(i + j), i.expand(H, W)] = t
        return s

    lo = [skew(band(o)) for o in offs]
    up = [skew(band(-o)) for o in offs]
    i = torch.arange(H, device=val.device)[:, None]
    j = torch.arange(W, device=val.device)[None, :]
    diag, b = skew(band(0)), skew(r.reshape(H, W))
    ok = skew(torch.ones(H, W, dtype=torch.float64, device=val.device)) > 0
    D = H + W - 1

    def before(s, d, q):
        # neighbour (i-1, j-1), (i-1, j), (i, j-1) of diagonal d
        o = d - 2 if q == 0 else d - 1
        if o < 0:
            return torch.zeros(H, dtype=torch.float64, device=s.device)
        return s[o] if q == 2 else torch.cat([s[o, :1] * 0, s[o, :-1]])

    def after(s, d, q):
        o = d + 2 if q == 0 else d + 1
        if o >= D:
            return torch.zeros(H, dtype=torch.float64, device=s.device)
        return s[o] if q == 2 else torch.cat([s[o, 1:], s[o, :1] * 0])

    piv = diag.clone()
    if prec == "ILU":
        inv = torch.zeros_like(diag)
        upn = up                      # a(k, i) for k before i, read at k
        for d in range(D):
            s = diag[d].clone()
            for q in range(3):
                s -= lo[q][d] * before(inv, d, q) * before(upn[q], d, q)
            inv[d] = torch.where(ok[d], 1.0 / torch.where(ok[d], s, 1.0), 0.0)
        piv = inv
    else:
        piv = torch.where(ok, 1.0 / torch.where(ok, diag, 1.0), 0.0)
    t = torch.zeros_like(b)
    for d in range(D):
        s = b[d].clone()
        for q in range(3):
            s -= lo[q][d] * before(t, d, q)
        t[d] = s * piv[d]
    z = torch.zeros_like(b)
    for d in range(D - 1, -1, -1):
        s = torch.zeros_like(b[d])
        for q in range(3):
            s += up[q][d] * after(z, d, q)
        z[d] = t[d] - s * piv[d]
    return z[(i + j), i.expand(H, W)].reshape(-1)


def exact(case, seed):
    fam = case["family"]
    if fam == "train":
        return None                       # an FP32 / BF16 network: no 64-bit value
    if fam == "batch":
        xs, es, cs, ks, fs, off = [], [], [], [], [], 0
        grp = []
        for q, (xy, elem, code, k, f) in enumerate(_batch_inputs(case, seed)):
            xs.append(xy)
            es.append(elem + off)
            cs.append(code)
            ks.append(k)
            fs.append(f)
            grp.append(torch.full((int((code == 0).sum()),), q, device=DEV))
            off += code.numel()
        code = torch.cat(cs)
        A, b, rows = _assembled(torch.cat(xs), torch.cat(es), code, torch.cat(ks), torch.cat(fs),
                                None)
        x = _tight_cg(A, b, 1.0 / _diag(A, rows), torch.cat(grp))
        return dict(u=_nodal(code, x))
    if fam == "prec" and case["mesh"] != "square":
        return None                       # no plain vectorised form on the cube
    d = _inputs(case, seed)
    if fam == "step":
        A, b, rows = _assembled(d["xy"], d["elem"], d["code"], None, None, None,
                                _cd_element(d["u"], d["v"]))
        x = _tight_bicgstab(A, b, torch.zeros_like(b), 1.0 / _diag(A, rows))
        return dict(u=_nodal(d["code"], x), x=x)
    A, b, rows = _assembled(d["xy"], d["elem"], d["code"], d["k"], d["f"], d["bc"])
    if fam == "mult":
        return A @ _uniform(_gen(seed + 7), b.numel())
    if fam == "assemble":
        return dict(values=A.values(), b=b)
    if fam == "prec":
        return _sweeps(A, rows, _uniform(_gen(seed + 7), b.numel()), case["nx"], case["ny"],
                       case["prec"])
    x = _tight_cg(A, b, 1.0 / _diag(A, rows))
    return dict(iterations=None, x=x, u=_nodal(d["code"], x))
