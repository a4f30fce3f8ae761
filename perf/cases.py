"""Performance cases of the op2 backend: what a simulation code built on it runs.

Eight kinds of work, each through the entry points a user's program calls:

* ``airfoil``: outer iterations of the airfoil finite-volume chain (direct
  loops, an indirect READ loop, indirect INC loops, Global reductions);
* ``p1``: P1 mass Mat and right-hand side on a triangle mesh;
* ``p2``: P2 stiffness and mass Mats by one loop, in FP64 or with FP32 element
  math and compensated FP64 accumulation;
* ``setup``: a new mesh from host arrays to its first assembled Mat and RHS
  (Map upload and checks, Sparsity build, every table a loop needs);
* ``solve``: a Jacobi-CG solve with a P2 mass Mat;
* ``vec``: Dat arithmetic and a norm;
* ``batch``: many uneven P1 meshes, three loops each, in batched launches;
* ``serve``: a mixed set of assembly and chain requests through the engine.

Loops run either one by one through ``op2.par_loop`` or, as a program with a
fixed step records them, as one CUDA graph (``graph``).
"""

import math

import numpy as np
import torch

from pyop2_b200 import b200, op2, serve
from pyop2_b200.batch import BatchLoop
from pyop2_b200.workloads import airfoil, batching, fem, meshes, serving


def listed():
    return [
        # the airfoil chain at the size of the OP2 demo's mesh, the step recorded once
        {"name": "airfoil 1200x600", "kind": "airfoil", "nx": 1200, "ny": 600, "iters": 1, "graph": True},
        # a small mesh stepped from Python: launches and host path count
        {"name": "airfoil 101x53 loops", "kind": "airfoil", "nx": 101, "ny": 53, "iters": 2, "graph": False},
        # the mass2d form on the unit square, re-assembled inside a recorded step
        {"name": "p1 256x256", "kind": "p1", "nx": 256, "ny": 256, "permute": False, "graph": True},
        # the largest served triangle mesh: a million elements, permuted numbering, odd sides
        {"name": "p1 1000x503 permuted", "kind": "p1", "nx": 1000, "ny": 503, "permute": True, "graph": False},
        # P2 stiffness and mass, the largest Mats in use: 48 million entries each
        {"name": "p2 1024", "kind": "p2", "n": 1024, "precision": "f64", "graph": False},
        # the same on a mesh that fits the L2, odd side, inside a recorded step
        {"name": "p2 181", "kind": "p2", "n": 181, "precision": "f64", "graph": True},
        # FP32 element math, compensated FP64 accumulation in element order
        {"name": "p2 512 f32", "kind": "p2", "n": 512, "precision": "f32", "graph": False},
        # remeshing: everything a new mesh costs up to its first assembly
        {"name": "setup p1 350x301", "kind": "setup", "nx": 350, "ny": 301},
        # the linear solve of an implicit step
        {"name": "solve p2 512", "kind": "solve", "n": 512, "rtol": 1e-10},
        # the vector updates between loops
        {"name": "vec 4198401", "kind": "vec", "n": 4198401, "dim": 1},
        # an ensemble of uneven meshes, one graph of three batched launches
        {"name": "batch 256 meshes", "kind": "batch", "nmesh": 256, "emax": 65536},
        # a burst of requests at a server with its meshes resident
        {"name": "serve 24 requests", "kind": "serve", "njobs": 24, "nmesh": 6, "p1_max": 200000.0, "quad_max": 100000.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["airfoil", "airfoil", "p1", "p1", "p2", "p2", "setup", "solve", "vec", "batch", "serve"])
    if kind == "airfoil":
        cells, r = _log(rng, 4e3, 7.2e5), _log(rng, 0.5, 4.0)
        nx = max(8, int(math.sqrt(cells * r)))
        ny = max(8, min(int(cells / nx), 720000 // nx))
        return {"kind": kind, "nx": nx, "ny": ny, "iters": 1 if cells > 1e5 else 2, "graph": rng.random() < 0.5}
    if kind in ("p1", "setup"):
        quads, r = _log(rng, 500, 5e5 if kind == "p1" else 2e5), _log(rng, 0.25, 4.0)
        nx = max(4, int(math.sqrt(quads * r)))
        ny = max(4, int(quads / nx))
        if kind == "setup":
            return {"kind": kind, "nx": nx, "ny": ny}
        return {"kind": kind, "nx": nx, "ny": ny, "permute": rng.random() < 0.5, "graph": rng.random() < 0.5}
    if kind == "p2":
        f32 = rng.random() < 0.3
        return {"kind": kind, "n": int(_log(rng, 16, 512 if f32 else 900)), "precision": "f32" if f32 else "f64",
                "graph": rng.random() < 0.5}
    if kind == "solve":
        return {"kind": kind, "n": int(_log(rng, 24, 512)), "rtol": 1e-10}
    if kind == "vec":
        dim = rng.choice([1, 2, 4])
        return {"kind": kind, "n": int(_log(rng, 1e4, 4e6)) // dim, "dim": dim}
    if kind == "batch":
        return {"kind": kind, "nmesh": int(_log(rng, 24, 256)), "emax": int(_log(rng, 4096, 65536))}
    return {"kind": kind, "njobs": rng.randint(6, 24), "nmesh": rng.randint(2, 6), "p1_max": _log(rng, 1e4, 2e5),
            "quad_max": _log(rng, 2e4, 1e5)}


# ------------------------------------------------------------- device views
class _Span(object):
    """Device memory of ``owner``, which the span keeps alive."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": None, "stream": None}


def _view(ptr, n, owner):
    """``n`` doubles of ``owner``'s device memory at ``ptr`` as a torch tensor (no copy)."""
    return torch.as_tensor(_Span(ptr, n, owner), device="cuda")


def _ints(ptr, n, owner):
    s = _Span(ptr, n, owner)
    s.__cuda_array_interface__["typestr"] = "<i4"
    return torch.as_tensor(s, device="cuda")


def _dat_view(d):
    return _view(d.array.ptr, d.dataset.total_size * d.cdim, d)


def _mat_view(m):
    return _view(m._device_values().ptr, int(m.sparsity.nz), m)


_CONSTS = []


def _init(**config):
    """Start the backend (once per process); later calls set the configuration."""
    op2.init(backend="b200", device=0, **dict({"inc_mode": "staged", "kahan": False}, **config))
    if not _CONSTS:
        _CONSTS.extend(serving.declare_consts(op2))


def _jitter(coords, nx, ny, rng):
    """Nodes moved by up to a tenth of the cell size."""
    return coords + rng.uniform(-0.1, 0.1, size=coords.shape) / max(nx, ny)


class _State(object):
    """A prepared case: ``call()`` runs one pass and returns its outputs."""


def _record(s, step, reset=None):
    """Record ``step`` as a CUDA graph (it has to run once before)."""
    step()
    b200.synchronize()
    with b200.capture() as g:
        step()
    if reset:
        reset()
    b200.synchronize()
    s.graph = g
    return g.launch


# ------------------------------------------------------------------ airfoil
def _airfoil_inputs(case, seed):
    g = meshes.airfoil_grid(case["nx"], case["ny"], seed)
    rng = np.random.default_rng(seed + 1)
    qinf = np.array([1.0, 0.5, 0.0, 2.625])
    return g, qinf * (1.0 + rng.uniform(-0.01, 0.01, size=(g.ncells, 4)))


def _prepare_airfoil(case, seed):
    _init()
    g, q0 = _airfoil_inputs(case, seed)
    s = _State()
    A = s.A = airfoil.build(op2, 0, 0, grid=g, consts=False, q0=q0.copy())
    iters = case["iters"]
    views = {"q": A.p_q, "qold": A.p_qold, "res": A.p_res, "adt": A.p_adt}
    if case["graph"]:
        rms = s.rms = op2.Global(1, 0.0, np.float64, "rms")

        def step():
            for _ in range(iters):
                rms.zero()
                airfoil.iteration(op2, A, rms)

        def reset():
            A.p_q.data[...] = q0
            for d in views.values():
                _dat_view(d)
        launch = _record(s, step, reset)
        out = {k: _dat_view(d) for k, d in views.items()}
        out["rms"] = _view(rms._device.ptr, 1, rms)

        def call():
            launch()
            return out
    else:
        out = {k: _dat_view(d) for k, d in views.items()}

        def call():
            # the demo's loop: a new rms Global per update, read at the end
            for _ in range(iters):
                rms = airfoil.iteration(op2, A)
            return dict(out, rms=float(rms.data[0]))
    s.call = call
    return s


def _exact_airfoil(case, seed):
    g, q0 = _airfoil_inputs(case, seed)
    return _airfoil_steps(g, q0, case["iters"], case["graph"])


def _airfoil_steps(g, q0, iters, both_rms, qold_first=False):
    """The chain in 64-bit torch arithmetic; ``both_rms``: rms sums both updates of an iteration."""
    gam, gm1, cfl, eps = 1.4, 0.4, 0.9, 0.05
    T = lambda a: torch.as_tensor(np.asarray(a), device="cuda")  # noqa: E731
    x, q = T(g.x), T(q0).clone()
    pc, pe, pec = T(g.pcell).long(), T(g.pedge).long(), T(g.pecell).long()
    pb, pbc, bnd = T(g.pbedge).long(), T(g.pbecell).long()[:, 0], T(g.p_bound)[:, 0]
    qinf = torch.tensor([1.0, 0.5, 0.0, 2.625], dtype=torch.float64, device="cuda")
    res = torch.zeros_like(q)
    adt = qold = rms = None

    def press(w):
        return gm1 * (w[..., 3] - 0.5 / w[..., 0] * (w[..., 1] ** 2 + w[..., 2] ** 2))

    def flux(w1, w2, p1, p2, dx, dy, mu):
        v1, v2 = (w1[..., 1] * dy - w1[..., 2] * dx) / w1[..., 0], (w2[..., 1] * dy - w2[..., 2] * dx) / w2[..., 0]
        z = torch.zeros_like(dx)
        f = 0.5 * (v1[:, None] * w1 + v2[:, None] * w2)
        f = f + 0.5 * torch.stack([z, (p1 + p2) * dy, -(p1 + p2) * dx, v1 * p1 + v2 * p2], dim=1)
        return f + mu[:, None] * (w1 - w2)

    for it in range(iters):
        if not qold_first or it == 0:
            qold = q.clone()
        total = 0.0
        for _ in range(1 if qold_first else 2):
            c = torch.sqrt(gam * gm1 * (q[:, 3] / q[:, 0] - 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0] ** 2))
            adt = torch.zeros_like(c)
            for k in range(4):
                d = x[pc[:, (k + 1) % 4]] - x[pc[:, k]]
                adt = adt + ((q[:, 1] * d[:, 1] - q[:, 2] * d[:, 0]) / q[:, 0]).abs() + c * d.norm(dim=1)
            adt = adt / cfl
            d = x[pe[:, 0]] - x[pe[:, 1]]
            w1, w2 = q[pec[:, 0]], q[pec[:, 1]]
            f = flux(w1, w2, press(w1), press(w2), d[:, 0], d[:, 1], 0.5 * (adt[pec[:, 0]] + adt[pec[:, 1]]) * eps)
            res.index_add_(0, pec[:, 0], f)
            res.index_add_(0, pec[:, 1], -f)
            d = x[pb[:, 0]] - x[pb[:, 1]]
            w1 = q[pbc]
            w2 = qinf.expand_as(w1)
            p1 = press(w1)
            f = flux(w1, w2, p1, press(w2), d[:, 0], d[:, 1], adt[pbc] * eps)
            z = torch.zeros_like(p1)
            wall = torch.stack([z, p1 * d[:, 1], -p1 * d[:, 0], z], dim=1)
            res.index_add_(0, pbc, torch.where((bnd == 1)[:, None], wall, f))
            dq = res / adt[:, None]
            q = qold - dq
            res = torch.zeros_like(q)
            rms = float((dq * dq).sum())
            total += rms
        if both_rms:
            rms = total
    return {"q": q.reshape(-1), "qold": qold.reshape(-1), "res": res.reshape(-1), "adt": adt,
            "rms": torch.tensor([rms], dtype=torch.float64) if both_rms else float(rms)}


def _work_airfoil(case):
    nx, ny = case["nx"], case["ny"]
    b = airfoil.bytes_per_iteration(nx * ny, (nx + 1) * (ny + 1), (nx - 1) * ny + nx * (ny - 1), 2 * (nx + ny))
    return {"bytes": b["iteration"] * case["iters"],
            "flops": case["iters"] * (2 * nx * ny * (45 + 2 * 95 + 17))}


# ---------------------------------------------------------------------- P1
_PHI1 = np.array([[2 / 3, 1 / 6, 1 / 6], [1 / 6, 1 / 6, 2 / 3], [1 / 6, 2 / 3, 1 / 6]])


def _p1_inputs(case, seed):
    coords, elem = meshes.rect_p1(case["nx"], case["ny"], seed if case.get("permute", True) else None)
    rng = np.random.default_rng(seed + 2)
    coords = _jitter(coords, case["nx"], case["ny"], rng)
    return coords, elem, rng.standard_normal(len(coords))


def _prepare_p1(case, seed):
    _init()
    coords, elem, f = _p1_inputs(case, seed)
    s = _State()
    P = s.P = fem.build_p1(op2, 0, coords=coords, elem=elem)
    P.f.data[...] = f.reshape(P.f.data.shape)

    def step():
        P.mat.zero()
        P.b.zero()
        fem.assemble_p1(op2, P)
    out = {"mat": _mat_view(P.mat), "b": _dat_view(P.b)}
    launch = _record(s, step) if case["graph"] else step

    def call():
        launch()
        return out
    s.call = call
    return s


def _csr(elem, local):
    """CSR of element matrices ``local`` [m][E, a, a]: rowptr, colidx, values per m."""
    e = torch.as_tensor(elem, device="cuda").long()
    n = int(e.max()) + 1
    keys, inv = torch.unique(e[:, :, None] * n + e[:, None, :], return_inverse=True)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(keys // n, minlength=n), 0)
    inv = inv.reshape(-1)
    vals = [torch.zeros(keys.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv, m.reshape(-1))
            for m in local]
    return rowptr.int(), (keys % n).int(), vals


def _jac(coords, elem):
    x = torch.as_tensor(coords, device="cuda")[torch.as_tensor(elem, device="cuda").long()[:, :3]]
    return x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]      # columns of the Jacobian


def _p1_local(coords, elem, f):
    a, b = _jac(coords, elem)
    det = (a[:, 0] * b[:, 1] - b[:, 0] * a[:, 1])
    phi = torch.as_tensor(_PHI1, device="cuda")
    ref = phi.T @ phi / 6.0
    rg = torch.tensor([[-1.0, -1.0], [1.0, 0.0], [0.0, 1.0]], dtype=torch.float64, device="cuda")
    g = torch.stack([b[:, 1:2] * rg[:, 0] - a[:, 1:2] * rg[:, 1],
                     a[:, 0:1] * rg[:, 1] - b[:, 0:1] * rg[:, 0]], dim=2) / det[:, None, None]
    area = det.abs()
    e = torch.as_tensor(elem, device="cuda").long()
    loc = (torch.as_tensor(f, device="cuda")[e] @ ref) * area[:, None]
    rhs = torch.zeros(len(coords), dtype=torch.float64, device="cuda").index_add_(0, e.reshape(-1), loc.reshape(-1))
    return area[:, None, None] * ref, 0.5 * area[:, None, None] * (g @ g.transpose(1, 2)), rhs


def _exact_p1(case, seed):
    coords, elem, f = _p1_inputs(case, seed)
    mass, _, rhs = _p1_local(coords, elem, f)
    return {"mat": _csr(elem, [mass])[2][0], "b": rhs}


def _p1_sizes(nx, ny):
    return 2 * nx * ny, (nx + 1) * (ny + 1), 7 * nx * ny + 3 * (nx + ny) + 1


def _work_p1(case):
    e, n, nnz = _p1_sizes(case["nx"], case["ny"])
    # one mesh and its coordinates, the pattern, f; the Mat and the RHS written
    return {"bytes": e * 12 + n * 16 + (n + 1) * 4 + nnz * 4 + n * 8 + nnz * 8 + n * 8, "flops": e * (9 * 15 + 3 * 30)}


# ---------------------------------------------------------------------- P2
def _prepare_p2(case, seed):
    f32 = case["precision"] == "f32"
    _init(**(dict(inc_mode="lma", kahan=True) if f32 else {}))
    s = _State()
    P = s.P = fem.build_p2(op2, case["n"], seed, precision=case["precision"])

    def step():
        P.K.zero()
        P.M.zero()
        fem.assemble_p2(op2, P)
    out = {"K": _mat_view(P.K), "M": _mat_view(P.M)}
    launch = _record(s, step) if case["graph"] else step

    def call():
        launch()
        return out
    s.call = call
    return s


def _p2_basis(s, t):
    l0, l1, l2 = 1 - s - t, s, t
    phi = [l0 * (2 * l0 - 1), l1 * (2 * l1 - 1), l2 * (2 * l2 - 1), 4 * l1 * l2, 4 * l0 * l2, 4 * l0 * l1]
    ds = [1 - 4 * l0, 4 * l1 - 1, 0 * s, 4 * l2, -4 * l2, 4 * (l0 - l1)]
    dt = [1 - 4 * l0, 0 * s, 4 * l2 - 1, 4 * l1, 4 * (l0 - l2), -4 * l1]
    return np.array(phi), np.array(ds), np.array(dt)


def _p2_mass_ref():
    a, b = 0.445948490915965, 0.091576213509771
    w = np.repeat([0.223381589678011 / 2, 0.109951743655322 / 2], 3)
    phi, _, _ = _p2_basis(np.array([a, 1 - 2 * a, a, b, 1 - 2 * b, b]), np.array([a, a, 1 - 2 * a, b, b, 1 - 2 * b]))
    return (phi * w) @ phi.T


def _p2_local(coords, elem):
    a, b = _jac(coords, elem)
    det = a[:, 0] * b[:, 1] - b[:, 0] * a[:, 1]
    _, ds, dt = _p2_basis(np.array([1 / 6, 2 / 3, 1 / 6]), np.array([1 / 6, 1 / 6, 2 / 3]))
    T = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
    ss, st, tt = T(ds @ ds.T / 6), T((ds @ dt.T + dt @ ds.T) / 6), T(dt @ dt.T / 6)
    w = det.abs() / det ** 2
    c = [w * (b * b).sum(1), -w * (a * b).sum(1), w * (a * a).sum(1)]
    K = sum(k[:, None, None] * m for k, m in zip(c, (ss, st, tt)))
    return K, det.abs()[:, None, None] * T(_p2_mass_ref())


def _exact_p2(case, seed):
    coords, elem = meshes.square_p2(case["n"], seed)
    K, M = _csr(elem, _p2_local(coords, elem))[2]
    return {"K": K, "M": M}


def _p2_sizes(n):
    return 2 * n * n, (2 * n + 1) ** 2, 46 * n * n + 16 * n + 1


def _work_p2(case):
    e, n, nnz = _p2_sizes(case["n"])
    return {"bytes": e * 24 + n * 16 + (n + 1) * 4 + nnz * 4 + 2 * nnz * 8, "flops": e * 36 * 40}


# ------------------------------------------------------------------- setup
def _prepare_setup(case, seed):
    _init()
    s = _State()
    coords, elem, f = _p1_inputs(case, seed)
    e, n, nnz = _p1_sizes(case["nx"], case["ny"])
    k_mass, k_rhs = op2.Kernel(fem.P1_MASS, "p1_mass"), op2.Kernel(fem.P1_RHS, "p1_rhs")

    def call():
        nodes, vnodes, elements = op2.Set(n, 1, "nodes"), op2.Set(n, 2, "vnodes"), op2.Set(e, 1, "elements")
        values = elem.copy()
        en = op2.Map(elements, nodes, 3, values, "elem_node")
        ev = op2.Map(elements, vnodes, 3, values, "elem_vnode")
        sp = op2.Sparsity((en, en), "p1_sparsity")
        mat = op2.Mat(sp, np.float64, "mass")
        x, fd = op2.Dat(vnodes, coords, np.float64, "coords"), op2.Dat(nodes, f, np.float64, "f")
        b = op2.Dat(nodes, None, np.float64, "b")
        b.zero()
        op2.par_loop(k_mass, elements(3, 3), mat((en[op2.i[0]], en[op2.i[1]]), op2.INC), x(ev, op2.READ))
        op2.par_loop(k_rhs, elements(3), b(en[op2.i[0]], op2.INC), x(ev, op2.READ), fd(en, op2.READ))
        s.last = (mat, b)
        return {"rowptr": _ints(sp._d_rowptr, n + 1, sp), "colidx": _ints(sp._d_colidx, nnz, sp), "mat": _mat_view(mat),
                "b": _dat_view(b)}
    s.call = call
    return s


def _exact_setup(case, seed):
    coords, elem, f = _p1_inputs(case, seed)
    mass, _, rhs = _p1_local(coords, elem, f)
    rowptr, colidx, (mat,) = _csr(elem, [mass])
    return {"rowptr": rowptr, "colidx": colidx, "mat": mat, "b": rhs}


def _work_setup(case):
    e, n, nnz = _p1_sizes(case["nx"], case["ny"])
    return {"bytes": e * 12 + n * 16 + n * 8 + (n + 1) * 4 + nnz * 4 + nnz * 8 + n * 8,
            "flops": e * (9 * 15 + 3 * 30)}


# ------------------------------------------------------------------- solve
def _solve_inputs(case, seed):
    coords, elem = meshes.square_p2(case["n"], seed)
    x = np.random.default_rng(seed + 3).standard_normal(len(coords))
    p = coords[elem[:, :3]]
    a, b = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    det = np.abs(a[:, 0] * b[:, 1] - b[:, 0] * a[:, 1])
    loc = (x[elem] @ _p2_mass_ref()) * det[:, None]
    return coords, elem, x, np.bincount(elem.ravel(), weights=loc.ravel(), minlength=len(coords))


def _prepare_solve(case, seed):
    _init()
    s = _State()
    coords, elem, x, rhs = _solve_inputs(case, seed)
    P = s.P = fem.build_p2(op2, case["n"], coords=coords, elem=elem)
    fem.assemble_p2(op2, P)
    s.x = op2.Dat(P.dofs, np.zeros(len(x)), np.float64, "x")
    s.b = op2.Dat(P.dofs, rhs, np.float64, "b")
    solver = op2.Solver(relative_tolerance=case["rtol"])
    out = _dat_view(s.x)

    def call():
        solver.solve(P.M, s.x, s.b)
        return out
    s.call = call
    return s


def _exact_solve(case, seed):
    return torch.as_tensor(_solve_inputs(case, seed)[2])


def _work_solve(case):
    _, n, nnz = _p2_sizes(case["n"])
    steps = 25      # about what the tolerance takes on these matrices
    return {"bytes": steps * (nnz * 12 + (n + 1) * 4 + n * 8 * 11), "flops": steps * (2 * nnz + 14 * n)}


# --------------------------------------------------------------------- vec
def _vec_inputs(case, seed):
    rng = np.random.default_rng(seed)
    shape = (case["n"], case["dim"])
    return rng.standard_normal(shape), rng.standard_normal(shape)


def _prepare_vec(case, seed):
    _init()
    s = _State()
    x, y = _vec_inputs(case, seed)
    s.set = op2.Set(case["n"], case["dim"], "dofs")
    s.x, s.y = op2.Dat(s.set, x, np.float64, "x"), op2.Dat(s.set, y, np.float64, "y")
    s.x.array
    out = _dat_view(s.y)

    def call():
        # y <- x + y / 2, the step of a relaxation, and its norm
        s.y *= 0.5
        s.y += s.x
        return {"y": out, "norm": s.y.norm}
    s.call = call
    return s


def _exact_vec(case, seed):
    x, y = _vec_inputs(case, seed)
    y = x + 0.5 * y
    return {"y": y.reshape(-1), "norm": float(np.sqrt((y * y).sum()))}


def _work_vec(case):
    n = case["n"] * case["dim"]
    return {"bytes": n * 24, "flops": 4 * n}


# ------------------------------------------------------------------- batch
def _batch_meshes(case, seed):
    shapes = batching.mesh_shapes(case["nmesh"], case["nmesh"] + 1, emax=case["emax"])   # sizes belong to the case
    out = []
    for m, (nx, ny) in enumerate(shapes):
        out.append(_p1_inputs({"nx": nx, "ny": ny}, seed * 4099 + m))
    return shapes, out


def _arena(shapes):
    """Offsets (in doubles) of each mesh's mass, stiffness and RHS, 256-byte aligned."""
    offs, o = [], 0
    for nx, ny in shapes:
        _, n, nnz = _p1_sizes(nx, ny)
        row = []
        for k in (nnz, nnz, n):
            row.append(o)
            o += (k + 31) // 32 * 32
        offs.append(row)
    return offs, o


def _prepare_batch(case, seed):
    _init()
    s = _State()
    shapes, inputs = _batch_meshes(case, seed)
    s.problems = []
    for coords, elem, f in inputs:
        P = fem.build_p1(op2, 0, coords=coords, elem=elem, stiffness=True)
        P.f.data[...] = f.reshape(P.f.data.shape)
        s.problems.append(P)
    offs, total = _arena(shapes)
    s.arena = b200.DeviceBuffer(total * 8)
    at = lambda o: s.arena.ptr + 8 * o  # noqa: E731
    groups = [[], [], []]
    for row, P, insts in zip(offs, s.problems, zip(*batching.instances(op2, s.problems))):
        for g, inst, obj, o in zip(groups, insts, (P.mat, P.stiff, P.b), row):
            g.append(inst.patch({obj: at(o)}))
    s.loops = [BatchLoop(g, block_size=256, elems_per_thread=2) for g in groups]

    def step():
        s.arena.memset(0)
        for bl in s.loops:
            bl.launch(sync_host=False)
    launch = _record(s, step)
    out = _view(s.arena.ptr, total, s.arena)

    def call():
        launch()
        return out
    s.call = call
    return s


def _exact_batch(case, seed):
    shapes, inputs = _batch_meshes(case, seed)
    offs, total = _arena(shapes)
    out = torch.zeros(total, dtype=torch.float64, device="cuda")
    for row, (coords, elem, f) in zip(offs, inputs):
        mass, stiff, rhs = _p1_local(coords, elem, f)
        for o, v in zip(row, _csr(elem, [mass, stiff])[2] + [rhs]):
            out[o:o + v.numel()] = v
    return out


def _work_batch(case):
    b = fl = 0
    for nx, ny in batching.mesh_shapes(case["nmesh"], case["nmesh"] + 1, emax=case["emax"]):
        e, n, nnz = _p1_sizes(nx, ny)
        b += e * 12 + n * 24 + (n + 1) * 4 + nnz * 4 + 2 * nnz * 8 + n * 8
        fl += e * (9 * 15 + 9 * 25 + 3 * 30)
    return {"bytes": b, "flops": fl}


# ------------------------------------------------------------------- serve
def _serve_inputs(case, seed):
    k = case["nmesh"]
    pool = serving.mesh_pool(k, k, seed=k, p1_range=(1e3, case["p1_max"]), quad_range=(1e4, case["quad_max"]))
    jobs = serving.trace(case["njobs"], 2000.0, pool, seed=case["njobs"])      # sizes and mix belong to the case
    rng = np.random.default_rng(seed)
    for j in jobs:
        j.seed = int(rng.integers(0, 2 ** 31))
    return pool, jobs


def _prepare_serve(case, seed):
    _init()
    s = _State()
    pool, s.jobs = _serve_inputs(case, seed)
    s.store = serve.MeshStore()
    serving.register(s.store, op2, pool, seed=1)
    for mid in sorted({j.mesh_id for j in s.jobs}):
        s.store.load(mid)

    def call():
        done = serve.Engine(s.store).run(serving.clone_trace(s.jobs, realtime=False), realtime=False)
        return {"%s %d" % (j.kind, j.rid): j.result for j in done}
    s.call = call
    return s


def _exact_serve(case, seed):
    pool, jobs = _serve_inputs(case, seed)
    made = {}
    for k, (mid, (kind, nx, ny)) in enumerate(sorted(pool.items())):
        made[mid] = (meshes.rect_p1(nx, ny, 7919 + k) if kind == "p1" else meshes.airfoil_grid(nx, ny, 7919 + k))
    out = {}
    qinf = np.array([1.0, 0.5, 0.0, 2.625])
    for j in jobs:
        scale = float(np.random.default_rng(j.seed).uniform(0.5, 2.0))
        if j.kind == "p1":
            coords, elem = made[j.mesh_id]
            f = scale * np.sin(np.pi * coords[:, 0]) * np.sin(np.pi * coords[:, 1])
            mass, _, rhs = _p1_local(coords, elem, f)
            out["p1 %d" % j.rid] = {"mat": _csr(elem, [mass])[2][0], "b": rhs}
        else:
            g = made[j.mesh_id]
            noise = np.random.default_rng(2).uniform(-0.01, 0.01, size=(g.ncells, 4))
            r = _airfoil_steps(g, qinf + scale * (qinf * (1.0 + noise) - qinf), j.iters, False, qold_first=True)
            # the engine's rms adds up over the chain's iterations
            out["quad %d" % j.rid] = {"q": r["q"].reshape(-1, 4), "rms": None}
    return out


def _work_serve(case):
    pool, jobs = _serve_inputs(case, 0)
    b = fl = 0
    for j in jobs:
        _, nx, ny = pool[j.mesh_id]
        if j.kind == "p1":
            w = _work_p1({"nx": nx, "ny": ny})
        else:
            w = _work_airfoil({"nx": nx, "ny": ny, "iters": j.iters / 2})
        b, fl = b + w["bytes"], fl + w["flops"]
    return {"bytes": b, "flops": fl}


# -------------------------------------------------------------- entry points
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state.call()


def work(case):
    return globals()["_work_" + case["kind"]](case)


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)
