"""The measured work: what programs built on pylith_b200 call again and again, over its real range.

Every case runs public entry points only (`pylith_b200.feassemble`, `pylith_b200.problems`,
`pylith_b200.materials`, `pylith_b200.greensfns`). Meshes are the package's own seeded boxes; a
program reads its mesh once, so a mesh depends on the case's sizes alone and is kept between
preparations, while every field, material and load comes from the seed.

Kinds of a case:
  apply      the matrix-free operators of a quasi-static step on one domain integrator: any of the
             FP64 residual, the FP64 Jacobian action and the FP32 Jacobian action
  visco      the state update that ends a generalized-Maxwell time step and the residual (domain and
             fault) that opens the next one
  assemble   the assembled Jacobian (3x3-block CSR) and one product with it
  output     the derived stress and strain fields of an output step
  static     a whole static solve: residual, multigrid-preconditioned CG with FP32 V-cycles
  greens     a tile of Green's-function impulses solved together
"""
import ctypes
import functools

import numpy as np
import torch

from pylith_b200 import _lib
from pylith_b200 import feassemble as FA
from pylith_b200 import greensfns as GF
from pylith_b200 import materials as MAT
from pylith_b200 import meshing as M
from pylith_b200 import multigrid as MG
from pylith_b200 import problems as P

DT = MAT.YEAR


def listed():
    return [
        # one residual and one Jacobian action on a mesh of a few thousand tetrahedra (the size of
        # a test mesh, or of one rank's share of a coarse level): launch latency counts
        dict(name="tet_small", kind="apply", mesh="delaunay", cells=4000, ops="residual,action", body_force=False),
        # an unstructured mesh of ordinary size, with the FP32 action of the refined solvers
        dict(name="tet_medium", kind="apply", mesh="delaunay", cells=60000, ops="residual,action,action32", body_force=False),
        # the production size: 1.2 million tetrahedra
        dict(name="tet_large", kind="apply", mesh="kuhn", nx=64, ny=64, nz=48, ops="residual,action", body_force=False),
        # the 16^3 hexahedral box of the closed-form test, under gravity
        dict(name="hex8_small", kind="apply", mesh="hex8", nx=16, ny=16, nz=16, ops="residual,action", body_force=True),
        # the 96x96x72 hexahedral box, both precisions of the action
        dict(name="hex8_large", kind="apply", mesh="hex8", nx=96, ny=96, nz=72, ops="residual,action,action32", body_force=False),
        # quadratic hexahedra, 6.4 million DOFs
        dict(name="hex27_large", kind="apply", mesh="hex27", nx=64, ny=64, nz=64, ops="residual,action", body_force=False),
        # viscoelastic relaxation around a fault: state update, then the next step's residual
        dict(name="visco_step", kind="visco", nx=48, ny=48, nz=36),
        # assembly for programs that hand the matrix to a direct or algebraic solver
        dict(name="assemble_hex8", kind="assemble", mesh="hex8", nx=32, ny=32, nz=24),
        dict(name="assemble_tet", kind="assemble", mesh="delaunay", cells=60000),
        # stress and strain of every cell for an output step, on a box with odd counts
        dict(name="output_hex8", kind="output", mesh="hex8", nx=61, ny=47, nz=35),
        # coseismic slip on a fault, solved from zero to full accuracy
        dict(name="static_solve", kind="static", nx=48, ny=48, nz=36),
        # eight unit-slip impulses in one tile on a tetrahedral mesh with a fault
        dict(name="greens_tile", kind="greens", nx=28, ny=28, nz=20, impulses=8),
    ]


def _box(rng, lo, hi):
    """Cells per direction of a box of about the proportions of the test boxes, each count its own."""
    n = lo * (hi / lo) ** rng.random()
    return [max(3, int(round(n * rng.uniform(0.8, 1.1)))) for _ in range(2)] + [max(3, int(round(n * rng.uniform(0.6, 0.9))))]


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "visco", "assemble", "output", "static", "greens"])
    if kind == "apply":
        mesh = rng.choice(["delaunay", "kuhn", "hex8", "hex27"])
        ops = rng.choice(["residual,action", "residual,action,action32"])
        c = dict(kind=kind, mesh=mesh, ops=ops, body_force=rng.random() < 0.3)
        if mesh == "delaunay":
            c["cells"] = int(3000 * 30 ** rng.random())
        else:
            lo, hi = {"kuhn": (6, 56), "hex8": (10, 86), "hex27": (4, 52)}[mesh]
            c["nx"], c["ny"], c["nz"] = _box(rng, lo, hi)
        if mesh == "hex27":
            c["ops"] = "residual,action"
        return c
    if kind == "visco":
        nx, ny, nz = _box(rng, 8, 46)
        return dict(kind=kind, nx=nx + nx % 2, ny=ny, nz=nz)
    if kind == "assemble":
        if rng.random() < 0.5:
            return dict(kind=kind, mesh="delaunay", cells=int(3000 * 20 ** rng.random()))
        nx, ny, nz = _box(rng, 8, 32)
        return dict(kind=kind, mesh="hex8", nx=nx, ny=ny, nz=nz)
    if kind == "output":
        mesh = rng.choice(["kuhn", "hex8"])
        nx, ny, nz = _box(rng, 8, 32 if mesh == "kuhn" else 60)
        return dict(kind=kind, mesh=mesh, nx=nx, ny=ny, nz=nz)
    nx, ny, nz = _box(rng, 10, 44 if kind == "static" else 26)
    c = dict(kind=kind, nx=4 * max(2, round(nx / 4)), ny=max(8, ny), nz=max(8, nz))
    if kind == "greens":
        c["impulses"] = rng.choice([4, 8])
    return c


# ---- meshes -----------------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _mesh_of(mesh, cells, nx, ny, nz, fault):
    if mesh == "delaunay":
        return M.box_tet_delaunay(cells, seed=1)
    if mesh == "kuhn":
        return M.box_tet_kuhn(nx, ny, nz, fault_x=0.0 if fault else None)
    if mesh == "hex27":
        return M.box_hex27(nx, ny, nz)
    return M.insert_fault_x(M.box_hex(nx, ny, nz)) if fault else M.box_hex(nx, ny, nz)


def _mesh(case, fault=False):
    mesh = case.get("mesh", "kuhn" if case["kind"] == "greens" else "hex8")
    return _mesh_of(mesh, case.get("cells", 0), case.get("nx", 0), case.get("ny", 0), case.get("nz", 0), fault)


@functools.lru_cache(maxsize=2)
def _levels(nx, ny, nz):
    return MG.build_hierarchy(nx, ny, nz, fault_x=0.0, constrained_faces=[(0, "neg", (0, 1, 2)), (0, "pos", (0, 1, 2))])


# ---- inputs from the seed ---------------------------------------------------------------------
def _elastic(mesh, seed):
    return MAT.lognormal_elastic(mesh.num_cells, seed=seed)


def _body_force(rho):
    return np.stack([0.0 * rho, 0.0 * rho, -9.80665 * rho], axis=1)


def _field(n, seed):
    return np.random.default_rng(seed + 1000).standard_normal(n)


def _maxwell(mesh, seed):
    rng = np.random.default_rng(seed + 2000)
    nc = mesh.num_cells
    rho, mu, K = _elastic(mesh, seed)
    tau = MAT.genmaxwell_times(rho, np.sqrt(mu / rho), [1e18, 1e19, 1e20], [0.3, 0.3, 0.3])
    visc = rng.standard_normal((nc, 8, 18), dtype=np.float32).astype(np.float64) * 1e-3
    total = rng.standard_normal((nc, 8, 6), dtype=np.float32).astype(np.float64) * 1e-3
    return rho, mu, K, tau, np.full((nc, 3), 0.3), visc, total


def _visco_fields(mesh, seed):
    """Displacements of metres, tractions (Lagrange multipliers) of MPa, slip of up to 2 m."""
    rng = np.random.default_rng(seed + 3000)
    u = _field(mesh.num_dof, seed)
    u[3 * mesh.num_nodes:] *= 1e7
    return u, np.stack([np.zeros(mesh.num_lagrange), 2.0 * rng.random(mesh.num_lagrange), rng.random(mesh.num_lagrange)], axis=1)


def _faces_fixed(mesh):
    cons = np.zeros((mesh.num_nodes, 3), dtype=bool)
    for side in ("neg", "pos"):
        cons[M.boundary_mask(mesh, 0, side)] = True
    return np.concatenate([cons.ravel(), np.zeros(3 * mesh.num_lagrange, dtype=bool)])


class _DeviceArray:
    """A device array of the library, by address, for torch; it keeps its owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _matrix_values(A):
    nrows, nnzb, val = ctypes.c_int64(), ctypes.c_int64(), ctypes.c_void_p()
    _lib.check(_lib.lib().pl_matrix_info(A.handle, ctypes.byref(nrows), ctypes.byref(nnzb), None, None, ctypes.byref(val)))
    return torch.as_tensor(_DeviceArray(A, val.value, (nnzb.value, 3, 3)), device="cuda")


# ---- prepare ----------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    ctx = FA.Context(0)
    s = {"kind": kind, "ctx": ctx}
    if kind in ("apply", "assemble", "output"):
        mesh = _mesh(case)
        rho, mu, K = _elastic(mesh, seed)
        mat = MAT.IsotropicLinearElasticity(rho, mu, K, _body_force(rho) if case.get("body_force") else None)
        dm = FA.DeviceMesh(ctx, mesh)
        s["ig"] = mat.create_integrator(dm)
        s["u"] = torch.from_numpy(_field(mesh.num_dof, seed)).cuda()
        if kind == "apply":
            s["ops"] = case["ops"].split(",")
            s["out"] = {op: torch.empty_like(s["u"]) for op in s["ops"] if op != "action32"}
            if "action32" in s["ops"]:
                s["v32"] = s["u"].float()
                s["out"]["action32"] = torch.empty_like(s["v32"])
        elif kind == "assemble":
            s["A"] = FA.Matrix(dm)
            s["val"] = _matrix_values(s["A"])
            s["y"] = torch.empty_like(s["u"])
        else:
            s["fields"] = torch.empty((mesh.num_cells, 12), dtype=torch.float64, device="cuda")
    elif kind == "visco":
        mesh = _mesh(case, fault=True)
        u, slip = _visco_fields(mesh, seed)
        dm = FA.DeviceMesh(ctx, mesh)
        s["ig"] = MAT.IsotropicLinearGenMaxwell(*_maxwell(mesh, seed)).create_integrator(dm, DT)
        s["fault"] = MAT.FaultCohesiveKin(slip).create_integrator(dm)
        s["u"] = torch.from_numpy(u).cuda()
        s["r"] = torch.empty_like(s["u"])
        s["nd"] = 3 * mesh.num_nodes
    elif kind == "static":
        levels = _levels(case["nx"], case["ny"], case["nz"])
        mesh = levels[0].mesh
        rng = np.random.default_rng(seed + 4000)
        slip = np.zeros((mesh.num_lagrange, 3))
        at = mesh.coords[mesh.cohesive[:, :4].ravel()]
        lag = mesh.cohesive[:, 8:].ravel()
        y0, z0 = rng.uniform(-3000.0, 0.0), rng.uniform(-7000.0, -4000.0)
        on = (at[:, 1] >= y0) & (at[:, 1] <= y0 + 4000.0) & (at[:, 2] >= z0) & (at[:, 2] <= z0 + 4000.0)
        slip[lag[on], 1] = rng.uniform(0.5, 3.0)
        mat = MAT.IsotropicLinearElasticity(*_elastic(mesh, seed))
        s["prob"] = P.QuasistaticProblem(ctx, mesh, [(mat, None)], levels[0].constrained, np.zeros(mesh.num_dof),
                                         faults=[MAT.FaultCohesiveKin(slip)], rtol=1e-12)
        s["mg"] = MG.attach(ctx, s["prob"].solver, levels, mat, fault_x=0.0, precision=FA.Solver.FP32_REFINED)
    else:
        mesh = _mesh(case, fault=True)
        mat = MAT.IsotropicLinearElasticity(*_elastic(mesh, seed))
        patches = GF.fault_patches(mesh, (-6000.0, 6000.0), (-9000.0, 0.0), 4, 3)
        g = GF.GreensFunctions(ctx, mesh, mat, _faces_fixed(mesh), patches, rtol=1e-12, inner_rtol=1e-4, tile=8)
        pick = np.random.default_rng(seed + 5000).choice(len(g.impulses), case["impulses"], replace=False)
        s["g"] = g
        s["b"] = [g.impulse_rhs(g.impulses[i])[1] for i in pick]
        s["x"] = [torch.empty_like(b) for b in s["b"]]
    return s


# ---- run --------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "apply":
        for op in s["ops"]:
            if op == "residual":
                s["ig"].compute_lhs_residual(0.0, 0.0, s["u"], s["out"][op])
            elif op == "action":
                s["ig"].compute_lhs_jacobian_action(0.0, 0.0, 0.0, s["u"], s["u"], s["out"][op])
            else:
                s["ig"].compute_lhs_jacobian_action_f32(0.0, 0.0, s["v32"], s["out"][op])
        return s["out"]
    if kind == "visco":
        s["ig"].update_state_vars(DT, DT, s["u"])
        s["ig"].compute_lhs_residual(2.0 * DT, DT, s["u"], s["r"])
        s["fault"].compute_lhs_residual(2.0 * DT, DT, s["u"], s["r"], mode=FA.ADD)
        return [s["r"][:s["nd"]], s["r"][s["nd"]:]]
    if kind == "assemble":
        s["A"].zero()
        s["ig"].compute_lhs_jacobian(0.0, 0.0, 0.0, s["u"], s["A"])
        s["A"].spmv(s["u"], s["y"])
        return [s["val"], s["y"]]
    if kind == "output":
        s["ig"].compute_derived_field(0.0, 0.0, s["u"], s["fields"])
        return s["fields"]
    if kind == "static":
        s["prob"].u.zero_()
        s["prob"].step(0.0)
        return s["prob"].u
    for x in s["x"]:
        x.zero_()
    s["g"].batch.solve(s["b"], s["x"])
    return s["x"]


# ---- work -------------------------------------------------------------------------------------
def work(case):
    """Unique bytes (each input once, each output once) and multiply-adds counted as two."""
    kind = case["kind"]
    mesh = _mesh(case, fault=kind in ("visco", "static", "greens"))
    nc, nn = mesh.num_cells, mesh.num_nodes
    nen, nq = mesh.cells.shape[1], M.QUAD_POINTS[mesh.cell_type]
    cell = nc * (4 * nen + 16)
    # per Gauss point: geometry, gradient, flux, test weights and, per node, the two contractions
    # (summed factor by factor for Q2)
    point = {4: 250, 8: 140 + 8 * 36, 27: 140 + 290}[nen] * nc * nq
    if kind == "apply":
        b = f = 0.0
        for op in case["ops"].split(","):
            b += cell + nn * (24 + (24 if op == "action32" else 48)) + (24 * nc if case["body_force"] and op == "residual" else 0)
            f += point
        return {"bytes": b, "flops": f}
    if kind == "visco":
        state = nc * nq * 24 * 8
        return {"bytes": 2 * (cell + 72 * nn) + 2 * 48 * nc + 3 * state, "flops": 2 * point + 400.0 * nc * nq}
    if kind == "assemble":
        nnzb = len(_pattern(case)[0])
        return {"bytes": cell + 24 * nn + nnzb * (2 * 72 + 4) + nn * 52, "flops": nc * nq * nen * nen * 40.0 + 18.0 * nnzb}
    if kind == "output":
        return {"bytes": cell + 48 * nn + 96 * nc, "flops": nc * 300.0}
    if kind == "static":  # about 12 iterations, each an FP64 operator and an FP32 V-cycle of 6 fine operators
        return {"bytes": 12 * (7 * cell + nn * (72 + 6 * 72)), "flops": 12 * 7.0 * point}
    n = case["impulses"]  # about 500 iterations, the cells read once per tile
    return {"bytes": 500.0 * (cell + nn * (24 + 24 * n + 60 * n)), "flops": 500.0 * n * point}


# ---- exact ------------------------------------------------------------------------------------
_CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _linear(x):
    return np.array([0.5 * (1 - x), 0.5 * (1 + x)]), np.array([-0.5, 0.5])


def _quadratic(x):
    return np.array([0.5 * x * (x - 1), 1 - x * x, 0.5 * x * (x + 1)]), np.array([x - 0.5, -2 * x, x + 0.5])


def _tensor(x, nodes, basis):
    """Values [n] and reference gradients [n, 3] of a tensor-product basis at the point x."""
    v, d = zip(*(basis(t) for t in x))
    val = np.array([v[0][a] * v[1][b] * v[2][c] for a, b, c in nodes])
    grad = np.array([[d[0][a] * v[1][b] * v[2][c], v[0][a] * d[1][b] * v[2][c], v[0][a] * v[1][b] * d[2][c]] for a, b, c in nodes])
    return val, grad


def _tables(cell_type, centre=False):
    """Per quadrature point: weight, geometry gradients, field values and gradients; corner columns."""
    if cell_type == M.CELL_TET4:
        g = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
        return np.array([1 / 6]), g[None], np.full((1, 4), 0.25), g[None], [0, 1, 2, 3]
    q2 = cell_type == M.CELL_HEX27
    x1, w1 = np.polynomial.legendre.leggauss(3 if q2 else 2)
    if centre:
        x1, w1 = np.array([0.0]), np.array([2.0])
    n1 = len(x1)
    w, gg, v, gf = [], [], [], []
    nodes = [(a, b, c) for c in range(3) for b in range(3) for a in range(3)] if q2 else _CORNERS
    for k in range(n1):
        for j in range(n1):
            for i in range(n1):
                x = (x1[i], x1[j], x1[k])
                w.append(w1[i] * w1[j] * w1[k])
                gg.append(_tensor(x, _CORNERS, _linear)[1])
                val, grad = _tensor(x, nodes, _quadratic if q2 else _linear)
                v.append(val)
                gf.append(grad)
    corner = [2 * a + 6 * b + 18 * c for a, b, c in _CORNERS] if q2 else list(range(8))
    return np.array(w), np.array(gg), np.array(v), np.array(gf), corner


def _cuda(*arrays):
    return [torch.as_tensor(np.asarray(a), device="cuda") for a in arrays]


def _chunks(mesh, size):
    return [slice(i, min(i + size, mesh.num_cells)) for i in range(0, mesh.num_cells, size)]


def _geometry(mesh, sl, coords, cells, tab):
    """(nodes, wdet [c, q], gradients [c, q, n, 3]) of the cells sl."""
    w, gg, _, gf, corner = tab
    cn = cells[sl].long()
    J = torch.einsum("cki,qkj->cqij", coords[cn[:, corner]], gg)
    grad = torch.einsum("qnj,cqjd->cqnd", gf, torch.linalg.inv(J))
    return cn, w * torch.linalg.det(J), grad


def _gpu_tables(mesh, centre=False):
    w, gg, v, gf, corner = _tables(mesh.cell_type, centre)
    return (*_cuda(w, gg, v, gf), corner)


def _stress(lam, mu, e):
    tr = e.diagonal(dim1=-2, dim2=-1).sum(-1)
    return (lam * tr)[..., None, None] * torch.eye(3, dtype=e.dtype, device=e.device) + 2 * mu[..., None, None] * e


def _apply_exact(mesh, u, mu, K, body_force):
    tab = _gpu_tables(mesh)
    coords, cells, un, mu, K = _cuda(mesh.coords, mesh.cells, u.reshape(-1, 3), mu, K)
    out = torch.zeros_like(un)
    bf = None if body_force is None else _cuda(body_force)[0]
    for sl in _chunks(mesh, 32768):
        cn, wdet, grad = _geometry(mesh, sl, coords, cells, tab)
        G = torch.einsum("cni,cqnd->cqid", un[cn], grad)
        e = 0.5 * (G + G.transpose(-1, -2))
        lam = (K - 2 * mu / 3)[sl, None]
        f1 = -_stress(lam.expand(wdet.shape), mu[sl, None].expand(wdet.shape), e)
        r = torch.einsum("cq,cqid,cqnd->cni", wdet, f1, grad)
        if bf is not None:
            r += torch.einsum("cq,qn,ci->cni", wdet, tab[2], bf[sl])
        out.index_add_(0, cn.reshape(-1), r.reshape(-1, 3))
    return out.reshape(-1)


def _sym(v):
    """[..., 6] (xx, yy, zz, xy, yz, xz) as [..., 3, 3]."""
    return v[..., [0, 3, 5, 3, 1, 4, 5, 4, 2]].reshape(v.shape[:-1] + (3, 3))


def _deviatoric(e):
    return e - (e.diagonal(dim1=-2, dim2=-1).sum(-1) / 3)[..., None, None] * torch.eye(3, dtype=e.dtype, device=e.device)


def _visco_exact(mesh, seed):
    rho, mu, K, tau, ratio, visc, total = _maxwell(mesh, seed)
    u, slip = _visco_fields(mesh, seed)
    tab = _gpu_tables(mesh)
    coords, cells, ut, mu, K, tau, ratio, visc, total, slip = _cuda(mesh.coords, mesh.cells, u, mu, K, tau, ratio, visc, total, slip)
    nn = mesh.num_nodes
    un, lag = ut[:3 * nn].reshape(-1, 3), ut[3 * nn:].reshape(-1, 3)
    out, lout = torch.zeros_like(un), torch.zeros_like(lag)
    for sl in _chunks(mesh, 16384):
        cn, wdet, grad = _geometry(mesh, sl, coords, cells, tab)
        G = torch.einsum("cni,cqnd->cqid", un[cn], grad)
        e = 0.5 * (G + G.transpose(-1, -2))
        de = _deviatoric(e)
        ef = torch.exp(-DT / tau[sl])[:, None, :, None, None]
        dq = (tau[sl] * (1 - torch.exp(-DT / tau[sl])) / DT)[:, None, :, None, None]
        old = _sym(visc[sl].reshape(visc[sl].shape[:2] + (3, 6)))
        new = ef * old + dq * (de - _deviatoric(_sym(total[sl])))[:, :, None]
        again = ef * new  # the strain has not changed since the update
        rr = ratio[sl][:, None, :, None, None]
        m = mu[sl][:, None, None, None]
        s = (K[sl][:, None] * e.diagonal(dim1=-2, dim2=-1).sum(-1))[..., None, None] * torch.eye(3, dtype=e.dtype, device=e.device)
        s = s + 2 * m * (1 - ratio[sl].sum(1))[:, None, None, None] * de + 2 * m * (rr * again).sum(2)
        out.index_add_(0, cn.reshape(-1), torch.einsum("cq,cqid,cqnd->cni", wdet, -s, grad).reshape(-1, 3))
    # the fault: bilinear quadrilaterals, normal +x, slip given as (opening, along y, along z)
    coh = _cuda(mesh.cohesive)[0].long()
    neg, pos, lg = coh[:, :4], coh[:, 4:8], coh[:, 8:]
    X = coords[neg]
    g = 1 / np.sqrt(3.0)
    for eta in (-g, g):
        for xi in (-g, g):
            (vx, dx), (vy, dy) = _linear(xi), _linear(eta)
            at = [(0, 0), (1, 0), (1, 1), (0, 1)]
            phi, = _cuda(np.array([vx[a] * vy[b] for a, b in at]))
            d, = _cuda(np.array([[dx[a] * vy[b], vx[a] * dy[b]] for a, b in at]))
            T = torch.einsum("cki,kj->cij", X, d)
            area = torch.linalg.cross(T[:, :, 0], T[:, :, 1]).norm(dim=1)
            lam = torch.einsum("k,cki->ci", phi, lag[lg])
            gap = torch.einsum("k,cki->ci", phi, un[pos] - un[neg] - slip[lg])
            w = area[:, None, None] * phi[None, :, None]
            out.index_add_(0, neg.reshape(-1), (-w * lam[:, None]).reshape(-1, 3))
            out.index_add_(0, pos.reshape(-1), (w * lam[:, None]).reshape(-1, 3))
            lout.index_add_(0, lg.reshape(-1), (w * gap[:, None]).reshape(-1, 3))
    return [out.reshape(-1), lout.reshape(-1)]


def _pattern(case):
    """Sorted block keys row * nodes + column of the assembled matrix, and each element block's index."""
    mesh = _mesh(case)
    nn = mesh.num_nodes
    c = mesh.cells.astype(np.int64)
    keys = (c[:, :, None] * nn + c[:, None, :]).ravel()
    diag = np.arange(nn, dtype=np.int64) * (nn + 1)
    return np.unique(np.concatenate([keys, diag])), keys


def _assemble_exact(case, seed):
    mesh = _mesh(case)
    rho, mu, K = _elastic(mesh, seed)
    uniq, keys = _pattern(case)
    tab = _gpu_tables(mesh)
    coords, cells, mu, K, x, uniq, keys = _cuda(mesh.coords, mesh.cells, mu, K, _field(mesh.num_dof, seed).reshape(-1, 3), uniq, keys)
    pos = torch.searchsorted(uniq, keys).reshape(mesh.num_cells, -1)
    val = torch.zeros((len(uniq), 3, 3), dtype=torch.float64, device="cuda")
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    for sl in _chunks(mesh, 8192):
        cn, wdet, grad = _geometry(mesh, sl, coords, cells, tab)
        lam = (K - 2 * mu / 3)[sl]
        H = torch.einsum("cq,cqaf,cqbg->cabfg", wdet, grad, grad)
        tr = H.diagonal(dim1=-2, dim2=-1).sum(-1)
        Ke = -(lam[:, None, None, None, None] * H + mu[sl][:, None, None, None, None] * (tr[..., None, None] * eye + H.transpose(-1, -2)))
        val.index_add_(0, pos[sl].reshape(-1), Ke.reshape(-1, 3, 3))
    y = torch.zeros_like(x)
    y.index_add_(0, uniq // mesh.num_nodes, torch.einsum("kfg,kg->kf", val, x[uniq % mesh.num_nodes]))
    return [val, y.reshape(-1)]


def _output_exact(mesh, u, mu, K):
    tab = _gpu_tables(mesh, centre=True)
    coords, cells, un, mu, K = _cuda(mesh.coords, mesh.cells, u.reshape(-1, 3), mu, K)
    out = []
    at = [0, 4, 8, 1, 5, 2]
    for sl in _chunks(mesh, 65536):
        cn, wdet, grad = _geometry(mesh, sl, coords, cells, tab)
        G = torch.einsum("cni,cnd->cid", un[cn], grad[:, 0])
        e = 0.5 * (G + G.transpose(-1, -2))
        s = _stress((K - 2 * mu / 3)[sl], mu[sl], e)
        out.append(torch.cat([s.reshape(-1, 9)[:, at], e.reshape(-1, 9)[:, at]], dim=1))
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("static", "greens"):
        return None  # a 3-D sparse system of this size takes minutes with plain torch
    if kind == "visco":
        return _visco_exact(_mesh(case, fault=True), seed)
    if kind == "assemble":
        return _assemble_exact(case, seed)
    mesh = _mesh(case)
    rho, mu, K = _elastic(mesh, seed)
    u = _field(mesh.num_dof, seed)
    if kind == "output":
        return _output_exact(mesh, u, mu, K)
    out = {}
    for op in case["ops"].split(","):
        v = u.astype(np.float32).astype(np.float64) if op == "action32" else u
        out[op] = _apply_exact(mesh, v, mu, K, _body_force(rho) if case["body_force"] and op == "residual" else None)
    return out
