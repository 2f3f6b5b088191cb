"""P1 tetrahedra on every layout their kernels have, with several blocks per CTA: pairs of cells with few
(cells along a Morton curve) and with many nodes per block (in grid order), and single cells (shuffled
within windows of 1,000: too scattered for pairs; throughout, they exceed the single cells' limits too).
Residual, actions, deterministic mode, batched operator, reduced fault space and the cached tangent."""
import os
import subprocess
import sys

import numpy as np
import pytest

from pylith_b200 import materials as MAT
from pylith_b200 import meshing as M

pytestmark = pytest.mark.gpu

TOL64 = 1e-12
ORDERS = ["morton", "grid", "shuffled"]


def _shuffled(num_cells):
    rng = np.random.default_rng(81)
    return np.concatenate([i + rng.permutation(min(1000, num_cells - i)) for i in range(0, num_cells, 1000)])


@pytest.fixture(scope="module")
def ctx():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pylith_b200 import feassemble as FA

    return FA.Context(0)


def _mesh(order, n, **kw):
    mesh = M.box_tet_kuhn(*n, reorder=order != "grid", **kw)
    if order == "shuffled":
        mesh.cells = np.ascontiguousarray(mesh.cells[_shuffled(mesh.num_cells)])
    return mesh


def _rel(a, b):
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("order", ORDERS)
def test_many_blocks_per_cta(ctx, order):
    """752,640 cells: more than 5 blocks of pairs (or of single cells) for every resident CTA of the FP64
    kernels, 3.5 of the FP32 ones, and not a whole number of them. Against the thread-per-cell kernels
    (FP64 1e-12, FP32 1e-5); the deterministic mode twice, bit for bit."""
    import torch
    from pylith_b200 import feassemble as FA

    mesh = _mesh(order, (56, 56, 40))
    rho, mu, K = MAT.lognormal_elastic(mesh.num_cells, seed=82)
    body = np.random.default_rng(83).standard_normal((mesh.num_cells, 3)) * 1e4
    ig = MAT.IsotropicLinearElasticity(rho, mu, K, body).create_integrator(FA.DeviceMesh(ctx, mesh))
    u = torch.from_numpy(np.random.default_rng(84).standard_normal(mesh.num_dof)).cuda()
    calls = [lambda o, m: ig.compute_lhs_residual(0.0, 0.0, u, o, mode=m),
             lambda o, m: ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, u, o, mode=m)]
    refs = [torch.zeros_like(u), torch.zeros_like(u)]
    ig.set_scatter(FA.SCATTER_ATOMIC)
    for call, ref in zip(calls, refs):
        call(ref, FA.ADD)
    for scatter in (FA.SCATTER_AUTO, FA.SCATTER_DETERMINISTIC):
        ig.set_scatter(scatter)
        for call, ref in zip(calls, refs):
            runs = [torch.full_like(u, np.nan) for _ in range(2)]
            for r in runs:
                call(r, FA.INSERT)
            ctx.synchronize()
            assert _rel(runs[0], ref) <= TOL64
            if scatter == FA.SCATTER_DETERMINISTIC:
                assert torch.equal(runs[0], runs[1])
            call(runs[1], FA.ADD)
            ctx.synchronize()
            assert _rel(runs[1], 2 * ref) <= TOL64
    out = torch.full_like(u.float(), np.nan)
    ig.compute_lhs_jacobian_action_f32(0.0, 0.0, u.float(), out)
    ctx.synchronize()
    assert _rel(out.double(), refs[1]) <= 1e-5


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("tile", [4, 8])
def test_batched_operator_with_many_blocks(ctx, order, tile):
    """Batched solves on 151,200 cells (more than two blocks of pairs for every CTA of a chunk of right-hand
    sides) match FP64 solves of one right-hand side at a time to <= 1e-8."""
    import torch
    from pylith_b200 import feassemble as FA

    mesh = _mesh(order, (30, 30, 28))
    cons = np.zeros((mesh.num_nodes, 3), dtype=bool)
    for side in ("neg", "pos"):
        cons[M.boundary_mask(mesh, 0, side)] = True
    dm = FA.DeviceMesh(ctx, mesh)
    ig = MAT.IsotropicLinearElasticity(*MAT.lognormal_elastic(mesh.num_cells, seed=85)).create_integrator(dm)
    rng = np.random.default_rng(86)
    bs = [torch.from_numpy(rng.standard_normal(mesh.num_dof)).cuda() for _ in range(tile)]
    refined = FA.Solver(dm, cons.ravel(), [ig], rtol=1e-11, precision=FA.Solver.FP32_REFINED, inner_rtol=1e-4)
    refined.setup()
    xs = [torch.zeros_like(b) for b in bs]
    FA.BatchSolver(refined, tile).solve(bs, xs)
    S = FA.Solver(dm, cons.ravel(), [ig], rtol=1e-11)
    S.setup()
    for b, x in list(zip(bs, xs))[::3]:
        ref = torch.zeros_like(b)
        S.solve(b, ref)
        ctx.synchronize()
        assert _rel(x, ref) <= 1e-8


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_reduced_fault_space_in_two_orders(ctx, precision):
    """A fault's slip problem on the same mesh along a Morton curve and in grid order: the displacements
    agree to 1e-8. (Solvers with faults refuse cells too scattered for pairs, see test_selectable_kernels
    for the single cells.)"""
    from pylith_b200 import feassemble as FA
    from pylith_b200 import problems as P

    base = M.box_tet_kuhn(12, 11, 10, fault_x=0.0, reorder=False)
    rho, mu, K = MAT.lognormal_elastic(base.num_cells, seed=87)
    cons = np.zeros((base.num_nodes, 3), dtype=bool)
    for side in ("neg", "pos"):
        cons[M.boundary_mask(base, 0, side)] = True
    cons = np.concatenate([cons.ravel(), np.zeros(3 * base.num_lagrange, dtype=bool)])
    slip = np.zeros((base.num_lagrange, 3))
    slip[: base.num_lagrange // 2, 1] = 2.0
    cells = base.cells.copy()
    got = []
    morton = np.argsort(M._morton_keys(base.coords[cells].mean(axis=1)), kind="stable")
    for order in ("morton", "grid"):
        # (the nodes keep their numbers, so that the fields compare entry by entry)
        at = {"grid": np.arange(len(cells)), "morton": morton}[order]
        base.cells = np.ascontiguousarray(cells[at])
        mat = MAT.IsotropicLinearElasticity(rho[at], mu[at], K[at])
        prob = P.QuasistaticProblem(ctx, base, [(mat, None)], cons, np.zeros(base.num_dof),
                                    faults=[MAT.FaultCohesiveKin(slip)], rtol=1e-11,
                                    precision=FA.Solver.FP64 if precision == "fp64" else FA.Solver.FP32_REFINED)
        prob.step(0.0)
        got.append(prob.u.clone())
        prob.close()
    assert _rel(got[0], got[1]) <= 1e-8


@pytest.mark.parametrize("rheology", ["elastic", "genmaxwell"])
@pytest.mark.parametrize("order", ["grid", "shuffled"])
def test_cached_tangent_on_every_layout(ctx, rheology, order):
    """The FP32 action with the per-cell tangent that a solver's setup caches, against the FP64 action."""
    import torch
    from pylith_b200 import feassemble as FA

    mesh = _mesh(order, (20, 20, 18))
    nc = mesh.num_cells
    rho, mu, K = MAT.lognormal_elastic(nc, seed=89)
    if rheology == "genmaxwell":
        tau = MAT.genmaxwell_times(rho, np.sqrt(mu / rho), [1e18, 1e19, 1e20], [0.3, 0.3, 0.3])
        mat = MAT.IsotropicLinearGenMaxwell(rho, mu, K, tau, np.full((nc, 3), 0.3), np.zeros((nc, 1, 18)), np.zeros((nc, 1, 6)))
    else:
        mat = MAT.IsotropicLinearElasticity(rho, mu, K)
    dm = FA.DeviceMesh(ctx, mesh)
    ig = mat.create_integrator(dm, MAT.YEAR) if rheology == "genmaxwell" else mat.create_integrator(dm)
    cons = np.zeros((mesh.num_nodes, 3), dtype=bool)
    cons[M.boundary_mask(mesh, 2, "neg")] = True
    S = FA.Solver(dm, cons.ravel(), [ig], precision=FA.Solver.FP32_REFINED)
    S.setup(0.0, MAT.YEAR)
    v = torch.from_numpy(np.random.default_rng(90).standard_normal(dm.num_dof)).cuda().float()
    out, ref = torch.full_like(v, np.nan), torch.empty_like(v.double())
    ig.compute_lhs_jacobian_action_f32(0.0, MAT.YEAR, v, out)
    ig.compute_lhs_jacobian_action(0.0, MAT.YEAR, 0.0, None, v.double(), ref)
    ctx.synchronize()
    assert _rel(out.double(), ref) <= 1e-5
    S.close()


@pytest.mark.parametrize("kernel", ["pair", "pad2", "pipe", "twophase"])
def test_selectable_kernels(ctx, kernel):
    """Each kernel that PYLITH_B200_TET_KERNEL names (read once per process) on 384,000 cells: residual,
    action and FP32 action, INSERT and ADD, against the thread-per-cell kernels; and a solve in the reduced
    fault space (not two-phase, which has none) against the one that unfolds and folds."""
    code = """
import numpy as np, torch
from pylith_b200 import feassemble as FA, materials as MAT, meshing as M
mesh = M.box_tet_kuhn(40, 40, 40)
ctx = FA.Context(0)
rho, mu, K = MAT.lognormal_elastic(mesh.num_cells, seed=91)
body = np.random.default_rng(92).standard_normal((mesh.num_cells, 3)) * 1e4
ig = MAT.IsotropicLinearElasticity(rho, mu, K, body).create_integrator(FA.DeviceMesh(ctx, mesh))
u = torch.from_numpy(np.random.default_rng(93).standard_normal(mesh.num_dof)).cuda()
calls = [lambda o, m: ig.compute_lhs_residual(0.0, 0.0, u, o, mode=m),
         lambda o, m: ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, u, o, mode=m),
         lambda o, m: ig.compute_lhs_jacobian_action_f32(0.0, 0.0, u.float(), o, mode=m)]
for i, call in enumerate(calls):
    ref = torch.zeros_like(u)
    ig.set_scatter(FA.SCATTER_ATOMIC)
    calls[min(i, 1)](ref, FA.ADD)
    ig.set_scatter(FA.SCATTER_AUTO)
    out = torch.full_like(u.float() if i == 2 else u, np.nan)
    call(out, FA.INSERT)
    torch.cuda.synchronize()
    tol = 1e-5 if i == 2 else 1e-12
    assert float((out.double() - ref).norm() / ref.norm()) <= tol, i
    call(out, FA.ADD)
    torch.cuda.synchronize()
    assert float((out.double() - 2 * ref).norm() / (2 * ref).norm()) <= tol, i
import os
from pylith_b200 import problems as P
if os.environ["PYLITH_B200_TET_KERNEL"] != "twophase":
    mesh = M.box_tet_kuhn(12, 11, 10, fault_x=0.0)
    cons = np.zeros((mesh.num_nodes, 3), dtype=bool)
    for side in ("neg", "pos"):
        cons[M.boundary_mask(mesh, 0, side)] = True
    cons = np.concatenate([cons.ravel(), np.zeros(3 * mesh.num_lagrange, dtype=bool)])
    slip = np.zeros((mesh.num_lagrange, 3))
    slip[: mesh.num_lagrange // 2, 1] = 2.0
    for precision in (FA.Solver.FP64, FA.Solver.FP32_REFINED):
        got = []
        for flag in ("1", "0"):
            os.environ["PYLITH_B200_REDUCED_KERNELS"] = flag
            mat = MAT.IsotropicLinearElasticity(*MAT.lognormal_elastic(mesh.num_cells, seed=94))
            prob = P.QuasistaticProblem(ctx, mesh, [(mat, None)], cons, np.zeros(mesh.num_dof),
                                        faults=[MAT.FaultCohesiveKin(slip)], rtol=1e-11, precision=precision)
            prob.step(0.0)
            got.append(prob.u.clone())
            prob.close()
        assert float((got[0] - got[1]).norm() / got[1].norm()) <= 1e-8, precision
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=root,
                       env=dict(os.environ, PYLITH_B200_TET_KERNEL=kernel))
    assert r.returncode == 0, r.stderr[-2000:]
