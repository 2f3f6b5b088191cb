"""GPU parity: the CUDA cell loop (called through the C ABI) against the oracle on the same
seeded meshes, fields and parameters. FP64 tolerance: relative L2 <= 1e-12 (the FP64
parity bar); FP32 Jacobian action: relative L2 <= 1e-5."""
import numpy as np
import pytest

import known_answers as KA
from pylith_b200 import materials as MAT
from pylith_b200 import meshing as M

pytestmark = pytest.mark.gpu

F1_ILE = "IsotropicLinearElasticity3D::f1v_infinitesimalStrain"
JF3_ILE = "IsotropicLinearElasticity3D::Jf3vu_infinitesimalStrain"
F1_GM = "IsotropicLinearGenMaxwell3D::f1v_infinitesimalStrain"
JF3_GM = "IsotropicLinearGenMaxwell3D::Jf3vu_infinitesimalStrain"
TOL64 = 1e-12


def rel_l2(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300)


@pytest.fixture(scope="module")
def torch_cuda():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.fixture(scope="module")
def ctx(torch_cuda):
    from pylith_b200 import feassemble as FA

    return FA.Context(0)


def dev(torch, a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a))
    if dtype is not None:
        t = t.to(dtype)
    return t.cuda()


MESHES = {
    "tet4": lambda: M.box_tet_delaunay(6000, seed=5),
    "hex8": lambda: M.box_hex(6, 5, 4),
    "hex27": lambda: M.box_hex27(3, 3, 2),
    "tet4_unsorted": lambda: M.box_tet_delaunay(3000, seed=9, reorder=False),
}


def elastic_setup(mesh, seed=0, body_force=False):
    rho, mu, K = MAT.lognormal_elastic(mesh.num_cells, seed=seed)
    bf = np.random.default_rng(seed + 1).standard_normal((mesh.num_cells, 3)) * 1e3 if body_force else None
    return MAT.IsotropicLinearElasticity(rho, mu, K, bf)


def oracle_aux(O, mat):
    fields = [(mat.density[:, None], "cell")]
    if mat.body_force is not None:
        fields.append((mat.body_force, "cell"))
    fields += [(mat.shear_modulus[:, None], "cell"), (mat.bulk_modulus[:, None], "cell")]
    return O.AuxFields(fields)


@pytest.mark.parametrize("kind", list(MESHES))
@pytest.mark.parametrize("scatter", [0, 1, 3])
def test_elastic_residual_matches_oracle(oracle_lib, torch_cuda, ctx, kind, scatter):
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = MESHES[kind]()
    mat = elastic_setup(mesh)
    u = np.random.default_rng(2).standard_normal(mesh.num_nodes * 3)
    r_ref = O.residual(mesh, u, oracle_aux(O, mat), f1=F1_ILE)
    dm = FA.DeviceMesh(ctx, mesh)
    ig = mat.create_integrator(dm)
    ig.set_scatter(scatter)
    du = dev(torch, u)
    dr = torch.full_like(du, np.nan)
    ig.compute_lhs_residual(0.0, 0.0, du, dr)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    # ADD mode accumulates on top of the existing values
    ig.compute_lhs_residual(0.0, 0.0, du, dr, mode=FA.ADD)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), 2 * r_ref) <= TOL64


@pytest.mark.parametrize("kind", ["tet4", "hex8", "hex27"])
def test_body_force_residual(oracle_lib, torch_cuda, ctx, kind):
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = MESHES[kind]()
    mat = elastic_setup(mesh, body_force=True)
    u = np.random.default_rng(3).standard_normal(mesh.num_nodes * 3) * 1e-3
    r_ref = O.residual(mesh, u, oracle_aux(O, mat), f0="Elasticity::g0v_bodyforce", f1=F1_ILE)
    dm = FA.DeviceMesh(ctx, mesh)
    ig = mat.create_integrator(dm)
    du = dev(torch, u)
    dr = torch.zeros_like(du)
    ig.compute_lhs_residual(0.0, 0.0, du, dr)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64


@pytest.mark.parametrize("kind", ["tet4", "hex8", "hex27"])
def test_jacobian_action_and_assembly_match_oracle(oracle_lib, torch_cuda, ctx, kind):
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = MESHES[kind]()
    mat = elastic_setup(mesh, seed=4)
    aux = oracle_aux(O, mat)
    J = O.assemble(mesh, O.jacobian_elements(mesh, aux, g3=JF3_ILE))
    v = np.random.default_rng(5).standard_normal(mesh.num_nodes * 3)
    jv_ref = J @ v
    dm = FA.DeviceMesh(ctx, mesh)
    ig = mat.create_integrator(dm)
    dv = dev(torch, v)
    djv = torch.zeros_like(dv)
    ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, dv, djv)
    ctx.synchronize()
    assert rel_l2(djv.cpu().numpy(), jv_ref) <= TOL64
    # FP32 action (FP32 operands and accumulation, FP64 geometry)
    dv32 = dv.float()
    djv32 = torch.zeros_like(dv32)
    ig.compute_lhs_jacobian_action_f32(0.0, 0.0, dv32, djv32)
    ctx.synchronize()
    assert rel_l2(djv32.double().cpu().numpy(), jv_ref) <= 1e-5
    # assembled block-CSR Jacobian
    A = FA.Matrix(dm)
    ig.compute_lhs_jacobian(0.0, 0.0, 0.0, None, A)
    Jg = A.to_scipy().tocsr()
    assert abs(Jg - J).max() <= TOL64 * abs(J).max()
    dy = torch.zeros_like(dv)
    A.spmv(dv, dy)
    ctx.synchronize()
    assert rel_l2(dy.cpu().numpy(), jv_ref) <= TOL64


def genmaxwell_setup(mesh, seed=0):
    rng = np.random.default_rng(seed)
    nc = mesh.num_cells
    nq = M.QUAD_POINTS[mesh.cell_type]
    rho, mu, K = MAT.lognormal_elastic(nc, seed=seed)
    tau = MAT.genmaxwell_times(rho, np.sqrt(mu / rho), [1e18, 1e19, 1e20], [0.3, 0.3, 0.3])
    ratio = np.tile([0.3, 0.3, 0.3], (nc, 1))
    visc = rng.standard_normal((nc, nq, 18)) * 1e-5
    total = rng.standard_normal((nc, nq, 6)) * 1e-5
    return MAT.IsotropicLinearGenMaxwell(rho, mu, K, tau, ratio, visc, total)


def genmaxwell_oracle_aux(O, g):
    return O.AuxFields([(g.density[:, None], "cell"), (g.shear_modulus[:, None], "cell"),
                        (g.bulk_modulus[:, None], "cell"), (g.maxwell_time, "cell"),
                        (g.shear_modulus_ratio, "cell"), (g.viscous_strain, "qp"), (g.total_strain, "qp")])


@pytest.mark.parametrize("kind", ["hex8", "tet4", "hex27"])
def test_genmaxwell_residual_jacobian_and_state_update(oracle_lib, torch_cuda, ctx, kind):
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = MESHES[kind]()
    g = genmaxwell_setup(mesh)
    dt = 1.0 * MAT.YEAR
    aux = genmaxwell_oracle_aux(O, g)
    u = np.random.default_rng(7).standard_normal(mesh.num_nodes * 3) * 1e-2
    r_ref = O.residual(mesh, u, aux, f1=F1_GM, constants=[dt])
    J = O.assemble(mesh, O.jacobian_elements(mesh, aux, g3=JF3_GM, constants=[dt]))
    v = np.random.default_rng(8).standard_normal(mesh.num_nodes * 3)
    visc_ref, total_ref = O.project_qp(
        mesh, u, aux, ["IsotropicLinearGenMaxwell3D::viscousStrain_infinitesimalStrain_asVector",
                       "Elasticity3D::infinitesimalStrain_asVector"], [18, 6], constants=[dt])
    dm = FA.DeviceMesh(ctx, mesh)
    ig = g.create_integrator(dm, dt)
    du, dv = dev(torch, u), dev(torch, v)
    dr, djv = torch.zeros_like(du), torch.zeros_like(du)
    ig.compute_lhs_residual(0.0, dt, du, dr)
    ig.compute_lhs_jacobian_action(0.0, dt, 0.0, du, dv, djv)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    assert rel_l2(djv.cpu().numpy(), J @ v) <= TOL64
    ig.update_state_vars(0.0, dt, du)
    ctx.synchronize()
    nq = M.QUAD_POINTS[mesh.cell_type]
    visc = ig.get_aux("viscous_strain", (mesh.num_cells, nq, 18))
    total = ig.get_aux("total_strain", (mesh.num_cells, nq, 6))
    assert rel_l2(visc, visc_ref) <= TOL64
    assert rel_l2(total, total_ref) <= TOL64


def test_genmaxwell_relaxation_known_answer_on_gpu(torch_cuda, ctx):
    """The analytic relaxation of axialstrain_genmaxwell_soln.py, stepped on the GPU."""
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    mesh = M.box_hex(2, 2, 2, lo=(-4000.0, -4000.0, -8000.0), hi=(4000.0, 4000.0, 0.0))
    mu, K, lam, tau = KA.genmaxwell_params()
    nc, nq, e0 = mesh.num_cells, 8, KA.GM_E0
    g = MAT.IsotropicLinearGenMaxwell(
        np.full(nc, KA.GM_DENSITY), np.full(nc, mu), np.full(nc, K), np.tile(tau, (nc, 1)),
        np.tile(KA.GM_RATIO, (nc, 1)), np.tile([-e0 / 3, -e0 / 3, 2 * e0 / 3, 0, 0, 0] * 3, (nc, nq, 1)),
        np.tile([0, 0, e0, 0, 0, 0.0], (nc, nq, 1)))
    dm = FA.DeviceMesh(ctx, mesh)
    ig = g.create_integrator(dm, KA.GM_DT)
    X = mesh.coords
    u = np.stack([0 * X[:, 0], 0 * X[:, 1], e0 * (X[:, 2] + 8000.0)], axis=1).ravel()
    du = dev(torch, u)
    dr = torch.zeros_like(du)
    for step in range(1, KA.GM_STEPS + 1):
        ig.compute_lhs_residual(step * KA.GM_DT, KA.GM_DT, du, dr)
        ig.update_state_vars(step * KA.GM_DT, KA.GM_DT, du)
        ctx.synchronize()
        sigma = KA.stress_from_residual(X, dr.cpu().numpy(), 8000.0**3)
        np.testing.assert_allclose(np.diag(sigma), KA.genmaxwell_stress(step * KA.GM_DT), rtol=1e-10)


def fault_setup(nx=4, ny=3, nz=3):
    mesh = M.insert_fault_x(M.box_hex(nx, ny, nz))
    rng = np.random.default_rng(11)
    slip = rng.standard_normal((mesh.num_lagrange, 3))
    fault = MAT.FaultCohesiveKin(slip, ref_dir_1=(0, 0, 1), ref_dir_2=(0.5, 0, 0.5))
    return mesh, fault


def test_cohesive_residual_jacobian_action_and_assembly(oracle_lib, torch_cuda, ctx):
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh, fault = fault_setup()
    u = np.random.default_rng(12).standard_normal(mesh.num_dof)
    r_ref = O.cohesive_residual(mesh, u, fault.slip, fault.constants)
    Jc = O.cohesive_jacobian(mesh, fault.constants)
    v = np.random.default_rng(13).standard_normal(mesh.num_dof)
    dm = FA.DeviceMesh(ctx, mesh)
    ig = fault.create_integrator(dm)
    du, dv = dev(torch, u), dev(torch, v)
    dr, djv = torch.zeros_like(du), torch.zeros_like(du)
    ig.compute_lhs_residual(0.0, 0.0, du, dr)
    ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, du, dv, djv)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    assert rel_l2(djv.cpu().numpy(), Jc @ v) <= TOL64
    A = FA.Matrix(dm)
    ig.compute_lhs_jacobian(0.0, 0.0, 0.0, None, A)
    Jg = A.to_scipy().tocsr()
    assert abs(Jg - Jc).max() <= 1e-12 * abs(Jc).max()


def test_full_fault_problem_residual(oracle_lib, torch_cuda, ctx):
    """Domain + interface integrators summed into one local vector (TimeDependent's loop over
    integrators, TimeDependent.cc:659-662)."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh, fault = fault_setup(6, 4, 3)
    mat = elastic_setup(mesh, seed=21)
    u = np.random.default_rng(14).standard_normal(mesh.num_dof)
    r_ref = np.zeros(mesh.num_dof)
    r_ref[:3 * mesh.num_nodes] = O.residual(mesh, u[:3 * mesh.num_nodes], oracle_aux(O, mat), f1=F1_ILE)
    O.cohesive_residual(mesh, u, fault.slip, fault.constants, r=r_ref)
    dm = FA.DeviceMesh(ctx, mesh)
    igs = [mat.create_integrator(dm), fault.create_integrator(dm)]
    du = dev(torch, u)
    dr = torch.zeros_like(du)
    for i, ig in enumerate(igs):
        ig.compute_lhs_residual(0.0, 0.0, du, dr, mode=FA.INSERT if i == 0 else FA.ADD)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64


def test_host_buffer_entry_point(oracle_lib, torch_cuda, ctx):
    from pylith_b200 import feassemble as FA

    O = oracle_lib
    mesh = MESHES["tet4"]()
    mat = elastic_setup(mesh)
    u = np.random.default_rng(2).standard_normal(mesh.num_nodes * 3)
    r_ref = O.residual(mesh, u, oracle_aux(O, mat), f1=F1_ILE)
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    r = np.zeros_like(u)
    ig.compute_lhs_residual_host(0.0, 0.0, u, r)
    assert rel_l2(r, r_ref) <= TOL64
    # the same call with both host buffers from pl_host_alloc
    hu, hr = ctx.host_empty(u.shape), ctx.host_empty(u.shape)
    hu[:] = u
    ig.compute_lhs_residual_host(0.0, 0.0, hu, hr)
    assert rel_l2(hr, r_ref) <= TOL64


def _page_nodes(ptr: int, nbytes: int):
    """NUMA node of every 64th page of [ptr, ptr + nbytes) (move_pages query; x86-64 / arm64)."""
    import ctypes
    import platform

    nr = {"x86_64": 279, "aarch64": 239}.get(platform.machine())
    if nr is None:
        return None
    libc = ctypes.CDLL(None, use_errno=True)
    addrs = list(range(ptr, ptr + nbytes, 64 * 4096))
    pages = (ctypes.c_void_p * len(addrs))(*addrs)
    status = (ctypes.c_int * len(addrs))()
    if libc.syscall(nr, 0, ctypes.c_ulong(len(addrs)), pages, None, status, 0) != 0:
        return None
    return list(status)


def test_numa_local_host_buffers(torch_cuda, ctx):
    """pl_host_alloc: aligned, zero-filled, page-locked (CUDA sees it as pinned host memory) and,
    where the host reports the GPU's NUMA node and lets the process use that node's memory,
    placed there; a round trip through the device returns the same bytes."""
    torch = torch_cuda
    n = 3 << 20
    a = ctx.host_empty((2, n))
    assert a.shape == (2, n) and a.dtype == np.float64
    assert a.ctypes.data % 256 == 0
    assert not a.any()
    t = torch.from_numpy(a)
    assert t.is_pinned()
    a[0] = np.arange(n, dtype=np.float64)
    a[1] = -a[0]
    d = t.to("cuda", non_blocking=True)
    back = ctx.host_empty((2, n))
    torch.from_numpy(back).copy_(d * 2.0, non_blocking=True)
    torch.cuda.synchronize()
    assert np.array_equal(back, 2.0 * a)
    node = ctx.numa_node
    allowed = ""
    with open("/proc/self/status") as f:
        for ln in f:
            if ln.startswith("Mems_allowed_list:"):
                allowed = ln.split(":", 1)[1].strip()
    mems = set()
    for part in filter(None, allowed.split(",")):
        lo, _, hi = part.partition("-")
        mems |= set(range(int(lo), int(hi or lo) + 1))
    nodes = _page_nodes(a.ctypes.data, a.nbytes)
    if node >= 0 and node in mems and len(mems) > 1 and nodes is not None:
        assert sum(x == node for x in nodes) >= 0.9 * len(nodes), (node, nodes[:16])


def test_unknown_kernel_is_rejected(torch_cuda, ctx):
    from pylith_b200 import _lib
    from pylith_b200 import feassemble as FA
    import oracle as O

    mesh = MESHES["hex8"]()
    ig = FA.IntegratorDomain(FA.DeviceMesh(ctx, mesh))
    # the oracle's restated kernel has the right signature but is not a registered kernel
    foreign = O.kernel(F1_ILE, "oracle")
    with pytest.raises(_lib.PylithB200Error) as e:
        ig.set_kernels_residual([FA.ResidualKernels("displacement", FA.LHS, None, foreign)])
    assert e.value.code == -2
    with pytest.raises(_lib.PylithB200Error) as e:
        ig.compute_lhs_residual(0.0, 0.0, None, None)
    assert e.value.code == -1


def test_more_than_eight_constants_are_rejected(torch_cuda, ctx):
    """Integrator::_setKernelConstants takes any number of constants; the library holds at most 8
    (the kernels on the path use 1 or 6) and rejects more with PL_ERR_UNSUPPORTED instead of
    dropping the extra ones; the previous constants stay in place."""
    from pylith_b200 import _lib
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    mesh = MESHES["hex8"]()
    mat = elastic_setup(mesh)
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    ig.set_constants([1.0] * 8)
    with pytest.raises(_lib.PylithB200Error) as e:
        ig.set_constants([1.0] * 9)
    assert e.value.code == -7
    du = torch.zeros(mesh.num_dof, dtype=torch.float64, device="cuda")
    ig.compute_lhs_residual(0.0, 0.0, du, torch.empty_like(du))
    ctx.synchronize()


def test_inverted_cell_is_reported(torch_cuda, ctx):
    from pylith_b200 import _lib
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    mesh = M.box_hex(2, 2, 2)
    mesh.cells[0] = mesh.cells[0][[1, 0, 3, 2, 5, 4, 7, 6]]  # mirror cell 0 -> negative |J|
    mat = elastic_setup(mesh)
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    du = torch.zeros(mesh.num_nodes * 3, dtype=torch.float64, device="cuda")
    dr = torch.zeros_like(du)
    ig.compute_lhs_residual(0.0, 0.0, du, dr)
    with pytest.raises(_lib.PylithB200Error) as e:
        ctx.synchronize()
    assert e.value.code == -6
    ctx.synchronize()  # the flag is cleared after it is reported


def test_destroy_in_any_order(torch_cuda):
    """Context, mesh and integrator handles may be released in any order (the C layer defers a
    destroy until no dependent object is left)."""
    from pylith_b200 import feassemble as FA

    c = FA.Context(0)
    mesh = M.box_hex(2, 2, 2)
    dm = FA.DeviceMesh(c, mesh)
    ig = elastic_setup(mesh).create_integrator(dm)
    A = FA.Matrix(dm)
    c.close()
    dm.close()
    du = torch_cuda.zeros(mesh.num_nodes * 3, dtype=torch_cuda.float64, device="cuda")
    ig.compute_lhs_residual(0.0, 0.0, du, du.clone())
    A.close()
    ig.close()


@pytest.mark.parametrize("kind", ["tet4", "hex8", "hex27"])
def test_derived_fields_match_oracle(oracle_lib, torch_cuda, ctx, kind, tmp_path):
    """pl_compute_derived_field (cauchy_stress, cauchy_strain of basis order 0 at the cell
    centroids, IntegratorDomain.cc:596-630) against the oracle's centroid projection; the fields
    and the solution written through DataWriterHDF5 read back unchanged."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = MESHES[kind]()
    mat = elastic_setup(mesh, seed=31)
    u = np.random.default_rng(32).standard_normal(mesh.num_dof)
    ref_s, ref_e = O.project_centroid(
        mesh, u, oracle_aux(O, mat),
        ["IsotropicLinearElasticity3D::cauchyStress_infinitesimalStrain_asVector",
         "Elasticity3D::infinitesimalStrain_asVector"], [6, 6])
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    out = torch.zeros((mesh.num_cells, 12), dtype=torch.float64, device="cuda")
    ig.compute_derived_field(0.0, 0.0, dev(torch, u), out)
    ctx.synchronize()
    got = out.cpu().numpy()
    assert rel_l2(got[:, :6], ref_s) <= TOL64
    assert rel_l2(got[:, 6:], ref_e) <= TOL64
    from pylith_b200 import hdf5 as H5
    from pylith_b200 import output as OUT

    w = OUT.DataWriterHDF5(filename=str(tmp_path / "out.h5"))
    w.open(mesh)
    w.write_vertex_field(1.0, "displacement", u[:3 * mesh.num_nodes].reshape(-1, 3))
    w.write_cell_field(1.0, "cauchy_stress", got[:, :6])
    w.write_cell_field(1.0, "cauchy_strain", got[:, 6:])
    w.close()
    f = H5.H5File(str(tmp_path / "out.h5"))
    assert np.array_equal(f.dataset("/vertex_fields/displacement")[0], u[:3 * mesh.num_nodes].reshape(-1, 3))
    assert np.array_equal(f.dataset("/cell_fields/cauchy_stress")[0], got[:, :6])
    assert np.array_equal(f.dataset("/cell_fields/cauchy_strain")[0], got[:, 6:])
    assert f.attrs("/cell_fields/cauchy_stress")["vector_field_type"] == "tensor"


def test_derived_genmaxwell_stress(oracle_lib, torch_cuda, ctx):
    """Generalized-Maxwell stress from the stored state (cauchyStress_stateVars) on P1 tets,
    whose single quadrature point is the centroid; hexahedra are rejected (-7)."""
    from pylith_b200 import _lib
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = MESHES["tet4"]()
    g = genmaxwell_setup(mesh, seed=33)
    dt = 0.1 * MAT.YEAR
    u = np.random.default_rng(34).standard_normal(mesh.num_dof) * 1e-2
    ref_s, ref_e = O.project_centroid(
        mesh, u, genmaxwell_oracle_aux(O, g),
        ["IsotropicLinearGenMaxwell3D::cauchyStress_infinitesimalStrain_asVector",
         "Elasticity3D::infinitesimalStrain_asVector"], [6, 6], constants=[dt])
    ig = g.create_integrator(FA.DeviceMesh(ctx, mesh), dt)
    out = torch.zeros((mesh.num_cells, 12), dtype=torch.float64, device="cuda")
    ig.compute_derived_field(0.0, dt, dev(torch, u), out)
    ctx.synchronize()
    got = out.cpu().numpy()
    assert rel_l2(got[:, :6], ref_s) <= TOL64
    assert rel_l2(got[:, 6:], ref_e) <= TOL64
    hexm = MESHES["hex8"]()
    ih = genmaxwell_setup(hexm, seed=35).create_integrator(FA.DeviceMesh(ctx, hexm), dt)
    with pytest.raises(_lib.PylithB200Error) as e:
        ih.compute_derived_field(0.0, dt, dev(torch, np.zeros(hexm.num_dof)),
                                 torch.zeros((hexm.num_cells, 12), dtype=torch.float64, device="cuda"))
    assert e.value.code == -7


@pytest.mark.parametrize("kind", ["tet4", "hex8", "hex27"])
def test_two_materials_on_cell_subsets(oracle_lib, torch_cuda, ctx, kind):
    """Two materials on complementary cell subsets (one IntegratorDomain per material label,
    IntegratorDomain.cc:422-453) summed into one residual and one Jacobian action; an integrator
    over an empty subset contributes nothing."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = MESHES[kind]()
    rng = np.random.default_rng(41)
    ids = [np.flatnonzero(mesh.coords[mesh.cells].mean(axis=1)[:, 0] < 0.0),
           np.flatnonzero(mesh.coords[mesh.cells].mean(axis=1)[:, 0] >= 0.0)]
    mats = [elastic_setup(M.Mesh(mesh.cell_type, mesh.coords, mesh.cells[i]), seed=42 + k) for k, i in enumerate(ids)]
    u = rng.standard_normal(mesh.num_dof)
    v = rng.standard_normal(mesh.num_dof)
    r_ref = np.zeros(mesh.num_dof)
    jv_ref = np.zeros(mesh.num_dof)
    for i, mat in zip(ids, mats):
        sub = M.Mesh(mesh.cell_type, mesh.coords, mesh.cells[i])
        aux = oracle_aux(O, mat)
        r_ref += O.residual(sub, u, aux, f1=F1_ILE)
        J = O.assemble(sub, O.jacobian_elements(sub, aux, g3=JF3_ILE))
        jv_ref += J @ v
    dm = FA.DeviceMesh(ctx, mesh)
    igs = [mat.create_integrator(dm, i) for i, mat in zip(ids, mats)]
    empty = elastic_setup(M.Mesh(mesh.cell_type, mesh.coords, mesh.cells[:0]), seed=9).create_integrator(
        dm, np.zeros(0, dtype=np.int32))
    du, dv = dev(torch, u), dev(torch, v)
    dr = torch.full_like(du, 7.0)
    djv = torch.full_like(du, 7.0)
    for k, ig in enumerate(igs + [empty]):
        mode = FA.INSERT if k == 0 else FA.ADD
        ig.compute_lhs_residual(0.0, 0.0, du, dr, mode=mode)
        ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, du, dv, djv, mode=mode)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    assert rel_l2(djv.cpu().numpy(), jv_ref) <= TOL64
    # the empty integrator alone in INSERT mode writes zeros
    empty.compute_lhs_residual(0.0, 0.0, du, dr, mode=FA.INSERT)
    ctx.synchronize()
    assert float(dr.abs().max()) == 0.0


def test_reference_compiled_kernels_drive_the_device_path(oracle_lib, torch_cuda, ctx):
    """The reference's own pointwise kernels compiled from libsrc/pylith/fekernels/*.hh
    (oracle/_ref) are registered under their names (pl_fekernel_register) and passed to the
    integrator exactly as PyLith passes them to PetscWeakForm: the device path runs with them and
    gives what it gives with the library's own addresses, for a material and a fault."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    if not O.ref_available():
        pytest.skip("reference kernels not built")
    for name in O.KERNELS:
        FA.register_fekernel(name, O.kernel(name, "ref"))
        assert FA.fekernel_name(O.kernel(name, "ref")) == name
    ref = lambda n: O.kernel(n, "ref")  # noqa: E731
    mesh = MESHES["tet4"]()
    mat = elastic_setup(mesh, seed=51)
    dm = FA.DeviceMesh(ctx, mesh)
    ig_lib = mat.create_integrator(dm)
    ig_ref = FA.IntegratorDomain(dm)
    for name, vals in (("density", mat.density), ("shear_modulus", mat.shear_modulus),
                       ("bulk_modulus", mat.bulk_modulus)):
        ig_ref.set_aux(name, FA.PER_CELL, vals[:, None])
    ig_ref.set_kernels_residual([FA.ResidualKernels("displacement", FA.LHS, None, ref(F1_ILE))])
    ig_ref.set_kernels_jacobian([FA.JacobianKernels("displacement", "displacement", FA.LHS, None, None, None,
                                                    ref(JF3_ILE))])
    u = dev(torch, np.random.default_rng(52).standard_normal(mesh.num_dof))
    outs = []
    for ig in (ig_lib, ig_ref):
        r, jv = torch.empty_like(u), torch.empty_like(u)
        ig.set_scatter(FA.SCATTER_DETERMINISTIC)
        ig.compute_lhs_residual(0.0, 0.0, u, r)
        ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, u, jv)
        outs.append((r, jv))
    ctx.synchronize()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    # a fault with the reference's FaultCohesiveKin kernels
    fmesh, fault = fault_setup()
    fdm = FA.DeviceMesh(ctx, fmesh)
    if_lib = fault.create_integrator(fdm)
    if_ref = FA.IntegratorInterface(fdm)
    if_ref.set_aux("slip", FA.PER_FAULT_NODE, fault.slip)
    if_ref.set_constants(fault.constants)
    if_ref.set_kernels_residual([
        FA.InterfaceResidualKernels("displacement", FA.LHS, FA.FACE_NEGATIVE, ref("FaultCohesiveKin::f0u_neg"), None),
        FA.InterfaceResidualKernels("displacement", FA.LHS, FA.FACE_POSITIVE, ref("FaultCohesiveKin::f0u_pos"), None),
        FA.InterfaceResidualKernels("lagrange_multiplier_fault", FA.LHS, FA.FACE_FAULT,
                                    ref("FaultCohesiveKin::f0l_slip"), None)])
    fu = dev(torch, np.random.default_rng(53).standard_normal(fmesh.num_dof))
    fr = [torch.zeros_like(fu), torch.zeros_like(fu)]
    if_lib.compute_lhs_residual(0.0, 0.0, fu, fr[0])
    if_ref.compute_lhs_residual(0.0, 0.0, fu, fr[1])
    ctx.synchronize()
    assert torch.equal(fr[0], fr[1])


def _hex_variant(mesh, order):
    """The box with jittered nodes, its cells in the given order: 'x' (as built: consecutive cells
    share a face), 'morton', or 'shuffled' (neighbouring lanes share nothing or single nodes)."""
    rng = np.random.default_rng(8)
    h = (mesh.coords.max(axis=0) - mesh.coords.min(axis=0)) / 16
    mesh.coords += rng.uniform(-0.05, 0.05, mesh.coords.shape) * np.minimum(h, 300.0)  # (Q2: corners count)
    if order == "morton":
        return M.reorder_for_locality(mesh)
    if order == "shuffled":
        mesh.cells = np.ascontiguousarray(mesh.cells[rng.permutation(mesh.num_cells)])
    return mesh


# Q1: one cell; less than, exactly and one more than a warp; a 64-cell block and a partial one; the
# first size with 64-cell blocks (more than 148 * 64 cells). Q2: one cell; one less than, exactly and
# one more than a warp's ten cells; two warps and three.
HEX_SIZES = [("hex8", n) for n in [(1, 1, 1), (31, 1, 1), (8, 4, 1), (33, 1, 1), (13, 5, 1), (7, 5, 3), (24, 21, 19)]]
HEX_SIZES += [("hex27", n) for n in [(1, 1, 1), (9, 1, 1), (10, 1, 1), (11, 1, 1), (5, 2, 2), (7, 3, 2)]]


@pytest.mark.parametrize("kind,n", HEX_SIZES)
@pytest.mark.parametrize("order", ["x", "morton", "shuffled"])
def test_hex_cell_kernel_sizes(oracle_lib, torch_cuda, ctx, kind, n, order):
    """The hexahedral kernels against the oracle at warp and block edges, for cell orders with and
    without faces shared by consecutive cells: residual with body force, action, FP32 action, cell
    subsets."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = _hex_variant(M.box_hex(*n) if kind == "hex8" else M.box_hex27(*n), order)
    mat = elastic_setup(mesh, seed=6, body_force=True)
    aux = oracle_aux(O, mat)
    u = np.random.default_rng(7).standard_normal(mesh.num_nodes * 3)
    plain = O.AuxFields([(a[:, None], "cell") for a in (mat.density, mat.shear_modulus, mat.bulk_modulus)])
    r_ref = O.residual(mesh, u, aux, f0="Elasticity::g0v_bodyforce", f1=F1_ILE)
    jv_ref = O.jacobian_action(mesh, u, plain, g3=JF3_ILE)
    dm = FA.DeviceMesh(ctx, mesh)
    ig = mat.create_integrator(dm)
    du = dev(torch, u)
    dr, djv, d32 = torch.full_like(du, np.nan), torch.full_like(du, np.nan), torch.full_like(du.float(), np.nan)
    ig.compute_lhs_residual(0.0, 0.0, du, dr)
    ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, du, djv)
    ig.compute_lhs_jacobian_action_f32(0.0, 0.0, du.float(), d32)
    # every second cell as an integrator of its own, then the others on top
    dsum = torch.zeros_like(du)
    for ids in [np.arange(s, mesh.num_cells, 2, dtype=np.int32) for s in (0, 1)]:
        part = MAT.IsotropicLinearElasticity(mat.density[ids], mat.shear_modulus[ids], mat.bulk_modulus[ids])
        part.create_integrator(dm, ids).compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, du, dsum, mode=FA.ADD)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    assert rel_l2(djv.cpu().numpy(), jv_ref) <= TOL64
    assert rel_l2(dsum.cpu().numpy(), jv_ref) <= TOL64
    assert rel_l2(d32.double().cpu().numpy(), jv_ref) <= 1e-5


# cells that do not fill a warp's 4 hexahedra or 8 tetrahedra, and rows of 1 to 125 blocks
ASSEMBLY = {
    "hex8_1": lambda: M.box_hex(1, 1, 1),
    "hex8_5": lambda: M.box_hex(5, 1, 1),
    "hex8_54": lambda: M.box_hex(3, 6, 3),
    "hex27_1": lambda: M.box_hex27(1, 1, 1),
    "hex27_12": lambda: M.box_hex27(2, 3, 2),
    "tet_6": lambda: M.box_tet_kuhn(1, 1, 1),
    "tet_510": lambda: M.box_tet_kuhn(5, 17, 1),
}


@pytest.mark.parametrize("kind", list(ASSEMBLY))
@pytest.mark.parametrize("genmaxwell", [False, True])
def test_assembly_and_product_sizes(oracle_lib, torch_cuda, ctx, kind, genmaxwell):
    """The assembled Jacobian of two integrators on complementary cell subsets added into one
    matrix, and its product with a vector, against the oracle's element matrices."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = ASSEMBLY[kind]()
    nc, nq = mesh.num_cells, M.QUAD_POINTS[mesh.cell_type]
    rho, mu, K = MAT.lognormal_elastic(nc, seed=12)
    ids = [np.arange(0, nc, 3, dtype=np.int32), np.array([c for c in range(nc) if c % 3], dtype=np.int32)]
    dm = FA.DeviceMesh(ctx, mesh)
    A = FA.Matrix(dm)
    if genmaxwell:
        tau = MAT.genmaxwell_times(rho, np.sqrt(mu / rho), [1e18, 1e19, 1e20], [0.3, 0.2, 0.1])
        ratio = np.tile([0.3, 0.2, 0.1], (nc, 1))
        state = [np.zeros((nc, nq, 18)), np.zeros((nc, nq, 6))]
        aux = O.AuxFields([(a, "cell") for a in (rho[:, None], mu[:, None], K[:, None], tau, ratio)] + [(a, "qp") for a in state])
        J = O.assemble(mesh, O.jacobian_elements(mesh, aux, g3=JF3_GM, constants=[MAT.YEAR]))
        for i in ids:
            MAT.IsotropicLinearGenMaxwell(rho[i], mu[i], K[i], tau[i], ratio[i], state[0][i], state[1][i]).create_integrator(
                dm, MAT.YEAR, i).compute_lhs_jacobian(0.0, MAT.YEAR, 0.0, None, A)
    else:
        aux = O.AuxFields([(a[:, None], "cell") for a in (rho, mu, K)])
        J = O.assemble(mesh, O.jacobian_elements(mesh, aux, g3=JF3_ILE))
        for i in ids:
            MAT.IsotropicLinearElasticity(rho[i], mu[i], K[i]).create_integrator(dm, i).compute_lhs_jacobian(0.0, 0.0, 0.0, None, A)
    ctx.synchronize()
    assert abs(A.to_scipy().tocsr() - J).max() <= TOL64 * abs(J).max()
    x = np.random.default_rng(13).standard_normal(3 * mesh.num_nodes)
    dx = dev(torch, x)
    dy = torch.full_like(dx, np.nan)
    A.spmv(dx, dy)
    ctx.synchronize()
    assert rel_l2(dy.cpu().numpy(), J @ x) <= TOL64


# one cell; one more than a warp; one more than a block; the first size with 64-cell blocks, whose
# state copies take more than the default shared memory
@pytest.mark.parametrize("n", [(1, 1, 1), (11, 3, 1), (13, 5, 1), (24, 21, 19)])
@pytest.mark.parametrize("subset", [False, True])
def test_genmaxwell_hex8_sizes(oracle_lib, torch_cuda, ctx, n, subset):
    """Generalized-Maxwell residual and state update of Q1 hexahedra at warp and block edges, for
    all cells in one integrator and in two on complementary subsets."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = M.box_hex(*n)
    nc = mesh.num_cells
    g = genmaxwell_setup(mesh, seed=14)
    aux = genmaxwell_oracle_aux(O, g)
    u = np.random.default_rng(15).standard_normal(mesh.num_nodes * 3) * 1e-2
    r_ref = O.residual(mesh, u, aux, f1=F1_GM, constants=[MAT.YEAR])
    visc_ref, total_ref = O.project_qp(
        mesh, u, aux, ["IsotropicLinearGenMaxwell3D::viscousStrain_infinitesimalStrain_asVector",
                       "Elasticity3D::infinitesimalStrain_asVector"], [18, 6], constants=[MAT.YEAR])
    dm = FA.DeviceMesh(ctx, mesh)
    du = dev(torch, u)
    dr = torch.full_like(du, np.nan)
    sets = [np.arange(0, nc, 2, dtype=np.int32), np.arange(1, nc, 2, dtype=np.int32)] if subset else [None]
    visc, total = np.zeros((nc, 8, 18)), np.zeros((nc, 8, 6))
    for k, ids in enumerate(sets):
        at = slice(None) if ids is None else ids
        if ids is not None and len(ids) == 0:
            continue
        ig = MAT.IsotropicLinearGenMaxwell(
            g.density[at], g.shear_modulus[at], g.bulk_modulus[at], g.maxwell_time[at], g.shear_modulus_ratio[at],
            g.viscous_strain[at], g.total_strain[at]).create_integrator(dm, MAT.YEAR, ids)
        ig.compute_lhs_residual(0.0, MAT.YEAR, du, dr, mode=FA.ADD if k else FA.INSERT)
        ig.update_state_vars(0.0, MAT.YEAR, du)
        ctx.synchronize()
        m = nc if ids is None else len(ids)
        visc[at] = ig.get_aux("viscous_strain", (m, 8, 18))
        total[at] = ig.get_aux("total_strain", (m, 8, 6))
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    assert rel_l2(visc, visc_ref) <= TOL64
    assert rel_l2(total, total_ref) <= TOL64


@pytest.mark.parametrize("ny,nz", [(1, 1), (7, 1), (8, 1), (3, 3), (17, 1)])
def test_cohesive_kernel_sizes(oracle_lib, torch_cuda, ctx, ny, nz):
    """Cohesive residual and actions for cell counts that do and do not fill a warp's eight cells."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh, fault = fault_setup(2, ny, nz)
    u = np.random.default_rng(16).standard_normal(mesh.num_dof)
    r_ref = O.cohesive_residual(mesh, u, fault.slip, fault.constants)
    jv_ref = O.cohesive_jacobian(mesh, fault.constants) @ u
    ig = fault.create_integrator(FA.DeviceMesh(ctx, mesh))
    du = dev(torch, u)
    dr, djv, d32 = torch.full_like(du, np.nan), torch.full_like(du, np.nan), torch.full_like(du.float(), np.nan)
    ig.compute_lhs_residual(0.0, 0.0, du, dr)
    ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, du, du, djv)
    ig.compute_lhs_jacobian_action_f32(0.0, 0.0, du.float(), d32)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    assert rel_l2(djv.cpu().numpy(), jv_ref) <= TOL64
    assert rel_l2(d32.double().cpu().numpy(), jv_ref) <= 1e-5


# one cell; one pair; one more than an item's two; one less than, exactly and one more than a block of
# pairs; several blocks; mixed within windows (more nodes per block than consecutive cells have); mixed
# throughout (the layout of single cells)
@pytest.mark.parametrize("nc,window", [(1, 0), (2, 0), (3, 0), (239, 0), (240, 0), (241, 0), (1296, 0), (1296, 432), (1296, 1296)])
def test_tet_pair_kernel_sizes(oracle_lib, torch_cuda, ctx, nc, window):
    """The tetrahedral kernels on pairs of cells at item and block edges and for mixed cell orders:
    residual with body force (INSERT and ADD), action, FP32 action and the deterministic mode; nodes
    outside the first nc cells belong to no cell."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    rng = np.random.default_rng(17)
    mesh = M.box_tet_kuhn(6, 6, 6)
    mesh.cells = mesh.cells[:nc].copy()
    for i in range(0, nc if window else 0, window or 1):
        rng.shuffle(mesh.cells[i:i + window])
    mat = elastic_setup(mesh, seed=18, body_force=True)
    aux = oracle_aux(O, mat)
    plain = O.AuxFields([(a[:, None], "cell") for a in (mat.density, mat.shear_modulus, mat.bulk_modulus)])
    u = rng.standard_normal(mesh.num_nodes * 3)
    r_ref = O.residual(mesh, u, aux, f0="Elasticity::g0v_bodyforce", f1=F1_ILE)
    jv_ref = O.jacobian_action(mesh, u, plain, g3=JF3_ILE)
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    du = dev(torch, u)
    dr, djv, d32 = torch.full_like(du, np.nan), torch.full_like(du, np.nan), torch.full_like(du.float(), np.nan)
    ig.compute_lhs_residual(0.0, 0.0, du, dr)
    ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, du, djv)
    ig.compute_lhs_jacobian_action_f32(0.0, 0.0, du.float(), d32)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), r_ref) <= TOL64
    assert rel_l2(djv.cpu().numpy(), jv_ref) <= TOL64
    assert rel_l2(d32.double().cpu().numpy(), jv_ref) <= 1e-5
    ig.compute_lhs_residual(0.0, 0.0, du, dr, mode=FA.ADD)
    ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, du, djv, mode=FA.ADD)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), 2 * r_ref) <= TOL64
    assert rel_l2(djv.cpu().numpy(), 2 * jv_ref) <= TOL64
    ig.set_scatter(FA.SCATTER_DETERMINISTIC)
    runs = []
    for _ in range(2):
        dr.fill_(np.nan)
        ig.compute_lhs_residual(0.0, 0.0, du, dr)
        ctx.synchronize()
        runs.append(dr.cpu().numpy())
    assert np.array_equal(runs[0], runs[1])
    assert rel_l2(runs[0], r_ref) <= TOL64
    ig.compute_lhs_residual(0.0, 0.0, du, dr, mode=FA.ADD)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), 2 * r_ref) <= TOL64


# the smallest output, one block of the zeroing kernel and several; small and large cell grids
@pytest.mark.parametrize("kind,n", [("tet4", (1, 1, 1)), ("tet4", (9, 8, 7)), ("hex8", (1, 1, 1)), ("hex8", (13, 11, 9)),
                                    ("hex27", (1, 1, 1)), ("hex27", (7, 5, 3))])
def test_insert_zeroes_stale_output(oracle_lib, torch_cuda, kind, n):
    """INSERT over stale outputs, issued back to back and replayed from a CUDA graph: the cell kernels
    start while the zeros are being written and read the output only after them; each application
    reads the one before it (v = J u, w = J v)."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = {"tet4": M.box_tet_kuhn, "hex8": M.box_hex, "hex27": M.box_hex27}[kind](*n)
    mat = elastic_setup(mesh, seed=31)
    aux = oracle_aux(O, mat)
    u = np.random.default_rng(32).standard_normal(mesh.num_nodes * 3)
    v_ref = O.jacobian_action(mesh, u, aux, g3=JF3_ILE)
    w_ref = O.jacobian_action(mesh, v_ref, aux, g3=JF3_ILE)
    ctx = FA.Context(0)
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    du = dev(torch, u)
    u32 = du.float()
    v, w, r, v32 = (torch.empty_like(x) for x in (du, du, du, u32))

    def spoil():
        for x in (v, w, r, v32):
            x.fill_(np.nan)

    def apply():
        ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, du, v)
        ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, v, w)
        ig.compute_lhs_residual(0.0, 0.0, v, r)
        ig.compute_lhs_jacobian_action_f32(0.0, 0.0, u32, v32)

    def check():
        torch.cuda.synchronize()
        assert rel_l2(v.cpu().numpy(), v_ref) <= TOL64
        assert rel_l2(w.cpu().numpy(), w_ref) <= TOL64
        assert rel_l2(r.cpu().numpy(), w_ref) <= TOL64  # linear elasticity: F(v) = J v
        assert rel_l2(v32.double().cpu().numpy(), v_ref) <= 1e-5

    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        spoil()
        for _ in range(3):
            apply()
        check()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            apply()
        for _ in range(2):
            spoil()
            graph.replay()
            check()
    del graph


# one to four kernels (6 to 24 values per cell) on one cell, one less than, exactly and one more than a
# warp's and a block's cells, and several blocks
@pytest.mark.parametrize("num", [1, 2, 3, 4])
@pytest.mark.parametrize("nc", [1, 31, 32, 33, 127, 128, 129, 1000])
def test_derived_rows(oracle_lib, torch_cuda, ctx, nc, num):
    """The rows of pl_compute_derived_field for every number of kernels and at warp and block edges;
    nothing is written past the last row."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = M.box_hex(10, 10, 10)
    mesh.cells = mesh.cells[:nc].copy()
    mat = elastic_setup(mesh, seed=41)
    stress = "IsotropicLinearElasticity3D::cauchyStress_infinitesimalStrain_asVector"
    strain = "Elasticity3D::infinitesimalStrain_asVector"
    names = [stress, strain, strain, stress][:num]
    k = FA.fekernels
    fn = {stress: k.IsotropicLinearElasticity3D.cauchyStress_infinitesimalStrain_asVector,
          strain: k.Elasticity3D.infinitesimalStrain_asVector}
    u = np.random.default_rng(42).standard_normal(mesh.num_dof)
    ref = np.concatenate(O.project_centroid(mesh, u, oracle_aux(O, mat), names, [6] * num), axis=1)
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    ig.set_kernels_derived_field([FA.ProjectKernels(f"field_{i}", fn[n]) for i, n in enumerate(names)])
    out = torch.full((nc + 1, 6 * num), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ig.compute_derived_field(0.0, 0.0, dev(torch, u), out)
    ctx.synchronize()
    got = out.cpu().numpy()
    assert np.isnan(got[nc]).all()
    for i in range(num):
        assert rel_l2(got[:nc, 6 * i:6 * i + 6], ref[:, 6 * i:6 * i + 6]) <= TOL64


def test_fp32_action_allocates_nothing_once_the_layout_is_there():
    """The FP32 action of integrators in the deterministic mode, whose FP64 partial sums it does not
    use: after the first call has built the mesh's layout, free device memory stays as it is. (A
    process of its own, whose memory pool holds nothing to hand out again; 6 integrators would take
    17 MB each.)"""
    import os
    import subprocess
    import sys

    code = """
import torch
from pylith_b200 import feassemble as FA, materials as MAT, meshing as M
mesh = M.box_tet_kuhn(64, 64, 48)
ctx = FA.Context(0)
dm = FA.DeviceMesh(ctx, mesh)
mat = MAT.IsotropicLinearElasticity(*MAT.lognormal_elastic(mesh.num_cells, seed=1))
igs = [mat.create_integrator(dm) for _ in range(6)]
v = torch.ones(mesh.num_dof, dtype=torch.float32, device="cuda")
out = torch.empty_like(v)
igs[0].compute_lhs_jacobian_action_f32(0.0, 0.0, v, out)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
for ig in igs:
    ig.set_scatter(FA.SCATTER_DETERMINISTIC)
    ig.compute_lhs_jacobian_action_f32(0.0, 0.0, v, out)
torch.cuda.synchronize()
print("taken", free - torch.cuda.mem_get_info()[0])
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=root)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) == 0, r.stdout


@pytest.mark.parametrize("kind", ["tet4", "hex8", "hex27"])
@pytest.mark.parametrize("scale", [1e-13, 1e-7, 1.0, 1e7])
def test_fp32_action_over_length_scales(torch_cuda, ctx, kind, scale):
    """The FP32 action on boxes from nanometres to astronomic sizes with moduli in Pa: it agrees with the
    FP64 action to 1e-5 as at the usual size (no factor of a cell leaves FP32's range)."""
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    mesh = {"tet4": M.box_tet_kuhn, "hex8": M.box_hex, "hex27": M.box_hex27}[kind](4, 4, 3)
    mesh.coords *= scale
    ig = elastic_setup(mesh, seed=51).create_integrator(FA.DeviceMesh(ctx, mesh))
    v = torch.from_numpy(np.random.default_rng(52).standard_normal(mesh.num_dof)).cuda().float()
    d64, d32 = torch.empty_like(v.double()), torch.empty_like(v)
    ig.compute_lhs_jacobian_action(0.0, 0.0, 0.0, None, v.double(), d64)
    ig.compute_lhs_jacobian_action_f32(0.0, 0.0, v, d32)
    ctx.synchronize()
    assert rel_l2(d32.double().cpu().numpy(), d64.cpu().numpy()) <= 1e-5


# calls whose kernel is launched behind the zeroing, not under it, and outputs of a few values
ONE_LAUNCH = {
    "tet4_atomic": (lambda: M.box_tet_kuhn(6, 5, 4), "atomic", "rjf"),
    "tet4_subset": (lambda: M.box_tet_kuhn(6, 5, 4), "subset", "rjf"),
    "tet4_genmaxwell": (lambda: M.box_tet_kuhn(6, 5, 4), "genmaxwell", "rjf"),
    "tet4_scattered": (lambda: M.box_tet_kuhn(9, 9, 9, reorder=False), "scattered", "f"),
    "hex8_atomic": (lambda: M.box_hex(6, 5, 4), "atomic", "rjf"),
    "hex8_genmaxwell": (lambda: M.box_hex(6, 5, 4), "genmaxwell", "r"),
    "hex8_few": (lambda: M.box_hex(2, 2, 2), "", "rjf"),
    "hex27": (lambda: M.box_hex27(3, 3, 3), "", "f"),
    "tet4_few": (lambda: M.box_tet_kuhn(1, 1, 1), "", "rjf"),
}


@pytest.mark.parametrize("case", list(ONE_LAUNCH))
def test_insert_takes_one_launch_where_nothing_starts_early(torch_cuda, ctx, case):
    """INSERT zeroes by a memset wherever no kernel starts under the zeroing (one launch per call), and
    gives what ADD into zeros gives."""
    from pylith_b200 import _lib
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    make, form, calls = ONE_LAUNCH[case]
    mesh = make()
    if form == "scattered":
        np.random.default_rng(60).shuffle(mesh.cells)
    dm = FA.DeviceMesh(ctx, mesh)
    if form == "genmaxwell":
        ig = genmaxwell_setup(mesh, seed=61).create_integrator(dm, MAT.YEAR)
    elif form == "subset":
        ids = np.arange(0, mesh.num_cells, 2, dtype=np.int32)
        mat = elastic_setup(mesh, seed=61)
        ig = MAT.IsotropicLinearElasticity(mat.density[ids], mat.shear_modulus[ids], mat.bulk_modulus[ids]).create_integrator(dm, ids)
    else:
        ig = elastic_setup(mesh, seed=61).create_integrator(dm)
    if form == "atomic":
        ig.set_scatter(FA.SCATTER_ATOMIC)
    u = torch.from_numpy(np.random.default_rng(62).standard_normal(mesh.num_dof)).cuda()
    run = {"r": lambda o, m: ig.compute_lhs_residual(0.0, MAT.YEAR, u, o, mode=m),
           "j": lambda o, m: ig.compute_lhs_jacobian_action(0.0, MAT.YEAR, 0.0, None, u, o, mode=m),
           "f": lambda o, m: ig.compute_lhs_jacobian_action_f32(0.0, MAT.YEAR, u.float(), o, mode=m)}
    for c in calls:
        ref = torch.zeros_like(u.float() if c == "f" else u)
        out = torch.full_like(ref, np.nan)
        run[c](ref, FA.ADD)  # (builds the layout)
        ctx.synchronize()
        n0 = _lib.lib().pl_kernel_launches()
        run[c](out, FA.INSERT)
        ctx.synchronize()
        assert _lib.lib().pl_kernel_launches() - n0 == 1, c
        assert rel_l2(out.double().cpu().numpy(), ref.double().cpu().numpy()) <= (1e-6 if c == "f" else TOL64)


# Q2: the last size by lines and the first by planes of each rheology and call (26, 36 and 44 cells per
# multiprocessor), a part of a line warp's three cells, and one cell more than a block's six
@pytest.mark.parametrize("genmaxwell", [False, True])
@pytest.mark.parametrize("per_sm,extra", [(0, 2), (0, 7), (26, 0), (26, 1), (36, 0), (36, 1), (44, 0), (44, 1)])
def test_q2_kernels_on_both_sides_of_their_rules(torch_cuda, ctx, genmaxwell, per_sm, extra):
    """Residual (body force; INSERT and ADD) and action of Q2 hexahedra where the kernel changes, against
    the thread-per-cell kernels."""
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    nc = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    n = max(2, int(np.ceil(nc ** (1 / 3))))
    mesh = M.box_hex27(n, n, n)
    mesh.cells = mesh.cells[:nc].copy()
    rng = np.random.default_rng(71)
    dm = FA.DeviceMesh(ctx, mesh)
    if genmaxwell:
        ig = genmaxwell_setup(mesh, seed=72).create_integrator(dm, MAT.YEAR)
    else:
        ig = elastic_setup(mesh, seed=72, body_force=True).create_integrator(dm)
    u = torch.from_numpy(rng.standard_normal(mesh.num_dof)).cuda()
    calls = [lambda o, m: ig.compute_lhs_residual(0.0, MAT.YEAR, u, o, mode=m),
             lambda o, m: ig.compute_lhs_jacobian_action(0.0, MAT.YEAR, 0.0, None, u, o, mode=m)]
    refs = []
    ig.set_scatter(FA.SCATTER_ATOMIC)
    for call in calls:
        refs.append(torch.zeros_like(u))
        call(refs[-1], FA.ADD)
    ig.set_scatter(FA.SCATTER_AUTO)
    for call, ref in zip(calls, refs):
        out = torch.full_like(u, np.nan)
        call(out, FA.INSERT)
        ctx.synchronize()
        assert rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= TOL64
        call(out, FA.ADD)
        ctx.synchronize()
        assert rel_l2(out.cpu().numpy(), 2 * ref.cpu().numpy()) <= TOL64


# a part of a warp's four cells and of a block's 32; the last size with a lane per point and the next
@pytest.mark.parametrize("per_sm,extra", [(0, 3), (0, 33), (32, 0), (32, 1)])
@pytest.mark.parametrize("body_force", [False, True])
def test_genmaxwell_hex8_residual_on_both_sides_of_its_rule(oracle_lib, torch_cuda, ctx, per_sm, extra, body_force):
    """The generalized-Maxwell residual of Q1 hexahedra (INSERT and ADD, with and without a body force)
    where the kernel changes, against the oracle."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    nc = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    n = max(2, int(np.ceil(nc ** (1 / 3))))
    mesh = M.box_hex(n, n, n)
    mesh.cells = mesh.cells[:nc].copy()
    g = genmaxwell_setup(mesh, seed=73)
    aux = genmaxwell_oracle_aux(O, g)
    u = np.random.default_rng(74).standard_normal(mesh.num_dof) * 1e-2
    ig = g.create_integrator(FA.DeviceMesh(ctx, mesh), MAT.YEAR)
    ref = O.residual(mesh, u, aux, f1=F1_GM, constants=[MAT.YEAR])
    if body_force:
        b = np.random.default_rng(75).standard_normal((nc, 3)) * 1e3
        ig.set_aux("body_force", FA.PER_CELL, b)
        k = FA.fekernels
        ig.set_kernels_residual([FA.ResidualKernels("displacement", FA.LHS, k.Elasticity.g0v_bodyforce,
                                                    k.IsotropicLinearGenMaxwell3D.f1v_infinitesimalStrain)])
        plain = elastic_setup(mesh, seed=73)
        with_b = O.AuxFields([(plain.density[:, None], "cell"), (b, "cell"), (plain.shear_modulus[:, None], "cell"),
                              (plain.bulk_modulus[:, None], "cell")])
        ref = ref + O.residual(mesh, 0 * u, with_b, f0="Elasticity::g0v_bodyforce", f1=F1_ILE)
    du = dev(torch, u)
    dr = torch.full_like(du, np.nan)
    ig.compute_lhs_residual(0.0, MAT.YEAR, du, dr)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), ref) <= TOL64
    ig.compute_lhs_residual(0.0, MAT.YEAR, du, dr, mode=FA.ADD)
    ctx.synchronize()
    assert rel_l2(dr.cpu().numpy(), 2 * ref) <= TOL64


# the last size whose state fits 128 MB and the first that does not
@pytest.mark.parametrize("nc", [87381, 87382])
def test_genmaxwell_hex8_state_update_on_both_sides_of_its_rule(oracle_lib, torch_cuda, ctx, nc):
    """The state update of Q1 hexahedra where the kernel changes, against the oracle."""
    from pylith_b200 import feassemble as FA

    O, torch = oracle_lib, torch_cuda
    mesh = M.box_hex(45, 45, 44)
    mesh.cells = mesh.cells[:nc].copy()
    g = genmaxwell_setup(mesh, seed=76)
    u = np.random.default_rng(77).standard_normal(mesh.num_dof) * 1e-2
    visc, total = O.project_qp(
        mesh, u, genmaxwell_oracle_aux(O, g), ["IsotropicLinearGenMaxwell3D::viscousStrain_infinitesimalStrain_asVector",
                                               "Elasticity3D::infinitesimalStrain_asVector"], [18, 6], constants=[MAT.YEAR])
    ig = g.create_integrator(FA.DeviceMesh(ctx, mesh), MAT.YEAR)
    ig.update_state_vars(0.0, MAT.YEAR, dev(torch, u))
    ctx.synchronize()
    assert rel_l2(ig.get_aux("viscous_strain", (nc, 8, 18)), visc) <= TOL64
    assert rel_l2(ig.get_aux("total_strain", (nc, 8, 6)), total) <= TOL64


# Q2: one cell, a warp and a block and one more of each; the last size without staged rows and the next
@pytest.mark.parametrize("per_sm,extra", [(0, 1), (0, 33), (0, 129), (128, 0), (128, 1)])
@pytest.mark.parametrize("num", [2, 4])
def test_derived_rows_of_q2(torch_cuda, ctx, per_sm, extra, num):
    """Derived fields of Q2 hexahedra where the kernel changes, for a displacement of constant gradient:
    every cell's strain is that gradient's, its stress follows, and nothing is written past the last row."""
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    nc = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    n = max(2, int(np.ceil(nc ** (1 / 3))))
    mesh = M.box_hex27(n, n, n)
    mesh.cells = mesh.cells[:nc].copy()
    mat = elastic_setup(mesh, seed=95)
    G = np.random.default_rng(96).standard_normal((3, 3)) * 1e-3
    e = 0.5 * (G + G.T)
    strain = np.tile(e[[0, 1, 2, 0, 1, 0], [0, 1, 2, 1, 2, 2]], (nc, 1))
    lam = mat.bulk_modulus - 2.0 / 3.0 * mat.shear_modulus
    stress = 2.0 * mat.shear_modulus[:, None] * strain
    stress[:, :3] += (lam * np.trace(e))[:, None]
    k = FA.fekernels
    f_stress = k.IsotropicLinearElasticity3D.cauchyStress_infinitesimalStrain_asVector
    f_strain = k.Elasticity3D.infinitesimalStrain_asVector
    ig = mat.create_integrator(FA.DeviceMesh(ctx, mesh))
    ig.set_kernels_derived_field([FA.ProjectKernels(f"field_{i}", f_strain if i % 2 else f_stress) for i in range(num)])
    out = torch.full((nc + 1, 6 * num), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ig.compute_derived_field(0.0, 0.0, dev(torch, (mesh.coords @ G.T).ravel()), out)
    ctx.synchronize()
    got = out.cpu().numpy()
    assert np.isnan(got[nc]).all()
    # (differences of displacements of up to 20 m over cells of 400 m and more, u and x rounded: 1e-11)
    for i in range(num):
        assert rel_l2(got[:nc, 6 * i:6 * i + 6], strain if i % 2 else stress) <= 1e-10


@pytest.mark.parametrize("kind,n", [("hex8", (7, 6, 5)), ("hex8", (46, 45, 43)), ("hex27", (4, 3, 3)), ("hex27", (19, 17, 13))])
@pytest.mark.parametrize("genmaxwell", [False, True])
def test_hexahedra_far_from_the_origin(torch_cuda, ctx, kind, n, genmaxwell):
    """The hexahedral kernels on a box 2^26 m from the origin and, Q1, displaced by 2^20 m as a whole:
    residual, action and Q1 state update agree with those of the box at the origin to 1e-12. (Cells of 256 m
    and displacements of whole multiples of 2^-20: all differences are exact in both, so only the kernels'
    own rounding is left; sums of absolute coordinates would lose 2^26 / 256 times 1e-16, of displacements
    2^20 times.)"""
    from pylith_b200 import feassemble as FA

    torch = torch_cuda
    got = []
    for far in (False, True):
        mesh = (M.box_hex if kind == "hex8" else M.box_hex27)(*n, (0.0, 0.0, 0.0), tuple(256.0 * k for k in n))
        u = np.round(np.random.default_rng(97).standard_normal((mesh.num_nodes, 3)) * 2.0**20) / 2.0**20
        if far:
            mesh.coords += np.array([2.0**26, -2.0**25, 2.0**24])
            u += np.array([2.0**20, -2.0**19, 2.0**18]) * (kind == "hex8")
        mat = genmaxwell_setup(mesh, seed=98) if genmaxwell else elastic_setup(mesh, seed=98)
        dm = FA.DeviceMesh(ctx, mesh)
        ig = mat.create_integrator(dm, MAT.YEAR) if genmaxwell else mat.create_integrator(dm)
        du = dev(torch, u.ravel())
        r, jv = torch.empty_like(du), torch.empty_like(du)
        ig.compute_lhs_residual(0.0, MAT.YEAR, du, r)
        ig.compute_lhs_jacobian_action(0.0, MAT.YEAR, 0.0, None, du, jv)
        fields = [r.cpu().numpy(), jv.cpu().numpy()]
        if genmaxwell and kind == "hex8":
            ig.update_state_vars(0.0, MAT.YEAR, du)
            ctx.synchronize()
            fields += [ig.get_aux("viscous_strain", (mesh.num_cells, 8, 18)), ig.get_aux("total_strain", (mesh.num_cells, 8, 6))]
        got.append(fields)
    for a, b in zip(*got):
        assert rel_l2(b, a) <= TOL64
