"""Solves of field-dependent operators in every form of their apply: the merged streams in
the coloured launches (the form of production sizes, here by lane_cells 0 and on a
stream beyond the operator's workspaces) as in two launches, with the velocity as a
constant and as a DoF vector.  The residual under the oracle's operator is the solver's
tolerance with 5 % for its own rounding; the forms return the same bits.  And the
constraint kernels of mapped meshes above the size where copy and interpolation are
one launch."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, rng
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LAW = dict(rho=(3925.0, 7850.0, 7000.0), cp=(230.0, 460.0, 700.0), k=(27.8, 55.6, 17.0), solidus=1900.0, liquidus=2000.0)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("perturb", [0.0, 0.1])
@pytest.mark.parametrize("case", ["law", "law nodal", "full", "kT"])
@pytest.mark.parametrize("mixed", [False, True])
def test_solves_in_every_form_of_the_apply(cuda, p, perturb, case, mixed):
    import torch
    import meltpooldg_b200 as M
    nc = (5, 4, 3)
    mask = M.boundary_mask(nc, p, faces=[(2, 0)])
    gm, om = meshes(nc, p, perturb, seed=5, mask=mask)
    x = om.dof_coordinates()
    N = gm.n_dofs
    T = 1950.0 + 60.0 * np.sin(3.0 * x[:, 0]) + rng(1).uniform(-1, 1, N)
    T_old, H = T - 1.0, 0.5 + 0.4 * np.sin(4.0 * x[:, 1])
    U = np.stack([0.3 + 0.1 * x[:, 1], -0.2 * np.cos(x[:, 0]), 0.1 + x[:, 2]])
    prec = ("fp64", "fp32") if mixed else ("fp64",)
    vel, ov = (0.3, -0.2, 0.1), dict(vel_kind=O.VEL_CONST, vel_param=(0.3, -0.2, 0.1))
    if case == "law nodal":
        vel, ov = "nodal", dict(vel_kind=O.VEL_NODAL, vel_nodal=U)
    if case.startswith("law"):
        op = M.HeatDiffuseOperator(gm, 1e-4, velocity=vel, precisions=prec, material=dict(LAW, kind="gas_liquid_solid"))
        okw = dict(temperature_old=T_old, heaviside=H, material=dict(LAW, kind=O.MAT_GAS_LIQUID_SOLID), **ov)
    elif case == "full":
        op = M.HeatDiffuseOperator(gm, 1e-4, k_alpha=1e-3, full_tangent=True, velocity=vel, precisions=prec)
        okw = dict(k_alpha=1e-3, full_tangent=True, **ov)
    else:
        op = M.HeatDiffuseOperator(gm, 1e-4, k_alpha=1e-3, velocity=vel, precisions=prec)
        okw = dict(k_alpha=1e-3, **ov)
    fields = [dev(a) for a in (T, T_old, H, U.reshape(-1))]
    if case == "law nodal":
        op.set_velocity(fields[3])
    op.set_temperature(fields[0])
    if case.startswith("law"):
        op.set_temperature_old(fields[1])
        op.set_heaviside(fields[2])
    b = rng(3).uniform(-1, 1, N)
    b[mask == 1] = 0.0
    data = M.LinearSolverData(solver_type="GMRES", rel_tolerance=1e-9, mixed_precision=mixed)
    oop = O.Operator(O.HEAT, 1e-4, temperature=T, dirichlet=mask, **okw)

    def solve():
        sol = torch.zeros(N, dtype=torch.float64, device="cuda")
        rhs = dev(b)
        torch.cuda.synchronize()
        M.LinearSolver.solve(op, sol, rhs, data)
        sol = sol.cpu().numpy()
        r = b - O.vmult(om, oop, sol)
        assert np.linalg.norm(r) <= 1.05e-9 * np.linalg.norm(b)
        return sol

    two = solve()
    keep = [torch.cuda.Stream() for _ in range(5)]
    for st in keep:
        op.set_stream(st)
    assert np.array_equal(solve(), two)
    op.set_stream(None)
    for pr in prec:
        op.set_schedule(precision=pr, **dict(op.schedule(pr), lane_cells=0))
    assert np.array_equal(solve(), two)
    assert op.device_error() == 0


@pytest.mark.parametrize("p", [1, 2])
@pytest.mark.parametrize("masked", [False, True])
def test_constraints_above_the_fused_size(cuda, p, masked):
    """The same mesh with a million DoFs of no cell behind its own."""
    import torch
    import meltpooldg_b200 as M
    m2 = O.Mesh2(p, (2, 3, 2), 2, perturb=0.1, seed=20 + p)
    mm = O.mapped_from_mesh2(m2)
    mask = m2.boundary_face_mask() if masked else None
    n = mm.n_dofs
    x = rng(60 + p).uniform(-1, 1, n)
    out = {}
    for extra in (0, 1 << 20):
        mk = None if mask is None else np.concatenate([mask, np.zeros(extra, np.uint8)])
        gm = M.MappedMesh(mm.cell_vertices, mm.cell_dofs, n + extra, p, dirichlet_mask=mk, constraints=mm.constraints)
        op = M.HeatDiffuseOperator(gm, 1e-2, precisions=("fp64", "fp32"))
        for dtype in (torch.float64, torch.float32):
            s = dev(np.concatenate([x, np.ones(extra)]), dtype)
            d = torch.full_like(s, float("nan"))
            op.vmult(d, s)
            out[extra, dtype] = d.cpu().numpy()
    oop = O.Operator(O.HEAT, 1e-2, dirichlet=mask)
    ref = O.mapped_vmult(mm, oop, x)
    for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        got = out[1 << 20, dtype]
        assert np.array_equal(got[:n], out[0, dtype])
        assert not got[n:].any()
        assert np.abs(got[:n] - ref).max() < tol * np.abs(ref).max()
