"""Linear solves of operators whose coefficients follow the fields: in a solve the
terms are merged into the apply's streams once, outside it every apply evaluates
them; the solution's residual under the oracle's operator is the solver's, for the
phase laws, the full tangent and k(T) on uniform cells, all degrees, FP64 and
FP32-inner, and a second solve sees fields changed in place.  The residual bound
is the solve's tolerance with 5 % for its own rounding."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, rng
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LAW = dict(rho=(3925.0, 7850.0, 7000.0), cp=(230.0, 460.0, 700.0), k=(27.8, 55.6, 17.0), solidus=1900.0, liquidus=2000.0)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("perturb", [0.0, 0.1])
@pytest.mark.parametrize("case", ["law", "gas_liquid", "full", "kT"])
@pytest.mark.parametrize("mixed", [False, True])
def test_solve_residual_under_the_oracle(cuda, p, perturb, case, mixed):
    import torch
    import meltpooldg_b200 as M
    nc = (5, 4, 3)
    mask = M.boundary_mask(nc, p, faces=[(2, 0)])
    gm, om = meshes(nc, p, perturb, seed=5, mask=mask)
    x = om.dof_coordinates()
    T = 1950.0 + 60.0 * np.sin(3.0 * x[:, 0]) + rng(1).uniform(-1, 1, gm.n_dofs)
    T_old, H = T - 1.0, 0.5 + 0.4 * np.sin(4.0 * x[:, 1])
    prec = ("fp64", "fp32") if mixed else ("fp64",)
    vel, ov = (0.3, -0.2, 0.1), dict(vel_kind=O.VEL_CONST, vel_param=(0.3, -0.2, 0.1))
    if case in ("law", "gas_liquid"):
        kind, ok = (("gas_liquid_solid", O.MAT_GAS_LIQUID_SOLID) if case == "law" else ("gas_liquid", O.MAT_GAS_LIQUID))
        op = M.HeatDiffuseOperator(gm, 1e-4, velocity=vel, precisions=prec, material=dict(LAW, kind=kind))
        okw = dict(temperature_old=T_old, heaviside=H, material=dict(LAW, kind=ok), **ov)
    elif case == "full":
        op = M.HeatDiffuseOperator(gm, 1e-4, k_alpha=1e-3, full_tangent=True, precisions=prec)
        okw = dict(k_alpha=1e-3, full_tangent=True)
    else:
        op = M.HeatDiffuseOperator(gm, 1e-4, k_alpha=1e-3, velocity=vel, precisions=prec)
        okw = dict(k_alpha=1e-3, **ov)
    Td, Od, Hd = dev(T), dev(T_old), dev(H)
    op.set_temperature(Td)
    if case in ("law", "gas_liquid"):
        op.set_temperature_old(Od)
        op.set_heaviside(Hd)
    b = rng(3).uniform(-1, 1, gm.n_dofs)
    b[mask == 1] = 0.0
    data = M.LinearSolverData(solver_type="GMRES", rel_tolerance=1e-9, mixed_precision=mixed)
    for step in range(2):
        sol = torch.zeros(gm.n_dofs, dtype=torch.float64, device="cuda")
        M.LinearSolver.solve(op, sol, dev(b), data)
        oop = O.Operator(O.HEAT, 1e-4, temperature=T, dirichlet=mask, **okw)
        r = b - O.vmult(om, oop, sol.cpu().numpy())
        assert np.linalg.norm(r) <= 1.05e-9 * np.linalg.norm(b), step
        if case == "kT" and perturb:
            break  # this operator holds its fields from set_temperature
        T = T + 3.0  # the fields change in place: applies and solves read them as they are
        Td.copy_(dev(T))
        if mixed:
            op.set_temperature(Td)  # the FP32 copies are made here
