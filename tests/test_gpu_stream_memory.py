"""Memory of the streams that a solve merges from an operator's fields: a solve that may
not have them evaluates the fields in every apply, precision by precision, with the same
solution; whether it may does not depend on what else is on the device; large streams
go back when the solve ends.  Residuals under the oracle's operator, bounded by the
solves' tolerance with 5 % for its own rounding."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, rng
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LAW = dict(rho=(3925.0, 7850.0, 7000.0), cp=(230.0, 460.0, 700.0), k=(27.8, 55.6, 17.0), solidus=1900.0, liquidus=2000.0)


def _problem(nc, p, perturb):
    import meltpooldg_b200 as M
    mask = M.boundary_mask(nc, p, faces=[(2, 0)])
    gm, om = meshes(nc, p, perturb, seed=5, mask=mask)
    x = om.dof_coordinates()
    T = 1950.0 + 60.0 * np.sin(3.0 * x[:, 0])
    T_old, H = T - 1.0, 0.5 + 0.4 * np.sin(4.0 * x[:, 1])
    vel, ov = (0.3, -0.2, 0.1), dict(vel_kind=O.VEL_CONST, vel_param=(0.3, -0.2, 0.1))
    op = M.HeatDiffuseOperator(gm, 1e-4, velocity=vel, precisions=("fp64", "fp32"), material=dict(LAW, kind="gas_liquid_solid"))
    fields = [dev(T), dev(T_old), dev(H)]
    op.set_temperature(fields[0])
    op.set_temperature_old(fields[1])
    op.set_heaviside(fields[2])
    oop = O.Operator(O.HEAT, 1e-4, temperature=T, temperature_old=T_old, heaviside=H, dirichlet=mask,
                     material=dict(LAW, kind=O.MAT_GAS_LIQUID_SOLID), **ov)
    b = rng(3).uniform(-1, 1, gm.n_dofs)
    b[mask == 1] = 0.0
    return gm, om, op, oop, b, fields


@pytest.mark.parametrize("perturb", [0.0, 0.1])
@pytest.mark.parametrize("allowed", ["none", "fp32 alone", "both"])
def test_solves_without_the_streams(cuda, perturb, allowed):
    import torch
    import meltpooldg_b200 as M
    from meltpooldg_b200 import _capi as A
    gm, om, op, oop, b, _ = _problem((5, 4, 3), 2, perturb)
    # 60 cells of 192 + 168 values
    limit = {"none": 0, "fp32 alone": 60 * 360 * 4, "both": -1}[allowed]
    A.check(A.lib().mpdg_debug_set_stream_limit(op._h, limit), "mpdg_debug_set_stream_limit")
    before = A.allocations()
    x = torch.zeros(gm.n_dofs, dtype=torch.float64, device="cuda")
    data = M.LinearSolverData(solver_type="GMRES", rel_tolerance=1e-9, mixed_precision=True)
    M.LinearSolver.solve(op, x, dev(b), data)
    # pinned memory, two precisions' vectors, the basis, and the streams (or the FP32
    # geometry that the block kernel reads on general cells)
    assert A.allocations() - before == 4 + {"none": int(perturb > 0), "fp32 alone": 1, "both": 2}[allowed]
    r = b - O.vmult(om, oop, x.cpu().numpy())
    assert np.linalg.norm(r) <= 1.05e-9 * np.linalg.norm(b)


def test_large_streams_are_given_back(cuda):
    """116^3 Q2 cells: 4.5 GB of streams, against 0.6 GB of vectors that stay."""
    import torch
    import meltpooldg_b200 as M
    nc = (116, 116, 116)
    gm = M.Mesh(M.box_vertices(nc), nc, 2)
    op = M.HeatDiffuseOperator(gm, 1e-4, material=dict(LAW, kind="gas_liquid_solid"))
    T = torch.full((gm.n_dofs,), 1950.0, dtype=torch.float64, device="cuda")
    T_old, H, b, x = T - 1.0, torch.full_like(T, 0.5), torch.ones_like(T), torch.zeros_like(T)
    op.set_temperature(T)
    op.set_temperature_old(T_old)
    op.set_heaviside(H)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    data = M.LinearSolverData(solver_type="GMRES", rel_tolerance=1e-3, gmres_restart=3)
    M.LinearSolver.solve(op, x, b, data)
    assert free - torch.cuda.mem_get_info()[0] < 2.5e9
