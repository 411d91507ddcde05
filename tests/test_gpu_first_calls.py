"""What a first call on a new operator allocates: the arrays it needs come in few driver
allocations (0.3 ms each), and the room of the two-launch apply behind one of them.
Counted by the library's own counter."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, rng

pytestmark = pytest.mark.gpu

LAW = dict(kind="gas_liquid_solid", rho=(3925.0, 7850.0, 7000.0), cp=(230.0, 460.0, 700.0), k=(27.8, 55.6, 17.0),
           solidus=1900.0, liquidus=2000.0)


def allocated(f):
    from meltpooldg_b200 import _capi as A
    before = A.allocations()
    f()
    return A.allocations() - before


@pytest.mark.parametrize("p,nc,perturb,vel,count", [
    (2, (9, 8, 7), 0.1, None, 1),          # the coefficient stream
    (4, (5, 4, 3), 0.1, "nodal", 1),
    (2, (9, 8, 7), 0.0, "nodal", 0),       # the velocity stream came with the field
    (3, (9, 8, 7), 0.0, "vortex", 0),      # nothing per cell
    (4, (5, 4, 3), 0.0, ("rotation", 0.8), 0),
    (2, (9, 8, 7), 0.0, "vortex", 0)])     # the band apply
def test_first_applies(cuda, p, nc, perturb, vel, count):
    import torch
    import meltpooldg_b200 as M
    gm, _ = meshes(nc, p, perturb, seed=3)
    op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=vel)
    if vel == "nodal":
        op.set_velocity(dev(rng(5).uniform(-1, 1, 3 * gm.n_dofs)))
    s = dev(rng(4).uniform(-1, 1, gm.n_dofs))
    d, e = torch.empty_like(s), torch.empty_like(s)
    assert allocated(lambda: op.vmult(d, s)) == count
    # the same on another stream, with room of its own
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    op.set_stream(st)
    op.vmult(e, s)
    torch.cuda.synchronize()
    op.set_stream(None)
    assert torch.equal(d, e)


def test_first_apply_of_a_mapped_mesh(cuda):
    import torch
    import meltpooldg_b200 as M
    n = 6
    i, j, k = (a.reshape(-1) for a in np.meshgrid(*[np.arange(n)] * 3, indexing="ij"))
    at = np.stack([k, j, i], 1)[:, None] + np.stack([(np.arange(8) >> d) & 1 for d in range(3)], 1)[None]
    gm = M.MappedMesh(at / n, at @ np.array([1, n + 1, (n + 1) ** 2]), (n + 1) ** 3, 1)
    op = M.HeatDiffuseOperator(gm, 1e-3)
    s = dev(rng(4).uniform(-1, 1, gm.n_dofs))
    assert allocated(lambda: op.vmult(torch.empty_like(s), s)) == 1


@pytest.mark.parametrize("solver,mixed,count", [("CG", False, 2), ("GMRES", False, 3), ("CG", True, 3), ("GMRES", True, 4)])
def test_first_solves(cuda, solver, mixed, count):
    """Constant coefficients: pinned memory, the vectors of each precision, the basis."""
    import torch
    import meltpooldg_b200 as M
    gm, _ = meshes((9, 8, 7), 2, 0.0)
    op = M.HeatDiffuseOperator(gm, 1e-3, precisions=("fp64", "fp32"))
    b = dev(rng(3).uniform(-1, 1, gm.n_dofs))
    x = torch.zeros_like(b)
    data = M.LinearSolverData(solver_type=solver, rel_tolerance=1e-9, mixed_precision=mixed)
    assert allocated(lambda: M.LinearSolver.solve(op, x, b, data)) == count
    y = torch.zeros_like(b)
    assert allocated(lambda: M.LinearSolver.solve(op, y, b, data)) == 0
    assert torch.equal(x, y)


@pytest.mark.parametrize("perturb", [0.0, 0.1])
def test_first_solve_of_a_field_dependent_operator(cuda, perturb):
    """The merged streams and the room of the two-launch apply in one more."""
    import torch
    import meltpooldg_b200 as M
    gm, om = meshes((9, 8, 7), 2, perturb, seed=5)
    op = M.HeatDiffuseOperator(gm, 1e-4, velocity=(0.3, -0.2, 0.1), material=LAW)
    T = dev(1950.0 + 60.0 * np.sin(3.0 * om.dof_coordinates()[:, 0]))
    H, T_old = torch.full_like(T, 0.5), T - 1.0
    op.set_temperature(T)
    op.set_temperature_old(T_old)
    op.set_heaviside(H)
    b = dev(rng(3).uniform(-1, 1, gm.n_dofs))
    x = torch.zeros_like(b)
    data = M.LinearSolverData(solver_type="GMRES", rel_tolerance=1e-9)
    assert allocated(lambda: M.LinearSolver.solve(op, x, b, data)) == 4
