"""CG whose sums end in the last block of their kernel, and (above 400,000 DoFs, in a
replayed graph) in a kernel of their own: the oracle's iteration counts and solution at
the sizes on both sides, with both preconditioners, and an iteration limit inside a
batch of iterations.  Bounds as for the other solves: the solver's residual, the Jacobi
form's solution to 1e-9 against the oracle's (the same iterates), and the residual of
the Chebyshev form under the oracle's operator with 5 % for its rounding."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, relerr, rng
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [(36, 36, 36), (37, 37, 36)])
def test_cg_on_both_sides_of_the_line(cuda, nc):
    import torch
    import meltpooldg_b200 as M
    mask = M.boundary_mask(nc, 2)
    gm, om = meshes(nc, 2, mask=mask)
    assert (gm.n_dofs > 400000) == (nc == (37, 37, 36))
    xs = rng(1).uniform(-1, 1, gm.n_dofs)
    xs[mask == 1] = 0.0
    oop = O.Operator(O.HEAT, 1e-3, dirichlet=mask)
    b = O.vmult(om, oop, xs)
    xo, it_o, hist, ok = O.cg(om, oop, b, inv_diag=O.inverse_diagonal(om, oop), rel_tol=1e-10, abs_tol=1e-20)
    assert ok
    op = M.HeatDiffuseOperator(gm, 1e-3)

    def solve(**kw):
        x = torch.zeros(gm.n_dofs, dtype=torch.float64, device="cuda")
        it = M.LinearSolver.solve(op, x, dev(b), M.LinearSolverData(solver_type="CG", rel_tolerance=1e-10,
                                                                   abs_tolerance=1e-20, **kw))
        return x, it, M.LinearSolver.last_report

    x, it, rep = solve(preconditioner_type="Diagonal")
    assert it == it_o
    assert rep["final_residual"] <= 1e-10 * rep["initial_residual"]
    assert relerr(x.cpu().numpy(), xo) < 1e-9
    x2, it2, rep2 = solve(preconditioner_type="Diagonal")
    assert it2 == it and torch.equal(x, x2) and rep2["final_residual"] == rep["final_residual"]
    x, _, rep = solve(preconditioner_type="Chebyshev")
    assert rep["final_residual"] <= 1e-10 * rep["initial_residual"]
    assert np.linalg.norm(b - O.vmult(om, oop, x.cpu().numpy())) <= 1.05e-10 * np.linalg.norm(b)
    # not converged after 10: two batches of four and one of two
    with pytest.raises(Exception):
        solve(preconditioner_type="Diagonal", max_iterations=10)
    rep = M.LinearSolver.last_report
    assert rep["iterations"] == 10
    assert abs(rep["final_residual"] - hist[10]) < 1e-6 * hist[0]
