"""Small lattices apply in two launches (local results, one gather per DoF).  The
sums run in the order of the colours, so the bits are those of the coloured
launches, which a caller's stream capture keeps; the workspace is one per stream,
streams beyond the operator's workspaces take the coloured launches, and a
precision change leaves it in place."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, relerr, rng
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,nc", [(1, (1, 1, 1)), (1, (7, 2, 5)), (2, (1, 4, 3)), (2, (33, 3, 2)), (3, (5, 1, 2)),
                                  (4, (4, 3, 5))])
@pytest.mark.parametrize("vel", [None, "vortex"])
def test_eager_applies_equal_captured_ones_on_every_stream(cuda, p, nc, vel):
    import torch
    import meltpooldg_b200 as M
    mask = M.boundary_mask(nc, p, faces=[(0, 0), (2, 1)])
    gm, om = meshes(nc, p, 0.1, seed=3, mask=mask)
    op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=vel, precisions=("fp64", "fp32"))
    ov = dict(vel_kind=O.VEL_VORTEX) if vel else {}
    oop = O.Operator(O.ADVDIFF, 1e-3, theta=0.5, diffusivity=1e-2, dirichlet=mask, **ov)
    src = rng(4).uniform(-1, 1, gm.n_dofs)
    ref = O.vmult(om, oop, src)
    for dtype, tol in ((torch.float32, 2e-5), (torch.float64, 1e-12)):
        s = dev(src, dtype)
        eager = torch.full_like(s, float("nan"))
        op.vmult(eager, s)
        assert relerr(eager.cpu().numpy().astype(np.float64), ref) < tol
        captured = torch.full_like(s, float("nan"))
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            op.set_stream(torch.cuda.current_stream())
            op.vmult(captured, s)
        op.set_stream(None)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, eager)
        # more streams than workspaces, applies in flight side by side
        streams = [torch.cuda.Stream() for _ in range(6)]
        outs = [torch.full_like(s, float("nan")) for _ in streams]
        torch.cuda.synchronize()
        for _ in range(3):
            for st, o in zip(streams, outs):
                op.set_stream(st)
                op.vmult(o, s)
        torch.cuda.synchronize()
        op.set_stream(None)
        for o in outs:
            assert torch.equal(o, eager)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("vel", [None, "vortex"])
def test_mapped_applies_equal_captured_ones(cuda, p, vel):
    """Mapped meshes, renumbered, with Dirichlet DoFs and DoFs of no cell (result 0)."""
    import torch
    import meltpooldg_b200 as M
    nc = (3, 4, 5)
    _, om = meshes(nc, p, 0.1, seed=p)
    R = rng(50 + p)
    perm = R.permutation(om.n_dofs)
    mm = O.mapped_from_mesh(om, perm=perm, cell_order=R.permutation(om.n_cells))
    N = om.n_dofs + 7
    mask = (R.uniform(size=N) < 0.1).astype(np.uint8)
    gm = M.MappedMesh(mm.cell_vertices, mm.cell_dofs, N, p, dirichlet_mask=mask)
    op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=vel, precisions=("fp64", "fp32"))
    ov = dict(vel_kind=O.VEL_VORTEX) if vel else {}
    oop = O.Operator(O.ADVDIFF, 1e-3, theta=0.5, diffusivity=1e-2, dirichlet=mask[:om.n_dofs], **ov)
    src = R.uniform(-1, 1, N)
    ref = np.concatenate([O.mapped_vmult(mm, oop, src[:om.n_dofs]), np.zeros(7)])
    for dtype, tol in ((torch.float32, 2e-5), (torch.float64, 1e-12)):
        s = dev(src, dtype)
        eager, captured = torch.full_like(s, float("nan")), torch.full_like(s, float("nan"))
        op.vmult(eager, s)
        assert relerr(eager.cpu().numpy().astype(np.float64), ref) < tol
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            op.set_stream(torch.cuda.current_stream())
            op.vmult(captured, s)
        op.set_stream(None)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, eager)
