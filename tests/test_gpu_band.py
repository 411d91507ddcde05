"""The band apply (uniform lattices, constant coefficients: sums of line products)
at the sizes where its strips, slots and chunks end: one cell, one strip, the
largest strip and one unit more, a z chunk's recomputed layer; every velocity
it serves; Dirichlet DoFs as whole faces, on some faces, and scattered.  FP64
against the oracle to 1e-12, FP32 to 2e-5 (the tolerances of every apply)."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, relerr, rng
from oracle import oracle as O

pytestmark = pytest.mark.gpu

VEL = {"none": (None, {}), "const": ((0.7, -0.4, 0.25), dict(vel_kind=O.VEL_CONST, vel_param=(0.7, -0.4, 0.25))),
       "vortex": ("vortex", dict(vel_kind=O.VEL_VORTEX)),
       "rotation": (("rotation", 0.8), dict(vel_kind=O.VEL_ROTATION, vel_param=(0.8, 0.0, 0.0)))}


@pytest.mark.parametrize("p,nc", [(1, (1, 1, 1)), (1, (61, 3, 2)), (1, (62, 9, 5)), (2, (29, 4, 3)), (2, (30, 5, 7)),
                                  (2, (31, 1, 9)), (3, (19, 3, 4)), (3, (20, 9, 2)), (4, (13, 2, 3)), (4, (14, 5, 3)),
                                  (4, (1, 9, 2))])
@pytest.mark.parametrize("vel", sorted(VEL))
@pytest.mark.parametrize("mask", ["none", "all", "some_faces", "scattered"])
def test_band_apply_matches_the_oracle(cuda, p, nc, vel, mask):
    import torch
    import meltpooldg_b200 as M
    m = {"none": lambda: None, "all": lambda: M.boundary_mask(nc, p),
         "some_faces": lambda: M.boundary_mask(nc, p, faces=[(0, 1), (2, 0)]),
         "scattered": lambda: (rng(5).uniform(size=int(np.prod([n * p + 1 for n in nc]))) < 0.1).astype(np.uint8)}[mask]()
    gm, om = meshes(nc, p, 0.0, seed=3, mask=m, hi=(1.0, 0.8, 1.3))
    v, ov = VEL[vel]
    op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=v, precisions=("fp64", "fp32"))
    oop = O.Operator(O.ADVDIFF, 1e-3, theta=0.5, diffusivity=1e-2, dirichlet=m, **ov)
    src = rng(70 + p).uniform(-1, 1, gm.n_dofs)
    ref = O.vmult(om, oop, src)
    for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        out = torch.full((gm.n_dofs,), float("nan"), dtype=dtype, device="cuda")
        op.vmult(out, dev(src, dtype))
        assert relerr(out.cpu().numpy().astype(np.float64), ref) < tol


@pytest.mark.parametrize("p,nc", [(1, (1, 2, 1)), (1, (63, 3, 2)), (2, (31, 5, 3)), (3, (7, 4, 3)), (4, (5, 3, 4))])
@pytest.mark.parametrize("vel", sorted(VEL))
@pytest.mark.parametrize("mask", ["none", "some_faces", "scattered"])
def test_band_diagonal_and_rhs_match_the_oracle(cuda, p, nc, vel, mask):
    """The diagonal as products of line diagonals, and the theta-scheme right-hand
    side added into a vector, constrained entries untouched."""
    import torch
    import meltpooldg_b200 as M
    m = {"none": lambda: None, "some_faces": lambda: M.boundary_mask(nc, p, faces=[(0, 1), (2, 0)]),
         "scattered": lambda: (rng(5).uniform(size=int(np.prod([n * p + 1 for n in nc]))) < 0.1).astype(np.uint8)}[mask]()
    gm, om = meshes(nc, p, 0.0, seed=3, mask=m, hi=(1.0, 0.8, 1.3))
    v, ov = VEL[vel]
    op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=v)
    oop = O.Operator(O.ADVDIFF, 1e-3, theta=0.5, diffusivity=1e-2, dirichlet=m, **ov)
    d = torch.empty(gm.n_dofs, dtype=torch.float64, device="cuda")
    op.compute_diagonal(d)
    assert relerr(d.cpu().numpy(), O.diagonal(om, oop)) < 1e-12
    phi, start = rng(8).uniform(-1, 1, gm.n_dofs), rng(9).uniform(-1, 1, gm.n_dofs)
    out = dev(start.copy())
    op.create_rhs(out, dev(phi))
    ref = O.rhs_advdiff(om, oop, phi, dst=np.zeros(gm.n_dofs))
    if m is not None:
        ref = np.where(m == 1, 0.0, ref)
    assert np.abs(out.cpu().numpy() - (start + ref)).max() < 1e-12 * max(1.0, np.abs(ref).max())
