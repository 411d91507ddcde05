"""Which launches an apply takes: the forms that replace the coloured launches return
their results, and are not slower than what they replace, on lattices that are thin
in one or two directions.  Times are the best of several event-timed batches, with
half as much again allowed for the machine."""
import numpy as np
import pytest

from gpu_helpers import dev, meshes, relerr, rng
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SLACK = 1.5


def best_us(*calls, n=20, batches=9):
    """Best time of each call, batches in turn."""
    import torch
    e0, e1, best = torch.cuda.Event(True), torch.cuda.Event(True), [float("inf")] * len(calls)
    for f in calls:
        f()
    for _ in range(batches):
        for i, f in enumerate(calls):
            torch.cuda.synchronize()
            e0.record()
            for _ in range(n):
                f()
            e1.record()
            torch.cuda.synchronize()
            best[i] = min(best[i], 1e3 * e0.elapsed_time(e1) / n)
    return best


def colours(op, p):
    """The default schedule's coloured launches."""
    op.set_schedule(1, False, "fp64", overlap_colours=True, cta_cell_groups=p in (2, 4), lane_cells=0)
    return op


def launches(f):
    import meltpooldg_b200 as M
    f()
    before = M.kernel_launches()
    f()
    return M.kernel_launches() - before


def coloured(op, dst, src):
    """A graph of one apply: a caller's capture keeps the coloured launches."""
    import torch
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        op.set_stream(torch.cuda.current_stream())
        op.vmult(dst, src)
    op.set_stream(None)
    return g


@pytest.mark.parametrize("p,nc", [(1, (1, 1, 300)), (2, (1, 70, 2)), (3, (43, 1, 1)), (4, (2, 1, 65)), (2, (3, 33, 7))])
def test_thin_lattices_in_two_launches_equal_the_colours(cuda, p, nc):
    """Rows that do not fill a block of the gather, blocks that end inside a row."""
    import torch
    import meltpooldg_b200 as M
    gm, _ = meshes(nc, p, 0.1, seed=3, mask=M.boundary_mask(nc, p, faces=[(0, 0), (2, 1)]))
    op = M.HeatDiffuseOperator(gm, 1e-3, precisions=("fp64", "fp32"))
    for dtype in (torch.float64, torch.float32):
        s = dev(rng(4).uniform(-1, 1, gm.n_dofs), dtype)
        two, eight = torch.full_like(s, float("nan")), torch.full_like(s, float("nan"))
        op.vmult(two, s)
        coloured(op, eight, s).replay()
        torch.cuda.synchronize()
        assert torch.equal(two, eight)


@pytest.mark.parametrize("p,nc", [(1, (2, 170, 180)), (2, (2, 90, 100))])
def test_two_launches_on_thin_lattices_are_not_slower_than_the_colours(cuda, p, nc):
    import torch
    import meltpooldg_b200 as M
    gm, _ = meshes(nc, p, 0.1, seed=3)
    op, ref = M.HeatDiffuseOperator(gm, 1e-3), colours(M.HeatDiffuseOperator(gm, 1e-3), p)
    s = dev(rng(4).uniform(-1, 1, gm.n_dofs))
    d = torch.empty_like(s)
    two, eight = best_us(lambda: op.vmult(d, s), lambda: ref.vmult(d, s))
    assert two < SLACK * eight, (two, eight)


def test_host_time_of_an_apply_does_not_grow_with_the_layers(cuda):
    """The band apply's search for its chunks on 4,000 cell layers against 40."""
    import time
    import torch
    import meltpooldg_b200 as M
    host = []
    for nz in (40, 4000):
        gm, _ = meshes((16, 4, nz), 1, 0.0)
        op = M.HeatDiffuseOperator(gm, 1e-3)
        s = dev(rng(4).uniform(-1, 1, gm.n_dofs))
        d = torch.empty_like(s)
        assert launches(lambda: op.vmult(d, s)) == 1
        best = float("inf")
        for _ in range(30):
            torch.cuda.synchronize()
            t = time.perf_counter()
            for _ in range(5):
                op.vmult(d, s)
            best = min(best, time.perf_counter() - t)
        host.append(best)
    assert host[1] < 2.5 * host[0], host


@pytest.mark.parametrize("p,nc,vel", [(4, (8, 60, 40), ("rotation", 0.8)), (4, (24, 24, 24), ("rotation", 0.8)),
                                      (3, (2, 100, 100), None), (4, (2, 100, 100), None), (3, (4, 16, 500), None),
                                      (2, (4, 4, 4000), ("rotation", 0.8)), (1, (4, 16, 4000), "vortex"),
                                      (4, (1, 1, 100), None), (3, (30, 1, 1), ("rotation", 0.8)),
                                      (3, (1000, 1, 1), None)])
def test_the_default_apply_is_not_slower_than_the_colours(cuda, p, nc, vel):
    """Uniform lattices whose strips of the band apply would stay nearly empty, or whose
    products spill: the default takes the launches that are faster there."""
    import torch
    import meltpooldg_b200 as M
    gm, _ = meshes(nc, p, 0.0)
    op, ref = (M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=vel) for _ in range(2))
    colours(ref, p)
    s = dev(rng(4).uniform(-1, 1, gm.n_dofs))
    d, e = torch.empty_like(s), torch.empty_like(s)
    default, eight = best_us(lambda: op.vmult(d, s), lambda: ref.vmult(e, s))
    assert (d - e).abs().max() <= 1e-13 * e.abs().max()
    assert default < SLACK * eight, (default, eight)


@pytest.mark.parametrize("p,nc", [(3, (20, 20, 10)), (3, (19, 3, 70)), (4, (13, 20, 16)), (4, (27, 10, 16))])
@pytest.mark.parametrize("mask", ["none", "some_faces", "scattered"])
def test_band_apply_of_degrees_3_and_4(cuda, p, nc, mask):
    import torch
    import meltpooldg_b200 as M
    m = {"none": lambda: None, "some_faces": lambda: M.boundary_mask(nc, p, faces=[(0, 1), (2, 0)]),
         "scattered": lambda: (rng(5).uniform(size=int(np.prod([n * p + 1 for n in nc]))) < 0.1).astype(np.uint8)}[mask]()
    gm, om = meshes(nc, p, 0.0, mask=m, hi=(1.0, 0.8, 1.3))
    op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=(0.7, -0.4, 0.25),
                                      precisions=("fp64", "fp32"))
    oop = O.Operator(O.ADVDIFF, 1e-3, theta=0.5, diffusivity=1e-2, dirichlet=m, vel_kind=O.VEL_CONST,
                     vel_param=(0.7, -0.4, 0.25))
    src = rng(70 + p).uniform(-1, 1, gm.n_dofs)
    ref = O.vmult(om, oop, src)
    for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        out = torch.full((gm.n_dofs,), float("nan"), dtype=dtype, device="cuda")
        before = M.kernel_launches()
        op.vmult(out, dev(src, dtype))
        assert M.kernel_launches() - before == 1
        assert relerr(out.cpu().numpy().astype(np.float64), ref) < tol


@pytest.mark.parametrize("p,nc,vel", [(2, (4, 2000, 4), "vortex"), (2, (64, 64, 64), "vortex"), (2, (100, 100, 2), "vortex"),
                                      (4, (32, 32, 32), ("rotation", 0.8)), (3, (1, 1, 1000), None),
                                      (4, (4, 1000, 4), ("rotation", 0.8))])
def test_diagonal_from_line_factors_is_not_slower_than_from_the_cells(cuda, p, nc, vel):
    """The same lattice as general cells takes the cells' element diagonals."""
    import torch
    import meltpooldg_b200 as M
    d, us = [], []
    for geometry in ("auto", "general"):
        gm, _ = meshes(nc, p, 0.0, geometry=geometry)
        op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=vel)
        d.append(torch.empty(gm.n_dofs, dtype=torch.float64, device="cuda"))
        us += best_us(lambda: op.compute_diagonal(d[-1]))
    assert (d[0] - d[1]).abs().max() <= 1e-12 * d[1].abs().max()
    assert us[0] < SLACK * us[1], us


@pytest.mark.parametrize("p,nc", [(2, (1, 1, 2000)), (3, (1, 1, 1000)), (4, (1, 1, 1000)), (4, (4, 4, 2000)), (3, (20, 9, 4)), (4, (13, 6, 5))])
def test_rhs_as_line_products_is_not_slower_than_from_the_cells(cuda, p, nc):
    """The same lattice as general cells takes the cells' block kernel."""
    import torch
    import meltpooldg_b200 as M
    d, us = [], []
    for geometry in ("auto", "general"):
        gm, _ = meshes(nc, p, 0.0, geometry=geometry, mask=M.boundary_mask(nc, p, faces=[(0, 0)]))
        op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=(0.3, 0.1, -0.2))
        phi = dev(rng(8).uniform(-1, 1, gm.n_dofs))
        d.append(torch.zeros(gm.n_dofs, dtype=torch.float64, device="cuda"))
        op.create_rhs(d[-1], phi)
        spare = torch.zeros_like(phi)
        us += best_us(lambda: op.create_rhs(spare, phi))
    assert (d[0] - d[1]).abs().max() <= 1e-12 * d[1].abs().max()
    assert us[0] < SLACK * us[1], us


def test_two_launches_up_to_the_measured_sizes(cuda):
    """900,000 local values; uniform Q4 cells with a velocity vector 650,000 in FP64."""
    import torch
    import meltpooldg_b200 as M
    for nc, count in (((32, 32, 32), 2), ((33, 32, 32), 8)):
        gm, _ = meshes(nc, 2, 0.1, seed=3)
        op = M.HeatDiffuseOperator(gm, 1e-3, precisions=("fp64", "fp32"))
        for dtype in (torch.float64, torch.float32):
            s = dev(rng(4).uniform(-1, 1, gm.n_dofs), dtype)
            d = torch.empty_like(s)
            assert launches(lambda: op.vmult(d, s)) == count
    for nc, fp64 in (((17, 17, 17), 2), ((18, 18, 18), 8)):
        gm, _ = meshes(nc, 4, 0.0)
        op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity="nodal", precisions=("fp64", "fp32"))
        U = dev(rng(5).uniform(-1, 1, 3 * gm.n_dofs))
        op.set_velocity(U)
        for dtype, n in ((torch.float64, fp64), (torch.float32, 2)):
            s = dev(rng(4).uniform(-1, 1, gm.n_dofs), dtype)
            d = torch.empty_like(s)
            assert launches(lambda: op.vmult(d, s)) == n


@pytest.mark.parametrize("n,order,count", [(40, "lexicographic", 2), (50, "lexicographic", 8), (50, "shuffled", 2)])
def test_mapped_q1_in_two_launches_where_its_colours_are_many(cuda, n, order, count):
    import torch
    import meltpooldg_b200 as M
    i, j, k = (a.reshape(-1) for a in np.meshgrid(*[np.arange(n)] * 3, indexing="ij"))
    cell = np.stack([k, j, i], 1)
    corner = np.stack([(np.arange(8) >> d) & 1 for d in range(3)], 1)
    at = cell[:, None] + corner[None]
    dofs = at @ np.array([1, n + 1, (n + 1) ** 2])
    if order == "shuffled":
        p = rng(2).permutation(len(cell))
        at, dofs = at[p], dofs[p]
    gm = M.MappedMesh(at / n, dofs, (n + 1) ** 3, 1)
    op = M.HeatDiffuseOperator(gm, 1e-3)
    s = dev(rng(4).uniform(-1, 1, gm.n_dofs))
    d = torch.empty_like(s)
    assert launches(lambda: op.vmult(d, s)) == count


@pytest.mark.parametrize("p,nc,perturb", [(1, (9, 8, 7), 0.0), (2, (40, 9, 8), 0.0), (3, (20, 20, 10), 0.0),
                                          (4, (13, 20, 16), 0.0), (2, (9, 8, 7), 0.1), (4, (5, 4, 3), 0.1)])
def test_setting_the_reported_schedule_changes_nothing(cuda, p, nc, perturb):
    """get, set: the same launches and bits; lane_cells 0: the coloured launches."""
    import torch
    import meltpooldg_b200 as M
    gm, _ = meshes(nc, p, perturb, seed=3)
    op = M.HeatDiffuseOperator(gm, 1e-3, precisions=("fp64", "fp32"))
    for prec, dtype in (("fp64", torch.float64), ("fp32", torch.float32)):
        s = dev(rng(4).uniform(-1, 1, gm.n_dofs), dtype)
        a, b = torch.empty_like(s), torch.empty_like(s)
        default = launches(lambda: op.vmult(a, s))
        assert default == (2 if perturb else 1)
        sc = op.schedule(prec)
        op.set_schedule(precision=prec, **sc)
        assert op.schedule(prec) == sc
        assert launches(lambda: op.vmult(b, s)) == default
        assert torch.equal(a, b)
        op.set_schedule(precision=prec, **dict(sc, lane_cells=0))
        assert launches(lambda: op.vmult(b, s)) == 8
        if perturb:
            assert torch.equal(a, b)


@pytest.mark.parametrize("p,nc", [(3, (19, 3, 4)), (3, (20, 9, 2)), (4, (13, 2, 3)), (4, (14, 5, 3)), (4, (1, 9, 2)),
                                  (2, (1, 1, 9)), (1, (1, 3, 70))])
@pytest.mark.parametrize("vel", ["none", "const", "rotation"])
def test_band_apply_wherever_it_is_built(cuda, p, nc, vel):
    """lane_cells 2 on lattices that the default gives to the other launches."""
    import torch
    import meltpooldg_b200 as M
    v, ov = {"none": (None, {}), "const": ((0.7, -0.4, 0.25), dict(vel_kind=O.VEL_CONST, vel_param=(0.7, -0.4, 0.25))),
             "rotation": (("rotation", 0.8), dict(vel_kind=O.VEL_ROTATION, vel_param=(0.8, 0.0, 0.0)))}[vel]
    m = M.boundary_mask(nc, p, faces=[(0, 1), (2, 0)])
    gm, om = meshes(nc, p, 0.0, mask=m, hi=(1.0, 0.8, 1.3))
    op = M.AdvectionDiffusionOperator(gm, 1e-3, theta=0.5, diffusivity=1e-2, velocity=v, precisions=("fp64", "fp32"))
    oop = O.Operator(O.ADVDIFF, 1e-3, theta=0.5, diffusivity=1e-2, dirichlet=m, **ov)
    src = rng(70 + p).uniform(-1, 1, gm.n_dofs)
    ref = O.vmult(om, oop, src)
    for prec, dtype, tol in (("fp64", torch.float64, 1e-12), ("fp32", torch.float32, 2e-5)):
        op.set_schedule(1, False, prec, overlap_colours=True, lane_cells=2)
        s = dev(src, dtype)
        out = torch.full_like(s, float("nan"))
        if not (p == 4 and vel == "rotation"):
            assert launches(lambda: op.vmult(out, s)) == 1
        op.vmult(out, s)
        assert relerr(out.cpu().numpy().astype(np.float64), ref) < tol


@pytest.mark.parametrize("p,nc,perturb,count,best", [(2, (40, 9, 8), 0.0, 9, 1), (3, (20, 20, 10), 0.0, 5, 1),
                                                     (2, (9, 8, 7), 0.1, 17, 2)])
def test_autotuner_times_each_form_once_and_finds_the_default_again(cuda, p, nc, perturb, count, best):
    """From the default schedule, and from one that took the coloured launches."""
    import meltpooldg_b200 as M
    gm, _ = meshes(nc, p, perturb, seed=3)
    op = M.HeatDiffuseOperator(gm, 1e-3)
    s = dev(rng(4).uniform(-1, 1, gm.n_dofs))
    d = s.clone()
    sc, _, times = op.autotune("fp64", reps=20)
    assert len(times) == count and sc["lane_cells"] == 1
    op.set_schedule(precision="fp64", **dict(sc, lane_cells=0))
    assert launches(lambda: op.vmult(d, s)) == 8
    sc, _, times = op.autotune("fp64", reps=20)
    assert len(times) == count and sc["lane_cells"] == 1
    assert launches(lambda: op.vmult(d, s)) == best


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_default_schedule(cuda, p):
    """One slab, overlapping colours, CTA cell groups for Q2 and FP64 Q4, the evict-first
    hint in FP32, the faster form of the apply."""
    import meltpooldg_b200 as M
    gm, _ = meshes((3, 3, 3), p, 0.1, seed=3)
    op = M.HeatDiffuseOperator(gm, 1e-3, precisions=("fp64", "fp32"))
    common = dict(slabs=1, overlap_colours=True, lane_cells=1)
    assert op.schedule("fp64") == dict(common, l2_evict_first=False, cta_cell_groups=p in (2, 4))
    assert op.schedule("fp32") == dict(common, l2_evict_first=True, cta_cell_groups=p == 2)


@pytest.mark.parametrize("p,nc", [(2, (4, 4, 60)), (4, (5, 4, 20)), (3, (9, 8, 17))])
def test_host_pipeline_of_small_lattices_takes_one_launch_a_range(cuda, p, nc):
    """Eight ranges of layers (as many as pairs of layers allow), one launch each."""
    import meltpooldg_b200 as M
    gm, om = meshes(nc, p, 0.0)
    op = M.HeatDiffuseOperator(gm, 1e-3)
    src = rng(4).uniform(-1, 1, gm.n_dofs)
    out = np.empty_like(src)
    assert launches(lambda: op.vmult_host(out, src)) == 8
    assert relerr(out, O.vmult(om, O.Operator(O.HEAT, 1e-3), src)) < 1e-12
