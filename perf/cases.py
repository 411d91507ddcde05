"""Measured cases of the operator library: what a heat / level-set host program
calls, over the sizes, degrees, meshes and precisions it calls it with.

A case is a dict of plain values; `kind` names the call:

  vmult   one operator apply (OperatorMatrixFree::vmult): the call a Krylov
          solver makes once per iteration, on a mesh and operator it keeps
  mapped  the same on an unstructured mesh with hanging nodes (one 2:1
          refined block), handed over cell by cell as an adaptive host does
  newton  one Newton step of the melt-pool heat equation: new temperature,
          heaviside and old temperature, residual, GMRES + Jacobi solve
  cg      a CG + Jacobi solve of the heat equation
  cheb    a CG + Chebyshev(5)/Jacobi solve in the FP32-inner / FP64-refined form
  step    one theta-scheme step of the level set: right-hand side, GMRES(30) +
          Jacobi solve
  batch   independent heat solves of mixed sizes and degrees, submitted with
          host right-hand sides, advanced together, solutions taken to the host
"""
import functools
import math

import numpy as np
import torch

import meltpooldg_b200 as M
from meltpooldg_b200.batch import Batch, Problem

DT = 1e-3
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    def vm(name, **kw):
        c = dict(name=name, kind="vmult", op="heat", p=2, nx=16, ny=16, nz=16, perturb=0.0, kT=False,
                 velocity="none", fp32=False, dirichlet=True)
        c.update(kw)
        return c

    return [
        # the smallest call: a coarse-grid apply, where launches and latency are the time
        vm("heat_q2_16"),
        # the large heat operator of a printed part: distorted cells, k(T), FP64
        vm("heat_q4_64_kT", p=4, nx=64, ny=64, nz=64, perturb=0.1, kT=True),
        # the same operator in the FP32 form the refined solves iterate with
        vm("heat_q4_64_kT_fp32", p=4, nx=64, ny=64, nz=64, perturb=0.1, kT=True, fp32=True),
        # the level-set transport on a regular grid with its prescribed vortex velocity
        vm("levelset_q2_128", op="advdiff", nx=128, ny=128, nz=128, velocity="vortex", dirichlet=False),
        # the level set moved by a flow solver's velocity vector on distorted cells, odd sizes
        vm("levelset_q2_flow", op="advdiff", nx=61, ny=47, nz=83, perturb=0.1, velocity="nodal", dirichlet=False),
        # constant-coefficient heat on a regular grid of odd size, degree 3
        vm("heat_q3_ragged", p=3, nx=45, ny=39, nz=52),
        # an adaptively refined host mesh
        dict(name="heat_q2_refined", kind="mapped", p=2, nx=32, ny=28, nz=30, fp32=False),
        # one Newton step of gas/liquid/solid heat with the flow's velocity
        dict(name="newton_q2_meltpool", kind="newton", p=2, nx=40, ny=32, nz=24, perturb=0.0),
        # the small linear solve of an inner time loop
        dict(name="cg_q2_16", kind="cg", p=2, nx=16, ny=16, nz=16),
        # the refined-precision solve on distorted cells with k(T)
        dict(name="cheb_q4_32_mixed", kind="cheb", p=4, nx=32, ny=32, nz=32),
        # a time step of the level set at production size
        dict(name="levelset_step_q2_128", kind="step", p=2, nx=128, ny=128, nz=128),
        # many small independent solves at once
        dict(name="batch_24", kind="batch", count=24, lo=8, hi=28, advdiff=False),
    ]


def draw(rng):
    def size(lo, hi):
        return max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    kind = rng.choice(["vmult", "vmult", "vmult", "vmult", "vmult", "mapped", "newton", "cg", "cheb", "step",
                       "batch"])
    if kind == "vmult":
        p = rng.choice([1, 2, 3, 4])
        hi = 256 // p
        op = rng.choice(["heat", "heat", "advdiff"])
        kT = op == "heat" and rng.random() < 0.5
        return dict(kind="vmult", op=op, p=p, nx=size(6, hi), ny=size(6, hi), nz=size(6, hi),
                    perturb=rng.choice([0.0, 0.1]), kT=kT,
                    velocity="none" if op == "heat" else rng.choice(["vortex", "nodal"]),
                    fp32=rng.random() < 0.4, dirichlet=op == "heat" or rng.random() < 0.5)
    if kind == "mapped":
        return dict(kind="mapped", p=rng.choice([1, 2]), nx=size(6, 32), ny=size(6, 32), nz=2 * size(3, 15),
                    fp32=rng.random() < 0.4)
    if kind == "newton":
        p = rng.choice([1, 2, 2])
        return dict(kind="newton", p=p, nx=size(8, 40), ny=size(8, 32), nz=size(6, 24), perturb=rng.choice([0.0, 0.1]))
    if kind == "cg":
        p = rng.choice([1, 2, 3, 4])
        return dict(kind="cg", p=p, nx=size(4, 64 // p), ny=size(4, 64 // p), nz=size(4, 64 // p))
    if kind == "cheb":
        return dict(kind="cheb", p=rng.choice([2, 3, 4]), nx=size(8, 32), ny=size(8, 32), nz=size(8, 32))
    if kind == "step":
        return dict(kind="step", p=rng.choice([1, 2]), nx=size(12, 128), ny=size(12, 128), nz=size(12, 128))
    return dict(kind="batch", count=rng.randint(4, 24), lo=8, hi=rng.randint(10, 28), advdiff=rng.random() < 0.3)


def _nc(c):
    return (c["nx"], c["ny"], c["nz"])


def _shape(c):
    return tuple(n * c["p"] + 1 for n in _nc(c))


def _n_dofs(c):
    return int(np.prod(_shape(c)))


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, lo, hi, gen):
    return torch.rand(n, dtype=F64, device="cuda", generator=gen) * (hi - lo) + lo


def _box_mask(shape):
    m = np.zeros(shape[::-1], np.uint8)
    m[0], m[-1], m[:, 0], m[:, -1], m[:, :, 0], m[:, :, -1] = 1, 1, 1, 1, 1, 1
    return m.reshape(-1)


def _nodes(c):
    """Nodal coordinates per axis of the undistorted unit box."""
    z = _gll(c["p"])
    out = []
    for n in _nc(c):
        g = (np.arange(n)[:, None] + z[None, :-1]).reshape(-1)
        out.append(np.append(g, n) / n)
    return out


def _coords(c):
    x, y, z = (torch.tensor(a, device="cuda") for a in _nodes(c))
    return (x[None, None, :].expand(len(z), len(y), len(x)), y[None, :, None].expand(len(z), len(y), len(x)),
            z[:, None, None].expand(len(z), len(y), len(x)))


def _flow(c, gen):
    """A smooth swirling velocity with a seeded amplitude and phase, component-major."""
    X, Y, Z = _coords(c)
    a, s = (float(v) for v in torch.rand(2, dtype=F64, device="cuda", generator=gen).cpu())
    pi = math.pi
    u = (1 + a) * torch.sin(pi * X + s) * torch.cos(pi * Y)
    v = -(1 + a) * torch.cos(pi * X + s) * torch.sin(pi * Y)
    w = 0.3 * torch.sin(2 * pi * (X + Y)) * (1 - Z)
    return torch.stack([t.reshape(-1) for t in (u, v, w)]).contiguous().reshape(-1)


def _level_set(c, gen):
    X, Y, Z = _coords(c)
    o = [float(v) for v in torch.rand(3, dtype=F64, device="cuda", generator=gen).cpu()]
    d = 0.25 - torch.sqrt((X - 0.4 - 0.2 * o[0]) ** 2 + (Y - 0.6 - 0.2 * o[1]) ** 2 + (Z - 0.4 - 0.2 * o[2]) ** 2)
    return d.reshape(-1)


LAW = dict(kind="gas_liquid_solid", rho=(3925.0, 7850.0, 7000.0), cp=(230.0, 460.0, 700.0), k=(27.7815, 55.563, 17.0),
           solidus=1900.0, liquidus=2000.0)


def _vmult_inputs(c, seed):
    gen = _generator(seed)
    N = _n_dofs(c)
    V = M.box_vertices(_nc(c), perturb=c["perturb"], seed=int(seed) & 0x7fffffff)
    mask = _box_mask(_shape(c)) if c["dirichlet"] else None
    return dict(V=V, mask=mask, src=_uniform(N, -1, 1, gen), T=_uniform(N, 300, 3000, gen) if c["kT"] else None,
                U=_flow(c, gen) if c["velocity"] == "nodal" else None)


def _newton_inputs(c, seed):
    gen = _generator(seed)
    V = M.box_vertices(_nc(c), perturb=c["perturb"], seed=int(seed) & 0x7fffffff)
    d = _level_set(c, gen)
    N = _n_dofs(c)
    T = 1950.0 + 200.0 * torch.tanh(4.0 * d) + _uniform(N, -0.5, 0.5, gen)
    return dict(V=V, T=T, T_old=T - 2.0 - _uniform(N, 0, 1, gen), H=0.5 + 0.5 * torch.tanh(d / 0.1), U=_flow(c, gen),
                q=1e9 * torch.exp(-40.0 * (d - 0.1) ** 2))


def _problems(c, seed):
    r = np.random.Generator(np.random.PCG64(int(seed)))
    out = []
    for i in range(c["count"]):
        # sizes and degrees are the case's own (the work does not change with the seed)
        s = np.random.Generator(np.random.PCG64(1000 * c["count"] + i))
        n, p = int(s.integers(c["lo"], c["hi"] + 1)), int(s.integers(2, 5))
        k0 = float(np.exp(s.uniform(0.0, np.log(100.0))))
        kind = M._capi.OP_ADVDIFF if c["advdiff"] and i % 2 else M._capi.OP_HEAT
        pr = Problem(kind=kind, degree=p, nc=n, dt=DT, k0=k0, rel_tolerance=1e-12)
        b = r.uniform(-1.0, 1.0, (n * p + 1,) * 3)
        b[0], b[-1], b[:, 0], b[:, -1], b[:, :, 0], b[:, :, -1] = 0, 0, 0, 0, 0, 0
        out.append((pr, b.reshape(-1)))
    return out


@functools.lru_cache(maxsize=4)
def _refined(p, nx, ny, nz):
    """A box whose upper half (in z) is refined once: cells' corner weights,
    their DoFs, the hanging-node constraints and the boundary mask.  Nodes are
    identified on the finest integer lattice; equidistant nodes, degree 1 or 2."""
    half = nz // 2
    ix, iy, iz = (a.reshape(-1) for a in np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"))
    low = iz < half
    t = np.arange(p + 1)
    k, j, i = (a.reshape(-1) for a in np.meshgrid(t, t, t, indexing="ij"))
    node = np.stack([i, j, k], 1)  # x fastest
    unit = 2 * p  # lattice units of a coarse cell
    parent = np.stack([ix, iy, iz], 1)
    coarse = parent[low][:, None, :] * unit + 2 * node[None]
    oz, oy, ox = (a.reshape(-1) for a in np.meshgrid([0, 1], [0, 1], [0, 1], indexing="ij"))
    off = np.stack([ox, oy, oz], 1)
    fine = (parent[~low][:, None, None, :] * unit + off[None, :, None, :] * p + node[None, None]).reshape(-1, node.shape[0], 3)
    dims = np.array([nx, ny, nz]) * unit + 1
    at = np.concatenate([coarse, fine])
    key = at[..., 0] + dims[0] * (at[..., 1] + dims[1] * at[..., 2])
    ids, cells = np.unique(key, return_inverse=True)
    cells = cells.reshape(key.shape)
    pos = np.stack([ids % dims[0], ids // dims[0] % dims[1], ids // (dims[0] * dims[1])], 1)
    # hanging: on the interface plane, off the coarse node lattice
    on = np.nonzero((pos[:, 2] == half * unit) & np.any(pos[:, :2] % 2 != 0, axis=1))[0]
    z = np.linspace(0.0, 1.0, p + 1)
    cons = {}
    for g in on:
        x, y = pos[g, 0], pos[g, 1]
        cx, cy = min(x // unit, nx - 1), min(y // unit, ny - 1)
        wx, wy = _basis(z, (x - cx * unit) / unit), _basis(z, (y - cy * unit) / unit)
        ent = []
        for b in range(p + 1):
            for a in range(p + 1):
                w = wx[a] * wy[b]
                if abs(w) > 1e-13:
                    q = (cx * unit + 2 * a) + dims[0] * ((cy * unit + 2 * b) + dims[1] * half * unit)
                    ent.append((int(np.searchsorted(ids, q)), float(w)))
        cons[int(g)] = ent
    bnd = np.any((pos == 0) | (pos == dims - 1), axis=1).astype(np.uint8)
    cons = {g: e for g, e in cons.items() if not bnd[g]}
    # corners: coarse vertices, or their trilinear midpoints in a child
    c8 = np.stack([(np.arange(8) >> d) & 1 for d in range(3)], 1)
    ref = 0.5 * (off[:, None, :] + c8[None])  # child, corner
    wt = np.prod(np.where(c8[None, None] == 1, ref[:, :, None, :], 1 - ref[:, :, None, :]), axis=3)
    return dict(parent=parent, low=low, weights=wt, c8=c8, cells=cells, cons=cons, bnd=bnd, n=len(ids))


def _mapped_inputs(c, seed):
    t = _refined(c["p"], c["nx"], c["ny"], c["nz"])
    nc = _nc(c)
    V = M.box_vertices(nc, perturb=0.1, seed=int(seed) & 0x7fffffff).reshape(nc[2] + 1, nc[1] + 1, nc[0] + 1, 3)
    at = t["parent"][:, None, :] + t["c8"][None]
    C = V[at[..., 2], at[..., 1], at[..., 0]]
    corners = np.concatenate([C[t["low"]], np.einsum("kvw,ewd->ekvd", t["weights"], C[~t["low"]]).reshape(-1, 8, 3)])
    return dict(corners=corners, src=_uniform(t["n"], -1, 1, _generator(seed)), **t)


def _solver(kind, prec, **kw):
    # the library's default tolerances (1e-12 relative)
    return M.LinearSolverData(solver_type=kind, preconditioner_type=prec, **kw)


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    c, s = case, dict(case=case)
    if c["kind"] == "vmult":
        i = _vmult_inputs(c, seed)
        s["mesh"] = M.Mesh(i["V"], _nc(c), c["p"], i["mask"])
        prec = ("fp64", "fp32") if c["fp32"] else ("fp64",)
        vel = None if c["velocity"] == "none" else c["velocity"]
        if c["op"] == "heat":
            s["op"] = M.HeatDiffuseOperator(s["mesh"], DT, k_alpha=1e-3 if c["kT"] else 0.0, velocity=vel, precisions=prec)
            if c["kT"]:
                s["op"].set_temperature(i["T"])
        else:
            s["op"] = M.AdvectionDiffusionOperator(s["mesh"], DT, theta=0.5, diffusivity=1e-3, velocity=vel, precisions=prec)
            if c["velocity"] == "nodal":
                s["op"].set_velocity(i["U"])
        s["src"] = i["src"].float() if c["fp32"] else i["src"]
        s["dst"] = torch.empty_like(s["src"])
    elif c["kind"] == "mapped":
        i = _mapped_inputs(c, seed)
        s["mesh"] = M.MappedMesh(i["corners"], i["cells"], i["n"], c["p"], i["bnd"], i["cons"])
        s["op"] = M.HeatDiffuseOperator(s["mesh"], DT, precisions=("fp64", "fp32") if c["fp32"] else ("fp64",))
        s["src"] = i["src"].float() if c["fp32"] else i["src"]
        s["dst"] = torch.empty_like(s["src"])
    elif c["kind"] == "newton":
        i = _newton_inputs(c, seed)
        s["mesh"] = M.Mesh(i["V"], _nc(c), c["p"], _box_mask(_shape(c)))
        s["op"] = M.HeatDiffuseOperator(s["mesh"], 1e-5, velocity="nodal", material=LAW)
        s["op"].set_velocity(i["U"])
        s.update(T=i["T"], T_old=i["T_old"], H=i["H"], q=i["q"], rhs=torch.empty_like(i["T"]), dx=torch.empty_like(i["T"]),
                 data=_solver("GMRES", "Diagonal"))
    elif c["kind"] in ("cg", "cheb"):
        cheb = c["kind"] == "cheb"
        gen = _generator(seed)
        V = M.box_vertices(_nc(c), perturb=0.1 if cheb else 0.0, seed=int(seed) & 0x7fffffff)
        mask = _box_mask(_shape(c))
        s["mesh"] = M.Mesh(V, _nc(c), c["p"], mask)
        s["op"] = M.HeatDiffuseOperator(s["mesh"], DT, k_alpha=1e-3 if cheb else 0.0,
                                        precisions=("fp64", "fp32") if cheb else ("fp64",))
        N = _n_dofs(c)
        if cheb:
            s["T"] = _uniform(N, 300, 3000, gen)
            s["op"].set_temperature(s["T"])
        s["b"] = _uniform(N, -1, 1, gen) * torch.tensor(1.0 - mask, device="cuda")
        s["x"] = torch.empty_like(s["b"])
        s["data"] = _solver("CG", "Chebyshev", mixed_precision=True) if cheb else _solver("CG", "Diagonal")
    elif c["kind"] == "step":
        s["mesh"] = M.Mesh(M.box_vertices(_nc(c)), _nc(c), c["p"])
        s["op"] = M.AdvectionDiffusionOperator(s["mesh"], DT, theta=0.5, diffusivity=1e-3, velocity="vortex")
        s["phi"] = torch.tanh(_level_set(c, _generator(seed)) / 0.03)
        s.update(rhs=torch.empty_like(s["phi"]), x=torch.empty_like(s["phi"]), data=_solver("GMRES", "Diagonal"))
    else:
        s["problems"] = _problems(c, seed)
        s["batch"] = Batch(40 * 10**9, capacity=c["count"])
    return s


def run(s):
    c = s["case"]
    if c["kind"] in ("vmult", "mapped"):
        s["op"].vmult(s["dst"], s["src"])
        return s["dst"]
    if c["kind"] == "newton":
        op = s["op"]
        op.set_heaviside(s["H"])
        op.set_temperature_old(s["T_old"])
        op.set_temperature(s["T"])
        s["rhs"].zero_()
        op.create_rhs(s["rhs"], s["T_old"], s["q"])
        s["dx"].zero_()
        M.LinearSolver.solve(op, s["dx"], s["rhs"], s["data"])
        return s["rhs"], s["dx"]
    if c["kind"] in ("cg", "cheb"):
        s["x"].zero_()
        M.LinearSolver.solve(s["op"], s["x"], s["b"], s["data"])
        return s["x"]
    if c["kind"] == "step":
        s["rhs"].zero_()
        s["op"].create_rhs(s["rhs"], s["phi"])
        s["x"].copy_(s["phi"])
        M.LinearSolver.solve(s["op"], s["x"], s["rhs"], s["data"])
        return s["rhs"], s["x"]
    b = s["batch"]
    tickets = [b.submit(pr, rhs) for pr, rhs in s["problems"]]
    b.run()
    return [b.take(t, pr.n_dofs)[0] for t, (pr, _) in zip(tickets, s["problems"])]


# ------------------------------------------------------------------ the work of a pass
def work(case):
    """Inputs read once, outputs written once; the sum-factorised arithmetic of
    an apply is 24 n^4 + c n^3 per cell.  The solves count one apply and the
    vectors of a Krylov step for each of a typical number of iterations."""
    c = case

    def flops(p, cells, cq):
        return cells * (24.0 * (p + 1) ** 4 + cq * (p + 1) ** 3)

    if c["kind"] == "vmult":
        N, E, r = _n_dofs(c), int(np.prod(_nc(c))), 4 if c["fp32"] else 8
        vert = 8 * 3 * int(np.prod([n + 1 for n in _nc(c)])) if c["perturb"] else 0
        by = 2 * r * N + (8 * N if c["kT"] else 0) + (24 * N if c["velocity"] == "nodal" else 0) + vert
        return dict(bytes=by, flops=flops(c["p"], E, 45 if c["perturb"] else 20 + (40 if c["velocity"] != "none" else 0)))
    if c["kind"] == "mapped":
        E = c["nx"] * c["ny"] * (c["nz"] // 2 + 8 * (c["nz"] - c["nz"] // 2))
        N, r = E * c["p"] ** 3, 4 if c["fp32"] else 8
        return dict(bytes=2 * r * N + 4 * E * (c["p"] + 1) ** 3 + 24 * E, flops=flops(c["p"], E, 45))
    if c["kind"] == "batch":
        N = sum(pr.n_dofs for pr, _ in _problems(c, 0))
        f = sum(flops(pr.degree, pr.nc**3, 20) for pr, _ in _problems(c, 0))
        return dict(bytes=200 * 40.0 * N, flops=200 * f)
    N, E = _n_dofs(c), int(np.prod(_nc(c)))
    its, vec, cq = {"newton": (20, 200, 90), "cg": (27, 88, 20), "cheb": (90 * 5, 60, 45), "step": (18, 200, 60)}[c["kind"]]
    return dict(bytes=float(its) * vec * N, flops=its * flops(c["p"], E, cq))


# ------------------------------------------------------------------ values in 64 bits
def _gll(p):
    if p == 1:
        return np.array([0.0, 1.0])
    c = np.zeros(p + 1)
    c[p] = 1.0
    r = np.polynomial.legendre.legroots(np.polynomial.legendre.legder(c))
    return np.concatenate([[0.0], 0.5 * (np.sort(r) + 1.0), [1.0]])


def _basis(z, x):
    return np.array([np.prod([(x - z[k]) / (z[i] - z[k]) for k in range(len(z)) if k != i]) for i in range(len(z))])


def _tables(p):
    """Values and derivatives of the nodal basis at the Gauss points of [0,1]; points and weights."""
    z = _gll(p)
    x, w = np.polynomial.legendre.leggauss(p + 1)
    x, w = 0.5 * (x + 1.0), 0.5 * w
    S = np.array([_basis(z, t) for t in x])
    D = np.zeros_like(S)
    for q, t in enumerate(x):
        for i in range(p + 1):
            for l in range(p + 1):
                if l != i:
                    D[q, i] += np.prod([(t - z[k]) / (z[i] - z[k]) for k in range(p + 1) if k not in (i, l)]) / (z[i] - z[l])
    return S, D, x, w


class _Cells:
    """Element-wise operators in plain torch: corners (E, 8, 3), cell DoFs (E, n^3), x fastest."""

    def __init__(self, p, corners, dofs, N, chunk=8192):
        S, D, x, w = _tables(p)
        self.p, self.N, self.chunk = p, N, chunk
        self.S, self.D = (torch.tensor(a, device="cuda") for a in (S, D))
        self.x, self.w = x, torch.tensor(np.einsum("k,j,i->kji", w, w, w), device="cuda")
        self.corners, self.dofs = torch.as_tensor(corners, device="cuda"), torch.as_tensor(dofs, device="cuda").long()

    def chunks(self):
        for a in range(0, self.dofs.shape[0], self.chunk):
            yield slice(a, a + self.chunk)

    def geometry(self, sl):
        n = self.p + 1
        C = self.corners[sl]
        X = torch.tensor(self.x, device="cuda")
        J = torch.zeros((C.shape[0], n, n, n, 3, 3), dtype=F64, device="cuda")
        for v in range(8):
            b = [(v >> d) & 1 for d in range(3)]
            f = [X if b[d] else 1 - X for d in range(3)]
            g = [torch.ones_like(X) * (1.0 if b[d] else -1.0) for d in range(3)]
            for d in range(3):
                q = [g[e] if e == d else f[e] for e in range(3)]
                J[..., :, d] += C[:, v][:, None, None, None, :] * (q[2][:, None, None] * q[1][None, :, None] * q[0][None, None, :])[None, ..., None]
        det = torch.linalg.det(J)
        return det * self.w, torch.linalg.inv(J)

    def values(self, u, sl):
        n = self.p + 1
        v = u[self.dofs[sl]].reshape(-1, n, n, n)
        return torch.einsum("ck,bj,ai,ekji->ecba", self.S, self.S, self.S, v)

    def gradients(self, u, sl):
        n = self.p + 1
        v = u[self.dofs[sl]].reshape(-1, n, n, n)
        S, D = self.S, self.D
        return torch.stack([torch.einsum("ck,bj,ai,ekji->ecba", S, S, D, v), torch.einsum("ck,bj,ai,ekji->ecba", S, D, S, v),
                            torch.einsum("ck,bj,ai,ekji->ecba", D, S, S, v)], -1)

    def test(self, out, sl, val, flux):
        """out += the tests with N (val) and reference grad N (flux)."""
        S, D = self.S, self.D
        r = torch.einsum("ck,bj,ai,ecba->ekji", S, S, S, val)
        r += torch.einsum("ck,bj,ai,ecba->ekji", S, S, D, flux[..., 0])
        r += torch.einsum("ck,bj,ai,ecba->ekji", S, D, S, flux[..., 1])
        r += torch.einsum("ck,bj,ai,ecba->ekji", D, S, S, flux[..., 2])
        out.index_add_(0, self.dofs[sl].reshape(-1), r.reshape(-1))

    def operator(self, terms):
        """terms(sl, JxW, Ji) -> (m, b, k, f): weights of u N, (b . grad u) N, k grad u . grad N and (f u) . grad N."""
        kept = []
        for sl in self.chunks():
            JxW, Ji = self.geometry(sl)
            kept.append((sl, JxW, Ji, terms(sl, JxW, Ji)))

        def apply(u):
            out = torch.zeros(self.N, dtype=F64, device="cuda")
            for sl, JxW, Ji, (m, b, k, f) in kept:
                g = torch.einsum("ecbaxd,ecbax->ecbad", Ji, self.gradients(u, sl))
                uq = self.values(u, sl)
                val = m * JxW * uq
                if b is not None:
                    val = val + JxW * (b * g).sum(-1)
                fl = k[..., None] * g if torch.is_tensor(k) else k * g
                if f is not None:
                    fl = fl + f * uq[..., None]
                self.test(out, sl, val, torch.einsum("ecbaxd,ecbad->ecbax", Ji, JxW[..., None] * fl))
            return out

        return apply


def _lattice(c, V):
    nc, p = _nc(c), c["p"]
    iz, iy, ix = (a.reshape(-1) for a in np.meshgrid(*[np.arange(n) for n in nc[::-1]], indexing="ij"))
    c8 = np.stack([(np.arange(8) >> d) & 1 for d in range(3)], 1)
    at = np.stack([ix, iy, iz], 1)[:, None, :] + c8[None]
    corners = V.reshape(nc[2] + 1, nc[1] + 1, nc[0] + 1, 3)[at[..., 2], at[..., 1], at[..., 0]]
    t = np.arange(p + 1)
    k, j, i = (a.reshape(-1) for a in np.meshgrid(t, t, t, indexing="ij"))
    sh = _shape(c)
    dofs = (ix[:, None] * p + i) + sh[0] * ((iy[:, None] * p + j) + sh[1] * (iz[:, None] * p + k).astype(np.int64))
    return _Cells(p, corners, dofs, _n_dofs(c))


def _points(cells, sl):
    C = cells.corners[sl]
    X = torch.tensor(cells.x, device="cuda")
    out = 0
    for v in range(8):
        f = [X if (v >> d) & 1 else 1 - X for d in range(3)]
        out = out + C[:, v][:, None, None, None, :] * (f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :])[None, ..., None]
    return out


def _velocity(c, cells, sl, U):
    if c["velocity"] == "none":
        return None
    if c["velocity"] == "nodal":
        return torch.stack([cells.values(U.reshape(3, -1)[d], sl) for d in range(3)], -1)
    x = _points(cells, sl) * math.pi
    return torch.stack([torch.sin(x[..., 0]) * torch.cos(x[..., 1]), -torch.cos(x[..., 0]) * torch.sin(x[..., 1]),
                        torch.zeros_like(x[..., 0])], -1)


def _masked(apply, mask):
    if mask is None:
        return apply
    keep = torch.tensor(1.0 - mask.astype(np.float64), device="cuda")
    return lambda u: keep * apply(keep * u)


def _krylov(apply, b, x, invd, free=None, tol=1e-13, most=3000):
    """BiCGStab on the Jacobi-scaled system."""
    dot = lambda p, q: float(torch.dot(p, q))  # noqa: E731
    r = b - apply(x)
    target = tol * float(torch.linalg.vector_norm(r))
    for _ in range(4):  # restarts with the true residual
        rh, p, v = r.clone(), torch.zeros_like(r), torch.zeros_like(r)
        rho = al = om = 1.0
        for _ in range(most):
            new = dot(rh, r)
            if new == 0.0:
                break
            p = r + (new / rho) * (al / om) * (p - om * v)
            rho = new
            ph = invd * p
            v = apply(ph)
            al = rho / dot(rh, v)
            s = r - al * v
            sh = invd * s
            t = apply(sh)
            tt = dot(t, t)
            om = dot(t, s) / tt if tt else 0.0
            x = x + al * ph + om * sh
            r = s - om * t
            if om == 0.0 or float(torch.linalg.vector_norm(r)) <= 0.5 * target:
                break
        r = b - apply(x)
        if float(torch.linalg.vector_norm(r)) <= target:
            break
    return x


def _jacobi(cells, kept, mask):
    """Inverse of a lumped estimate of the diagonal: element mass and stiffness weights."""
    d = torch.zeros(cells.N, dtype=F64, device="cuda")
    S2, D2 = cells.S**2, cells.D**2
    for sl, JxW, Ji, m, k in kept:
        G = torch.einsum("ecbaxd,ecbaxd->ecbax", Ji, Ji) * JxW[..., None] * (k[..., None] if torch.is_tensor(k) else k)
        r = torch.einsum("ck,bj,ai,ecba->ekji", S2, S2, S2, m * JxW)
        r += torch.einsum("ck,bj,ai,ecba->ekji", S2, S2, D2, G[..., 0])
        r += torch.einsum("ck,bj,ai,ecba->ekji", S2, D2, S2, G[..., 1])
        r += torch.einsum("ck,bj,ai,ecba->ekji", D2, S2, S2, G[..., 2])
        d.index_add_(0, cells.dofs[sl].reshape(-1), r.reshape(-1))
    if mask is not None:
        d[torch.tensor(mask.astype(bool), device="cuda")] = 1.0
    return 1.0 / d


def _solve_cells(cells, terms, mask, b, x0):
    kept = []

    def keep(sl, JxW, Ji):
        t = terms(sl, JxW, Ji)
        kept.append((sl, JxW, Ji, t[0], t[2]))
        return t

    A = _masked(cells.operator(keep), mask)
    return _krylov(A, b, x0, _jacobi(cells, kept, mask))


def _line_matrices(p, n, weight=None):
    """1D mass (weighted at the points), stiffness and advection matrices on n cells of [0,1]."""
    S, D, x, w = _tables(p)
    N = n * p + 1
    Mm, K, A = np.zeros((N, N)), np.zeros((N, N)), np.zeros((N, N))
    for e in range(n):
        f = np.ones(p + 1) if weight is None else weight((e + x) / n)
        sl = slice(e * p, e * p + p + 1)
        Mm[sl, sl] += np.einsum("q,qi,qj->ij", w * f / n, S, S)
        K[sl, sl] += np.einsum("q,qi,qj->ij", w * f * n, D, D)
        A[sl, sl] += np.einsum("q,qi,qj->ij", w * f, S, D)
    return tuple(torch.tensor(a, device="cuda") for a in (Mm, K, A))


def _kron(az, ay, ax, u):
    v = torch.matmul(u, ax.T)
    v = torch.matmul(ay, v)
    return torch.matmul(az, v.reshape(v.shape[0], -1)).reshape(v.shape)


def _box_heat_solve(p, nc, k0, b):
    """(M/dt + k0 K) x = b on the unit box with zero boundary values, by the lines' eigenvectors."""
    Q, lam = [], []
    for n in nc:
        Mm, K, _ = _line_matrices(p, n)
        L = torch.linalg.cholesky(Mm[1:-1, 1:-1])
        Li = torch.linalg.inv(L)
        e, W = torch.linalg.eigh(Li @ K[1:-1, 1:-1] @ Li.T)
        Q.append(Li.T @ W)
        lam.append(e)
    sh = tuple(n * p + 1 for n in nc)[::-1]
    r = torch.as_tensor(b, device="cuda").reshape(sh)[1:-1, 1:-1, 1:-1].contiguous()
    t = _kron(Q[2].T, Q[1].T, Q[0].T, r)
    t = t / (1.0 / DT + k0 * (lam[2][:, None, None] + lam[1][None, :, None] + lam[0][None, None, :]))
    x = torch.zeros(sh, dtype=F64, device="cuda")
    x[1:-1, 1:-1, 1:-1] = _kron(Q[2], Q[1], Q[0], t)
    return x.reshape(-1)


def _box_level_set(c):
    """The vortex level-set forms on the unit box as sums of line products."""
    p, (nx, ny, nz) = c["p"], _nc(c)
    sin, cos = (lambda x: np.sin(np.pi * x)), (lambda x: np.cos(np.pi * x))
    X, Xs, Xc = _line_matrices(p, nx), _line_matrices(p, nx, sin), _line_matrices(p, nx, cos)
    Y, Ys, Yc = _line_matrices(p, ny), _line_matrices(p, ny, sin), _line_matrices(p, ny, cos)
    Z = _line_matrices(p, nz)

    def form(mass, adv, diff):
        def apply(u):
            v = u.reshape(_shape(c)[::-1])
            r = _kron(Z[0], Y[0], mass * X[0] + diff * X[1], v) + _kron(Z[0], diff * Y[1], X[0], v)
            r += _kron(diff * Z[1], Y[0], X[0], v)
            r += _kron(Z[0], Yc[0], adv * Xs[2], v) - _kron(Z[0], adv * Ys[2], Xc[0], v)
            return r.reshape(-1)

        return apply

    d = [m[0].diag() for m in (Z, Y, X)], [m[1].diag() for m in (Z, Y, X)]
    o = lambda a, b, e: (a[:, None, None] * b[None, :, None] * e[None, None, :]).reshape(-1)  # noqa: E731
    M3, K3 = d
    diag = o(M3[0], M3[1], M3[2]) / DT + 0.5e-3 * (o(K3[0], M3[1], M3[2]) + o(M3[0], K3[1], M3[2]) + o(M3[0], M3[1], K3[2]))
    return form, 1.0 / diag


def _law(T, H):
    """Density, capacity and conductivity of the gas/liquid/solid law and their T derivatives."""
    dT = LAW["liquidus"] - LAW["solidus"]
    fs = torch.clamp((LAW["liquidus"] - T) / dT, 0.0, 1.0)
    inside = ((fs > 0) & (fs < 1)).to(F64)
    s, ds = 3 * fs**2 - 2 * fs**3, -(6 * fs - 6 * fs**2) / dT * inside
    out = []
    for g, l, so in (LAW["rho"], LAW["cp"], LAW["k"]):
        out.append(((1 - H) * g + H * (l + (so - l) * s), H * (so - l) * ds))
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "vmult":
        i = _vmult_inputs(c, seed)
        cells = _lattice(c, i["V"])

        def terms(sl, JxW, Ji):
            b = _velocity(c, cells, sl, i["U"])
            if c["op"] == "heat":
                return 1.0 / DT, b, 1.0 + 1e-3 * cells.values(i["T"], sl) if c["kT"] else 1.0, None
            return 1.0 / DT, 0.5 * b, 0.5e-3, None

        src = i["src"].float().double() if c["fp32"] else i["src"]
        out = torch.zeros_like(src)
        keep = 1.0 if i["mask"] is None else torch.tensor(1.0 - i["mask"].astype(np.float64), device="cuda")
        for sl in cells.chunks():  # chunk by chunk: the whole geometry of the largest mesh is tens of GB
            part = _Cells(c["p"], cells.corners[sl], cells.dofs[sl], cells.N, cells.chunk)
            part_terms = lambda s_, J_, I_, sl=sl: terms(sl, J_, I_)  # noqa: E731
            out += part.operator(part_terms)(keep * src)
        return keep * out
    if c["kind"] == "mapped":
        i = _mapped_inputs(c, seed)
        cells = _Cells(c["p"], i["corners"], i["cells"], i["n"])
        src = i["src"].float().double() if c["fp32"] else i["src"]
        keep = torch.tensor(1.0 - i["bnd"].astype(np.float64), device="cuda")
        g = torch.tensor([k for k, e in i["cons"].items() for _ in e], device="cuda")
        m = torch.tensor([q for e in i["cons"].values() for q, _ in e], device="cuda")
        w = torch.tensor([v for e in i["cons"].values() for _, v in e], dtype=F64, device="cuda")
        u = keep * src
        u[g] = 0.0
        u = u.index_add(0, g, w * u[m])
        out = torch.zeros_like(u)
        for sl in cells.chunks():
            part = _Cells(c["p"], cells.corners[sl], cells.dofs[sl], cells.N, cells.chunk)
            out += part.operator(lambda s_, J_, I_: (1.0 / DT, None, 1.0, None))(u)
        out = out.index_add(0, m, w * out[g])
        out[g] = 0.0
        return keep * out
    if c["kind"] == "newton":
        i = _newton_inputs(c, seed)
        cells, mask, dt = _lattice(c, i["V"]), _box_mask(_shape(c)), 1e-5
        keep = torch.tensor(1.0 - mask.astype(np.float64), device="cuda")
        rhs = torch.zeros_like(i["T"])

        def fields(sl, Ji):
            T, H, b = cells.values(i["T"], sl), cells.values(i["H"], sl), _velocity(dict(velocity="nodal"), cells, sl, i["U"])
            g = torch.einsum("ecbaxd,ecbax->ecbad", Ji, cells.gradients(i["T"], sl))
            (r, dr), (cp, dc), (k, dk) = _law(T, H)
            return T, g, b, r * cp, dr * cp + r * dc, k, dk

        def terms(sl, JxW, Ji):
            T, g, b, rc, drc, k, dk = fields(sl, Ji)
            inc = (T - cells.values(i["T_old"], sl)) / dt + (b * g).sum(-1)
            val = rc * inc - cells.values(i["q"], sl)
            cells.test(rhs, sl, -JxW * val, -torch.einsum("ecbaxd,ecbad->ecbax", Ji, (JxW * k)[..., None] * g))
            return rc / dt + drc * inc, rc[..., None] * b, k, dk[..., None] * g

        kept = []

        def both(sl, JxW, Ji):
            t = terms(sl, JxW, Ji)
            kept.append((sl, JxW, Ji, t[0], t[2]))
            return t

        A = _masked(cells.operator(both), mask)
        rhs = keep * rhs
        return rhs, _krylov(A, rhs, torch.zeros_like(rhs), _jacobi(cells, kept, mask))
    if c["kind"] == "cg":
        b = _uniform(_n_dofs(c), -1, 1, _generator(seed)) * torch.tensor(1.0 - _box_mask(_shape(c)), device="cuda")
        return _box_heat_solve(c["p"], _nc(c), 1.0, b)
    if c["kind"] == "cheb":
        gen, mask = _generator(seed), _box_mask(_shape(c))
        cells = _lattice(c, M.box_vertices(_nc(c), perturb=0.1, seed=int(seed) & 0x7fffffff))
        T = _uniform(_n_dofs(c), 300, 3000, gen)
        b = _uniform(_n_dofs(c), -1, 1, gen) * torch.tensor(1.0 - mask, device="cuda")
        return _solve_cells(cells, lambda sl, J, I: (1.0 / DT, None, 1.0 + 1e-3 * cells.values(T, sl), None), mask, b,
                            torch.zeros_like(b))
    if c["kind"] == "step":
        phi = torch.tanh(_level_set(c, _generator(seed)) / 0.03)
        form, invd = _box_level_set(c)
        rhs = form(1.0 / DT, -0.5, -0.5e-3)(phi)
        return rhs, _krylov(form(1.0 / DT, 0.5, 0.5e-3), rhs, phi.clone(), invd)
    if c["advdiff"]:
        return None
    return [_box_heat_solve(pr.degree, (pr.nc,) * 3, pr.k0, b) for pr, b in _problems(c, seed)]
