"""The work that programs have this library do, as cases that can be timed and checked.

Each case is one call (or the few calls of one step) through the public entry points, at sizes from
the repository's own workloads: heat cubes of 8 to 100 hexes per side, the 64x32x32 elasticity beam,
uneven batches of 8..40 hexes per side, a 40^3 transient, GMRES(30) on a convection-diffusion grid,
several right-hand sides of one matrix, the numeric assembly of a 6M-tet mesh and one application of
the learned preconditioner.

  kind       what runs
  solve      Context.solve on a device-resident matrix, right-hand side and solution
  dropin     Solver.solve from host arrays, the mirror of RMatrixSolver::solve: values and b in, x out
  refresh    Matrix.update_values + Context.solve from host arrays (same pattern, new values)
  transient  one backward-Euler step: numeric assembly, solve from the previous temperatures, write-back
  beam       elasticity: numeric assembly and solve
  gmres      Context.solve with GMRES(30) on a nonsymmetric matrix, device-resident
  batch      Batch.solve: many systems of uneven size at once, device-resident
  multi      Context.solve_multi: k right-hand sides of one matrix, device-resident
  assemble   numeric assembly of a heat system from device-resident element fields
  learned    one application of the learned preconditioner (inference)

Matrices, right-hand sides and fields are made from the seed; the mesh and the assembly plan of a size
are made once and kept, as a program keeps them.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "range-solver-lib_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import rsg  # noqa: E402
from rsg import workloads as W  # noqa: E402
from rsg.learned import Learned  # noqa: E402

PREC = {"none": 0, "jacobi": rsg.PREC_JACOBI, "amg": rsg.PREC_AMG}
RHO_C, DT = 1.0, 1.0e-3


def listed():
    return [
        # the smallest call: a coarse model or a cell problem, where launches and latency are all there is
        dict(name="heat8_fp64", kind="solve", hexes=8, sigma=1.0, precision="fp64", prec="jacobi"),
        # a small steady conduction model through the drop-in interface, host arrays in and out
        dict(name="heat20_dropin", kind="dropin", hexes=20, sigma=0.0, precision="fp64", prec="jacobi"),
        # one step of a 40^3 transient: re-assembly, solve, write-back, nothing leaves the GPU
        dict(name="heat40_transient", kind="transient", hexes=40, sigma=0.0, precision="mixed", prec="jacobi"),
        # the plain FP64 drop-in on a 1M-unknown heterogeneous conduction system
        dict(name="heat100_fp64", kind="solve", hexes=100, sigma=1.5, precision="fp64", prec="jacobi"),
        # the same system with the fastest solver: mixed precision and the multilevel preconditioner
        dict(name="heat100_amg", kind="solve", hexes=100, sigma=1.5, precision="mixed", prec="amg"),
        # a mid-size system whose new values and right-hand side come from the host each time
        dict(name="heat60_refresh_amg", kind="refresh", hexes=60, sigma=1.5, precision="mixed", prec="amg"),
        # linear elasticity: assembly and FP64 solve of the clamped beam
        dict(name="beam64", kind="beam", nx=64, ny=32, nz=32),
        # the nonsymmetric systems of the fluid solver: restarted GMRES with Jacobi, a ragged grid size
        dict(name="gmres61", kind="gmres", grid=61, precision="fp64"),
        # independent meshes of uneven size in one call
        dict(name="batch24", kind="batch", systems=24, lo=8, hi=40, sigma=1.0, precision="mixed"),
        # several load cases of one stiffness matrix
        dict(name="multi60x8", kind="multi", hexes=60, sigma=1.5, k=8),
        # re-assembly of a 6M-tet mesh
        dict(name="assemble100", kind="assemble", hexes=100, sigma=1.5),
        # one application of the shipped learned preconditioner
        dict(name="learned60", kind="learned", hexes=60, sigma=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "dropin", "refresh", "transient", "beam", "gmres", "batch", "multi",
                       "assemble", "learned"])
    sigma = round(rng.uniform(0.5, 1.5), 2)
    if kind == "solve":
        precision, prec = rng.choice([("fp64", "jacobi"), ("mixed", "jacobi"), ("mixed", "amg")])
        return dict(kind=kind, hexes=_log_int(rng, 6, 96), sigma=sigma, precision=precision, prec=prec)
    if kind == "dropin":
        return dict(kind=kind, hexes=_log_int(rng, 6, 40), sigma=sigma, precision="fp64", prec="jacobi")
    if kind == "refresh":
        precision, prec = rng.choice([("fp64", "jacobi"), ("mixed", "amg")])
        return dict(kind=kind, hexes=_log_int(rng, 20, 60), sigma=sigma, precision=precision, prec=prec)
    if kind == "transient":
        return dict(kind=kind, hexes=_log_int(rng, 10, 50), sigma=sigma, precision=rng.choice(["fp64", "mixed"]),
                    prec="jacobi")
    if kind == "beam":
        ny = _log_int(rng, 5, 30)
        return dict(kind=kind, nx=2 * ny + rng.randint(0, 3), ny=ny, nz=ny + rng.randint(0, 2))
    if kind == "gmres":
        return dict(kind=kind, grid=_log_int(rng, 12, 60), precision=rng.choice(["fp64", "mixed"]))
    if kind == "batch":
        return dict(kind=kind, systems=_log_int(rng, 4, 24), lo=rng.randint(6, 12), hi=rng.randint(20, 40), sigma=sigma,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "multi":
        return dict(kind=kind, hexes=_log_int(rng, 10, 60), sigma=sigma, k=rng.choice([2, 3, 4, 7, 8]))
    if kind == "assemble":
        return dict(kind=kind, hexes=_log_int(rng, 10, 96), sigma=sigma)
    return dict(kind="learned", hexes=_log_int(rng, 10, 60), sigma=sigma)


# ---------------------------------------------------------------- inputs --------------------


@functools.lru_cache(maxsize=None)
def _ctx():
    ctx = rsg.Context(torch.cuda.current_device())
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)  # torch's copies and the library's kernels in one order
    return ctx, stream


@functools.lru_cache(maxsize=4)
def _cube(n):
    return W.heat_cube(n, source="unit")


@functools.lru_cache(maxsize=4)
def _beam(nx, ny, nz):
    return W.stress_beam(nx, ny, nz)


@functools.lru_cache(maxsize=2)
def _plan(n):
    """Assembly plan of the unit cube and its pattern on the device."""
    ctx, stream = _ctx()
    p = _cube(n)
    asm = rsg.Assembly.heat(ctx, p)
    fields = {k: torch.from_numpy(getattr(p, k)).cuda() for k in ("k_e", "q_e", "rhoc_e", "node_t")}
    b = torch.empty(p.n_free, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    A = asm.assemble(p, b, inputs_on_device=fields)
    rp, ci, _ = A.to_host()
    pattern = (torch.from_numpy(rp.view(np.int32)).cuda(), torch.from_numpy(ci.view(np.int32)).cuda())
    torch.cuda.synchronize()
    return p, asm, pattern, (rp, ci)


class _DeviceArray:
    def __init__(self, ptr, count, owner):
        self.owner = owner  # the tensor made of it keeps the memory's owner
        self.__cuda_array_interface__ = dict(shape=(count,), typestr="<f8", data=(ptr, False), version=3)


def _values(A, owner):
    """The value array of the matrix that `owner` holds, as a tensor."""
    return torch.as_tensor(_DeviceArray(A.device_arrays()[2], A.nnz, owner), device="cuda")


def _fields(n, sigma, seed):
    """Element conductivity (lognormal), nodal source averaged per tet, on the device."""
    p = _cube(n)
    g = torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1))
    nt = p.mesh.n_tets
    f64 = dict(dtype=torch.float64, device="cuda")
    if sigma:
        k_e = torch.exp(sigma * torch.randn(nt, generator=g, **f64))
        s = torch.rand(p.mesh.n_nodes, generator=g, **f64)
        q_e = s[torch.from_numpy(p.mesh.tets.astype(np.int64)).cuda()].mean(dim=1)
    else:  # uniform material and load, their size set by the seed
        k_e = torch.full((nt,), 0.5 + float(torch.rand(1, generator=g, **f64)), **f64)
        q_e = torch.full((nt,), 0.5 + float(torch.rand(1, generator=g, **f64)), **f64)
    return dict(k_e=k_e.contiguous(), q_e=q_e.contiguous(), rhoc_e=torch.full((nt,), RHO_C, **f64),
                node_t=torch.from_numpy(p.node_t).cuda())


def _start_temperature(n, seed):
    """A smooth temperature field between the two faces, as a transient has after some steps."""
    p = _cube(n)
    ph = 0.1 + (seed % 97) / 97.0
    x, y, z = (torch.from_numpy(np.ascontiguousarray(p.mesh.xyz[:, i])).cuda() for i in range(3))
    t = x + 0.3 * torch.sin(math.pi * x) * torch.cos(math.pi * (y + ph)) * torch.cos(2 * math.pi * z)
    fixed = torch.from_numpy(p.disabled).cuda()
    return torch.where(fixed, torch.from_numpy(p.node_t).cuda(), t).contiguous()


def _heat_values(n, sigma, seed):
    """(values, b) of one heat system as device tensors, from the kept plan."""
    p, asm, _, _ = _plan(n)
    f = _fields(n, sigma, seed)
    b = torch.empty(p.n_free, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    A = asm.assemble(p, b, inputs_on_device=f)
    _ctx()[0].sync()
    return _values(A, asm).clone(), b


def _conv_diff(m, seed):
    """7-point convection-diffusion on an m^3 grid with a swirling field: (rp, ci, val, b) on the device."""
    n, h = m ** 3, 1.0 / (m + 1)
    g = torch.Generator(device="cuda").manual_seed(7919 * (seed + 1))
    f64 = dict(dtype=torch.float64, device="cuda")
    t = (torch.arange(m, **f64) + 1) * h
    X, Y, Z = torch.meshgrid(t, t, t, indexing="ij")
    amp = 2.0 * (0.6 + 0.4 * float(torch.rand(1, generator=g, **f64))) / h
    w = torch.stack([torch.sin(math.pi * Y), -torch.sin(math.pi * X), 0.5 * torch.cos(math.pi * Z)]) * amp
    idx = torch.arange(n, device="cuda").reshape(m, m, m)
    rows, cols, vals = [idx.reshape(-1)], [idx.reshape(-1)], [torch.full((n,), 6.0 / h ** 2, **f64)]
    for ax in range(3):
        a, b = idx.narrow(ax, 0, m - 1).reshape(-1), idx.narrow(ax, 1, m - 1).reshape(-1)
        wa = w[ax].reshape(-1)
        rows += [a, b]
        cols += [b, a]
        vals += [-1.0 / h ** 2 + wa[a] / (2.0 * h), -1.0 / h ** 2 - wa[b] / (2.0 * h)]
    S = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals), (n, n)).coalesce()
    r, c = S.indices()
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    rhs = torch.randn(n, generator=g, **f64)
    return rp.to(torch.int32), c.to(torch.int32).contiguous(), S.values().contiguous(), rhs


def _batch_sizes(case, seed):
    """Hexes per side of the batch's systems: fixed by the case, spread over [lo, hi]."""
    g = np.random.default_rng(17)
    return [int(v) for v in g.integers(case["lo"], case["hi"] + 1, case["systems"])]


def _beam_fields(case, seed):
    """The beam with its modulus and traction set by the seed."""
    p = _beam(case["nx"], case["ny"], case["nz"])
    g = np.random.default_rng(seed + 5)
    e = 210e9 * (0.8 + 0.4 * g.random())
    t = np.array([0.2e6 * g.standard_normal(), 0.2e6 * g.standard_normal(), -1.0e6])
    nt = p.mesh.n_tets
    f64 = dict(dtype=torch.float64, device="cuda")
    return p, dict(e_mod=torch.full((nt,), e, **f64), nu=torch.full((nt,), 0.3, **f64),
                   rho_e=torch.full((nt,), 7850.0, **f64), gravity=torch.zeros(3, **f64),
                   texp_e=torch.zeros(nt, **f64), dtemp_e=torch.zeros(nt, **f64),
                   traction=torch.from_numpy(np.tile(t, (p.tris.shape[0], 1))).cuda(),
                   node_u=torch.zeros(3 * p.mesh.n_nodes, **f64))


def _conf(case, **kw):
    return rsg.make_conf(n_outer=50000, stop_rule="true", rtol=case.get("rtol", 1e-10),
                         precision=case.get("precision", "fp64"), **kw)


# ---------------------------------------------------------------- prepare / run --------------


def prepare(case, seed):
    ctx, stream = _ctx()
    kind = case["kind"]
    s = dict(kind=kind, ctx=ctx, stream=stream)
    if kind in ("solve", "multi", "learned"):
        p, _, (rp, ci), _ = _plan(case["hexes"])
        val, b = _heat_values(case["hexes"], case["sigma"], seed)
        s.update(A=ctx.matrix(rp, ci, val))
        if kind == "solve":
            s.update(b=b, x=torch.zeros_like(b), conf=_conf(case), prec=PREC[case["prec"]])
        elif kind == "multi":
            B = _load_cases(case, seed, b)
            s.update(B=B, X=torch.zeros_like(B), conf=_conf(case))
        else:
            g = torch.Generator(device="cuda").manual_seed(31 * seed + 7)
            r = torch.randn(p.n_free, generator=g, dtype=torch.float64, device="cuda")
            s.update(M=_model(ctx), r=r, z=torch.empty_like(r), xyz=_free_xyz(p))
    elif kind in ("dropin", "refresh"):
        _, _, (drp, dci), (rp, ci) = _plan(case["hexes"])
        val, b = _heat_values(case["hexes"], case["sigma"], seed)
        s.update(val=val.cpu().numpy(), b=b.cpu().numpy(), conf=_conf(case), prec=PREC[case["prec"]])
        if kind == "dropin":
            s.update(solver=rsg.Solver(ctx, s["conf"]), rp=rp, ci=ci)
        else:
            s.update(A=ctx.matrix(drp, dci, val))
    elif kind == "transient":
        p, f = _transient_inputs(case, seed)
        free = np.flatnonzero(p.book != 0xFFFFFFFF)
        order = torch.from_numpy(free[np.argsort(p.book[free])]).cuda()
        s.update(p=p, asm=rsg.Assembly.heat(ctx, p), f=f, t=f["node_t"].clone(), conf=_conf(case),
                 x0=f["node_t"][order].contiguous(), x=torch.empty(p.n_free, dtype=torch.float64, device="cuda"),
                 b=torch.empty(p.n_free, dtype=torch.float64, device="cuda"))
        s["f"] = dict(f, node_t=s["t"])
        s["t0"] = f["node_t"]
    elif kind == "beam":
        p, f = _beam_fields(case, seed)
        s.update(p=p, asm=rsg.Assembly.stress(ctx, p), f=f, conf=_conf(case),
                 x=torch.zeros(p.n_free, dtype=torch.float64, device="cuda"),
                 b=torch.empty(p.n_free, dtype=torch.float64, device="cuda"))
    elif kind == "gmres":
        rp, ci, val, b = _conv_diff(case["grid"], seed)
        torch.cuda.synchronize()
        s.update(A=ctx.matrix(rp, ci, val), b=b, x=torch.zeros_like(b), prec=rsg.PREC_JACOBI,
                 conf=_conf(case, solver="gmres", n_inner=30))
    elif kind == "batch":
        systems, bs = [], []
        for i, n in enumerate(_batch_sizes(case, seed)):
            val, b = _heat_values(n, case["sigma"], 1000 * seed + i)
            rp, ci = _plan(n)[3]
            systems.append((rp, ci, val.cpu().numpy()))
            bs.append(b)
        b = torch.cat(bs)
        s.update(batch=rsg.Batch(ctx, systems), b=b, x=torch.zeros_like(b), conf=_conf(case))
    else:
        p = _cube(case["hexes"])
        s.update(p=p, asm=rsg.Assembly.heat(ctx, p), f=_fields(case["hexes"], case["sigma"], seed),
                 b=torch.empty(p.n_free, dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "dropin":
        x, _ = s["solver"].solve((s["rp"], s["ci"], s["val"]), s["b"], prec=s["prec"])
        return x
    if kind == "refresh":
        s["A"].update_values(s["val"])
        x, _ = ctx.solve(s["A"], s["b"], conf=s["conf"], prec=s["prec"])
        return x
    with torch.cuda.stream(s["stream"]):
        if kind in ("solve", "gmres"):
            s["x"].zero_()
            ctx.solve(s["A"], s["b"], s["x"], conf=s["conf"], prec=s["prec"])
            return s["x"]
        if kind == "transient":
            s["t"].copy_(s["t0"])
            s["x"].copy_(s["x0"])
            A = s["asm"].assemble(s["p"], s["b"], inputs_on_device=s["f"])
            ctx.solve(A, s["b"], s["x"], conf=s["conf"])
            ctx.check(ctx.lib.rsg_assembly_scatter(ctx.h, s["asm"].h, rsg._ptr(s["x"]), rsg._ptr(s["t"])), "scatter")
            return s["t"]
        if kind == "beam":
            s["x"].zero_()
            A = s["asm"].assemble(s["p"], s["b"], inputs_on_device=s["f"])
            ctx.solve(A, s["b"], s["x"], conf=s["conf"])
            return s["x"]
        if kind == "batch":
            s["x"].zero_()
            s["batch"].solve(s["b"], s["x"], conf=s["conf"])
            return s["x"]
        if kind == "multi":
            s["X"].zero_()
            ctx.solve_multi(s["A"], s["B"], s["X"], conf=s["conf"])
            return s["X"]
        if kind == "assemble":
            A = s["asm"].assemble(s["p"], s["b"], inputs_on_device=s["f"])
            return {"b": s["b"], "values": _values(A, s["asm"])}
        s["M"].apply(s["A"], s["r"], s["z"], s["xyz"])
        return s["z"]


def _load_cases(case, seed, b):
    g = torch.Generator(device="cuda").manual_seed(131 * seed + 3)
    B = torch.randn(case["k"], b.numel(), generator=g, dtype=torch.float64, device="cuda") * float(b.abs().mean())
    B[0] = b
    return B.contiguous()


def _transient_inputs(case, seed):
    import copy
    p = copy.copy(_cube(case["hexes"]))
    p.transient, p.alpha, p.dt = True, 1.0, DT
    f = _fields(case["hexes"], case["sigma"], seed)
    f["node_t"] = _start_temperature(case["hexes"], seed)
    return p, f


@functools.lru_cache(maxsize=1)
def _model(ctx):
    return Learned.load(ctx, os.path.join(_PKG, "rsg", "models", "heat_family_60.npz"))


@functools.lru_cache(maxsize=4)
def _free_xyz_of(n):
    p = _cube(n)
    free = np.flatnonzero(p.book != 0xFFFFFFFF)
    return torch.from_numpy(np.ascontiguousarray(p.mesh.xyz[free[np.argsort(p.book[free])]])).cuda()


def _free_xyz(p):
    return _free_xyz_of(p.mesh.nx)


# ---------------------------------------------------------------- work ----------------------

# CG iterations to 1e-10 grow with the hexes per side: measured 799 at 100 hexes (sigma 1.5, Jacobi).
# The work of a solve is one matrix pass and the vector passes of its iterations.


def _heat_size(n):
    rows = (n - 1) * (n + 1) ** 2
    return rows, int(14.76 * rows)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "dropin", "refresh", "transient"):
        n, nnz = _heat_size(case["hexes"])
        vb = 8 if case["precision"] == "fp64" else 4
        if case["prec"] == "amg":
            its, passes, vecs = 32, 4, 20
        else:
            its = int((8.0 if case["sigma"] else 3.5) * case["hexes"]) if kind != "transient" else 55
            passes, vecs = 1, 12
        per = passes * nnz * (vb + 2) + vecs * n * vb
        extra = nnz * 8 + 2 * n * 8 if kind in ("dropin", "refresh", "transient") else 0
        return dict(bytes=its * per + extra, flops=its * (passes * 2 * nnz + vecs * n))
    if kind == "beam":
        n = 3 * case["nx"] * (case["ny"] + 1) * (case["nz"] + 1)
        nnz, its = 43 * n, 19 * case["nx"]
        return dict(bytes=its * (nnz * 10 + 12 * n * 8), flops=its * (2 * nnz + 12 * n))
    if kind == "gmres":
        n, vb = case["grid"] ** 3, 8 if case["precision"] == "fp64" else 4
        its = 9 * case["grid"]
        return dict(bytes=its * (7 * n * (vb + 2) + (2 * 16 + 5) * n * vb), flops=its * (14 + 4 * 16) * n)
    if kind == "batch":
        per = 0.0
        vb = 8 if case["precision"] == "fp64" else 4
        for h in _batch_sizes(case, 0):
            n, nnz = _heat_size(h)
            per += 8.0 * h * (nnz * (vb + 2) + 12 * n * vb)
        return dict(bytes=per, flops=per / 4)
    if kind == "multi":
        n, nnz = _heat_size(case["hexes"])
        its = 8 * case["hexes"]
        return dict(bytes=its * (nnz * 10 + case["k"] * 12 * n * 8), flops=its * case["k"] * (2 * nnz + 12 * n))
    if kind == "assemble":
        n, nnz = _heat_size(case["hexes"])
        nt = 6 * case["hexes"] ** 3
        return dict(bytes=nt * (16 + 3 * 8) + n * 32 + nnz * 8 + n * 8, flops=nt * 150)
    n, nnz = _heat_size(case["hexes"])
    return dict(bytes=6 * (n * 256 + nnz * 8) + n * 48, flops=6 * (2 * nnz * 64 + 2 * n * 128 * 64))


# ---------------------------------------------------------------- 64-bit values --------------


def _csr(rows, cols, vals, n):
    A = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n, n)).coalesce()
    return A.to_sparse_csr(), A


def _tet_geometry(p):
    xyz = torch.from_numpy(p.mesh.xyz).cuda()
    t = torch.from_numpy(p.mesh.tets.astype(np.int64)).cuda()
    E = xyz[t[:, 1:]] - xyz[t[:, :1]]  # rows: edges from node 0
    det = torch.linalg.det(E)
    g = torch.linalg.inv(E).transpose(1, 2)  # gradients of the shape functions 1..3
    G = torch.cat([-g.sum(dim=1, keepdim=True), g], dim=1)
    return t, G, det.abs() / 6.0


def _heat_system(p, f, transient=False):
    """Linear-tetrahedron heat conduction (theta = 1 when transient) with fixed nodes lifted: (A csr, A coo, b)."""
    t, G, V = _tet_geometry(p)
    K = torch.einsum("emi,eni->emn", G, G) * (f["k_e"] * V)[:, None, None]
    fe = (f["q_e"] * V / 4.0)[:, None].expand(-1, 4)
    T = f["node_t"][t]
    if transient:
        M = (torch.ones(4, 4, dtype=V.dtype, device=V.device) + torch.eye(4, dtype=V.dtype, device=V.device)) / 20.0
        M = M[None] * (f["rhoc_e"] * V)[:, None, None]
        be = p.dt * fe + torch.einsum("emn,en->em", M, T)
        K = M + p.dt * K
    else:
        be = fe
    book = torch.from_numpy(p.book.astype(np.int64)).cuda()
    pos = torch.where(book == 0xFFFFFFFF, torch.full_like(book, -1), book)[t]
    fixed = pos < 0
    be = be - torch.einsum("emn,en->em", K, torch.where(fixed, T, torch.zeros_like(T)))
    b = torch.zeros(p.n_free, dtype=torch.float64, device="cuda")
    b.index_add_(0, pos[~fixed], be[~fixed])
    r, c = pos[:, :, None].expand(-1, 4, 4), pos[:, None, :].expand(-1, 4, 4)
    keep = (r >= 0) & (c >= 0)
    A, coo = _csr(r[keep], c[keep], K[keep], p.n_free)
    return A, coo, b


def _beam_system(p, f):
    t, G, V = _tet_geometry(p)
    E, nu = f["e_mod"], f["nu"]
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    GG = torch.einsum("emi,enj->eminj", G, G)  # [m, i, n, j] = d_i N_m d_j N_n
    dot = torch.einsum("emi,eni->emn", G, G)
    eye = torch.eye(3, dtype=V.dtype, device=V.device)
    K = lam[:, None, None, None, None] * GG + mu[:, None, None, None, None] * (
        GG.permute(0, 1, 4, 3, 2) + dot[:, :, None, :, None] * eye[None, None, :, None, :])
    K = K * V[:, None, None, None, None]
    book = torch.from_numpy(p.book.astype(np.int64)).cuda()
    book = torch.where(book == 0xFFFFFFFF, torch.full_like(book, -1), book)
    d = torch.arange(3, device="cuda")
    pos = book[3 * t[:, :, None] + d]  # (e, 4, 3)
    r, c = pos[:, :, :, None, None].expand(-1, 4, 3, 4, 3), pos[:, None, None, :, :].expand(-1, 4, 3, 4, 3)
    keep = (r >= 0) & (c >= 0)
    A, coo = _csr(r[keep], c[keep], K[keep], p.n_free)
    tri = torch.from_numpy(p.tris.astype(np.int64)).cuda()
    xyz = torch.from_numpy(p.mesh.xyz).cuda()
    area = 0.5 * torch.linalg.cross(xyz[tri[:, 1]] - xyz[tri[:, 0]], xyz[tri[:, 2]] - xyz[tri[:, 0]]).norm(dim=1)
    load = (f["traction"] * (area / 3.0)[:, None])[:, None, :].expand(-1, 3, -1)
    tp = book[3 * tri[:, :, None] + d]
    b = torch.zeros(p.n_free, dtype=torch.float64, device="cuda")
    b.index_add_(0, tp[tp >= 0], load[tp >= 0])
    return A, coo, b


def _diagonal(coo):
    r, c = coo.indices()
    on = r == c
    d = torch.zeros(coo.shape[0], dtype=torch.float64, device="cuda")
    d[r[on]] = coo.values()[on]
    return d


def _cg(A, d, b, rounds=3, limit=30000):
    """Jacobi-preconditioned CG restarted from the true residual until it no longer falls."""
    x = torch.zeros_like(b)
    for _ in range(rounds):
        r = b - A @ x
        r0 = float(r.norm())
        if r0 <= 1e-15 * float(b.norm()):
            break
        y, p, rho = torch.zeros_like(b), torch.zeros_like(b), None
        for i in range(limit):
            z = r / d
            new = torch.dot(r, z)
            p = z if rho is None else z + (new / rho) * p
            rho = new
            q = A @ p
            alpha = rho / torch.dot(p, q)
            y += alpha * p
            r -= alpha * q
            if i % 20 == 19 and not float(r.norm()) > 1e-13 * r0:
                break
        x = x + y
    return x


def _bicgstab(A, d, b, rounds=4, limit=5000):
    x = torch.zeros_like(b)
    for _ in range(rounds):
        r = b - A @ x
        r0 = float(r.norm())
        if r0 <= 1e-15 * float(b.norm()):
            break
        y, p, h = torch.zeros_like(b), r.clone(), r.clone()
        rho = torch.dot(h, r)
        for i in range(limit):
            v = A @ (p / d)
            alpha = rho / torch.dot(h, v)
            s = r - alpha * v
            t = A @ (s / d)
            om = torch.dot(t, s) / torch.dot(t, t)
            y += (alpha * p + om * s) / d
            r = s - om * t
            new = torch.dot(h, r)
            p = r + (new / rho) * (alpha / om) * (p - om * v)
            rho = new
            if i % 10 == 9 and not float(r.norm()) > 1e-12 * r0:
                break
        x = x + y
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "dropin", "refresh", "multi", "assemble", "learned"):
        p = _cube(case["hexes"])
        A, coo, b = _heat_system(p, _fields(case["hexes"], case["sigma"], seed))
        if kind == "assemble":
            return {"b": b, "values": coo.values()}
        if kind == "learned":
            return _network(coo, A, case, seed)
        d = _diagonal(coo)
        if kind == "multi":
            return torch.stack([_cg(A, d, row) for row in _load_cases(case, seed, b)])
        x = _cg(A, d, b)
        return x if kind == "solve" else x.cpu().numpy()
    if kind == "transient":
        p, f = _transient_inputs(case, seed)
        A, coo, b = _heat_system(p, f, transient=True)
        x = _cg(A, _diagonal(coo), b)
        book = torch.from_numpy(p.book.astype(np.int64)).cuda()
        free = book != 0xFFFFFFFF
        t = f["node_t"].clone()
        t[free] = x[book[free]]
        return t
    if kind == "beam":
        A, coo, b = _beam_system(*_beam_fields(case, seed))
        return _cg(A, _diagonal(coo), b)
    if kind == "gmres":
        rp, ci, val, b = _conv_diff(case["grid"], seed)
        A = torch.sparse_csr_tensor(rp.long(), ci.long(), val, (b.numel(), b.numel()))
        return _bicgstab(A, torch.full_like(b, 6.0 * (case["grid"] + 1) ** 2), b)
    xs = []
    for i, n in enumerate(_batch_sizes(case, seed)):
        A, coo, b = _heat_system(_cube(n), _fields(n, case["sigma"], 1000 * seed + i))
        xs.append(_cg(A, _diagonal(coo), b))
    return torch.cat(xs)


def _network(coo, A, case, seed):
    """The message-passing network of the shipped model in 64 bits."""
    m = np.load(os.path.join(_PKG, "rsg", "models", "heat_family_60.npz"))
    prm, layers, H = torch.from_numpy(m["params"].astype(np.float64)).cuda(), int(m["layers"]), int(m["hidden"])
    at = 0

    def take(*shape):
        nonlocal at
        v = prm[at:at + math.prod(shape)].reshape(shape)
        at += math.prod(shape)
        return v

    w_in, b_in = take(8, H), take(H)
    blocks = [(take(2 * H, H), take(H)) for _ in range(layers)]
    w_out, b_out = take(H), take(1)
    p = _cube(case["hexes"])
    n = p.n_free
    g = torch.Generator(device="cuda").manual_seed(31 * seed + 7)
    r = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    d = _diagonal(coo)
    s = 1.0 / d.sqrt()
    i, j = coo.indices()
    off = i != j
    G = torch.sparse_coo_tensor(coo.indices()[:, off], -coo.values()[off] * s[i[off]] * s[j[off]], (n, n)).to_sparse_csr()
    u = r * s
    rms = u.square().mean().sqrt()
    one = torch.ones_like(r)
    f = torch.stack([u / rms, d.log() - d.log().mean(), (A @ one) / d, *_free_xyz(p).T, one, 0 * one], dim=1)
    h = torch.relu(f @ w_in + b_in)
    for w, b in blocks:
        h = h + torch.relu(torch.cat([h, G @ h], dim=1) @ w + b)
    return (h @ w_out + b_out) * rms * s
