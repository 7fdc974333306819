"""The work that programs built on this package have it do, as cases that can be timed and checked.

A case names one of these calls and its sizes:

  ip        VonMisesBatch.update_and_stiffness: the stress update and the consistent tangent of n integration points,
            for a program that keeps its own elements
  tangent   VonMisesBatch.stiffness: the tangents alone, as at the start of a load step
  ep        ElastoplasticBatch.update_stress: the general (ODE based) elastoplastic update
  step      Elements.update_and_assemble on device buffers: the element work of one Newton iteration
  start     Elements.assemble_f_int and assemble_kk: the two calls that open a load step
  dropin    Elements.update_and_assemble on host arrays: the same Newton iteration for a host program that solves the
            linear system itself
  solve     BatchSolver: one load step of many independent problems, Newton and PCG on the device

Everything is FP64, the only type of the package.  The exact values restate the element, the return map and the Newton
loop with dense matrices in plain torch.
"""
import math

import numpy as np
import torch

from pmsim_b200 import mesh as M
from pmsim_b200.batch import BatchSolver
from pmsim_b200.elements import Elements, Material
from pmsim_b200.footing import block_problem, footing_problem
from pmsim_b200.material import ElastoplasticBatch, VonMisesBatch

YOUNG, POISSON, HARDENING, YIELD = 2e5, 0.3, 1e3, 250.0  # the large block's material


def listed():
    return [
        # the 1,800 points of the 20x10 strip footing: a call that is all latency
        dict(name="ip footing", call="ip", ndim=2, n=1800),
        # the stress-update benchmark: 16M points, the largest array call
        dict(name="ip 16M", call="ip", ndim=3, n=16777216),
        # the general plasticity model over the points of a mid-sized 3D mesh
        dict(name="ep 3d", call="ep", ndim=3, n=1048576),
        # Newton iteration of the 20x10 strip footing (3x3 points): small meshes are solved by the thousand
        dict(name="step footing", call="step", kind="qua8", nx=20, ny=10, ngauss=9),
        # a large plane-strain mesh with odd sides: bound by memory in principle
        dict(name="step plane", call="step", kind="qua8", nx=701, ny=350, ngauss=9),
        # an axisymmetric mesh with the 2x2 rule, as for pressurised vessels and plates
        dict(name="step ring", call="step", kind="qua8", nx=160, ny=81, ngauss=4, axisymmetric=True),
        # the large single problem: 64x64x32 Hex20, 27 points, 1.6M equations
        dict(name="step block", call="step", kind="hex20", nx=64, ny=64, nz=32, ngauss=27),
        # the largest block of the served mix, with the lower triangle that a symmetric direct solver takes
        dict(name="step served", call="step", kind="hex8", nx=40, ny=40, nz=40, ngauss=8, sym="lower"),
        # the start of a load step on a tetrahedral mesh, linear elastic
        dict(name="start tets", call="start", kind="tet4", nx=24, ny=23, nz=21, ngauss=4, elastic=True),
        # the drop-in call with host arrays, as a host Newton loop around a direct solver makes it
        dict(name="dropin block", call="dropin", kind="hex20", nx=16, ny=15, nz=9, ngauss=27),
        # one load step of 32 footings of uneven size, the batched solver
        dict(name="solve footings", call="solve", problem="footing", count=32, lo=8, hi=32, device_loop=False),
        # one load step of one 3D block with the Newton loop on the device, as a single served request
        dict(name="solve block", call="solve", problem="block", count=1, lo=20, hi=20, device_loop=True),
    ]


RULES = {"tri3": (3,), "tri6": (3,), "qua4": (4,), "qua8": (4, 9), "qua9": (9,), "tet4": (1, 4), "hex8": (8,), "hex20": (8, 27)}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["ip", "ip", "tangent", "ep", "step", "step", "step", "step", "start", "dropin", "solve"])
    if call in ("ip", "tangent"):
        return dict(call=call, ndim=rng.choice([2, 3]), n=_log(rng, 1000, 12000000))
    if call == "ep":
        return dict(call=call, ndim=rng.choice([2, 3]), n=_log(rng, 2000, 1000000))
    if call == "solve":
        if rng.random() < 0.5:
            lo = rng.randint(8, 16)
            return dict(call=call, problem="footing", count=_log(rng, 1, 24), lo=lo, hi=lo + rng.randint(0, 12), device_loop=rng.random() < 0.5)
        lo = rng.randint(8, 18)
        return dict(call=call, problem="block", count=rng.randint(1, 3), lo=lo, hi=lo + rng.randint(0, 2), device_loop=rng.random() < 0.5)
    kind = rng.choice(["tri3", "tri6", "qua4", "qua8", "qua8", "qua9", "tet4", "hex8", "hex8", "hex20", "hex20"])
    case = dict(call=call, kind=kind, ngauss=rng.choice(RULES[kind]))
    points = _log(rng, 500, 60000 if call == "dropin" else 1500000)  # integration points of the mesh
    squares = max(2.0, points / case["ngauss"] / {"tri3": 2, "tri6": 2, "tet4": 6}.get(kind, 1))
    if kind in ("tet4", "hex8", "hex20"):
        side = squares ** (1.0 / 3.0)
        nx, ny = (max(1, round(side * rng.uniform(0.7, 1.4))) for _ in range(2))
        case.update(nx=nx, ny=ny, nz=max(1, round(squares / (nx * ny))))
    else:
        nx = max(1, round(math.sqrt(squares) * rng.uniform(0.6, 1.7)))
        case.update(nx=nx, ny=max(1, round(squares / nx)))
        if rng.random() < 0.2:
            case["axisymmetric"] = True
    if rng.random() < 0.25:
        case["elastic"] = True
    if rng.random() < 0.25:
        case["sym"] = rng.choice(["lower", "upper"])
    elif rng.random() < 0.2:
        case["assembly"] = "direct"
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------
def _points(case, seed):
    """The arrays of n integration points: stress free or on the yield surface, strain increments of which most yield."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nd, n = case["ndim"], case["n"]
    nc = 2 * nd
    shear = YOUNG / (2.0 * (1.0 + POISSON))

    def normal(*shape):
        return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")

    def uniform(*shape):
        return torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda")

    s = dict(sig=torch.zeros(nc, n, dtype=torch.float64, device="cuda"), z=torch.full((n,), YIELD, dtype=torch.float64, device="cuda"),
             elastic=torch.ones(n, dtype=torch.uint8, device="cuda"), deps=normal(nc, n) * (1.5 * YIELD / (2.0 * shear)))
    if case["call"] == "ep":
        # half of the points on the yield surface, the others inside it, in random directions, loaded further on the whole:
        # the model refuses a path that turns back during the plastic part
        dirs = normal(nc, n)
        dirs[:3] -= dirs[:3].mean(0)
        on = uniform(n) < 0.5
        s["sig"] += dirs * (torch.where(on, torch.ones_like(s["z"]), uniform(n)) * YIELD / torch.sqrt(1.5 * (dirs * dirs).sum(0)))
        s["sig"][:3] += YIELD * uniform(n)
        s["elastic"][on] = 0
        s["deps"] = 0.15 * s["deps"] + (0.6 * YIELD / (2.0 * shear)) * dirs
    else:
        s["hh"] = 2e3 * uniform(n)
        s["lam"] = torch.zeros(n, dtype=torch.float64, device="cuda")
        s["dd"] = torch.empty(nc * (nc + 1) // 2, n, dtype=torch.float64, device="cuda")
    if nd == 2:
        s["deps"][2] = 0.0  # plane strain
    if case["call"] == "ep":
        s["deps"] *= torch.where((dirs * s["deps"]).sum(0) < 0.0, -1.0, 1.0)
    if case["call"] == "tangent":
        dirs = normal(nc, n)
        s["sig"] += dirs * (YIELD / torch.sqrt((dirs * dirs).sum(0)))
        s["elastic"] = (uniform(n) < 0.6).to(torch.uint8)
        s["lam"] = torch.where(s["elastic"] == 0, uniform(n) * (YIELD / (3.0 * shear)), s["lam"])
    return s


def _mesh(case, seed):
    """Cells of unit size, the interior nodes moved a little, and two displacement increments: to the state at the start
    of the load step and from there on.  The indentation of a central footing, decaying with depth and across its edge."""
    sizes = [case["nx"], case["ny"]] + ([case["nz"]] if "nz" in case else [])
    make, kind = (M.structured_3d, M.structured_2d)[len(sizes) == 2], M.kind_from_name(case["kind"])
    m = make(kind, *sizes, *map(float, sizes))
    rng = np.random.default_rng(seed)
    c = m.coords.copy()
    inside = np.all((c > 1e-9) & (c < np.array(sizes) - 1e-9), axis=1)
    c[inside] += rng.uniform(-0.05, 0.05, (int(inside.sum()), m.ndim))
    if case.get("axisymmetric"):
        c[:, 0] += 0.25 * sizes[0]  # a ring: the axis lies outside
    m = M.Mesh(m.ndim, c, m.cells, kind)
    x = m.coords
    u = np.zeros_like(x)
    plate = np.ones(len(x))
    for d, n in enumerate(sizes[:-1]):
        plate *= 0.5 * (np.tanh((n / 4.0 - np.abs(x[:, d] - x[:, d].mean())) / 2.0) + 1.0)
    depth = np.exp(-(sizes[-1] - x[:, -1]) / (0.5 * sizes[-1]))
    u[:, -1] = -0.00175 * sizes[-1] * plate * depth
    first = 0.7 * u + rng.normal(0.0, 2e-4, u.shape)
    return m, first.reshape(-1), (u + rng.normal(0.0, 2e-4, u.shape)).reshape(-1)


def _material(case):
    return Material.linear_elastic(YOUNG, POISSON) if case.get("elastic") else Material.von_mises(YOUNG, POISSON, HARDENING, YIELD)


def _problems(case, seed):
    """Problems of the batched and served populations, with a hardening material; the sizes are the case's."""
    sizes, rng = np.random.default_rng(case["lo"] + 100 * case["hi"] + 10000 * case["count"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        young, z0 = 1e4 * math.exp(rng.normal(0.0, 0.3)), rng.uniform(8.0, 20.0)
        if case["problem"] == "footing":
            nx = int(sizes.integers(case["lo"], case["hi"] + 1))
            ny = max(4, nx // 2 + int(sizes.integers(-2, 3)))
            out.append(footing_problem(nx, ny, young, z0, rng.uniform(0.5, 2.0), nsteps=10, hh=0.05 * young))
        else:
            n = [int(v) for v in sizes.integers(case["lo"], case["hi"] + 1, size=3)]
            out.append(block_problem(*n, young, z0, nsteps=10, hh=0.05 * young))
    return out


_stream = []  # all meshes of a program share one stream


def prepare(case, seed):
    call = case["call"]
    if call in ("ip", "tangent", "ep"):
        s = _points(case, seed)
        if call == "ep":
            s["model"] = ElastoplasticBatch(YOUNG, POISSON, HARDENING, YIELD, ndim=case["ndim"])
            s["cases"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
            s["start"] = {k: s[k].clone() for k in ("sig", "z", "elastic")}
        else:
            s["model"] = VonMisesBatch(YOUNG, POISSON, HARDENING, YIELD, ndim=case["ndim"])
        return dict(s, call=call)
    if call == "solve":
        return dict(call=call, solver=BatchSolver(_problems(case, seed)), device_loop=case["device_loop"])
    m, first, ddu = _mesh(case, seed)
    el = Elements(m, _material(case), ngauss=case["ngauss"], axisymmetric=case.get("axisymmetric", False))
    el.set_assembly(case.get("assembly", "gather"))
    el.set_symmetry(case.get("sym", "full"))
    el.initialize_internal_values()
    el.update_secondary_values(first)
    el.reset_algorithmic_variables()
    el.backup_secondary_values()
    el.sync()
    s = dict(call=call, el=el)
    if call == "dropin":
        return dict(s, ddu=ddu, ff=np.zeros(el.ndof), kk=np.zeros(el.nnz))
    if not _stream:
        _stream.append(torch.cuda.Stream())
    el.set_stream(_stream[0])
    empty = dict(dtype=torch.float64, device="cuda")
    return dict(s, ddu=torch.tensor(ddu, **empty), ff=torch.empty(el.ndof, **empty), kk=torch.empty(el.nnz, **empty))


def run(s):
    call = s["call"]
    if call == "ip":
        s["model"].update_and_stiffness(s["sig"], s["z"], s["lam"], s["elastic"], s["deps"], hh=s["hh"], dd=s["dd"])
        return {k: s[k] for k in ("sig", "z", "lam", "elastic", "dd")}
    if call == "tangent":
        s["model"].stiffness(s["sig"], s["lam"], s["elastic"], s["dd"], hh=s["hh"])
        return {"dd": s["dd"]}
    if call == "ep":
        for k, v in s["start"].items():  # a Newton iteration starts from the state at the start of the load step
            s[k].copy_(v)
        s["model"].update_stress(s["sig"], s["z"], s["elastic"], s["deps"], cases=s["cases"])
        return {k: s[k] for k in ("sig", "z", "elastic", "cases")}
    if call == "solve":
        solver = s["solver"]
        solver.reset()
        iterations, _, status, _ = solver.solve_step(device_loop=s["device_loop"])
        sig, ivs, elastic = solver.elements.get_state()
        return dict(u=solver.u(), sig=sig, ivs=ivs, elastic=elastic, iterations=iterations, status=status)
    if call == "start":
        s["el"].assemble_f_int(s["ff"])
        s["el"].assemble_kk(s["kk"])
    else:
        s["el"].update_and_assemble(s["ddu"], s["ff"], s["kk"])
    return {"ff": s["ff"], "kk": s["kk"]}


# ---- the work of one pass ----------------------------------------------------------------------------------------
def _sizes(kind, dims):
    """(nodes, cells, nodes per cell, node pairs of the matrix) of a structured mesh."""
    nn, nd = M.KIND_NNODE[M.kind_from_name(kind)], len(dims)
    corners = math.prod(n + 1 for n in dims)
    edges = sum(n * math.prod(m + 1 for j, m in enumerate(dims) if j != i) for i, n in enumerate(dims))
    squares = math.prod(dims)
    cells = squares * {"tri3": 2, "tri6": 2, "tet4": 6}.get(kind, 1)
    nodes = {"tri3": corners, "qua4": corners, "hex8": corners, "tet4": corners, "qua8": corners + edges, "hex20": corners + edges,
             "qua9": corners + edges + squares, "tri6": corners + edges + squares}[kind]
    per = {"tri3": 7, "tri6": 11.5, "qua4": 9, "qua8": 14, "qua9": 16, "tet4": 15, "hex8": 27, "hex20": 57}[kind]  # blocks a row, away from the sides
    return nodes, cells, nn, int(nodes * min(per, nodes)), nd


def _step_work(kind, dims, ngauss, sym, update):
    nodes, cells, nn, pairs, nd = _sizes(kind, dims)
    nc, ips, values = 2 * nd, cells * ngauss, pairs * nd * nd * (1.0 if sym == "full" else 0.5)
    state = ips * ((8 * nc + 8) + (8 * nc + 17) if update else 8 * nc + 9)
    # D B, B^T D B of the node pairs a <= b, the Jacobian and the gradients
    flops = 2.0 * ips * (nd * nc * nd * nn + nd ** 3 * nn * (nn + 1) // 2 + 2 * nn * nd * nd)
    return nodes * nd * 8 * (3 if update else 2) + cells * nn * 4 + state + 8 * values, flops


def work(case):
    call = case["call"]
    if call in ("ip", "tangent", "ep"):
        nc = 2 * case["ndim"]
        nt = nc * (nc + 1) // 2
        doubles = {"ip": 3 * nc + 4 + nt, "tangent": nc + 2 + nt, "ep": 3 * nc + 2}[call]
        # ep: about 30 steps of six stages a point, each the rates of the three scalars that the flow comes down to
        return {"bytes": case["n"] * (8.0 * doubles + {"ip": 1, "tangent": 1, "ep": 6}[call]), "flops": case["n"] * (4500.0 if call == "ep" else 200.0)}
    if call == "solve":
        # seven Newton iterations; a PCG iteration reads the matrix once, and its count grows with the side of the mesh
        total = {"bytes": 0.0, "flops": 0.0}
        for p in _problems(case, 0):
            meta = p.meta
            kind, dims = ("qua8", [meta["nx"], meta["ny"]]) if "width" in meta else ("hex8", [meta["nx"], meta["ny"], meta["nz"]])
            b, f = _step_work(kind, dims, p.ngauss, "full", True)
            nodes, _, _, pairs, nd = _sizes(kind, dims)
            rounds = 7.0 * {2: 10.0, 3: 4.0}[nd] * max(dims)
            total["bytes"] += 7.0 * b + rounds * (pairs * (8.0 * nd * nd + 4) + 80.0 * nodes * nd)
            total["flops"] += 7.0 * f + rounds * 2.0 * pairs * nd * nd
        return total
    dims = [case["nx"], case["ny"]] + ([case["nz"]] if "nz" in case else [])
    b, f = _step_work(case["kind"], dims, case["ngauss"], case.get("sym", "full"), call != "start")
    return {"bytes": float(b), "flops": float(f)}


# ---- exact values ------------------------------------------------------------------------------------------------
ROOT2 = math.sqrt(2.0)


def _moduli(young, poisson):
    return young / (3.0 * (1.0 - 2.0 * poisson)), young / (2.0 * (1.0 + poisson))


def _split(v):
    """Mean and deviator of Mandel vectors (last axis)."""
    m = v[..., :3].sum(-1, keepdim=True) / 3.0
    s = v.clone()
    s[..., :3] -= m
    return m, s


def _return_map(mat, sig, z, lam, el, deps):
    """The radial return: (sig, z, lam, el) after deps.  mat: (young, poisson, hh, z_ini or None where linear elastic)."""
    k, g = _moduli(*mat[:2])
    m, s = _split(deps)
    trial = sig + 2.0 * g * s
    trial[..., :3] += 3.0 * k * m
    if mat[3] is None:
        return trial, z, lam, el
    m, s = _split(trial)
    sd = torch.sqrt(1.5 * (s * s).sum(-1))
    f = sd - z
    yields = f / mat[3] > 1e-6
    dl = torch.where(yields, f / (3.0 * g + mat[2]), torch.zeros_like(f))
    s = s * torch.where(yields, 1.0 - dl * 3.0 * g / sd, torch.ones_like(f))[..., None]
    out = s.clone()
    out[..., :3] += m
    return torch.where(yields[..., None], out, trial), z + mat[2] * dl, dl, ~yields


def _tangent(mat, sig, lam, el):
    """The consistent tangent D[..., nc, nc] in Mandel form."""
    k, g = _moduli(*mat[:2])
    nc = sig.shape[-1]
    one = torch.zeros(nc, dtype=sig.dtype, device=sig.device)
    one[:3] = 1.0
    dev = torch.eye(nc, dtype=sig.dtype, device=sig.device) - one[:, None] * one / 3.0
    a, b = torch.full_like(lam, 2.0 * g), torch.zeros_like(lam)
    _, s = _split(sig)
    if mat[3] is not None:
        ss = (s * s).sum(-1)
        trial = torch.sqrt(1.5 * ss) + 3.0 * g * lam
        a = torch.where(el, a, 2.0 * g * (1.0 - 3.0 * g * lam / trial))
        b = torch.where(el, b, 6.0 * g * g * (lam / trial - 1.0 / (3.0 * g + mat[2])) / ss)
    return a[..., None, None] * dev + b[..., None, None] * s[..., :, None] * s[..., None, :] + k * one[:, None] * one


def _nodes(kind):
    """Natural coordinates of the nodes and the exponents of the monomials that span the shape functions."""
    if kind in ("tri3", "tri6"):
        r = [(0, 0), (1, 0), (0, 1)] + ([(0.5, 0), (0.5, 0.5), (0, 0.5)] if kind == "tri6" else [])
        return r, [(i, j) for i in range(3) for j in range(3) if i + j <= (1 if kind == "tri3" else 2)]
    if kind == "tet4":
        return [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)], [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
    square = [(-1, -1), (1, -1), (1, 1), (-1, 1)]
    if kind in ("qua4", "qua8", "qua9"):
        r = square + ([(0, -1), (1, 0), (0, 1), (-1, 0)] if kind != "qua4" else []) + ([(0, 0)] if kind == "qua9" else [])
        top = 1 if kind == "qua4" else 2
        return r, [(i, j) for i in range(top + 1) for j in range(top + 1) if kind != "qua8" or i + j < 4]
    r = [(x, y, -1) for x, y in square] + [(x, y, 1) for x, y in square]
    if kind == "hex20":
        mids = [(0, -1), (1, 0), (0, 1), (-1, 0)]
        r += [(x, y, -1) for x, y in mids] + [(x, y, 1) for x, y in mids] + [(x, y, 0) for x, y in square]
    top = 1 if kind == "hex8" else 2
    return r, [e for e in np.ndindex(top + 1, top + 1, top + 1) if sum(v == 2 for v in e) <= 1]


def _rule(kind, n):
    """Points and weights, the first coordinate running fastest."""
    if kind in ("tri3", "tri6"):
        return [(1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3)], [1 / 6] * 3
    if kind == "tet4":
        if n == 1:
            return [(0.25,) * 3], [1 / 6]
        a, b = (5.0 + 3.0 * math.sqrt(5.0)) / 20.0, (5.0 - math.sqrt(5.0)) / 20.0
        return [(a, b, b), (b, a, b), (b, b, a), (b, b, b)], [1 / 24] * 4
    nd = 3 if kind.startswith("hex") else 2
    x, w = np.polynomial.legendre.leggauss(round(n ** (1.0 / nd)))
    index = [e[::-1] for e in np.ndindex(*[len(x)] * nd)]
    return [tuple(x[i] for i in e) for e in index], [math.prod(w[i] for i in e) for e in index]


def _shapes(kind, ngauss, device):
    """N[p, m], dN[p, m, j] and w[p] from the Vandermonde matrix of the nodes."""
    nodes, powers = _nodes(kind)
    points, w = _rule(kind, ngauss)
    powers = np.array(powers)

    def mono(x, d=None):
        out = np.ones((len(x), len(powers)))
        for j in range(powers.shape[1]):
            e = powers[:, j]
            out *= (e * x[:, j, None] ** np.maximum(e - 1, 0)) if j == d else x[:, j, None] ** e
        return out

    nodes, points = np.array(nodes, dtype=np.float64), np.array(points)
    inverse = np.linalg.inv(mono(nodes))
    grads = np.stack([mono(points, d) @ inverse for d in range(powers.shape[1])], axis=-1)
    return [torch.tensor(v, dtype=torch.float64, device=device) for v in (mono(points) @ inverse, grads, np.array(w))]


class _Dense:
    """Element vectors and matrices of a mesh with dense strain-displacement matrices, some cells at a time."""

    def __init__(self, mesh, kind, ngauss, mat, axisymmetric=False):
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        self.mat, self.axisymmetric, self.nd, self.npoint = mat, axisymmetric, mesh.ndim, mesh.npoint
        self.nc = 2 * self.nd
        self.x = torch.tensor(mesh.coords, device=self.device)
        self.cells = torch.tensor(mesh.cells, device=self.device)
        self.shapes = _shapes(kind, ngauss, self.device)
        shape = (mesh.ncell, ngauss)
        zero = torch.zeros(shape, dtype=torch.float64, device=self.device)
        self.state = (torch.zeros(*shape, self.nc, dtype=torch.float64, device=self.device), zero + (mat[3] or 0.0), zero.clone(),
                      torch.ones(shape, dtype=torch.bool, device=self.device))

    def chunks(self):
        per = max(1, 1 + 60000000 // (self.state[0].shape[1] * self.nc * self.cells.shape[1] * self.nd))
        return [slice(i, i + per) for i in range(0, len(self.cells), per)]

    def strain_matrix(self, part):
        """B[c, p, nc, nn*nd] and the weights |J| w (r)."""
        n, dn, w = self.shapes
        x = self.x[self.cells[part]]
        jac = torch.einsum("cmi,pmj->cpij", x, dn)
        g = torch.einsum("pmj,cpji->cpmi", dn, torch.linalg.inv(jac))
        b = torch.zeros(*g.shape[:2], self.nc, g.shape[2], self.nd, dtype=g.dtype, device=g.device)
        for i in range(self.nd):
            b[:, :, i, :, i] = g[..., i]
        for c, (i, j) in enumerate(((0, 1), (1, 2), (0, 2))[: self.nc - 3]):
            b[:, :, 3 + c, :, i] = g[..., j] / ROOT2
            b[:, :, 3 + c, :, j] = g[..., i] / ROOT2
        w = torch.linalg.det(jac) * w
        if self.axisymmetric:
            r = torch.einsum("pm,cm->cp", n, x[..., 0])
            b[:, :, 2, :, 0] = n / r[..., None]
            w = w * r
        return b.flatten(3), w

    def dofs(self, part):
        return (self.cells[part][..., None] * self.nd + torch.arange(self.nd, device=self.device)).flatten(1)

    def update(self, state, ddu):
        out = [v.clone() for v in state]
        for part in self.chunks():
            b, _ = self.strain_matrix(part)
            new = _return_map(self.mat, *(v[part] for v in state), torch.einsum("cpne,ce->cpn", b, ddu[self.dofs(part)]))
            for o, v in zip(out, new):
                o[part] = v
        return tuple(out)

    def vectors(self, state):
        """F_int and, some cells at a time, (slice, K_e)."""
        ff, kk = torch.zeros(self.npoint * self.nd, dtype=torch.float64, device=self.device), []
        for part in self.chunks():
            b, w = self.strain_matrix(part)
            ff.index_add_(0, self.dofs(part).flatten(), torch.einsum("cpne,cpn,cp->ce", b, state[0][part], w).flatten())
            db = (_tangent(self.mat, state[0][part], state[2][part], state[3][part]) * w[..., None, None]) @ b
            kk.append((part, b.flatten(1, 2).transpose(1, 2) @ db.flatten(1, 2)))
        return ff, kk

    def csr_values(self, kk, sym):
        nd, nn, n = self.nd, self.cells.shape[1], self.npoint
        keys, where = torch.unique((self.cells[:, :, None] * n + self.cells[:, None, :]).flatten(), return_inverse=True)
        where = where.view(-1, nn * nn)
        blocks = torch.zeros(len(keys), nd, nd, dtype=torch.float64, device=self.device)
        for part, ke in kk:
            blocks.index_add_(0, where[part].flatten(), ke.view(-1, nn, nd, nn, nd).transpose(2, 3).reshape(-1, nd, nd))
        row, col = keys // n, keys % n
        count = torch.bincount(row, minlength=n)
        start = torch.cumsum(count, 0) - count
        i = torch.arange(nd, device=self.device)
        at = (nd * nd * start[row] + nd * (torch.arange(len(keys), device=self.device) - start[row]))[:, None, None] + nd * count[row][:, None, None] * i[:, None] + i
        values = torch.empty(len(keys) * nd * nd, dtype=torch.float64, device=self.device)
        values[at.flatten()] = blocks.flatten()
        if sym == "full":
            return values
        keep = torch.empty(len(values), dtype=torch.bool, device=self.device)
        r, c = (row * nd)[:, None, None] + i[:, None], (col * nd)[:, None, None] + i
        keep[at.flatten()] = (c <= r if sym == "lower" else c >= r).flatten()
        return values[keep]


def _exact_solve(case, seed):
    problems = _problems(case, seed)
    if sum((p.mesh.ndof / 1e4) ** 3 for p in problems) > 5.0:
        return None
    out = {k: [] for k in ("u", "sig", "ivs")}
    for p in problems:
        kind = "qua8" if p.mesh.ndim == 2 else "hex8"
        el = _Dense(p.mesh, kind, p.ngauss, (p.material.young, p.material.poisson, p.material.hh, p.material.z_ini))
        n = p.mesh.ndof
        want = {int(eq): c for eq, c, _ in p.essential}
        at = torch.tensor(sorted(want), device=el.device)
        c = torch.tensor([want[k] for k in sorted(want)], dtype=torch.float64, device=el.device)
        free = torch.ones(n, dtype=torch.bool, device=el.device)
        free[at] = False
        u, lam = torch.zeros(n, dtype=torch.float64, device=el.device), torch.zeros_like(c)
        state = start = el.state
        first = None
        for it in range(20):
            rr, kk = el.vectors(state)
            rr[at] += lam
            if max(rr.abs().max(), (u[at] - c).abs().max()) < 1e-10:
                break
            full = torch.zeros(n, n, dtype=torch.float64, device=el.device)
            for part, ke in kk:
                d = el.dofs(part)
                full.view(-1).index_add_(0, (d[:, :, None] * n + d[:, None, :]).flatten(), ke.flatten())
            du = torch.zeros_like(u)
            du[at] = u[at] - c
            du[free] = torch.linalg.solve(full[free][:, free], (rr - full @ du)[free])
            both = torch.cat([du, (rr - full @ du)[at]])
            if first is None:
                first = both
            elif (both.abs() / (1.0 + first.abs())).max() < 1e-8:
                break
            u, lam = u - du, lam - both[n:]
            state = el.update(start, u)
        else:
            return None
        out["u"].append(u)
        out["sig"].append(state[0].flatten(0, 1))
        out["ivs"].append(torch.stack([state[1].flatten(), state[2].flatten()], 1))
    return {**{k: torch.cat(v) for k, v in out.items()}, "elastic": None, "iterations": None, "status": None}


def _exact_points(case, seed):
    s = _points(case, seed)
    nc = 2 * case["ndim"]
    i, j = np.triu_indices(nc)
    out = {k: torch.empty_like(s[k]) for k in (("dd",) if case["call"] == "tangent" else ("sig", "z", "lam", "dd"))}
    for a in range(0, case["n"], 1 << 20):
        part = slice(a, a + (1 << 20))
        mat = (YOUNG, POISSON, s["hh"][part], YIELD)
        state = (s["sig"][:, part].T, s["z"][part], s["lam"][part], s["elastic"][part] != 0)
        if case["call"] == "ip":
            state = _return_map(mat, *state, s["deps"][:, part].T)
            out["sig"][:, part], out["z"][part], out["lam"][part] = state[0].T, state[1], state[2]
        out["dd"][:, part] = _tangent(mat, state[0], state[2], state[3])[:, i, j].T
    return dict(out, elastic=None) if case["call"] == "ip" else out


def _exact_ep(case, seed):
    """The elastic part up to the yield surface, then the flow at the constant rate deps, integrated with the classical
    fourth-order Runge-Kutta method in the plane of the two deviators it stays in."""
    s = _points(case, seed)
    k, g = _moduli(YOUNG, POISSON)
    sig, deps, z = s["sig"].T, s["deps"].T, s["z"]
    em, e = _split(deps)
    sm, s0 = _split(sig)
    a, b = 4.0 * g * g * (e * e).sum(-1), 2.0 * g * (s0 * e).sum(-1)
    c = (s0 * s0).sum(-1) - 2.0 / 3.0 * z * z
    t0 = torch.where(s["elastic"] == 0, torch.zeros_like(z), (-b + torch.sqrt((b * b - a * c).clamp(min=0.0))) / a)
    t0 = t0.clamp(0.0, 1.0)
    s1 = s0 + 2.0 * g * t0[:, None] * e
    # s = p s1 + q e at the rates dp = -w (s:e) p, dq = 2G - w (s:e) q with w = (2G)^2 (3/2) / (sd^2 (1 + H / 3G)) / 2G
    ss, se, ee = (s1 * s1).sum(-1), (s1 * e).sum(-1), (e * e).sum(-1)

    def rate(p, q):
        n2 = p * p * ss + 2.0 * p * q * se + q * q * ee
        w = (2.0 * g / (1.0 + HARDENING / (3.0 * g))) * (p * se + q * ee) / n2
        dz = HARDENING * 2.0 * g * 1.5 * (p * se + q * ee) / torch.sqrt(1.5 * n2) / (3.0 * g + HARDENING)
        return -w * p, 2.0 * g - w * q, dz

    p, q, zz = torch.ones_like(z), torch.zeros_like(z), z.clone()
    steps = 3000
    h = (1.0 - t0) / steps
    for _ in range(steps):
        k1 = rate(p, q)
        k2 = rate(p + 0.5 * h * k1[0], q + 0.5 * h * k1[1])
        k3 = rate(p + 0.5 * h * k2[0], q + 0.5 * h * k2[1])
        k4 = rate(p + h * k3[0], q + h * k3[1])
        p, q, zz = (v + h / 6.0 * (k1[i] + 2.0 * (k2[i] + k3[i]) + k4[i]) for i, v in enumerate((p, q, zz)))
    out = p[:, None] * s1 + q[:, None] * e
    out[:, :3] += sm + 3.0 * k * em
    return dict(sig=out.T.contiguous(), z=zz, elastic=None, cases=None)


def exact(case, seed):
    call = case["call"]
    if call == "ep":
        return _exact_ep(case, seed)
    if call in ("ip", "tangent"):
        return _exact_points(case, seed)
    if call == "solve":
        return _exact_solve(case, seed)
    m, first, ddu = _mesh(case, seed)
    mat = (YOUNG, POISSON, 0.0, None) if case.get("elastic") else (YOUNG, POISSON, HARDENING, YIELD)
    el = _Dense(m, case["kind"], case["ngauss"], mat, case.get("axisymmetric", False))
    state = el.update(el.state, torch.tensor(first, device=el.device))
    state = (state[0], state[1], torch.zeros_like(state[2]), state[3])
    if call != "start":
        state = el.update(state, torch.tensor(ddu, device=el.device))
    ff, kk = el.vectors(state)
    return {"ff": ff, "kk": el.csr_values(kk, case.get("sym", "full"))}
