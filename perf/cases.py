"""Performance cases of the SIMP / voxel-FEM path, each one pass through public entry points.

The kinds and what they stand for:

``apply``     K(x) p on a structured grid (``Engine.apply``): the operator a caller's own solver
              or eigen-analysis runs.
``edof``      the drop-in kernels over an element -> DOF table (``cuda_kernels.fused_spmv`` and
              ``simp_sensitivity``), as the reference's solver calls them once per iteration.
``update``    the design update of one SIMP iteration without its solve: sensitivities, their
              filter, the OC bisection with the filtered densities.
``solve``     one forward FEM solve of a fresh design to rtol 1e-8 (``Engine.solve``).
``simp``      a SIMP run of a few iterations (``Engine.simp_run``).
``batch``     forward solves of several designs of different sizes at once (``BatchFEM``).
``evaluate``  the evaluator on a batch of latents: decode, resample and smooth, solve
              (``VoxelFEMEvaluator.evaluate_batch``).
``generate``  the data generator's batch of small uneven SIMP problems (``BatchSIMP``).
``prep``      the evaluator's input step alone (``Engine.voxel_prep``).

Displacements are returned in single precision, the type in which the reference's solver holds
and returns them; the solves behind them run to their relative residual.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs as B
from genpipeline_gb300 import cuda_kernels
from genpipeline_gb300.batch import BatchFEM, FEMDesign
from genpipeline_gb300.engine import get_engine
from genpipeline_gb300.fem.voxel_fem import VoxelFEMEvaluator
from genpipeline_gb300.schema import DesignParameters
from genpipeline_gb300.topology.batch_simp import BatchSIMP, SimpCase
from genpipeline_gb300.topology.topo_data_gen import TopoDataGenerator

EXACT_ELEMENTS = 300_000  # above, a solve in 64 bits takes too long to be a reference here


def listed():
    return [
        # the smallest call: SIMPSolver's default grid, a latency-bound loop
        dict(name="simp 32x8x8", kind="simp", nx=32, ny=8, nz=8, load="cantilever", law="ref", rmin=1.5, volfrac=0.4,
             iters=3, preserve=False),
        # the benchmark problem: 64^3, top patch, 33-point filter
        dict(name="simp 64x64x64", kind="simp", nx=64, ny=64, nz=64, load="top_patch", law="modified", rmin=2.0,
             volfrac=0.25, iters=2, preserve=False),
        # the largest problem of the benchmark: 1.8 million elements, vectors larger than L2
        dict(name="simp 192x96x96", kind="simp", nx=192, ny=96, nz=96, load="edge_line", law="modified", rmin=3.0,
             volfrac=0.2, iters=1, preserve=False),
        # one forward solve of an odd, elongated grid
        dict(name="solve 95x47x33", kind="solve", nx=95, ny=47, nz=33, load="torsion"),
        # the benchmark's batch: 4 x 64^3 and 4 x 32^3 designs served together
        dict(name="batch 4x64 4x32", kind="batch", sizes="64,64,64,64,32,32,32,32", load="cantilever"),
        # the evaluator's batch of 16 latents on 64^3 decodes, 32^3 solves
        dict(name="evaluate 16", kind="evaluate", batch=16, size=64),
        # the generator's medium grids, eight samples
        dict(name="generate 8", kind="generate", samples=8, pick=0, iters=2),
        # the design update of the largest grid, and of an odd one with preserved elements
        dict(name="update 192x96x96", kind="update", nx=192, ny=96, nz=96, law="modified", rmin=3.0, volfrac=0.2,
             preserve=False),
        dict(name="update 61x37x23", kind="update", nx=61, ny=37, nz=23, law="ref", rmin=1.5, volfrac=0.35,
             preserve=True),
        # the operator at the largest grid with a clamped face
        dict(name="apply 192x96x96", kind="apply", nx=192, ny=96, nz=96, law="modified", masked=True),
        # the table-driven kernels of the drop-in module, int64 tables as the reference builds
        dict(name="edof 64x32x32", kind="edof", nx=64, ny=32, nz=32, penal=3.0),
        # the input step of a batch of decoded grids
        dict(name="prep 16x64", kind="prep", batch=16, D=64, H=64, W=64, d=32, h=32, w=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most, lo=6, hi=160):
    while True:
        nx, ny, nz = _log(rng, lo, hi), _log(rng, lo, hi), _log(rng, lo, hi)
        if nx * ny * nz <= most:
            return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    kind = rng.choice(["simp", "simp", "solve", "batch", "evaluate", "generate", "update", "update", "apply", "edof",
                       "prep"])
    load = rng.choice(["cantilever", "top_patch", "torsion", "edge_line"])
    if kind == "simp":
        return dict(kind=kind, **_grid(rng, 280_000, 8, 96), load=load, law=rng.choice(["ref", "modified"]),
                    rmin=rng.choice([1.5, 2.0, 2.5, 3.0]), volfrac=round(rng.uniform(0.2, 0.5), 3),
                    iters=rng.choice([1, 2, 3]), preserve=rng.random() < 0.3)
    if kind == "solve":
        return dict(kind=kind, **_grid(rng, 290_000, 8, 128), load=load)
    if kind == "batch":
        sizes = [_log(rng, 12, 64) for _ in range(rng.randint(2, 9))]
        return dict(kind=kind, sizes=",".join(map(str, sizes)), load=rng.choice(["cantilever", "top_patch", "torsion"]))
    if kind == "evaluate":
        return dict(kind=kind, batch=rng.randint(1, 20), size=rng.choice([40, 48, 56, 64]))
    if kind == "generate":
        return dict(kind=kind, samples=rng.randint(2, 8), pick=rng.randrange(1000), iters=rng.choice([1, 2]))
    if kind == "update":
        return dict(kind=kind, **_grid(rng, 1_700_000), law=rng.choice(["ref", "modified"]),
                    rmin=rng.choice([1.5, 2.0, 2.5, 3.0]), volfrac=round(rng.uniform(0.2, 0.5), 3),
                    preserve=rng.random() < 0.4)
    if kind == "apply":
        return dict(kind=kind, **_grid(rng, 1_700_000), law=rng.choice(["ref", "modified"]), masked=rng.random() < 0.5)
    if kind == "edof":
        return dict(kind=kind, **_grid(rng, 400_000), penal=rng.choice([1.0, 3.0, 3.5]))
    D, H, W = (_log(rng, 24, 96) for _ in range(3))
    half = rng.random() < 0.7  # the evaluator halves every extent; smoothing alone keeps them
    return dict(kind="prep", batch=rng.randint(1, 16), D=D, H=H, W=W, d=round(D / 2) if half else D,
                h=round(H / 2) if half else H, w=round(W / 2) if half else W)


# ---- inputs ------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _smooth(shape, g, scale=6.0):
    """A Gaussian random field: white noise under a Gaussian of `scale` voxels, unit variance."""
    k = torch.meshgrid(*(torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) for n in shape), indexing="ij")
    t = torch.exp(-2.0 * math.pi ** 2 * scale ** 2 * sum(a * a for a in k))
    z = torch.fft.ifftn(torch.fft.fftn(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)) * t).real
    return (z - z.mean()) / (z.std() + 1e-30)


def _density(shape, g, lo=1e-3):
    """Densities of the serving workload: a sigmoid of a smooth field, mean 0.2 to 0.5."""
    s = torch.sigmoid(_smooth(shape, g))
    m = 0.2 + 0.3 * torch.rand((), generator=g, device="cuda", dtype=torch.float64)
    return (s * (m / s.mean())).clamp(lo, 1.0).float().reshape(-1)


def _grid_of(c):
    return c["nx"], c["ny"], c["nz"]


def _load(c, grid):
    f, fixed = B.LOAD_CASES[c["load"]](*grid)
    return torch.as_tensor(f, device="cuda"), torch.as_tensor(B.node_mask(*grid, fixed), device="cuda")


def _law(c):
    return L.make_law(c.get("law", "modified"), 3.0)


def _preserved(c, grid):
    """A bolt pattern's worth of elements kept solid: two corners of the x faces."""
    if not c["preserve"]:
        return None
    p = torch.zeros(grid, dtype=torch.uint8, device="cuda")
    p[:2, :2, :2] = 1
    p[-2:, -2:, -2:] = 1
    return p.reshape(-1)


def _edof(grid):
    nx, ny, nz = grid
    i, j, k = torch.meshgrid(*(torch.arange(n, device="cuda") for n in grid), indexing="ij")
    corner = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    n = torch.stack([((i + a) * (ny + 1) + j + b) * (nz + 1) + k + c for a, b, c in corner], -1).reshape(-1, 8, 1)
    return (3 * n + torch.arange(3, device="cuda")).reshape(-1, 24)


class _Decoder:
    """The caller's decoder: latents to densities through a fixed basis of smooth fields."""

    def __init__(self, size, latent_dim=16):
        g = _gen(1234)
        self.size = size
        self.fields = torch.stack([_smooth((size,) * 3, g).reshape(-1) for _ in range(latent_dim)]).float()

    def parameters(self):
        return iter([self.fields])

    def decode(self, z):
        v = torch.sigmoid(1.5 * (z.to(self.fields.dtype) @ self.fields) / math.sqrt(self.fields.shape[0]))
        return v.reshape(-1, 1, self.size, self.size, self.size)


def _latents(c, seed):
    return np.random.default_rng(seed).standard_normal((c["batch"], 16)).astype(np.float32)


def _samples(c, seed):
    """The generator's draws at its medium grid size (organic mode, penal 3.5): the geometries and
    grids are the case's, volume fractions and forces the seed's."""
    r, v = np.random.default_rng(c["pick"]), np.random.default_rng(seed)
    out = []
    for geom in r.choice(["bridge", "arch", "offset", "center", "cantilever", "lbracket", "branch"], c["samples"]):
        if geom in ("lbracket", "bridge", "arch", "center"):
            grid = r.integers(16, 24), r.integers(6, 10), r.integers(12, 18)
        elif geom == "branch":
            grid = r.integers(22, 32), r.integers(10, 16), r.integers(10, 16)
        else:
            grid = r.integers(20, 32), r.integers(6, 10), r.integers(6, 10)
        out.append((str(geom), tuple(int(n) for n in grid), float(v.uniform(0.12, 0.35)), float(v.uniform(200, 5000))))
    return out


def _displacement(shape, g):
    """A displacement field of a bent body: smooth, with a fixed x = 0 face."""
    u = torch.stack([_smooth(shape, g, 8.0) for _ in range(3)], -1)
    ramp = torch.linspace(0, 1, shape[0], device="cuda", dtype=torch.float64) ** 2
    return (10.0 * u * ramp[:, None, None, None]).reshape(-1).contiguous()


def _nodes(grid):
    return tuple(n + 1 for n in grid)


def prepare(case, seed):
    c, s, g = case, {"case": case}, _gen(seed)
    kind = c["kind"]
    if kind in ("simp", "solve", "update", "apply", "edof"):
        grid = s["grid"] = _grid_of(c)
        s["x"] = _density(grid, g)
    if kind != "generate":
        s["eng"] = get_engine()
    if kind in ("simp", "solve"):
        s["f"], s["mask"] = _load(c, grid)
    if kind in ("simp", "update"):
        s["pres"] = _preserved(c, grid)
        if s["pres"] is not None:
            s["x"][s["pres"].bool()] = 1.0
    if kind == "update":
        eng = s["eng"]
        s["u"] = _displacement(_nodes(grid), g)
        s["key"] = "oc:%s:%s:%s" % (grid, c["rmin"], c["preserve"])
        s["hs"] = eng.filter_hs(grid, c["rmin"])
        eng.oc_prepare(grid, c["rmin"], s["pres"], key=s["key"])
    elif kind == "apply":
        s["p"] = _displacement(_nodes(grid), g).float()
        s["mask"] = None
        if c["masked"]:
            s["mask"] = torch.as_tensor(B.node_mask(*grid, B.clamp_face(*grid, "x_min")), device="cuda")
    elif kind == "edof":
        s["p"] = _displacement(_nodes(grid), g).float()
        s["edof"] = _edof(grid)
        s["Ke"] = torch.as_tensor(get_engine().get_ke(), device="cuda")
    elif kind == "batch":
        s["batch"] = BatchFEM(s["eng"])
        s["designs"] = []
        for n in map(int, c["sizes"].split(",")):
            f, fixed = B.LOAD_CASES[c["load"]](n, n, n)
            s["designs"].append(s["batch"].upload(FEMDesign((n, n, n), _density((n, n, n), g), f, fixed)))
    elif kind == "evaluate":
        s["ev"] = VoxelFEMEvaluator(use_gpu=True, vae_model=_Decoder(c["size"]), engine=s["eng"])
        s["params"] = [DesignParameters(8.0, 2.0, latent_z=z) for z in _latents(c, seed)]
    elif kind == "generate":
        s["samples"] = _samples(c, seed)
    elif kind == "prep":
        s["vol"] = torch.stack([torch.sigmoid(1.5 * _smooth((c["D"], c["H"], c["W"]), g)).float()
                                for _ in range(c["batch"])])
    return s


# ---- one pass ----------------------------------------------------------------------------
def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "simp":
        x, u = s["x"].clone(), torch.zeros_like(s["f"])
        xphys, obj, _ = s["eng"].simp_run(s["grid"], _law(c), s["f"], s["mask"], x, u, c["volfrac"], c["rmin"],
                                          c["iters"], preserved=s["pres"])
        return {"x": x, "xphys": xphys, "u": u.float(), "objective": torch.tensor(obj)}
    if kind == "solve":
        u = torch.zeros_like(s["f"])
        s["eng"].solve(s["grid"], _law(c), s["x"], s["f"], s["mask"], u)
        return u.float()
    if kind == "update":
        eng, grid, law = s["eng"], s["grid"], _law(c)
        dc = eng.sensitivity(grid, law, s["x"], s["u"])
        dcf = eng.filter(grid, c["rmin"], dc, hs=s["hs"], transpose=True)
        xnew, xphys = eng.oc(grid, c["rmin"], c["volfrac"], s["x"], dcf, s["pres"], key=s["key"], prepared=True)
        return {"dc": dc, "dcf": dcf, "xnew": xnew, "xphys": xphys}
    if kind == "apply":
        return s["eng"].apply(s["grid"], _law(c), s["x"], s["p"], s["mask"])
    if kind == "edof":
        a = (s["Ke"], s["edof"], c["penal"], *s["grid"])
        return {"y": cuda_kernels.fused_spmv(s["x"], s["p"], *a), "dc": cuda_kernels.simp_sensitivity(s["x"], s["p"], *a)}
    if kind == "batch":
        for d in s["designs"]:
            d.du.zero_()
        s["batch"].solve_all(s["designs"])
        return {"u": [d.du.float() for d in s["designs"]], "compliance": torch.tensor([d.compliance for d in s["designs"]])}
    if kind == "evaluate":
        r = s["ev"].evaluate_batch(s["params"])
        return {k: torch.tensor([getattr(v, k) for v in r]) for k in ("compliance", "stress_max", "mass")}
    if kind == "generate":
        cases = [SimpCase(grid, v, f, dict(TopoDataGenerator.GEOM_BCS[geom]), 3.5, 1.5) for geom, grid, v, f in s["samples"]]
        BatchSIMP(cases, bc_fn=B.generator).run(c["iters"])
        return {"density": [k.density for k in cases], "history": torch.tensor([h for k in cases for h in k.history])}
    return s["eng"].voxel_prep(s["vol"], (c["d"], c["h"], c["w"]))


# ---- what a pass cannot do without ---------------------------------------------------------
APPLY_FLOPS = 2 * 24 * 24  # one element's dense product; the modal form needs 210


def _solve_work(ne, nd):
    """Inputs once (densities, load, mask), the displacement once; the products of one residual,
    since how many iterations it takes is the method's choice."""
    return 4 * ne + 8 * nd + nd // 3 + 8 * nd, APPLY_FLOPS * ne


def work(case):
    c, kind = case, case["kind"]
    if "nx" in c:
        ne, nd = math.prod(_grid_of(c)), 3 * math.prod(_nodes(_grid_of(c)))
        taps = sum(1 for i in range(-4, 5) for j in range(-4, 5) for k in range(-4, 5)
                   if i * i + j * j + k * k < c.get("rmin", 0) ** 2)
        update = 4 * ne + 8 * nd + 4 * 4 * ne, (APPLY_FLOPS + 50 + 4 * taps) * ne
    if kind == "simp":
        b, f = _solve_work(ne, nd)
        return {"bytes": c["iters"] * (b + 3 * 4 * ne), "flops": c["iters"] * (f + update[1])}
    if kind == "solve":
        b, f = _solve_work(ne, nd)
    elif kind == "update":
        b, f = update
    elif kind == "apply":
        b, f = 4 * ne + 8 * nd, APPLY_FLOPS * ne
    elif kind == "edof":
        b, f = 2 * (24 * 8 * ne + 8 * ne + 8 * nd), 2 * APPLY_FLOPS * ne
    elif kind == "batch":
        w = [_solve_work(n ** 3, 3 * (n + 1) ** 3) for n in map(int, c["sizes"].split(","))]
        b, f = sum(v[0] for v in w), sum(v[1] for v in w)
    elif kind == "evaluate":
        n = c["size"] // 2
        sb, sf = _solve_work(n ** 3, 3 * (n + 1) ** 3)
        b, f = c["batch"] * (4 * c["size"] ** 3 + sb) + 64 * c["size"] ** 3, c["batch"] * (sf + 32 * c["size"] ** 3)
    elif kind == "generate":
        sb, sf = _solve_work(20 * 9 * 12, 3 * 21 * 10 * 13)
        b, f = c["samples"] * c["iters"] * 2 * sb, c["samples"] * c["iters"] * 2 * sf
    else:
        vi, vo = c["batch"] * c["D"] * c["H"] * c["W"], c["batch"] * c["d"] * c["h"] * c["w"]
        b, f = 4 * (vi + vo), 60 * vo
    return {"bytes": int(b), "flops": int(f)}


# ---- the same in 64 bits -------------------------------------------------------------------
def _ke64():
    """Trilinear unit-cube hexahedron, E = 1, nu = 0.3, by 2x2x2 Gauss quadrature."""
    nu = 0.3
    D = np.zeros((6, 6))
    D[:3, :3] = nu
    D[range(3), range(3)] = 1 - nu
    D[range(3, 6), range(3, 6)] = (1 - 2 * nu) / 2
    D /= (1 + nu) * (1 - 2 * nu)
    corner = np.array([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]) * 2.0 - 1
    K = np.zeros((24, 24))
    for p in corner / math.sqrt(3):
        t = 1 + corner * p
        dN = 2 * 0.125 * np.stack([corner[:, d] * np.prod(np.delete(t, d, 1), 1) for d in range(3)])
        Bm = np.zeros((6, 24))
        for d in range(3):
            Bm[d, d::3] = dN[d]
        for r, (a, b) in enumerate(((0, 1), (1, 2), (0, 2))):
            Bm[3 + r, a::3], Bm[3 + r, b::3] = dN[b], dN[a]
        K += Bm.T @ D @ Bm / 8
    return torch.as_tensor(K, device="cuda")


def _E64(x, law, penal=3.0):
    x = x.double()
    return x.clamp(min=1e-3) ** penal if law == "ref" else 1e-9 + x ** penal * (1.0 - 1e-9)


def _dE64(x, law, penal=3.0):
    x = x.double()
    return penal * x.clamp(min=1e-3) ** (penal - 1) if law == "ref" else penal * x ** (penal - 1) * (1.0 - 1e-9)


def _K64(E, edof, K, p):
    return torch.zeros_like(p).index_add_(0, edof.reshape(-1), ((p[edof] @ K) * E[:, None]).reshape(-1))


def _solve64(grid, E, f, fixed, rtol=1e-12):
    """Jacobi-preconditioned conjugate gradients in 64 bits."""
    edof, K = _edof(grid), _ke64()
    free = torch.ones_like(f)
    free[torch.as_tensor(fixed, device="cuda")] = 0.0
    diag = torch.zeros_like(f).index_add_(0, edof.reshape(-1), (E[:, None] * K.diagonal()).reshape(-1))
    minv = torch.where((free > 0) & (diag > 0), 1.0 / diag.clamp(min=1e-300), torch.zeros_like(diag))
    u, r = torch.zeros_like(f), f * free
    z = minv * r
    p, rz, stop = z.clone(), torch.dot(r, z), rtol * torch.linalg.norm(r)
    for i in range(40000):
        q = _K64(E, edof, K, p) * free
        a = rz / torch.dot(p, q)
        u += a * p
        r -= a * q
        if i % 20 == 19 and bool(torch.linalg.norm(r) < stop):
            break
        z = minv * r
        rz, old = torch.dot(r, z), rz
        p = z + (rz / old) * p
    return u


def _ce64(grid, u):
    edof, K = _edof(grid), _ke64()
    return torch.cat([((v @ K) * v).sum(1) for v in (u[e] for e in edof.split(1 << 18))])


def _filter64(grid, rmin):
    """v -> H v for the cone filter of radius rmin (zero outside the grid)."""
    r = math.ceil(rmin)
    d = torch.arange(-r, r + 1, device="cuda", dtype=torch.float64)
    w = (rmin - torch.sqrt(d[:, None, None] ** 2 + d[:, None] ** 2 + d ** 2)).clamp(min=0)

    def H(v):
        pad = torch.nn.functional.pad(v.reshape(grid), (r,) * 6)
        out = torch.zeros(grid, dtype=torch.float64, device="cuda")
        for i in range(2 * r + 1):
            for j in range(2 * r + 1):
                for k in range(2 * r + 1):
                    if float(w[i, j, k]) > 0:
                        out += w[i, j, k] * pad[i:i + grid[0], j:j + grid[1], k:k + grid[2]]
        return out.reshape(-1)

    return H


def _oc64(H, Hs, x, dc, volfrac, pres, gpu_variant=False):
    x = x.double()
    l1, l2, steps, tol, eps, floor = 0.0, 1e9, 50, 1e-4, 1e-12, 1e-12
    if gpu_variant:
        l2, steps, tol, eps, floor = 2.0 * max(float((-dc).max()), 1.0), 30, 1e-5, 1e-15, 1e-15
    keep = None if pres is None else pres.bool()

    def physical(lam):
        v = (x * torch.sqrt((-dc / lam).clamp(min=floor))).clamp(0.0, 1.0)
        v = torch.minimum(torch.maximum(v, x - 0.2), x + 0.2)
        if keep is not None:
            v[keep] = 1.0
        ph = H(v) / Hs
        if keep is not None:
            ph[keep] = 1.0
        return v, ph

    for _ in range(steps):
        lam = 0.5 * (l1 + l2)
        if (l2 - l1) / (l1 + l2 + eps) < tol:
            break
        if float(physical(lam)[1].mean()) > volfrac:
            l1 = lam
        else:
            l2 = lam
    return physical(lam)


def _prep64(vol, shape, sigma=0.5, sharpness=15.0):
    """scipy's zoom(order=1) along each axis, a Gaussian with mirrored edges, the logistic."""
    v = vol.double()
    r = int(4 * sigma + 0.5)
    t = torch.arange(-r, r + 1, device="cuda", dtype=torch.float64)
    g = torch.exp(-0.5 / sigma ** 2 * t * t)
    g = g / g.sum()
    for axis, n in zip((1, 2, 3), shape):
        m = v.shape[axis]
        p = torch.arange(n, device="cuda", dtype=torch.float64) * ((m - 1) / (n - 1))
        i = p.floor().long().clamp(max=m - 1)
        w = (p - i).reshape([-1 if a == axis else 1 for a in range(4)])
        v = v.index_select(axis, i) * (1 - w) + v.index_select(axis, (i + 1).clamp(max=m - 1)) * w
        j = (torch.arange(n, device="cuda")[None] + t.long()[:, None]) % (2 * n)
        j = torch.where(j < n, j, 2 * n - 1 - j)
        v = sum(g[q] * v.index_select(axis, j[q]) for q in range(2 * r + 1))
    return torch.sigmoid(sharpness * (v - 0.5))


def exact(case, seed):
    c, kind, g = case, case["kind"], _gen(seed)
    if kind == "generate":
        return _generate64(c, seed)
    if kind == "evaluate":
        return _evaluate64(c, seed)
    if kind == "prep":
        vol = torch.stack([torch.sigmoid(1.5 * _smooth((c["D"], c["H"], c["W"]), g)).float() for _ in range(c["batch"])])
        return _prep64(vol, (c["d"], c["h"], c["w"]))
    if kind == "batch":
        out = {"u": [], "compliance": []}
        for n in map(int, c["sizes"].split(",")):
            x = _density((n, n, n), g)
            f, fixed = B.LOAD_CASES[c["load"]](n, n, n)
            f = torch.as_tensor(f, device="cuda")
            out["u"].append(_solve64((n, n, n), _E64(x, "modified"), f, fixed))
            out["compliance"].append(torch.dot(f, out["u"][-1]))
        out["compliance"] = torch.stack(out["compliance"])
        return out
    grid = _grid_of(c)
    x = _density(grid, g)
    law = c.get("law", "modified")
    if kind == "apply":
        p = _displacement(_nodes(grid), g).float().double()
        clamped = torch.as_tensor(B.clamp_face(*grid, "x_min"), device="cuda") if c["masked"] else None
        if clamped is not None:
            p[clamped] = 0.0
        y = _K64(_E64(x, law), _edof(grid), _ke64(), p)
        if clamped is not None:
            y[clamped] = 0.0
        return y
    if kind == "edof":
        p = _displacement(_nodes(grid), g).float().double()
        return {"y": _K64(_E64(x, "ref", c["penal"]), _edof(grid), _ke64(), p),
                "dc": -_dE64(x, "ref", c["penal"]) * _ce64(grid, p)}
    if kind in ("simp", "solve"):
        if math.prod(grid) > EXACT_ELEMENTS:
            return None
        f, fixed = B.LOAD_CASES[c["load"]](*grid)
        f = torch.as_tensor(f, device="cuda")
    if kind == "solve":
        return _solve64(grid, _E64(x, law), f, fixed)
    pres = _preserved(c, grid)
    if pres is not None:
        x[pres.bool()] = 1.0
    H = _filter64(grid, c["rmin"])
    Hs = H(torch.ones(math.prod(grid), dtype=torch.float64, device="cuda"))
    if kind == "update":
        dc = -_dE64(x, law) * _ce64(grid, _displacement(_nodes(grid), g))
        dcf = H(dc / Hs)
        xnew, xphys = _oc64(H, Hs, x, dcf, c["volfrac"], pres)
        return {"dc": dc, "dcf": dcf, "xnew": xnew, "xphys": xphys}
    x, obj = x.double(), []
    xphys = x
    for _ in range(c["iters"]):
        u = _solve64(grid, _E64(xphys, law), f, fixed)
        ce = _ce64(grid, u)
        obj.append((_E64(xphys, law) * ce).sum())
        x, xphys = _oc64(H, Hs, x, H(-_dE64(xphys, law) * ce / Hs), c["volfrac"], pres)
    return {"x": x, "xphys": xphys, "u": u, "objective": torch.stack(obj)}


def _evaluate64(c, seed):
    n = round(c["size"] * 0.5)
    dec = _Decoder(c["size"])
    dec.fields = dec.fields.double()
    z = torch.as_tensor(_latents(c, seed), device="cuda")
    rho = _prep64(dec.decode(z)[:, 0], (n, n, n))
    f, fixed = B.reference_gpu(n, n, n, {"fixed_face": "x_min", "load_face": "x_max", "load_dof": 2}, 1000.0)
    f = torch.as_tensor(f, device="cuda")
    out = {"compliance": [], "stress_max": [], "mass": []}
    for v in rho:
        comp = float(torch.dot(f, _solve64((n, n, n), v.reshape(-1).clamp(min=1e-3), f, fixed)))
        solid = int((v > 0.5).sum())
        ok = solid >= 50 and comp >= 1.0
        out["compliance"].append(min(comp, 1e8) if ok else 1e6)
        out["stress_max"].append(min(comp / max(solid, 1) * 10.0, 1e4) if ok else 1e4)
        out["mass"].append(float(n ** 3) * (solid / n ** 3) * 7900 / 1e9)
    return {k: torch.tensor(v, dtype=torch.float64) for k, v in out.items()}


def _generate64(c, seed):
    out = {"density": [], "history": []}
    for geom, grid, volfrac, force in _samples(c, seed):
        f, fixed = B.generator(*grid, dict(TopoDataGenerator.GEOM_BCS[geom]), force)
        f = torch.as_tensor(f, device="cuda")
        H = _filter64(grid, 1.5)
        ne = math.prod(grid)
        Hs = H(torch.ones(ne, dtype=torch.float64, device="cuda"))
        x = xphys = torch.full((ne,), volfrac, dtype=torch.float32, device="cuda").double()
        for _ in range(c["iters"]):
            u = _solve64(grid, _E64(xphys, "ref", 3.5), f, fixed)
            dc = -_dE64(xphys, "ref", 3.5) * _ce64(grid, u)
            x, xphys = _oc64(H, Hs, x, H(dc / Hs), volfrac, None, gpu_variant=True)
            out["history"].append(torch.dot(f, _solve64(grid, _E64(xphys, "ref", 3.5), f, fixed)))
        out["density"].append(xphys.reshape(grid))
    out["history"] = torch.stack(out["history"])
    return out
