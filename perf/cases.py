"""The work that users of this framework have it do, as measurable cases.

Every case goes through the public entry points of fcgpu.py (or, for calls
whose arrays live on the device, through the C ABI that module declares).
The kinds:

  poisson   the pressure equation: laplacian() and ICCG on the mesh system,
            FP64 or with the multicolour mixed-precision inner solve
  csrsolve  the drop-in csrsolve call on the host arrays of a Fortran program
  simple    one outer SIMPLE iteration of the lid-driven cavity (hexahedra or
            tetrahedra): gradients, momentum and pressure assembly, BiCGStab
            and ICCG
  piso      one PISO time step of the same cavity
  sst       one k-omega SST update (gradients, strain, two scalar equations)
  grad      one cell gradient, with the case's limiter
  batch     independent convection-diffusion systems solved in one launch
  adjoint   assembly, forward solve and discrete adjoint of a scalar equation

Cell counts per side run from 9 to 128, odd and unequal sides among them.
"""
import importlib
import math

import numpy as np
import torch

fc = importlib.import_module("freecappuccino-dev_gb300.fcgpu")

PERTURB = 0.15        # interior vertices moved by up to this share of the spacing
LID = 3               # the ymax patch of the box generator
SCHEMES = {"gauss": fc.FC_GRAD_GAUSS, "lsq": fc.FC_GRAD_LSQ, "lsq_dm": fc.FC_GRAD_LSQ_DM}
LIMITERS = {"none": fc.FC_LIMITER_NONE, "bj": fc.FC_LIMITER_BJ, "venkat": fc.FC_LIMITER_VENKAT}
TWO_PI = 2.0 * math.pi


def listed():
    return [
        # the benchmark's pressure solve at its own size: the largest solve
        {"name": "poisson_128", "kind": "poisson", "nx": 128, "ny": 128, "nz": 128, "mode": "fp64"},
        # an ordinary pressure solve on an odd, uneven box
        {"name": "poisson_61x47x53", "kind": "poisson", "nx": 61, "ny": 47, "nz": 53, "mode": "fp64"},
        # the same equation with FP32 inner solves inside FP64 refinement
        {"name": "poisson_mixed_101", "kind": "poisson", "nx": 101, "ny": 96, "nz": 88, "mode": "coloured"},
        # the smallest calls: a host program's csrsolve, where latency counts
        {"name": "csrsolve_host_small", "kind": "csrsolve", "nx": 14, "ny": 11, "nz": 9, "solver": "bicgstab",
         "pe": 1.0},
        # the full SIMPLE iteration of the benchmark on perturbed hexahedra
        {"name": "simple_hex_128", "kind": "simple", "nx": 128, "ny": 128, "nz": 128, "tets": False,
         "perturb": PERTURB},
        # the plain method: the uniform 64^3 cavity
        {"name": "simple_hex_64", "kind": "simple", "nx": 64, "ny": 64, "nz": 64, "tets": False, "perturb": 0.0},
        # tetrahedra (4 faces a cell, uneven dependency levels), least-squares
        # gradients and a bounded scheme
        {"name": "simple_tets_50", "kind": "simple", "nx": 50, "ny": 50, "nz": 50, "tets": True, "perturb": PERTURB},
        # a transient run's time step
        {"name": "piso_48", "kind": "piso", "nx": 48, "ny": 48, "nz": 48},
        # the turbulence model's share of an outer iteration
        {"name": "sst_96", "kind": "sst", "nx": 96, "ny": 96, "nz": 96},
        # a cell gradient by itself, limited, at the largest size
        {"name": "grad_lsq_venkat_128", "kind": "grad", "nx": 128, "ny": 128, "nz": 128, "scheme": "lsq",
         "limiter": "venkat"},
        # many uneven scalar problems at once
        {"name": "batch_16", "kind": "batch", "count": 16, "lo": 20, "hi": 56, "sizes": 44},
        # sensitivities of a scalar equation
        {"name": "adjoint_56", "kind": "adjoint", "nx": 56, "ny": 56, "nz": 56},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """Three sides around a common size spread over the range's logarithm."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return {k: max(lo, min(hi, int(round(n * rng.uniform(0.8, 1.2))))) for k in ("nx", "ny", "nz")}


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "csrsolve", "simple", "simple", "piso", "sst", "grad", "batch", "adjoint"])
    if kind == "poisson":
        return {"kind": kind, **_sides(rng, 16, 120), "mode": rng.choice(["fp64", "fp64", "coloured"])}
    if kind == "csrsolve":
        return {"kind": kind, **_sides(rng, 9, 40), "solver": rng.choice(["bicgstab", "iccg", "dpcg"]),
                "pe": rng.lognormvariate(0.0, 1.0)}
    if kind == "simple":
        tets = rng.random() < 0.4
        return {"kind": kind, **_sides(rng, 12, 50 if tets else 112), "tets": tets,
                "perturb": rng.choice([0.0, PERTURB]) if not tets else PERTURB}
    if kind in ("piso", "adjoint"):
        return {"kind": kind, **_sides(rng, 16, 56)}
    if kind == "sst":
        return {"kind": kind, **_sides(rng, 16, 104)}
    if kind == "grad":
        return {"kind": kind, **_sides(rng, 16, 128), "scheme": rng.choice(sorted(SCHEMES)),
                "limiter": rng.choice(sorted(LIMITERS))}
    return {"kind": kind, "count": rng.randint(3, 16), "lo": 16, "hi": _log_int(rng, 24, 56),
            "sizes": rng.randrange(1 << 20)}


# ------------------------------------------------------ 7-point systems
def _box_index(nx, ny, nz):
    k, j, i = torch.meshgrid(torch.arange(nz, device="cuda"), torch.arange(ny, device="cuda"),
                             torch.arange(nx, device="cuda"), indexing="ij")
    return i.reshape(-1), j.reshape(-1), k.reshape(-1)


def _csr7(nx, ny, nz, w):
    """1-based CSR (ia, ja, diag) and values of a 7-point operator on the box
    nx x ny x nz, cells numbered x first; w: coefficients (n, 7) in column
    order -z, -y, -x, diagonal, +x, +y, +z, read where the neighbour exists."""
    i, j, k = _box_index(nx, ny, nz)
    n = nx * ny * nz
    one = torch.ones(n, dtype=torch.bool, device="cuda")
    has = torch.stack([k > 0, j > 0, i > 0, one, i < nx - 1, j < ny - 1, k < nz - 1], 1)
    off = torch.tensor([-nx * ny, -nx, -1, 0, 1, nx, nx * ny], device="cuda")
    ja = ((torch.arange(n, device="cuda")[:, None] + off)[has] + 1).to(torch.int32)
    cnt = has.sum(1)
    ia = torch.ones(n + 1, dtype=torch.int64, device="cuda")
    ia[1:] += torch.cumsum(cnt, 0)
    diag = (ia[:-1] + has[:, :3].sum(1)).to(torch.int32)
    return ia.to(torch.int32), ja, diag, w[has]


def _neighbours(v, nx, ny, nz):
    """The six neighbours' values of a cell field in the order -z, -y, -x,
    +x, +y, +z; the cell's own value where there is none."""
    v = v.view(nz, ny, nx)
    out = []
    for axis, step in ((0, -1), (1, -1), (2, -1), (2, 1), (1, 1), (0, 1)):
        m = v.shape[axis]
        idx = (torch.arange(m, device="cuda") + step).clamp(0, m - 1)
        out.append(v.index_select(axis, idx).reshape(-1))
    return out


def _poisson_inputs(case, seed):
    """Cell diffusivity (lognormal) and right-hand side (N(0,1), no mean)."""
    n = case["nx"] * case["ny"] * case["nz"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    mu = torch.exp(0.5 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    b = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return mu, b - b.mean()


def _poisson_matrix(case, mu):
    """The implicit Laplacian of the uniform unit box, Dirichlet on x = 0."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = [1.0 / nx, 1.0 / ny, 1.0 / nz]
    i, j, k = _box_index(nx, ny, nz)
    t = {"x": h[1] * h[2] / h[0], "y": h[0] * h[2] / h[1], "z": h[0] * h[1] / h[2]}
    has = [k > 0, j > 0, i > 0, i < nx - 1, j < ny - 1, k < nz - 1]
    w = torch.zeros(nx * ny * nz, 7, dtype=torch.float64, device="cuda")
    for e, (m, nb, ax) in enumerate(zip(has, _neighbours(mu, nx, ny, nz), "zyxxyz")):
        w[:, e if e < 3 else e + 1] = torch.where(m, 0.5 * (mu + nb) * t[ax], 0.0)
    w[:, 3] = -w.sum(1) - torch.where(i == 0, 2.0 * mu * t["x"], 0.0)
    return _csr7(nx, ny, nz, w)


def _cd_system(nx, ny, nz, pe, seed, symmetric=False):
    """Upwind convection-diffusion on [0, 2 pi]^3 with the velocity
    0.5 (sin x cos y, -cos x sin y, 0.3), cell Peclet number pe and a
    lognormal diffusivity, phi = 0 outside; right-hand side: a Gaussian blob
    and noise.  Returns the CSR system and the cell centres."""
    h = [TWO_PI / nx, TWO_PI / ny, TWO_PI / nz]
    i, j, k = _box_index(nx, ny, nz)
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = nx * ny * nz
    gam = 0.5 * h[0] / pe * torch.exp(0.3 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    x, y, z = (i + 0.5) * h[0], (j + 0.5) * h[1], (k + 0.5) * h[2]
    area = {"x": h[1] * h[2], "y": h[0] * h[2], "z": h[0] * h[1]}
    step = {"x": h[0], "y": h[1], "z": h[2]}
    has = [k > 0, j > 0, i > 0, i < nx - 1, j < ny - 1, k < nz - 1]
    flow = 0.0 if symmetric else 0.5
    w = torch.zeros(n, 7, dtype=torch.float64, device="cuda")
    edge = torch.zeros(n, dtype=torch.float64, device="cuda")
    for e, (m, nb, ax) in enumerate(zip(has, _neighbours(gam, nx, ny, nz), "zyxxyz")):
        s = -1.0 if e < 3 else 1.0
        xf, yf = (x + s * 0.5 * h[0] if ax == "x" else x), (y + s * 0.5 * h[1] if ax == "y" else y)
        u = {"x": torch.sin(xf) * torch.cos(yf), "y": -torch.cos(xf) * torch.sin(yf),
             "z": torch.full_like(x, 0.3)}[ax]
        out_flux = s * flow * u * area[ax]
        dif = 0.5 * (gam + nb) * area[ax] / step[ax]
        w[:, e if e < 3 else e + 1] = torch.where(m, -(dif + torch.clamp(-out_flux, min=0.0)), 0.0)
        edge += torch.where(m, 0.0, 2.0 * gam * area[ax] / step[ax])
    w[:, 3] = edge - w.sum(1)
    r2 = (x - math.pi) ** 2 + (y - math.pi) ** 2 + (z - math.pi) ** 2
    b = torch.exp(-2.0 * r2) + 0.05 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    ia, ja, diag, a = _csr7(nx, ny, nz, w)
    return ia, ja, diag, a, b * (h[0] * h[1] * h[2]), torch.cat([x, y, z])


def _cd_case_system(case, seed):
    return _cd_system(case["nx"], case["ny"], case["nz"], case["pe"], seed, case["solver"] != "bicgstab")


def _batch_sizes(case):
    r = np.random.default_rng(case["sizes"])
    side = r.integers(case["lo"], case["hi"] + 1, (case["count"], 3))
    return side.tolist(), r.lognormal(0.0, 1.0, case["count"]).tolist()


def _batch_systems(case, seed):
    side, pe = _batch_sizes(case)
    return [_cd_system(*s, p, seed * 1000 + q) for q, (s, p) in enumerate(zip(side, pe))]


# -------------------------------------------------------------- contexts
class _Field:
    """A field of a context as the device array it is; keeps the context."""

    def __init__(self, ctx, name, count):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "version": 3,
                                         "data": (ctx.field_ptr(name), False)}


def _fields(ctx, names):
    return {k: torch.as_tensor(_Field(ctx, k, ctx.field_len(k)), device="cuda") for k in names}


def _cavity(case, seed, viscos):
    """Lid-driven cavity: the mesh, a seeded smooth flow to start from, the
    lid at u = 1, mass fluxes from the velocity."""
    m = fc.Mesh.box(case["nx"], case["ny"], case["nz"], 1.0, 1.0, 1.0, perturb=case.get("perturb", PERTURB),
                    seed=seed + 1, tets=case.get("tets", False))
    ctx = fc.Context()
    ctx.set_mesh(m)
    r = np.random.default_rng(seed)
    xc, yc, zc = ctx.geometry("xc"), ctx.geometry("yc"), ctx.geometry("zc")
    ph = r.uniform(0.0, TWO_PI, 3)
    u, v, w = np.zeros(m.numTotal), np.zeros(m.numTotal), np.zeros(m.numTotal)
    bump = 16.0 * xc * (1.0 - xc) * yc * (1.0 - yc)
    u[:m.numCells] = 0.2 * bump * np.sin(TWO_PI * yc + ph[0])
    v[:m.numCells] = 0.2 * bump * np.sin(TWO_PI * zc + ph[1])
    w[:m.numCells] = 0.2 * bump * np.sin(TWO_PI * xc + ph[2])
    a = m.arrays()
    lid = m.numCells + int(a["startFace"][LID]) - m.numInnerFaces
    u[lid:lid + int(a["nfaces"][LID])] = 1.0
    for k, f in dict(u=u, v=v, w=w).items():
        ctx.field_set(k, f)
    for k, f in dict(p=0.0, pp=0.0, den=1.0, vis=viscos, visw=viscos, flmass=0.0, a=0.0, dUdxi=0.0, dVdxi=0.0,
                     dWdxi=0.0, dPdxi=0.0).items():
        ctx.field_fill(k, f)
    return m, ctx


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "poisson":
        m = fc.Mesh.box(case["nx"], case["ny"], case["nz"])
        ctx = fc.Context()
        ctx.set_mesh(m)
        if case["mode"] == "coloured":
            ctx.set_precision(fc.FC_PREC_MIXED_COLOURED, 1e-5, 0)
        mu, b = _poisson_inputs(case, seed)
        ctx.field_set("su", b.cpu().numpy())
        s.update(ctx=ctx, mu=mu, phi=torch.zeros(m.numTotal, dtype=torch.float64, device="cuda"))
        s["out"] = _fields(ctx, ["pp", "a"])
        s["out"]["pp"] = s["out"]["pp"][:m.numCells]
    elif kind == "csrsolve":
        ia, ja, diag, a, b, _ = (t.cpu().numpy() for t in _cd_case_system(case, seed))
        s.update(ctx=fc.Context(), sys=(ia, ja, a, diag), b=b, x0=np.zeros(len(b)))
    elif kind in ("simple", "piso"):
        tets = case.get("tets", False)
        viscos = 1.0 / 400.0 if tets else 0.01
        m, ctx = _cavity(case, seed, viscos)
        kw = dict(viscos=viscos)
        if tets:
            kw.update(scheme=19, grad=1, urfU=0.6, urfP=0.2)
        if kind == "piso":
            kw.update(urfU=1.0, urfP=1.0, maxiterU=20, maxiterP=100, tolRelU=1e-6, tolRelP=1e-6)
        ctx.simple_params(fc.SimpleParams.cavity(**kw))
        if kind == "piso":
            ctx.transient_params(0.1 / max(case["nx"], case["ny"], case["nz"]), fc.FC_TIME_BDF, 1, 2)
        ctx.init_flmass()
        s.update(ctx=ctx, out=_fields(ctx, ["u", "v", "w", "p", "flmass"]))
    elif kind == "sst":
        m, ctx = _cavity(case, seed, 1e-3)
        ctx.simple_params(fc.SimpleParams.cavity(viscos=1e-3))
        ctx.turbulence_params(fc.TurbulenceParams.defaults())
        ctx.init_flmass()
        ctx.wall_distance()
        s.update(ctx=ctx, out=_fields(ctx, ["te", "ed", "vis", "fsst", "magStrain"]))
        s["start"] = dict(te=1e-4, ed=1.0, fsst=0.0, vis=1e-3, visw=1e-3)
    elif kind == "grad":
        m = fc.Mesh.box(case["nx"], case["ny"], case["nz"], perturb=PERTURB, seed=seed + 1)
        ctx = fc.Context()
        ctx.set_mesh(m)
        ctx.set_gradient_limiter(LIMITERS[case["limiter"]])
        g = torch.Generator(device="cuda").manual_seed(seed)
        xyz = torch.from_numpy(np.stack([ctx.geometry(k) for k in ("xc", "yc", "zc")])).cuda()
        phi = torch.randn(m.numTotal, generator=g, device="cuda", dtype=torch.float64) * 0.01
        phi[:m.numCells] += torch.tanh(8.0 * (xyz[0] - 0.5)) * torch.cos(TWO_PI * xyz[1]) + xyz[2] ** 2
        s.update(ctx=ctx, phi=phi, out=torch.empty(3 * m.numTotal, dtype=torch.float64, device="cuda"))
    elif kind == "batch":
        ctx = fc.Context()
        batch = fc.Batch(ctx)
        systems = _batch_systems(case, seed)
        for ia, ja, diag, a, b, xyz in systems:
            batch.add(*(t.cpu().numpy() for t in (ia, ja, diag, xyz)))
        batch.plan()
        s.update(ctx=ctx, batch=batch, a=[t[3] for t in systems], b=[t[4] for t in systems],
                 x=[torch.zeros_like(t[4]) for t in systems], stream=torch.cuda.ExternalStream(ctx.stream()))
    elif kind == "adjoint":
        m = fc.Mesh.box(case["nx"], case["ny"], case["nz"], TWO_PI, TWO_PI, TWO_PI, perturb=PERTURB, seed=seed + 1)
        ctx = fc.Context()
        ctx.set_mesh(m)
        ctx.field_set("flmass", fc.stream_function_fluxes(m.arrays(), lambda x, y, z: 0.5 * np.sin(x) * np.sin(y)))
        xc, yc, zc, vol = (ctx.geometry(k) for k in ("xc", "yc", "zc", "vol"))
        gamma = np.exp(np.random.default_rng(seed).normal(-4.0, 0.5, m.numCells))
        src = np.exp(-2.0 * ((xc - math.pi) ** 2 + (yc - math.pi) ** 2 + (zc - math.pi) ** 2))
        weight = np.where(xc > math.pi, 2.0 * vol / vol[xc > math.pi].sum(), 0.0)
        s.update(ctx=ctx, gamma=gamma, src=src, weight=weight)
    torch.cuda.synchronize()
    return s


def run(s):
    kind, case, ctx = s["kind"], s["case"], s["ctx"]
    if kind == "poisson":
        ctx.laplacian(s["mu"], s["phi"], 0b1)
        ctx.field_fill("pp", 0.0)
        r0, _, _ = ctx.solve_field("iccg", "pp", "su", 20000, 0.0, 1e-10)
        return dict(s["out"], res0=r0)
    if kind == "csrsolve":
        ia, ja, a, diag = s["sys"]
        x, r0, _, _ = ctx.csrsolve(case["solver"], ia, ja, a, diag, s["x0"], s["b"], 500, 0.0, 1e-8)
        return {"x": x, "res0": r0}
    if kind == "simple":
        return dict(s["out"], resor=ctx.simple_iteration())
    if kind == "piso":
        ctx.time_shift()
        return dict(s["out"], resor=ctx.piso_iteration())
    if kind == "sst":
        for k, f in s["start"].items():  # the model's uniform start
            ctx.field_fill(k, f)
        return dict(s["out"], resor=ctx.kw_sst())
    if kind == "grad":
        st = fc.lib().fc_grad(ctx.h, SCHEMES[case["scheme"]], s["phi"].data_ptr(), s["out"].data_ptr())
        if st != 0:
            raise RuntimeError(ctx.error())
        return s["out"]
    if kind == "batch":
        with torch.cuda.stream(s["stream"]):
            for x in s["x"]:
                x.zero_()
        s["batch"].solve(s["a"], s["x"], s["b"], 500, 0.0, 1e-8)
        return s["x"]
    ctx.cd_assemble(s["gamma"], s["src"])
    phi, _ = ctx.cd_solve(2000, 1e-6)
    lam, grad, _ = ctx.cd_adjoint(s["weight"] * phi, 2000, 1e-6)
    return {"phi": phi, "lambda": lam, "dJdgamma": grad}


# ------------------------------------------------------------------ work
def _cells(case):
    return case["nx"] * case["ny"] * case["nz"] * (6 if case.get("tets") else 1)


def _nnz(n, tets=False):
    return (5 if tets else 7) * n


def work(case):
    """Bytes and operations of one pass: per solver iteration the matrix and
    the vectors once per pass over them (12 bytes an entry, 8 a value), with
    the iteration counts typical of the case; per assembly the fields and the
    geometry once."""
    kind = case["kind"]
    if kind == "batch":
        side, _ = _batch_sizes(case)
        n = sum(a * b * c for a, b, c in side)
        its = 30
        return {"bytes": its * n * (4 * 12 * 7 + 20 * 8.0), "flops": its * n * (8 * 7 + 30.0)}
    n = _cells(case)
    nnz = _nnz(n, case.get("tets", False))
    cg = (2 * 12 * nnz + 17 * 8 * n, 4 * nnz + 12 * n)           # one ICCG iteration
    bi = (4 * 12 * nnz + 30 * 8 * n, 8 * nnz + 24 * n)           # one BiCGStab iteration
    if kind == "poisson":
        its = 2.8 * max(case["nx"], case["ny"], case["nz"])
        half = 0.5 if case["mode"] == "coloured" else 1.0        # FP32 matrix and vectors
        return {"bytes": its * half * cg[0] + 20 * 8.0 * n, "flops": its * cg[1]}
    if kind == "csrsolve":
        its = max(case["nx"], case["ny"], case["nz"])
        return {"bytes": its * bi[0] + 12.0 * nnz, "flops": its * float(bi[1])}
    if kind == "simple":
        return {"bytes": 3 * 4 * bi[0] + 20 * cg[0] + 150 * 8.0 * n, "flops": 12 * bi[1] + 20 * cg[1] + 2500.0 * n}
    if kind == "piso":
        return {"bytes": 3 * 6 * bi[0] + 2 * 80 * cg[0] + 200 * 8.0 * n,
                "flops": 18 * bi[1] + 160 * cg[1] + 3000.0 * n}
    if kind == "sst":
        return {"bytes": 2 * 4 * bi[0] + 150 * 8.0 * n, "flops": 8 * bi[1] + 1500.0 * n}
    if kind == "grad":
        return {"bytes": 30 * 8.0 * n, "flops": 200.0 * n}
    return {"bytes": 2 * 60 * bi[0] + 40 * 8.0 * n, "flops": 120.0 * bi[1]}


# ----------------------------------------------------------------- exact
def _solve64(ia, ja, a, diag, b, symmetric):
    """A x = b to rounding: Jacobi-preconditioned CG or BiCGStab of torch's
    64-bit products, restarted on the true residual."""
    n = b.numel()
    A = torch.sparse_csr_tensor(ia.long() - 1, ja.long() - 1, a, size=(n, n))
    dinv = 1.0 / a[diag.long() - 1]
    x = torch.zeros_like(b)
    bn = float(b.norm())
    last = math.inf
    for _ in range(6):
        r = b - A @ x
        rn = float(r.norm())
        if rn <= 1e-15 * bn or rn > 0.5 * last:
            break
        last = rn
        x = x + (_cg(A, dinv, r) if symmetric else _bicgstab(A, dinv, r))
    return x


def _cg(A, dinv, b):
    x, r = torch.zeros_like(b), b.clone()
    z = dinv * r
    p, rz = z.clone(), torch.dot(r, z)
    stop = 1e-9 * float(b.norm())
    for it in range(6000):
        q = A @ p
        alpha = rz / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        if it % 20 == 19 and float(r.norm()) <= stop:
            break
        z = dinv * r
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _bicgstab(A, dinv, b):
    x, r = torch.zeros_like(b), b.clone()
    r0, p, rho = r.clone(), r.clone(), torch.dot(r, r)
    stop = 1e-8 * float(b.norm())
    for it in range(4000):
        ph = dinv * p
        v = A @ ph
        alpha = rho / torch.dot(r0, v)
        s = r - alpha * v
        sh = dinv * s
        t = A @ sh
        omega = torch.dot(t, s) / torch.dot(t, t)
        x += alpha * ph + omega * sh
        r = s - omega * t
        if it % 5 == 4 and not float(r.norm()) > stop:
            break
        new = torch.dot(r0, r)
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return x


def exact(case, seed):
    """64-bit values where the path computes the solution of a system that
    this file can state by itself; SIMPLE, PISO and SST steps, limited
    gradients and the adjoint have no such value."""
    kind = case["kind"]
    if kind == "poisson":
        mu, b = _poisson_inputs(case, seed)
        ia, ja, diag, a = _poisson_matrix(case, mu)
        return {"pp": _solve64(ia, ja, a, diag, b, True), "a": a, "res0": None}
    if kind == "csrsolve":
        ia, ja, diag, a, b, _ = _cd_case_system(case, seed)
        return {"x": _solve64(ia, ja, a, diag, b, case["solver"] != "bicgstab").cpu().numpy(), "res0": None}
    if kind == "batch":
        return [_solve64(ia, ja, a, diag, b, False) for ia, ja, diag, a, b, _ in _batch_systems(case, seed)]
    return None
