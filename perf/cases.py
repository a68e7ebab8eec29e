"""Workloads of the pressure path, as a program that uses this package calls it.

Every case is one call sequence through the public entry points on device
tensors: engine solves, the pressure-correction step, a batch of independent
problems, the reference-parity Krylov solvers, Gauss-Seidel and multigrid,
and the flow functions alone. Fields are bubbles in a liquid, with an upright
cylinder as a voxel body where the case has one: the shapes, density ratios
and right-hand sides of this repository's own generator, on grids of any
three extents.
"""
import math
import random

import torch

import psiboil_b200 as pb

DEV = "cuda"
F64 = torch.float64
RATIO = 1000.0   # liquid over vapour density of the single problems


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: a coarse test grid, one solve; latency and launches
        dict(name="solve_tiny", kind="solve", nx=20, ny=16, nz=18, body=False, precision="mixed",
             coarse_max=0),
        # the headline size: many right-hand sides on one matrix
        dict(name="solve_mixed_256", kind="solve", nx=256, ny=256, nz=256, body=True, precision="mixed",
             coarse_max=4096),
        # the same solver with every level in 64 bits
        dict(name="solve_fp64_128", kind="solve", nx=128, ny=128, nz=128, body=True, precision="fp64",
             coarse_max=0),
        # one time step of a two-phase run on a grid with odd extents:
        # assembly, right-hand side, solve, projection
        dict(name="step_odd", kind="step", nx=150, ny=117, nz=131, body=True, precision="mixed"),
        # a parameter study: independent uneven 2-D and 3-D problems at once
        dict(name="batch_mixed", kind="batch", count=48, two_d=24, s2lo=48, s2hi=256, s3lo=16, s3hi=64,
             pick=7, precision="mixed"),
        # the reference's plain CG, a fixed number of iterations
        dict(name="cg_di_128", kind="krylov", solver="cg", prec="di", nx=128, ny=128, nz=128, body=True,
             convect=False, iters=100),
        # the reference's usual pressure solver, CG with IC2
        dict(name="cg_ic2", kind="krylov", solver="cg", prec="ic2", nx=64, ny=56, nz=50, body=True,
             convect=False, iters=20),
        # a convected (non-symmetric) equation
        dict(name="bicgs_convected", kind="krylov", solver="bicgs", prec="di", nx=96, ny=80, nz=72,
             body=True, convect=True, iters=12),
        # CG whose sums are the reference's bit for bit
        dict(name="cg_exact", kind="exact_cg", nx=64, ny=64, nz=64, body=True, iters=40),
        # Gauss-Seidel sweeps
        dict(name="gauss_seidel", kind="gs", nx=64, ny=72, nz=60, body=True, iters=10),
        # the reference's multigrid, CG smoothing
        dict(name="ac_vcycle", kind="ac", nx=96, ny=96, nz=96, body=True, cycles=2),
        # the flow functions without a solve, on a grid that fills memory bandwidth:
        # a program that keeps its own solver
        dict(name="flow_large", kind="flow", nx=384, ny=320, nz=256, body=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi, cells):
    while True:
        d = [_log(rng, lo, hi) for _ in range(3)]
        if d[0] * d[1] * d[2] <= cells:
            return dict(nx=d[0], ny=d[1], nz=d[2])


def draw(rng):
    kind = rng.choice(["solve", "solve", "step", "step", "batch", "krylov", "krylov", "exact_cg", "gs",
                       "ac", "flow"])
    c = dict(kind=kind, body=rng.random() < 0.6)
    if kind == "solve":
        c.update(_dims(rng, 14, 256, 1 << 23))
        c.update(precision=rng.choice(["mixed", "mixed", "fp64"]), coarse_max=rng.choice([0, 0, 4096]))
    elif kind == "step":
        c.update(_dims(rng, 16, 220, 1 << 23), precision=rng.choice(["mixed", "mixed", "fp64"]))
    elif kind == "batch":
        n = rng.randint(4, 48)
        del c["body"]
        c.update(count=n, two_d=rng.randint(0, n), s2lo=32, s2hi=256, s3lo=12, s3hi=64,
                 pick=rng.randrange(1 << 16), precision=rng.choice(["mixed", "mixed", "fp64"]))
    elif kind == "krylov":
        solver = rng.choice(["cg", "cg", "bicgs"])
        prec = rng.choice(["di", "di", "ic0", "ic2"])
        c.update(_dims(rng, 24, 160 if prec == "di" else 96, 1 << 21 if prec == "di" else 1 << 18))
        c.update(solver=solver, prec=prec, convect=solver == "bicgs" and rng.random() < 0.7,
                 iters=rng.randint(6, 12 if solver == "bicgs" else 100 if prec == "di" else 20))
    elif kind == "exact_cg":
        c.update(_dims(rng, 20, 96, 1 << 18), iters=rng.randint(8, 40))
    elif kind == "gs":
        c.update(_dims(rng, 16, 96, 1 << 18), iters=rng.randint(2, 12))
    elif kind == "ac":
        for d in ("nx", "ny", "nz"):
            c[d] = rng.choice([4, 5, 6, 7, 8, 9, 10, 12]) * rng.choice([4, 4, 8])
        c.update(cycles=rng.randint(1, 2))
    else:
        c.update(_dims(rng, 32, 400, 31 << 20))
    return c


# ---------------------------------------------------------------- fields
def _centres(dims):
    x, y, z = (torch.arange(n, device=DEV, dtype=F64) + 0.5 for n in dims)
    return x.view(-1, 1, 1), y.view(1, -1, 1), z.view(1, 1, -1)


def _bubbles(dims, rng):
    """Centres and radii in cells, inside the domain: up to 32 bubbles of
    1/64 to 1/16 of the longest side, at least 1.5 cells and at most a
    quarter of the shortest side."""
    side, out = min(n for n in dims if n > 1), []
    for _ in range(32 if min(dims) >= 64 else 8):
        r = min(max(rng.uniform(1 / 64, 1 / 16) * max(dims), 1.5), 0.25 * side)
        out.append([rng.uniform(r, n - r) if n > 1 else 0.5 for n in dims] + [r])
    return out


def _colour(dims, bubbles, width):
    """1 in the liquid, 0 in the vapour; a ramp of `width` cells across each
    surface, sharp when width is 0."""
    x, y, z = _centres(dims)
    col = torch.ones(dims, device=DEV, dtype=F64)
    for cx, cy, cz, r in bubbles:
        d = torch.sqrt((x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2) - r
        col = torch.minimum(col, (d / width + 0.5).clamp(0, 1) if width else (d >= 0).to(F64))
    return col


def _solid(dims, body):
    x, y, z = _centres(dims)
    r = 0.17 * min(dims[0], dims[1]) if body else 0.0
    s = (x - 0.45 * dims[0]) ** 2 + (y - 0.55 * dims[1]) ** 2 < r * r
    return s.expand(dims).to(torch.uint8).contiguous()


def _bc(dims):
    """Walls, with p = 0 on the top (kmax; jmax in 2-D)."""
    bc = [pb.NEUMANN] * 6
    bc[5 if dims[2] > 1 else 3] = pb.DIRICHLET
    return bc


def _cut(a, axis, lo, hi):
    return a.narrow(axis, lo, a.shape[axis] + hi - lo)


def _matrix(dims, h, rho, solid, harmonic, wall=1.0):
    """The pressure matrix A p = c p - sum a_nb p_nb (c, w, e, s, n, b, t):
    couplings dS / dx / rho_face, walls Neumann, the top Dirichlet with
    dx = wall * h, voxel solid cells decoupled with c scaled by 1e-12."""
    A = {}
    sol = solid.bool()
    bc = _bc(dims)
    c = torch.zeros(dims, device=DEV, dtype=F64)
    for ax, (lo, hi) in enumerate((("w", "e"), ("s", "n"), ("b", "t"))):
        L = torch.zeros(dims, device=DEV, dtype=F64)
        H = torch.zeros(dims, device=DEV, dtype=F64)
        if dims[ax] > 1:
            ra, rb = _cut(rho, ax, 0, -1), _cut(rho, ax, 1, 0)
            f = 2 * ra * rb / (ra + rb) if harmonic else 0.5 * (ra + rb)
            a = (h / f) * (_cut(sol, ax, 0, -1) == _cut(sol, ax, 1, 0))
            _cut(L, ax, 1, 0).copy_(a)
            _cut(H, ax, 0, -1).copy_(a)
        c += L + H
        if bc[2 * ax + 1] == pb.DIRICHLET:
            top = rho.narrow(ax, dims[ax] - 1, 1)
            c.narrow(ax, dims[ax] - 1, 1).add_(h / wall / top)
        A[lo], A[hi] = L, H
    # a solid cell keeps the sum over all its faces, scaled; its value is 0 here
    A["c"] = torch.where(sol, 1e-12 * 6 * h / rho, c)
    for k in "wesnbt":
        A[k] = torch.where(sol, torch.zeros_like(c), A[k])
    return A


def _noise(dims, g):
    return torch.rand(dims, generator=g, device=DEV, dtype=F64)


def _rhs(dims, h, solid, g):
    """U[-1, 1] on fluid cells less its mean, over h^2; 0 on solid cells."""
    f = solid == 0
    b = (2 * _noise(dims, g) - 1) * f
    return torch.where(f, b - b.sum() / f.sum(), torch.zeros_like(b)) / h ** 2


def _problem(case, seed):
    """Fields of a single problem from the seed alone."""
    dims = (case["nx"], case["ny"], case["nz"])
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    bubbles = _bubbles(dims, random.Random(seed))
    return dims, 1.0 / max(dims), bubbles, _solid(dims, case["body"]), g


def _system(case, seed):
    """A single problem in the harmonic density, with its right-hand side."""
    dims, h, bubbles, solid, g = _problem(case, seed)
    rho = 1.0 + (RATIO - 1.0) * _colour(dims, bubbles, 0)
    return dims, h, rho, solid, _rhs(dims, h, solid, g)


def _krylov_matrix(case, dims, h, rho, solid):
    A = _matrix(dims, h, rho, solid, True)
    if case.get("convect"):
        # first-order upwind convection along +x between fluid cells
        flow = torch.zeros(dims, device=DEV, dtype=F64)
        flow[1:] = (0.3 * h / RATIO) * ((solid[1:] == 0) & (solid[:-1] == 0))
        A["w"] = A["w"] + flow
        A["c"] = A["c"] + flow
    return A


def _flow_fields(case, seed):
    dims, h, bubbles, solid, g = _problem(case, seed)
    vel = []
    for ax in range(3):
        shape = list(dims)
        shape[ax] += 1
        u = _noise(shape, g) - 0.5
        u.narrow(ax, 0, 1).zero_()
        u.narrow(ax, dims[ax], 1).zero_()
        vel.append(u)
    return dims, h, _colour(dims, bubbles, 3.0), solid, vel, g


def _batch_fields(case, seed):
    """The members of a batch: sizes from the case, fields from the seed."""
    sizes = random.Random(case["pick"])
    rng = random.Random(seed)
    out = []
    for q in range(case["count"]):
        flat = q < case["two_d"]
        n = _log(sizes, case["s2lo"], case["s2hi"]) if flat else _log(sizes, case["s3lo"], case["s3hi"])
        dims = (n, n, 1 if flat else n)
        g = torch.Generator(device=DEV)
        g.manual_seed(seed * 4099 + q)
        ratio = 10.0 ** rng.uniform(1, 3)
        bub = [[rng.uniform(r, n - r), rng.uniform(r, n - r), 0.5 if flat else rng.uniform(r, n - r), r]
               for r in (rng.uniform(0.05, 0.2) * n for _ in range(rng.randint(1, 8)))]
        rho = 1.0 + (ratio - 1.0) * _colour(dims, bub, 0)
        solid = torch.zeros(dims, device=DEV, dtype=torch.uint8)
        out.append((dims, 1.0 / n, rho, solid, _rhs(dims, 1.0 / n, solid, g)))
    return out


# ---------------------------------------------------------------- prepare and run
DT = 1e-3   # time step of the flow cases


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        prec = pb.FP64 if case["precision"] == "fp64" else pb.MIXED
        B = pb.Batch(precision=prec, slots=64)
        ids, out = [], []
        for dims, h, rho, solid, b in _batch_fields(case, seed):
            ids.append(B.add(dims, h, rho=rho, solid=solid, b=b))
            out.append(torch.empty(dims, device=DEV, dtype=F64))
        return dict(kind=kind, B=B, ids=ids, out=out)
    if kind in ("step", "flow"):
        dims, h, col, solid, vel, g = _flow_fields(case, seed)
        st = dict(kind=kind, s=pb.Session(*dims, h), col=col, solid=solid if case["body"] else None,
                  vel0=vel, vel=[u.clone() for u in vel])
        if kind == "flow":
            st.update(p=_noise(dims, g) * DT, rhs=torch.empty_like(col), res=torch.empty_like(col))
        else:
            st["p"] = torch.zeros_like(col)
            st["par"] = pb.default_params(pb.SOLVER_ENGINE)
            st["par"].precision = pb.FP64 if case["precision"] == "fp64" else pb.MIXED
            st["par"].x0_zero = 1
        return st
    dims, h, rho, solid, b = _system(case, seed)
    s = pb.Session(*dims, h)
    st = dict(kind=kind, s=s, b=b, x=torch.zeros_like(b))
    if kind == "solve":
        s.assemble_pressure(rho, solid)
        st.update(eng=pb.Engine(s), cm=case["coarse_max"],
                  prec=pb.FP64 if case["precision"] == "fp64" else pb.MIXED)
        return st
    s.upload_matrix(_krylov_matrix(case, dims, h, rho, solid))
    if kind == "ac":
        s.upload_active((1 - solid.int()).cpu().numpy())
        st["ac"] = pb.AC(s)
        st["ac"].max_cycles(case["cycles"])
    elif kind == "gs":
        st.update(lin=pb.GaussSeidel(s), iters=case["iters"])
    elif kind == "exact_cg":
        st.update(lin=pb.CG(s, exact_sums=True), iters=case["iters"])
    else:
        cls = pb.BiCGS if case["solver"] == "bicgs" else pb.CG
        st.update(lin=cls(s, prec=case["prec"]), iters=case["iters"])
    return st


def run(st):
    kind = st["kind"]
    if kind == "solve":
        ok = st["eng"].solve(st["x"], st["b"], tol=1e-8, precision=st["prec"], coarse_max=st["cm"],
                             x0_zero=True)
        return dict(x=st["x"], converged=int(ok))
    if kind == "batch":
        B = st["B"]
        for i in st["ids"]:
            B.set_x(i)   # cold start
        res = B.solve(st["ids"], tol=1e-8)
        for i, x in zip(st["ids"], st["out"]):
            B.get_x(i, x)
        return dict(x=st["out"], converged=sum(r.converged for r in res))
    if kind in ("step", "flow"):
        # the predicted velocity of the step, which the projection updates in place
        for u, u0 in zip(st["vel"], st["vel0"]):
            u.copy_(u0)
        s, (u, v, w) = st["s"], st["vel"]
        if kind == "step":
            r = s.pressure_step(st["col"], RATIO, 1.0, DT, u, v, w, st["p"], st["par"], solid=st["solid"])
            return dict(u=u, v=v, w=w, p=st["p"], converged=int(r.converged))
        s.assemble_mix(st["col"], RATIO, 1.0, solid=st["solid"])
        s.divergence(u, v, w, DT, st["rhs"], solid=st["solid"])
        s.residual(st["p"], st["rhs"], st["res"])
        s.project(st["p"], st["col"], RATIO, 1.0, DT, u, v, w, solid=st["solid"])
        return dict(rhs=st["rhs"], res=st["res"], u=u, v=v, w=w)
    st["x"].zero_()
    if kind == "ac":
        st["ac"].vcycle(st["x"], st["b"])
    else:
        st["lin"].solve(st["x"], st["b"], 1, st["iters"], None, 1e-12, 1e-30)
    return dict(x=st["x"])


# ---------------------------------------------------------------- work and tolerance
def _cells(case):
    if case["kind"] != "batch":
        return case["nx"] * case["ny"] * case["nz"]
    sizes = random.Random(case["pick"])
    total = 0
    for q in range(case["count"]):
        flat = q < case["two_d"]
        n = _log(sizes, case["s2lo"], case["s2hi"]) if flat else _log(sizes, case["s3lo"], case["s3hi"])
        total += n * n if flat else n ** 3
    return total


def work(case):
    """Inputs read once and outputs written once; operations of the fewest
    stencil applications that the call's result stands for."""
    n, kind = _cells(case), case["kind"]
    if kind == "flow":
        # colour, flag, pressure, six velocity passes (read and write), two outputs
        return dict(bytes=n * (8 + 1 + 8 + 48 + 16), flops=n * 120)
    if kind == "step":
        return dict(bytes=n * (8 + 1 + 48 + 8), flops=n * 120)
    if kind in ("solve", "batch"):
        return dict(bytes=n * (32 + 8 + 8), flops=n * 13)   # symmetric matrix, b, x
    mat = 56 if case.get("convect") else 32
    if kind == "ac":
        return dict(bytes=n * (mat + 16), flops=n * case["cycles"] * 40 * 25)
    per = {"di": 25, "ic0": 40, "ic2": 50}[case.get("prec", "di")]
    per = 15 if kind == "gs" else per * (2 if case.get("solver") == "bicgs" else 1)
    return dict(bytes=n * (mat + 16), flops=n * case["iters"] * per)


def tolerance(case):
    kind = case["kind"]
    if kind == "exact_cg":
        return "exact"
    if kind in ("flow", "gs"):
        return dict(rel=1e-15)
    if kind in ("solve", "step", "batch"):
        return dict(rel=1e-6)   # what a residual of 1e-8 leaves in p
    # fixed iteration counts: sums in another order, about four times the
    # largest difference seen over the ranges (the product method amplifies it)
    return dict(rel=1e-10 if case.get("solver") == "bicgs" else 1e-11)


# ---------------------------------------------------------------- 64-bit results
def _ax(A, x):
    y = A["c"] * x
    y[1:] -= A["w"][1:] * x[:-1]
    y[:-1] -= A["e"][:-1] * x[1:]
    y[:, 1:] -= A["s"][:, 1:] * x[:, :-1]
    y[:, :-1] -= A["n"][:, :-1] * x[:, 1:]
    y[:, :, 1:] -= A["b"][:, :, 1:] * x[:, :, :-1]
    y[:, :, :-1] -= A["t"][:, :, :-1] * x[:, :, 1:]
    return y


def _dot(a, b):
    return (a * b).sum()


def _cg(A, b, x, prec, iters):
    """`iters` preconditioned CG steps (a vanished residual ends them)."""
    r = b - _ax(A, x)
    p, rho_old = None, None
    for _ in range(iters):
        z = prec(r)
        rho = _dot(r, z)
        p = z if p is None else torch.where(rho_old > 0, z + (rho / rho_old) * p, z)
        q = _ax(A, p)
        pq = _dot(p, q)
        a = torch.where(pq > 0, rho / pq, torch.zeros_like(pq))
        x = x + a * p
        r = r - a * q
        rho_old = rho
    return x


def _bicgs(A, b, x, prec, iters):
    r = b - _ax(A, x)
    rt, p, v = r, None, None
    rho_old = alfa = omega = None
    for _ in range(iters):
        rho = _dot(rt, r)
        if p is None:
            p = r
        else:
            beta = rho / rho_old * (alfa / omega)
            p = r + beta * p - beta * omega * v
        ph = prec(p)
        v = _ax(A, ph)
        alfa = rho / _dot(rt, v)
        s = r - alfa * v
        sh = prec(s)
        t = _ax(A, sh)
        omega = _dot(t, s) / _dot(t, t)
        x = x + alfa * ph + omega * sh
        r = s - omega * t
        rho_old = rho
    return x


def _solve_tight(systems):
    """CG on several independent systems at once to 1e-13, on flat vectors
    with one scalar per system."""
    dims = [A["c"].shape for A, _ in systems]
    lens = torch.tensor([d.numel() for d in dims], device=DEV)
    flat = [torch.cat([A[k].reshape(-1) for A, _ in systems]) for k in "cwesnbt"]
    c, nb = flat[0], flat[1:]
    b = torch.cat([r.reshape(-1) for _, r in systems])
    at = torch.arange(b.numel(), device=DEV)
    SI = torch.cat([torch.full((d.numel(),), d[1] * d[2], device=DEV) for d in dims])
    SJ = torch.cat([torch.full((d.numel(),), d[2], device=DEV) for d in dims])
    idx = [torch.clamp(at + o, 0, b.numel() - 1) for o in (-SI, SI, -SJ, SJ, -1, 1)]
    one = len(systems) == 1
    seg = (lambda v: v.sum().view(1)) if one else (lambda v: torch.segment_reduce(v, "sum", lengths=lens))
    each = (lambda s: s) if one else (lambda s: torch.repeat_interleave(s, lens, output_size=b.numel()))
    x, r = torch.zeros_like(b), b.clone()
    rho_old, p = None, None
    bb = seg(b * b)
    for it in range(40000):
        z = r / c
        rho = seg(r * z)
        p = z if p is None else z + each(torch.nan_to_num(rho / rho_old)) * p
        q = c * p
        for a, i in zip(nb, idx):
            q -= a * p[i]
        alfa = each(torch.nan_to_num(rho / seg(p * q)))
        x += alfa * p
        r -= alfa * q
        rho_old = rho
        if it % 50 == 49 and bool((seg(r * r) <= 1e-26 * bb).all()):
            break
    return [v.view(d) for v, d in zip(torch.split(x, lens.tolist()), dims)]


def _planes(dims, wa, wb):
    """Cells of every plane wa i + wb j + k = h, as flat indices of a grid
    padded by one cell on each side."""
    ix = [torch.arange(n, device=DEV) for n in dims]
    h = (wa * ix[0].view(-1, 1, 1) + wb * ix[1].view(1, -1, 1) + ix[2].view(1, 1, -1)).reshape(-1)
    pad = (((ix[0] + 1).view(-1, 1, 1) * (dims[1] + 2) + (ix[1] + 1).view(1, -1, 1)) * (dims[2] + 2)
           + (ix[2] + 1).view(1, 1, -1)).reshape(-1)
    order = torch.argsort(h, stable=True)
    return torch.split(pad[order], torch.bincount(h).tolist())


def _padded(a):
    return torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1)).reshape(-1)


def _unpadded(v, dims):
    return v.view([n + 2 for n in dims])[1:-1, 1:-1, 1:-1]


def _incomplete_cholesky(A, dims, kind):
    """IC0 / IC2 of the symmetric pattern; returns the application."""
    SI, SJ = (dims[1] + 2) * (dims[2] + 2), dims[2] + 2
    planes = _planes(dims, 2, 2)
    ac, aw, as_, ab = (_padded(A[k]) for k in "cwsb")
    c = torch.ones_like(ac)
    w, s, b, tw, ts = (torch.zeros_like(ac) for _ in range(5))
    for p in planes:
        d = torch.sqrt(ac[p] - w[p] ** 2 - tw[p] ** 2 - s[p] ** 2 - ts[p] ** 2 - b[p] ** 2)
        c[p] = d
        w[p + SI] = -aw[p + SI] / d
        s[p + SJ] = -as_[p + SJ] / d
        if kind == "ic2":
            tw[p + SI - 1] = -w[p + SI - 1] * b[p] / d
            ts[p + SJ - 1] = -s[p + SJ - 1] * b[p] / d
            b[p + 1] = (-ab[p + 1] - w[p + 1] * tw[p] - s[p + 1] * ts[p]) / d
        else:
            b[p + 1] = -ab[p + 1] / d

    def apply(r):
        z = torch.zeros_like(ac)
        rp = _padded(r)
        for p in planes:
            z[p] = (rp[p] - w[p] * z[p - SI] - tw[p] * z[p - SI + 1] - s[p] * z[p - SJ]
                    - ts[p] * z[p - SJ + 1] - b[p] * z[p - 1]) / c[p]
        for p in reversed(planes):
            z[p] = (z[p] - w[p + SI] * z[p + SI] - tw[p + SI - 1] * z[p + SI - 1] - s[p + SJ] * z[p + SJ]
                    - ts[p + SJ - 1] * z[p + SJ - 1] - b[p + 1] * z[p + 1]) / c[p]
        return _unpadded(z, dims)
    return apply


def _gauss_seidel(A, b, dims, sweeps):
    SI, SJ = (dims[1] + 2) * (dims[2] + 2), dims[2] + 2
    P = {k: _padded(A[k]) for k in "cwesnbt"}
    bp = _padded(b)
    x = torch.zeros_like(bp)
    planes = _planes(dims, 1, 1)
    for _ in range(sweeps):
        for p in planes:
            x[p] = (bp[p] + P["w"][p] * x[p - SI] + P["e"][p] * x[p + SI] + P["s"][p] * x[p - SJ]
                    + P["n"][p] * x[p + SJ] + P["b"][p] * x[p - 1] + P["t"][p] * x[p + 1]) / P["c"][p]
    return _unpadded(x, dims)


def _first_factor(n):
    """The smallest divisor above 1 (n itself when prime)."""
    return next((f for f in range(2, n) if n % f == 0), n)


def _blocks(a, f):
    n = [a.shape[d] // f[d] for d in range(3)]
    return a.view(n[0], f[0], n[1], f[1], n[2], f[2])


def _block_sum(a, f):
    return _blocks(a, f).sum(dim=(1, 3, 5))


def _multigrid(A, b, active, cycles):
    """Additive-correction V-cycles with CG smoothing: 20 steps before and
    after each level, 100 on the coarsest, zero-mean coarse right-hand sides."""
    levels = [dict(A=A, act=active, phi=torch.zeros_like(b), f=b)]
    while True:
        L = levels[-1]
        n = list(L["phi"].shape)
        f = [_first_factor(m) if m > 4 and _first_factor(m) != m else 1 for m in n]
        if f == [1, 1, 1]:
            break
        H = {}
        c = _block_sum(L["A"]["c"], f)
        for ax, (lo, hi) in enumerate((("w", "e"), ("s", "n"), ("b", "t"))):
            for key, face in ((lo, 0), (hi, f[ax] - 1)):
                blk = _blocks(L["A"][key], f)
                out = blk.select(2 * ax + 1, face).sum(dim=[d if d < 2 * ax + 1 else d - 1
                                                           for d in (1, 3, 5) if d != 2 * ax + 1])
                c = c - (blk.sum(dim=(1, 3, 5)) - out)
                H[key] = out
        H["c"] = c
        levels.append(dict(A=H, act=_block_sum(L["act"].to(F64), f) > 0, f=torch.zeros_like(c),
                           phi=torch.zeros_like(c), fac=f))

    def smooth(L, its):
        L["phi"] = _cg(L["A"], L["f"], L["phi"], lambda r: r / L["A"]["c"], its)

    def visit(q):
        L = levels[q]
        if q == len(levels) - 1:
            smooth(L, 100)
        else:
            smooth(L, 20)
            H = levels[q + 1]
            f = _block_sum(L["f"] - _ax(L["A"], L["phi"]), H["fac"]) * H["act"]
            H["f"] = torch.where(H["act"], f - f.sum() / H["act"].sum(), f)
            visit(q + 1)
            smooth(L, 20)
        if q > 0:
            F = levels[q - 1]
            up = L["phi"]
            for d in range(3):
                up = up.repeat_interleave(L["fac"][d], dim=d)
            F["phi"] = F["phi"] + up

    for _ in range(cycles):
        visit(0)
    return levels[0]["phi"]


def _divergence(dims, h, vel, solid):
    """Fluxes in less fluxes out over dt; no flux through a face to a solid cell."""
    sol = solid.bool()
    f = torch.zeros(dims, device=DEV, dtype=F64)
    for ax, u in enumerate(vel):
        wet = torch.ones_like(u, dtype=torch.bool)
        _cut(wet, ax, 1, -1).copy_(~(_cut(sol, ax, 0, -1) | _cut(sol, ax, 1, 0)))
        flux = u * wet * (h * h / DT)
        f += _cut(flux, ax, 0, -1) - _cut(flux, ax, 1, 0)
    return torch.where(sol, torch.zeros_like(f), f)


def _projected(dims, h, p, rho, vel, solid):
    sol = solid.bool()
    out = []
    for ax, u in enumerate(vel):
        u = u.clone()
        wet = ~(_cut(sol, ax, 0, -1) | _cut(sol, ax, 1, 0))
        face = 0.5 * (_cut(rho, ax, 0, -1) + _cut(rho, ax, 1, 0))
        _cut(u, ax, 1, -1).add_((_cut(p, ax, 0, -1) - _cut(p, ax, 1, 0)) * wet * DT / face / h)
        out.append(u)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "step") and _cells(case) > 5 << 20:
        return None   # minutes of plain CG
    if kind == "batch":
        xs = _solve_tight([(_matrix(d, h, rho, sol, True), b)
                           for d, h, rho, sol, b in _batch_fields(case, seed)])
        return dict(x=xs, converged=None)
    if kind in ("step", "flow"):
        dims, h, col, solid, vel, g = _flow_fields(case, seed)
        rho = RATIO * col + 1.0 * (1.0 - col)
        if not case["body"]:
            solid = torch.zeros_like(solid)
        A = _matrix(dims, h, rho, solid, False, wall=0.5)
        rhs = _divergence(dims, h, vel, solid)
        if kind == "flow":
            p = _noise(dims, g) * DT
            u, v, w = _projected(dims, h, p, rho, vel, solid)
            res = rhs - _ax(A, p)
            return dict(rhs=rhs, res=res, u=u, v=v, w=w)
        p = _solve_tight([(A, rhs)])[0]
        u, v, w = _projected(dims, h, p, rho, vel, solid)
        return dict(u=u, v=v, w=w, p=p, converged=None)
    dims, h, rho, solid, b = _system(case, seed)
    A = _krylov_matrix(case, dims, h, rho, solid)
    if kind == "solve":
        return dict(x=_solve_tight([(A, b)])[0], converged=None)
    if kind == "ac":
        return dict(x=_multigrid(A, b, solid == 0, case["cycles"]))
    if kind == "gs":
        return dict(x=_gauss_seidel(A, b, dims, case["iters"]))
    if case.get("prec", "di") == "di":
        prec = lambda r: r / A["c"]   # noqa: E731
    else:
        prec = _incomplete_cholesky(A, dims, case["prec"])
    step = _bicgs if case.get("solver") == "bicgs" else _cg
    return dict(x=step(A, b, torch.zeros_like(b), prec, case["iters"]))
