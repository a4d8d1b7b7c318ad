"""The work this package does, as cases with one pass each through its public entry points.

Kinds of work:
  velocity   a scene's vortices set, its far field built, and the velocity evaluated at the vortices
             themselves or at separate points (Scene.set_vortices, build_far_field, eval / eval_f32)
  advect     one RK2 or Euler step of the vortices by their own velocity (Scene.advect)
  step       one vortex-segment time step with tracers (Scene.vortex_step)
  plume      one buoyant time step (Scene.solve_time_step)
  batch      several independent scenes of uneven sizes in one call (batch_run)
  potential  the scalar PPPM: far-field buffer and gradient or potential at points (PotentialFieldSolver)
  multigrid  the Poisson solver by itself (MultiGridSolver3DPeriod_double)

exact() restates the method in plain torch in 64 bits, with the float roundings that define the method's
inputs (cell size, hash cells, relative coordinates, stored positions) kept.
"""
import math

import torch

import pppm_vortex_bouyant_flow_sample_b200 as pb
from pppm_vortex_bouyant_flow_sample_b200.potential import PotentialFieldSolver

RING_R, RING_SIGMA = 0.25, 0.03
FOUR_PI = 12.5663706144          # the method's own literal
K_DIAG = 0.250580605913965       # the method's self-potential of a cell
DT, H_SEG, NU = 0.002, 0.1, 0.1
EDGES = (16, 24, 32, 40, 48, 56, 64, 80, 96, 112, 128, 160, 192, 224, 256)
MAX_PAIRS = 9.0e9                # about the largest listed case's near-field pairs
MAX_CELLS = 256 ** 3


def _v(name, n, N, dist="ring", K=1, a=0.0, a_cells=1.0, M=0, out="f64", domain="bbox3x", mg="reference", tol=1e-6):
    return dict(name=name, kind="velocity", n=n, N=N, dist=dist, K=K, a=a, a_cells=a_cells, M=M, out=out,
                domain=domain, mg=mg, tol=tol)


def listed():
    return [
        # the smallest scene of the tests: latency and launches
        _v("cloud_16", 16, 2000, "cloud", a=0.08, a_cells=0.0),
        # a small cloud in a fixed unit box, the multigrid iterated to a tolerance
        _v("cloud_32_fixed", 32, 16384, "cloud", domain="fixed", mg="converged"),
        # an odd number of vortices and tracers at separate points, float output, the method's own constants
        _v("ring_96_tracers", 96, 100003, M=50021, a=0.08, a_cells=0.0, out="f32"),
        # the most accurate preset: a wide near field and a converged multigrid
        _v("ring_64_accurate", 64, 65537, K=3, mg="converged"),
        # the ring at scale: one velocity evaluation of a million vortices
        _v("ring_128", 128, 1048576),
        # a large grid with about a vortex and a half per cell
        _v("cloud_256", 256, 1000003, "cloud"),
        # one RK2 step of a medium cloud, as in an advection loop
        dict(name="rk2_64", kind="advect", n=64, N=50000, dist="slow cloud", K=1, a=0.0, a_cells=1.0, method="rk2"),
        # one vortex-segment time step with tracers
        dict(name="step_128", kind="step", n=128, N=262144, dist="ring", K=1, a=0.08, a_cells=0.0, P=65537),
        # one buoyant time step on a large grid, the multigrid to 1e-10
        dict(name="plume_256", kind="plume", n=256, N=1048576, K=1, a=0.08, a_cells=0.0, tol=1e-10),
        # a mix of scenes of uneven edges and particle counts
        dict(name="batch_12", kind="batch", scenes=12, n_min=10000, n_max=200000, a=0.0, a_cells=1.0, K=1),
        # the scalar companion: sources on a sphere, gradient in a shell around it
        dict(name="potential_128", kind="potential", n=128, Ns=65536, M=262144, scalar=False, K=1),
        # the Poisson solver alone on 64-bit arrays
        dict(name="multigrid_128", kind="multigrid", n=128, mode="reference", tol=1e-10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    for _ in range(200):
        kind = rng.choice(("velocity",) * 4 + ("advect", "step", "plume", "batch", "potential", "multigrid"))
        n = rng.choice(EDGES)
        dist = rng.choice(("cloud", "ring"))
        smooth = rng.choice((dict(a=0.08, a_cells=0.0), dict(a=0.0, a_cells=1.0), dict(a=0.0, a_cells=1.5),
                             dict(a=0.03, a_cells=0.0)))
        if kind == "velocity":
            c = dict(kind=kind, n=n, N=_log(rng, 1000, 1048576), dist=dist, K=rng.choice((1, 1, 1, 2, 3, 0)),
                     M=rng.choice((0, 0, _log(rng, 500, 500000))), out=rng.choice(("f64", "f64", "f32")),
                     domain=rng.choice(("bbox3x", "bbox3x", "fixed")), mg=rng.choice(("reference", "reference", "converged")),
                     tol=1e-6, **smooth)
        elif kind == "advect":
            c = dict(kind=kind, n=n, N=_log(rng, 1000, 300000), dist=rng.choice(("slow cloud", "ring")), K=1, method=rng.choice(("rk2", "euler")), **smooth)
        elif kind == "step":
            c = dict(kind=kind, n=n, N=_log(rng, 1000, 300000), dist=rng.choice(("slow cloud", "ring")), K=1, P=_log(rng, 100, 100000), **smooth)
        elif kind == "plume":
            c = dict(kind=kind, n=n, N=_log(rng, 4000, 1048576), K=1, tol=1e-10, **smooth)
        elif kind == "batch":
            c = dict(kind=kind, scenes=rng.randint(2, 16), n_min=_log(rng, 1000, 10000), n_max=_log(rng, 12000, 200000), K=1, **smooth)
        elif kind == "potential":
            c = dict(kind=kind, n=rng.choice([e for e in EDGES if e <= 160]), Ns=_log(rng, 2000, 200000),
                     M=_log(rng, 2000, 500000), scalar=rng.random() < 0.4, K=rng.choice((1, 1, 2)))
        else:
            c = dict(kind=kind, n=n, mode=rng.choice(("reference", "reference", "converged", "vcycle")), tol=1e-10)
        if _pairs(c) <= MAX_PAIRS and _cells(c) <= MAX_CELLS:
            return c
    raise RuntimeError("no case drawn")


# ---- sizes ---------------------------------------------------------------

def _mix(case):
    """(edge, particles, distribution) of each scene of a batch: the edges and sizes cover their ranges."""
    edges, s = (32, 48, 64, 96, 128), case["scenes"]
    out = []
    for q in range(s):
        f = (q * 0.6180339887498949) % 1.0
        N = int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** f))
        n = edges[(q * 3) % 5]
        if N > 40000:
            n = max(n, 64)
        out.append((n, N | 1, "cloud" if q % 2 == 0 else "ring"))
    return out


def _extent(dist, N):
    return 1.0 if dist != "ring" else 2 * (RING_R + RING_SIGMA * math.sqrt(2 * math.log(max(N, 2) / 2.5)))


def _scene_pairs(n, N, M, dist, K, fixed=False):
    """Near-field pairs expected inside the (K + 0.5) h boxes of M points."""
    if K < 0:
        return 0.0
    h = (1.0 if fixed else 3.0 * _extent(dist, N)) / n
    w = (K + 0.5) * h
    if dist == "ring":
        f = math.erf(w / (2 * RING_SIGMA)) ** 2 * min(1.0, 2 * w / (2 * math.pi * RING_R))
    elif dist == "sphere":
        f = min(1.0, (2 * w) ** 3 / (math.pi / 6))
    else:
        f = (min(1.0, 2 * w - w * w) if w < 1 else 1.0) ** 3
    return float(M) * N * f


def _pairs(c):
    k = c["kind"]
    if k == "velocity":
        return _scene_pairs(c["n"], c["N"], c["M"] or c["N"], c["dist"], c["K"], c["domain"] == "fixed")
    if k == "advect":
        return (2 if c["method"] == "rk2" else 1) * _scene_pairs(c["n"], c["N"], c["N"], c["dist"], c["K"])
    if k == "step":
        return _scene_pairs(c["n"], c["N"], 2 * c["N"] + c["P"], c["dist"], c["K"])
    if k == "plume":
        return _scene_pairs(c["n"], c["N"], 2 * c["N"], "sphere", c["K"])
    if k == "batch":
        return sum(_scene_pairs(n, N, N, d, c["K"]) for n, N, d in _mix(c))
    if k == "potential":  # points of the shell near the sphere surface see sources within the box
        w = (c["K"] + 0.5) * 0.6 / c["n"]
        return c["M"] * c["Ns"] * min(1.0, 4 * w * w / (4 * math.pi * 0.15 ** 2)) * min(1.0, w / 0.13)
    return 0.0


def _cells(c):
    return sum(n ** 3 for n, _, _ in _mix(c)) if c["kind"] == "batch" else c["n"] ** 3


def work(case):
    """Inputs read once, outputs written once; 30 operations for a near-field pair and 400 for each component
    of each grid cell (two full-multigrid passes of eight half sweeps, transfers, curl and correction)."""
    k, p, cells = case["kind"], _pairs(case), _cells(case)
    if k == "velocity":
        M = case["M"] or case["N"]
        b = 40 * case["N"] + (16 if case["M"] else 0) * M + (24 if case["out"] == "f64" else 12) * M
    elif k == "advect":
        b = 56 * case["N"]
    elif k == "step":
        b = 80 * case["N"] + 56 * case["P"]
    elif k == "plume":
        b = 84 * case["N"]
    elif k == "batch":
        b = sum(64 * N for _, N, _ in _mix(case))
    elif k == "potential":
        b = 24 * case["Ns"] + (24 if case["scalar"] else 40) * case["M"]
    else:
        return {"bytes": 24 * cells, "flops": 400 * cells}
    return {"bytes": b, "flops": 30 * p + (3 if k != "potential" else 1) * 400 * cells}


def tolerance(case):
    """32-bit sums of up to some ten thousand terms, with 64-bit grids around them.  The strengths after a
    step are differences of stored float positions, so one rounding of a position shows in them: about four
    times the distance from the 64-bit values (plume 2.9e-4, step 1.2e-5)."""
    k = case["kind"]
    if k == "plume":
        return {"rel": 1.2e-3, "max": 0.05}
    if k == "step":
        return {"rel": 1e-4, "max": 0.02}
    if k in ("potential", "multigrid"):
        return {"rel": 2e-6, "max": 2e-4}
    return {"rel": 1e-5, "max": 1e-3}


# ---- inputs and passes ---------------------------------------------------

_GPU = torch.cuda.is_available()
_DEV = "cuda" if _GPU else "cpu"


def _gen(seed, salt=0):
    return torch.Generator(device=_DEV).manual_seed(int(seed) * 1000003 + salt)


def _u(g, *shape):
    return torch.rand(shape, generator=g, device=_DEV, dtype=torch.float64)


def _n(g, *shape):
    return torch.randn(shape, generator=g, device=_DEV, dtype=torch.float64)


def _pos4(p):
    out = torch.zeros((p.shape[0], 4), dtype=torch.float32, device=_DEV)
    out[:, :3] = p.to(torch.float32)
    return out


def _vortices(dist, N, seed, salt=0):
    """Positions (N, 4) float32 and strengths (3, N) float64."""
    g = _gen(seed, salt)
    if dist == "cloud":
        return _pos4(_u(g, N, 3)), _n(g, 3, N)
    if dist == "slow cloud":  # strengths for which a step moves a vortex by less than the spacing
        return _pos4(_u(g, N, 3)), _n(g, 3, N) / N
    if dist == "sphere":
        d = _n(g, N, 3)
        d = d / d.norm(dim=1, keepdim=True)
        return _pos4(torch.tensor([0.5, 0.15, 0.5], dtype=torch.float64, device=_DEV)
                     + 0.5 * d * _u(g, N, 1).pow(1.0 / 3.0)), torch.zeros((3, N), dtype=torch.float64, device=_DEV)
    phi = 2 * math.pi * _u(g, N)
    rad = RING_R + RING_SIGMA * _n(g, N)
    p = torch.stack([0.5 + rad * phi.cos(), 0.5 + rad * phi.sin(), 0.5 + RING_SIGMA * _n(g, N)], 1)
    t = torch.stack([-phi.sin(), phi.cos(), torch.zeros_like(phi)])
    return _pos4(p), (2 * math.pi * RING_R / N) * (t + 1e-3 * _n(g, 3, N))


def _points(dist, M, seed):
    """Tracers: around the ring, or through and somewhat beyond the cloud's box."""
    g = _gen(seed, 77)
    if dist == "ring":
        return _pos4(_vortices("ring", M, seed, 78)[0][:, :3].double() + 0.01 * _n(g, M, 3))
    return _pos4(-0.05 + 1.1 * _u(g, M, 3))


def _panels(case, seed):
    """Sources on a sphere with the sine layer of a uniform stream, and points in the shell around it."""
    g = _gen(seed, 5)
    Ns, M = case["Ns"], case["M"]
    k = torch.arange(Ns, dtype=torch.float64, device=_DEV) + 0.5
    y = 1 - 2 * k / Ns
    r = (1 - y * y).clamp_min(0).sqrt()
    phi = math.pi * (3 - math.sqrt(5)) * k + 2 * math.pi * _u(g, 1)
    src = _pos4(0.5 + 0.15 * torch.stack([r * phi.cos(), y, r * phi.sin()], 1))
    mass = (4 * math.pi * 0.15 ** 2 / Ns) * (y + 0.2) * (1 + 0.1 * _n(g, Ns))
    d = _n(g, M, 3)
    d = d / d.norm(dim=1, keepdim=True)
    pts = _pos4(0.5 + d * (0.16 ** 3 + (0.29 ** 3 - 0.16 ** 3) * _u(g, M, 1)).pow(1.0 / 3.0))
    return src, mass, pts


def _rhs(case, seed):
    d = case["n"]
    if case["mode"] == "vcycle":
        return 0.1 * _n(_gen(seed, 9), d ** 3), _n(_gen(seed, 8), d ** 3)
    return torch.zeros(d ** 3, dtype=torch.float64, device=_DEV), _n(_gen(seed, 8), d ** 3)


def _scene(case, n, N, M, **kw):
    return pb.Scene(n, K=case["K"], a=case["a"] or 0.08, a_cells=case["a_cells"], cap_vort=N, cap_eval=M, **kw)


def prepare(case, seed):
    k, s = case["kind"], {"case": case}
    if k == "velocity":
        s["pos"], s["al"] = _vortices(case["dist"], case["N"], seed)
        s["pts"] = _points(case["dist"], case["M"], seed) if case["M"] else None
        s["scene"] = _scene(case, case["n"], case["N"], case["M"] or case["N"], domain=case["domain"], mg=case["mg"],
                            mg_tol=case["tol"])
    elif k == "advect":
        s["pos"], s["al"] = _vortices(case["dist"], case["N"], seed)
        s["scene"] = _scene(case, case["n"], case["N"], case["N"])
    elif k == "step":
        s["pos"], s["al"] = _vortices(case["dist"], case["N"], seed)
        s["pts"] = _points(case["dist"], case["P"], seed)
        s["scene"] = _scene(case, case["n"], case["N"], max(2 * case["N"], case["P"]))
    elif k == "plume":
        s["pos"], s["al"] = _vortices("sphere", case["N"], seed)
        s["heat"] = (1 + 0.05 * _n(_gen(seed, 6), case["N"])).to(torch.float32)
        s["scene"] = _scene(case, case["n"], case["N"], 2 * case["N"], mg="converged", mg_tol=case["tol"])
    elif k == "batch":
        s["jobs"] = []
        for q, (n, N, dist) in enumerate(_mix(case)):
            pos, al = _vortices(dist, N, seed, 100 + q)
            s["jobs"].append((_scene(case, n, N, N), pos, al, None, None, 1))
    elif k == "potential":
        s["src"], s["mass"], s["pts"] = _panels(case, seed)
        s["solver"] = PotentialFieldSolver()
        s["solver"].initializeSolver(case["n"], case["n"], case["n"], case["K"], case["M"], case["Ns"])
    else:
        s["x"], s["b"] = _rhs(case, seed)
        s["solver"] = pb.MultiGridSolver3DPeriod_double()
        s["solver"].m_InitialSystem(case["n"], case["n"], case["n"])
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "velocity":
        sc = s["scene"]
        sc.set_vortices(s["pos"], s["al"])
        sc.build_far_field()
        ev = sc.eval if case["out"] == "f64" else sc.eval_f32
        return ev(s["pts"]) if s["pts"] is not None else ev(s["pos"], s["pos"], 1)
    if k == "advect":
        return s["scene"].advect(s["pos"].clone(), s["al"], DT, case["method"])
    if k == "step":
        pos, al, pts = s["pos"].clone(), s["al"].clone(), s["pts"].clone()
        pos, al, vel = s["scene"].vortex_step(pos, al, DT, H_SEG, NU, passive=pts)
        return {"pos": pos, "alpha": al, "passive": pts, "velocity": vel}
    if k == "plume":
        pos, al = s["scene"].solve_time_step(s["pos"].clone(), s["al"].clone(), DT, s["heat"])
        return {"pos": pos, "alpha": al}
    if k == "batch":
        return pb.batch_run(s["jobs"])
    if k == "potential":
        p = s["solver"]
        p.setMassParameter(case["Ns"], s["src"], s["mass"])
        p.setEvalParameter(case["M"], s["pts"])
        if case["scalar"]:
            p.computeFarFieldPotentialBuffer()
            p.evaluateScalarPotential()
            return p.getScalarPhi()
        p.computeFarFieldBuffer()
        p.evaluateGradient(True)
        return p.getGradPhi()
    x = s["x"].clone()
    if case["mode"] == "vcycle":
        s["solver"].m_Vcycle(x, s["b"])
    else:
        s["solver"].m_FullMultiGrid(x, s["b"], case["tol"], pb.MG_REFERENCE if case["mode"] == "reference" else pb.MG_CONVERGED)
    return x


# ---- the method in 64 bits -----------------------------------------------

def _f32(v):
    return float(torch.tensor(v, dtype=torch.float64).to(torch.float32))


class _Domain:
    def __init__(self, pos, n, K, a, a_cells, fixed=False, times=3.0):
        p = pos[:, :3].double()
        mn, mx = p.amin(0).tolist(), p.amax(0).tolist()
        self.n, self.K, self.C = n, K, n ** 3
        if fixed:
            self.L, self.origin = 1.0, [0.0, 0.0, 0.0]
        else:
            self.L = times * max(mx[c] - mn[c] for c in range(3))
            self.origin = [(mn[c] + 0.5 * (mx[c] - mn[c])) - 0.5 * self.L for c in range(3)]
        self.h = _f32(self.L / n)
        self.invh = 1.0 / self.h
        self.h2 = float(torch.tensor(self.h, dtype=torch.float32) ** 2)
        self.a = a_cells * self.h if a_cells > 0 else a
        self.bound = (K + 0.5) / self.invh

    def rel(self, pos):
        o = torch.tensor(self.origin, dtype=torch.float64, device=pos.device)
        return (pos[:, :3].double() - o).to(torch.float32)

    def hash(self, pos):
        of = torch.tensor(self.origin, dtype=torch.float64, device=pos.device).to(torch.float32)
        g = ((pos[:, :3] - of) / torch.tensor(self.h, dtype=torch.float32, device=pos.device)).floor().long() % self.n
        return (g[:, 2] * self.n + g[:, 1]) * self.n + g[:, 0]

    def cell(self, rel):
        return (rel.double() * self.invh).floor().long()

    def inside(self, c):
        return ((c >= 0) & (c < self.n)).all(1)


class _Sources:
    """Records sorted by hash cell, and the first record of every cell."""

    def __init__(self, dom, pos, values):
        key = dom.hash(pos)
        order = torch.argsort(key, stable=True)
        self.rel = dom.rel(pos)[order]
        self.val = [v[order] for v in values]
        self.first = torch.zeros(dom.C + 1, dtype=torch.long, device=pos.device)
        self.first[1:] = torch.bincount(key, minlength=dom.C).cumsum(0)
        self.order = order


def _pair_sums(dom, src, rt, lo, hi, bound, f, comps, chunk=24_000_000):
    """sum over the sources hashed into cells [lo, hi] of each target (within `bound` on each axis, if given)
    of f(target index, source index, float difference), a tuple of `comps` values."""
    n, M = dom.n, rt.shape[0]
    out = torch.zeros((comps, M), dtype=torch.float64, device=rt.device)
    if M == 0:
        return out
    lo, hi = lo.clamp_min(0), hi.clamp_max(n - 1)
    W = int((hi - lo).amax().item()) + 1
    if W < 1:
        return out
    d = torch.arange(W, device=rt.device)
    total = torch.zeros(M, dtype=torch.long, device=rt.device)
    runs = []
    for part in torch.arange(M, device=rt.device).split(200_000):
        y = lo[part, 1, None] + d
        z = lo[part, 2, None] + d
        ok = ((y <= hi[part, 1, None])[:, None, :] & (z <= hi[part, 2, None])[:, :, None] & (lo[part, 0] <= hi[part, 0])[:, None, None])
        row = ((z[:, :, None] * n + y[:, None, :]) * n).clamp(0, n ** 3 - n)
        s0 = src.first[(row + lo[part, 0, None, None].clamp(0, n - 1))]
        s1 = src.first[(row + hi[part, 0, None, None].clamp(0, n - 1)) + 1]
        cnt = torch.where(ok, (s1 - s0).clamp_min(0), torch.zeros_like(s0)).reshape(len(part), -1)
        runs.append((part, s0.reshape(len(part), -1).to(torch.int32), cnt.to(torch.int32)))
        total[part] = cnt.sum(1)
    for part, s0, cnt in runs:
        acc = total[part].cumsum(0)
        at, n_part = 0, len(part)
        while at < n_part:
            base = int(acc[at - 1]) if at else 0
            end = int(torch.searchsorted(acc, base + chunk, right=True))
            end = min(max(end, at + 1), n_part)
            c = cnt[at:end].reshape(-1).long()
            P = int(c.sum())
            if P:
                rid = torch.repeat_interleave(torch.arange(len(c), device=rt.device), c, output_size=P)
                off = s0[at:end].reshape(-1).long() - (c.cumsum(0) - c)
                p = torch.arange(P, device=rt.device) + off[rid]
                t = part[at] + torch.div(rid, cnt.shape[1], rounding_mode="floor")
                del rid
                diff = [rt[:, q][t] - src.rel[:, q][p] for q in range(3)]
                if bound is not None:
                    keep = ((diff[0].abs().double() < bound) & (diff[1].abs().double() < bound) & (diff[2].abs().double() < bound)).nonzero()[:, 0]
                    t, p, diff = t[keep], p[keep], [x[keep] for x in diff]
                edge = torch.searchsorted(t, torch.arange(at, end + 1, device=rt.device) + part[0])
                for q, v in enumerate(f(t, p, diff)):
                    s = torch.zeros(v.shape[0] + 1, dtype=torch.float64, device=rt.device)
                    torch.cumsum(v, 0, out=s[1:])
                    out[q, part[at:end]] = s[edge[1:]] - s[edge[:-1]]
            at = end
    return out


def _nb(x):
    """Sum of the six neighbours with zero ghost values; x is (components, z, y, x)."""
    s = torch.zeros_like(x)
    s[..., 1:] += x[..., :-1]
    s[..., :-1] += x[..., 1:]
    s[:, :, 1:] += x[:, :, :-1]
    s[:, :, :-1] += x[:, :, 1:]
    s[:, 1:] += x[:, :-1]
    s[:, :-1] += x[:, 1:]
    return s


class _Multigrid:
    def __init__(self, n):
        self.edges = [n]
        while self.edges[-1] ** 3 > 512:
            self.edges.append(self.edges[-1] // 2)
        self.odd = []
        for d in self.edges:
            i = torch.arange(d, device=_DEV)
            self.odd.append(((i[:, None, None] + i[:, None] + i) % 2 == 1))

    def smooth(self, lv, x, b):
        w, w1 = _f32(1.43), float(torch.tensor(1.0) - torch.tensor(1.43))
        for _ in range(4):
            for odd in (True, False):
                m = self.odd[lv] if odd else ~self.odd[lv]
                x = torch.where(m, w1 * x + w * (_nb(x) - b) / 6.0, x)
        return x

    @staticmethod
    def restrict(r):
        c, d = r.shape[0], r.shape[1] // 2
        return 0.5 * r.reshape(c, d, 2, d, 2, d, 2).sum((2, 4, 6))

    @staticmethod
    def prolong(x):
        return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    def coarse(self, b):
        x = torch.zeros_like(b)
        for _ in range(100):
            x = (_nb(x) - b) / 6.0
        return x

    def vcycle(self, lv, x, b):
        if lv == len(self.edges) - 1:
            return self.coarse(b)
        x = self.smooth(lv, x, b)
        r = self.restrict(b - (_nb(x) - 6 * x))
        x = x + self.prolong(self.vcycle(lv + 1, torch.zeros_like(r), r))
        return self.smooth(lv, x, b)

    def full(self, b):
        bs = [b]
        for _ in self.edges[1:]:
            bs.append(self.restrict(bs[-1]))
        x = self.coarse(bs[-1])
        for lv in range(len(self.edges) - 2, -1, -1):
            x = self.vcycle(lv, self.prolong(x), bs[lv])
        return x + self.vcycle(0, torch.zeros_like(b), b - (_nb(x) - 6 * x))

    def solve(self, b, converged):
        x = self.full(b)
        for _ in range(80 if converged else 0):
            r = b - (_nb(x) - 6 * x)
            if float(r.norm()) <= 1e-13 * float(b.norm()):
                break
            x = x + self.vcycle(0, torch.zeros_like(b), r)
        return x


def _shift(f, axis, d, periodic=False):
    """f at the neighbour d cells along an axis (x: -1, y: -2, z: -3), clamped or periodic."""
    n = f.shape[axis]
    i = torch.arange(n, device=f.device) + d
    return f.index_select(axis, i % n if periodic else i.clamp(0, n - 1))


def _curl(F, scale, K=None):
    d = lambda q, ax: _shift(F[q], ax, 1) - _shift(F[q], ax, -1)  # noqa: E731
    return scale * torch.stack([d(2, -2) - d(1, -3), d(0, -3) - d(2, -1), d(1, -1) - d(0, -2)])


def _green(K, h):
    """The central-difference gradient of 1 / (4 pi r) between a cell's centre and its neighbours'."""
    inv = lambda a, b: 1.0 / (FOUR_PI * math.dist(a, b) if math.dist(a, b) ** 2 > 1e-12 else 1e24)  # noqa: E731
    out, x = {}, [0.5 * h] * 3
    for k in range(-K, K + 1):
        for j in range(-K, K + 1):
            for i in range(-K, K + 1):
                if i or j or k:
                    p = [(i + 0.5) * h, (j + 0.5) * h, (k + 0.5) * h]
                    g = []
                    for c in range(3):
                        u, v = list(x), list(x)
                        u[c] += h
                        v[c] -= h
                        g.append(0.5 * (inv(u, p) - inv(v, p)) / h)
                    out[i, j, k] = g
    return out


def _window(f, i, j, k):
    """(slices of the cells whose neighbour at the offset is in the grid, that neighbour's values)."""
    n = f.shape[-1]
    s = lambda d: (slice(max(0, -d), n - max(0, d)), slice(max(0, d), n - max(0, -d)))  # noqa: E731
    (xi, xo), (yi, yo), (zi, zo) = s(i), s(j), s(k)
    return (Ellipsis, zi, yi, xi), f[..., zo, yo, xo]


def _interpolate(dom, grid, rel):
    """Hat-weighted values of (components, cells) at points; zero where the own cell is outside the grid."""
    n = dom.n
    q = rel.double() * dom.invh
    own = dom.inside(q.floor().long())
    t = q - 0.5
    b = t.floor()
    w = t - b
    b = b.long()
    out = torch.zeros((grid.shape[0], rel.shape[0]), dtype=torch.float64, device=rel.device)
    for c in range(8):
        o = torch.tensor([c & 1, (c >> 1) & 1, c >> 2], device=rel.device)
        g = b + o
        ok = dom.inside(g) & own
        wt = torch.where(o.bool(), w, 1 - w).prod(1) * ok
        g = g.clamp(0, n - 1)
        out += wt * grid[:, (g[:, 2] * n + g[:, 1]) * n + g[:, 0]]
    return out


class _Vortex:
    """The far field of a set of vortices, and velocities in it."""

    def __init__(self, case, n, pos, al, converged, fixed=False):
        self.d = d = _Domain(pos, n, case["K"], case["a"], case["a_cells"], fixed)
        c = d.cell(d.rel(pos))
        ok = d.inside(c)
        at = ((c[:, 2] * n + c[:, 1]) * n + c[:, 0])[ok]
        om = torch.zeros((3, d.C), dtype=torch.float64, device=pos.device)
        for q in range(3):
            om[q].index_add_(0, at, al[q][ok])
        om = (om * d.invh ** 3).reshape(3, n, n, n)
        psi = _Multigrid(n).solve(-om * d.h2, converged)
        far = _curl(psi, 0.5 * d.invh)
        if d.K >= 0:
            m = torch.zeros_like(om)
            for (i, j, k), (gx, gy, gz) in _green(d.K, d.h).items():
                w, o = _window(om, i, j, k)
                m[0][w[1:]] += gy * o[2] - gz * o[1]
                m[1][w[1:]] += gz * o[0] - gx * o[2]
                m[2][w[1:]] += gx * o[1] - gy * o[0]
            far = far - m * d.h ** 3 - _curl(om, 0.5 * d.invh * K_DIAG * d.h * d.h)
        self.far = far.reshape(3, d.C)
        self.src = _Sources(d, pos, list(al))

    def velocity(self, pts, other=None):
        d, src = self.d, self.src
        rt = d.rel(pts)
        u = _interpolate(d, self.far, rt)
        if d.K < 0:
            return u
        q = rt.double() * d.invh
        own = q.floor().long()
        lo = torch.maximum(own - d.K - 1, (q - (d.K + 0.5) - 1e-2).floor().long())
        hi = torch.minimum(own + d.K + 1, (q + (d.K + 0.5) + 1e-2).floor().long())
        rb = d.rel(other) if other is not None else None
        k4, ia3 = 1.0 / FOUR_PI, 1.0 / d.a ** 3

        def f(t, p, diff):
            x, y, z = (v.double() for v in diff)
            r3 = (x * x + y * y + z * z).pow(1.5)
            c = -torch.expm1(-r3 * ia3) / r3.clamp_min(1e-300) * k4
            c = torch.where(r3 > 1e-36, c, torch.zeros_like(c))
            if rb is not None:
                e = [rb[:, a][t] - src.rel[:, a][p] for a in range(3)]
                c = torch.where(e[0] * e[0] + e[1] * e[1] + e[2] * e[2] < 1e-24, torch.zeros_like(c), c)
            ax, ay, az = (v[p] for v in src.val)
            return (ay * z - az * y) * c, (az * x - ax * z) * c, (ax * y - ay * x) * c

        return u + _pair_sums(d, src, rt, lo, hi, d.bound, f, 3)


def _moved(pos, u, dt):
    out = torch.zeros_like(pos)
    out[:, :3] = (pos[:, :3].double() + u.t() * dt).to(torch.float32)
    return out


def _smooth(dom, pos, al):
    """Gaussian means of the strengths over the 5^3 hash cells around each vortex."""
    src = _Sources(dom, pos, list(al))
    rt = dom.rel(pos)
    c = dom.cell(rt)

    def f(t, p, diff):
        x, y, z = (v.double() for v in diff)
        w = torch.exp(-(x * x + y * y + z * z) / (2 * NU * NU))
        return w, w * src.val[0][p], w * src.val[1][p], w * src.val[2][p]

    s = _pair_sums(dom, src, rt, c - 2, c + 2, None, f, 4)
    tw = torch.where(s[0] < 1e-12, torch.full_like(s[0], 1e24), s[0])
    return s[1:] / tw


def _vortex_step(case, pos, al, pts, converged):
    n, N = case["n"], pos.shape[0]
    f = _Vortex(case, n, pos, al, converged)
    l = al.square().sum(0).sqrt()  # noqa: E741
    short = l < H_SEG
    half = torch.where(short, 0.5 * al, 0.5 * al / l.clamp_min(1e-300) * H_SEG).t()
    kappa = torch.where(short, torch.ones_like(l), l / H_SEG)
    b, a = pos.clone(), pos.clone()
    b[:, :3] = (pos[:, :3].double() + half).to(torch.float32)
    a[:, :3] = (pos[:, :3].double() - half).to(torch.float32)
    b, a = _moved(b, f.velocity(b, pos), DT), _moved(a, f.velocity(a, pos), DT)
    vel = None
    if pts is not None:
        vel = f.velocity(pts)
        pts = _moved(pts, vel, DT)
    new = pos.clone()
    new[:, :3] = (0.5 * (b[:, :3] + a[:, :3]).double()).to(torch.float32)
    mid = kappa * (b[:, :3] - a[:, :3]).double().t()
    return new, _smooth(_Domain(new, n, case["K"], case["a"], case["a_cells"]), new, mid), pts, vel


def _baroclinic(pos, heat, al):
    p = pos[:, :3].double()
    mn, mx = p.amin(0).tolist(), p.amax(0).tolist()
    L = 1.2 * max(mx[c] - mn[c] for c in range(3))
    n = min(int(math.floor(L / 0.2) + 1), 200)
    d = _Domain(pos, n, 1, 1.0, 0.0)
    d.L, d.h = L, L / n
    d.origin = [(mn[c] + 0.5 * (mx[c] - mn[c])) - 0.5 * L for c in range(3)]
    d.invh = 1.0 / d.h
    rel = d.rel(pos)
    q = rel.double() * d.invh
    own = q.floor().long()
    d.h = _f32(L / n)
    full = torch.bincount(d.hash(pos), minlength=n ** 3) == 0
    s = torch.zeros(n ** 3, dtype=torch.float64, device=pos.device)
    w = full.double()
    for k in (-1, 0, 1):
        for j in (-1, 0, 1):
            for i in (-1, 0, 1):
                g = own + torch.tensor([i, j, k], device=pos.device)
                ok = d.inside(g)
                r = (g.double() + 0.5 - q).square().sum(1)
                wt = torch.where(ok & (r < 1), (1 - r).pow(4), torch.zeros_like(r))
                g = g.clamp(0, n - 1)
                at = (g[:, 2] * n + g[:, 1]) * n + g[:, 0]
                s.index_add_(0, at, wt * heat.double())
                w.index_add_(0, at, wt)
    w = torch.where(w < 1e-12, torch.full_like(w, 1e24), w)
    rho = (s / w).to(torch.float32).double().reshape(n, n, n)
    g = torch.stack([(_shift(rho, ax, 1, True) - _shift(rho, ax, -1, True)) * 0.5 * d.invh for ax in (-1, -2, -3)])
    d.invh = 1.0 / d.h
    at = _interpolate_hat(d, g.to(torch.float32).double().reshape(3, -1), rel)
    zero = torch.zeros_like(at[0])
    return al + 5 * DT * 0.1 * torch.stack([-10.0 * at[2], zero, 10.0 * at[0]])


def _interpolate_hat(dom, grid, rel):
    """As _interpolate, for points whose own cell may lie outside the grid too."""
    n = dom.n
    t = rel.double() * dom.invh - 0.5
    b = t.floor()
    w = t - b
    out = torch.zeros((grid.shape[0], rel.shape[0]), dtype=torch.float64, device=rel.device)
    for c in range(8):
        o = torch.tensor([c & 1, (c >> 1) & 1, c >> 2], device=rel.device)
        g = b.long() + o
        wt = torch.where(o.bool(), w, 1 - w).prod(1) * dom.inside(g)
        g = g.clamp(0, n - 1)
        out += wt * grid[:, (g[:, 2] * n + g[:, 1]) * n + g[:, 0]]
    return out


def _potential(case, src, mass, pts):
    n, K = case["n"], case["K"]
    d = _Domain(src, n, K, 1.0, 0.0, times=2.0)
    c = d.cell(d.rel(src))
    ok = d.inside(c)
    rho = torch.zeros(d.C, dtype=torch.float64, device=src.device)
    rho.index_add_(0, ((c[:, 2] * n + c[:, 1]) * n + c[:, 0])[ok], mass[ok])
    rho = (rho * d.invh ** 3).reshape(n, n, n)
    am = mass.abs()
    centre = ((src[:, :3].double() * am[:, None]).sum(0) / am.sum()).tolist()
    total = float(mass.sum())
    rhs = -rho * d.h2
    x = [(torch.arange(n, device=src.device, dtype=torch.float64) + 0.5) * d.h + d.origin[q] for q in range(3)]
    for ax in range(3):  # ghost values of the monopole beyond each face
        for side in (0, 1):
            g = [x[0][None, None, :], x[1][None, :, None], x[2][:, None, None]]
            gx = ((-0.5) if side == 0 else (n + 0.5)) * d.h + d.origin[ax]
            g[ax] = torch.full_like(g[ax][..., :1] if ax == 0 else g[ax][:, :1] if ax == 1 else g[ax][:1], gx)
            r = ((g[0] - centre[0]) ** 2 + (g[1] - centre[1]) ** 2 + (g[2] - centre[2]) ** 2).sqrt() * FOUR_PI
            face = rhs.select(2 - ax, 0 if side == 0 else n - 1)
            face -= (total / r).squeeze(2 - ax)
    mg = _Multigrid(n)
    phi = torch.zeros((1, n, n, n), dtype=torch.float64, device=src.device)
    for _ in range(3):
        phi = phi + mg.full(rhs[None] - (_nb(phi) - 6 * phi))
    phi = phi[0]
    grad = lambda f: torch.stack([(_shift(f, ax, 1, True) - _shift(f, ax, -1, True)) * 0.5 * d.invh for ax in (-1, -2, -3)])  # noqa: E731
    h3 = d.h ** 3
    if case["scalar"]:
        m = 0.25 * rho * d.h ** 2
        for (i, j, k) in _green(K, d.h):
            w, o = _window(rho, i, j, k)
            m[w[1:]] += o * d.h ** 2 / (FOUR_PI * math.sqrt(i * i + j * j + k * k))
        far = (phi - m)[None]
    else:
        m = torch.zeros((3, n, n, n), dtype=torch.float64, device=src.device)
        for (i, j, k), g in _green(K, d.h).items():
            w, o = _window(rho, i, j, k)
            for q in range(3):
                m[q][w[1:]] += g[q] * o * h3
        far = grad(phi) - m - grad(K_DIAG * d.h ** 2 * rho)
    rt = d.rel(pts)
    out = _interpolate(d, far.reshape(far.shape[0], -1), rt)
    S = _Sources(d, src, [mass])
    q = rt.double() * d.invh
    own = q.floor().long()
    lo, hi = own - K - 1, own + K + 1
    if case["scalar"]:
        up = q > own.double() + 0.5
        lo, hi = torch.where(up, own - K, lo), torch.where(up, hi, own + K)

    def f(t, p, diff):
        x, y, z = (-v.double() for v in diff)
        r = (x * x + y * y + z * z).sqrt()
        core = 0.125 if case["scalar"] else 0.05
        e = 1 if case["scalar"] else 3
        den = torch.where(r > core, FOUR_PI * r.pow(e), torch.full_like(r, FOUR_PI * core ** e))
        den = torch.where(r < 1e-12, torch.full_like(r, 1e14), den)
        v = S.val[0][p] / den
        return (v,) if case["scalar"] else (x * v, y * v, z * v)

    out = out + _pair_sums(d, S, rt, lo, hi, d.bound, f, far.shape[0])
    return out[0] if case["scalar"] else out.t()


def exact(case, seed):
    k = case["kind"]
    if k == "velocity":
        pos, al = _vortices(case["dist"], case["N"], seed)
        v = _Vortex(case, case["n"], pos, al, case["mg"] == "converged", case["domain"] == "fixed")
        return v.velocity(_points(case["dist"], case["M"], seed) if case["M"] else pos).t()
    if k == "advect":
        pos, al = _vortices(case["dist"], case["N"], seed)
        u = _Vortex(case, case["n"], pos, al, False).velocity(pos)
        if case["method"] == "rk2":
            u = _Vortex(case, case["n"], _moved(pos, u, 0.5 * DT), al, False).velocity(_moved(pos, u, 0.5 * DT))
        return _moved(pos, u, DT)
    if k == "step":
        pos, al = _vortices(case["dist"], case["N"], seed)
        pos, al, pts, vel = _vortex_step(case, pos, al, _points(case["dist"], case["P"], seed), False)
        return {"pos": pos, "alpha": al, "passive": pts, "velocity": vel.t()}
    if k == "plume":
        pos, al = _vortices("sphere", case["N"], seed)
        heat = (1 + 0.05 * _n(_gen(seed, 6), case["N"])).to(torch.float32)
        pos, al, _, _ = _vortex_step(case, pos, _baroclinic(pos, heat, al), None, True)
        return {"pos": pos, "alpha": al}
    if k == "batch":
        out = []
        for q, (n, N, dist) in enumerate(_mix(case)):
            pos, al = _vortices(dist, N, seed, 100 + q)
            out.append(_Vortex(case, n, pos, al, False).velocity(pos).t())
        return out
    if k == "potential":
        return _potential(case, *_panels(case, seed))
    x, b = _rhs(case, seed)
    n, mg = case["n"], _Multigrid(case["n"])
    x, b = x.reshape(1, n, n, n), b.reshape(1, n, n, n)
    if case["mode"] == "vcycle":
        return mg.vcycle(0, x, b).reshape(-1)
    return mg.solve(b, case["mode"] == "converged").reshape(-1)
