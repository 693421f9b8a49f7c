"""Performance cases: the solves a user of this framework runs, through its public entry
points, over the range of sizes, kernels, precisions and options in use.

A case is a plain dict:
  entry    "solve"  fmm! on device buffers (fmm_solve through the ctypes binding)
           "host"   fmm! of a System object in host memory (fastmultipole_b200.fmm)
           "vjp"    forward solve + gradient of a loss (fmm_vjp), device buffers
           "direct" all pairs (fmm_direct), device buffers
  kind     "source" (Laplace point sources) or "vortex" (vortex particles)
  dist     "uniform", "clustered" (8 Gaussians, sigma 0.05, and 10% uniform) or "ring" (thin
           vortex ring, core sigma 0.05)
  n        sources; targets: separate targets (0: the sources are the targets)
  p, leaf, mac, tol   expansion order, leaf size, acceptance, PowerRelativeGradient tolerance
           (0: fixed order)
  phi, hess, precision   potential / velocity gradient requested; "f64" or "mixed"
"""
import ctypes as C
import math

import numpy as np
import torch

import fastmultipole_b200 as fm
from fastmultipole_b200 import _lib as L

FOUR_PI = 4.0 * math.pi


def _case(entry, kind, dist, n, p, leaf, mac, precision, targets=0, tol=0.0, phi=False, hess=False, name=None):
    c = dict(entry=entry, kind=kind, dist=dist, n=n, targets=targets, p=p, leaf=leaf, mac=mac, tol=tol, phi=phi,
             hess=hess, precision=precision)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest request of a serving stream, with the options fmm! has by default: latency
        _case("solve", "source", "uniform", 1_000, 5, 20, 0.4, "f64", name="source_1k_f64"),
        # the plain drop-in configuration: 1e4 uniform point sources, potential and gradient
        _case("solve", "source", "uniform", 10_000, 6, 50, 0.5, "f64", phi=True, name="source_10k_f64"),
        # a user's script on a System in host memory: gather, solve, scatter and the lists fmm! returns
        _case("host", "source", "uniform", 20_011, 5, 20, 0.4, "f64", phi=True, name="source_20k_host_f64"),
        # one step of a small vortex simulation: velocity and its gradient (stretching), ragged size
        _case("solve", "vortex", "ring", 30_011, 8, 50, 0.4, "mixed", hess=True, name="vortex_30k_mixed"),
        # a serving request with a tolerance, vortex particles: velocity
        _case("solve", "vortex", "uniform", 48_211, 16, 80, 0.5, "f64", tol=1e-6, name="vortex_48k_tol_f64"),
        # a serving request with a tight tolerance, point sources
        _case("solve", "source", "clustered", 150_001, 16, 64, 0.5, "f64", tol=1e-7, phi=True,
              name="source_150k_tol_f64"),
        # the headline problem in both precisions
        _case("solve", "source", "clustered", 1_000_000, 10, 64, 0.5, "mixed", tol=1e-6, phi=True,
              name="source_1m_tol_mixed"),
        _case("solve", "source", "clustered", 1_000_000, 10, 64, 0.5, "f64", tol=1e-6, phi=True,
              name="source_1m_tol_f64"),
        # vortex ring: a mid-sized one in the drop-in precision, the full one on the mixed path
        _case("solve", "vortex", "ring", 300_000, 12, 80, 0.4, "f64", hess=True, name="vortex_300k_f64"),
        _case("solve", "vortex", "ring", 2_000_000, 12, 80, 0.4, "mixed", hess=True, name="vortex_2m_mixed"),
        # gradient of a loss at probes with respect to 2e5 sources and the probes: forward + adjoint
        _case("vjp", "source", "uniform", 200_000, 8, 50, 0.5, "mixed", targets=10_000, phi=True,
              name="vjp_200k_mixed"),
        # the all-pairs check a user holds an FMM result against: a target subsample, all sources
        _case("direct", "source", "clustered", 200_003, 0, 0, 0.0, "f64", targets=20_000, phi=True,
              name="direct_20k_f64"),
    ]


def draw(rng):
    """One more case of the listed ranges."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["source", "source", "source_tol", "source_tol", "vortex", "vortex", "vortex_tol", "vjp", "direct",
                       "host"])
    precision = rng.choice(["f64", "mixed"])
    mac = rng.choice([0.4, 0.5])
    if what == "source":
        return _case("solve", "source", rng.choice(["uniform", "clustered"]), size(1_000, 1_000_000), rng.randint(4, 12),
                     rng.randint(20, 100), mac, precision, phi=rng.random() < 0.7)
    if what == "source_tol":
        return _case("solve", "source", rng.choice(["uniform", "clustered"]), size(1_000, 1_000_000),
                     rng.choice([10, 12, 16]), rng.randint(40, 80), 0.5, precision, tol=10.0 ** rng.uniform(-8, -4),
                     phi=rng.random() < 0.7)
    if what == "vortex":
        return _case("solve", "vortex", rng.choice(["ring", "uniform"]), size(1_000, 500_000), rng.randint(4, 12),
                     rng.randint(40, 100), mac, precision, hess=rng.random() < 0.7)
    if what == "vortex_tol":
        return _case("solve", "vortex", rng.choice(["uniform", "clustered"]), size(1_000, 200_000),
                     rng.choice([10, 12, 16]), rng.randint(60, 100), 0.5, precision, tol=10.0 ** rng.uniform(-8, -4))
    if what == "vjp":
        return _case("vjp", "source", "uniform", size(2_000, 300_000), rng.randint(4, 10), rng.randint(30, 80), 0.5,
                     precision, targets=size(500, 20_000), phi=True)
    if what == "direct":
        kind = rng.choice(["source", "vortex"])
        return _case("direct", kind, "clustered", size(1_000, 300_000), 0, 0, 0.0, precision, targets=size(500, 30_000),
                     phi=kind == "source", hess=kind == "vortex" and rng.random() < 0.5)
    return _case("host", "source", rng.choice(["uniform", "clustered"]), size(1_000, 100_000), rng.randint(4, 8),
                 rng.randint(20, 50), 0.4, precision, phi=True)


# ---------------------------------------------------------------------------
# inputs
def _bodies(case, seed):
    """Source rows x y z radius strength(s), as the reference's source buffers hold them."""
    g = torch.Generator(device="cuda").manual_seed(1 + int(seed))
    n = case["n"]
    kw = dict(generator=g, device="cuda", dtype=torch.float64)
    vortex = case["kind"] == "vortex"
    b = torch.zeros((n, 7 if vortex else 5), device="cuda", dtype=torch.float64)
    if case["dist"] == "ring":
        phi = 2 * math.pi * torch.rand(n, **kw)
        off = 0.05 * torch.randn((n, 2), **kw)
        r = 1.0 + off[:, 0]
        b[:, 0], b[:, 1], b[:, 2] = r * torch.cos(phi), r * torch.sin(phi), off[:, 1]
        b[:, 4], b[:, 5] = -torch.sin(phi) / n, torch.cos(phi) / n
        b[:, 4:7] += 1e-3 * torch.randn((n, 3), **kw) / n
        return b
    if case["dist"] == "clustered":
        nb = n // 10
        centres = torch.rand((8, 3), **kw)
        k = torch.randint(0, 8, (n - nb,), generator=g, device="cuda")
        b[: n - nb, :3] = centres[k] + 0.05 * torch.randn((n - nb, 3), **kw)
        b[n - nb:, :3] = torch.rand((nb, 3), **kw)
        signed = True
    else:
        b[:, :3] = torch.rand((n, 3), **kw)
        signed = False
    if vortex:
        b[:, 4:7] = (2 * torch.rand((n, 3), **kw) - 1) / n
    else:
        b[:, 4] = torch.rand(n, **kw) * (2.0 if signed else 1.0) - (1.0 if signed else 0.0)
    return b


def _targets(case, seed, bodies):
    """Separate targets: probes around the sources (vjp), or a subsample of the sources (direct)."""
    g = torch.Generator(device="cuda").manual_seed(1_000_003 + int(seed))
    m = case["targets"]
    if case["entry"] == "direct":
        ids = torch.randint(0, case["n"], (m,), generator=g, device="cuda")
        return bodies[ids, :3].contiguous()
    return 2.0 * torch.rand((m, 3), generator=g, device="cuda", dtype=torch.float64) - 0.5


_ctx = None


def _context():
    """The solver context a program keeps for all its calls."""
    global _ctx
    if _ctx is None:
        _ctx = fm.Context(torch.cuda.current_device())
    _ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return _ctx


def _kind(case):
    return L.FMM_POINT_SOURCE if case["kind"] == "source" else L.FMM_POINT_VORTEX


def prepare(case, seed):
    s = dict(case=case, ctx=_context())
    b = _bodies(case, seed)
    if case["entry"] == "host":
        h = b.cpu().numpy()
        s["system"] = fm.PointSources(h[:, :3], h[:, 4])
        return s
    m = case["targets"] or case["n"]
    s["bodies"] = b
    s["out"] = torch.zeros((m, 16), device="cuda", dtype=torch.float64)
    s["src"] = L.SourceSystem(_kind(case), case["n"], b.shape[1], b.data_ptr(), L.FMM_MEMORY_DEVICE)
    if case["targets"]:
        s["pos"] = _targets(case, seed, b)
        s["tgt"] = L.TargetSystem(m, s["pos"].data_ptr(), 3, s["out"].data_ptr(), L.FMM_MEMORY_DEVICE)
    else:
        s["tgt"] = L.TargetSystem(m, None, 0, s["out"].data_ptr(), L.FMM_MEMORY_DEVICE)
    s["res"] = L.Result()
    if case["entry"] == "direct":
        return s
    s["opt"] = fm.make_options(expansion_order=case["p"], leaf_size_source=case["leaf"],
                               multipole_acceptance=case["mac"],
                               error_tolerance=fm.PowerRelativeGradient(case["tol"]) if case["tol"] else None,
                               scalar_potential=case["phi"], gradient=True, hessian=case["hess"],
                               precision=case["precision"])
    if case["entry"] == "vjp":
        g = torch.Generator(device="cuda").manual_seed(2_000_003 + int(seed))
        s["cot"] = torch.zeros((m, 16), device="cuda", dtype=torch.float64)
        s["cot"][:, 3] = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
        s["dq"] = torch.zeros(case["n"], device="cuda", dtype=torch.float64)
        s["dx"] = torch.zeros((case["n"], 3), device="cuda", dtype=torch.float64)
        s["dy"] = torch.zeros((m, 3), device="cuda", dtype=torch.float64)
    return s


def _dptr(t):
    return C.cast(t.data_ptr(), L._dp)


def _rows(case, out):
    """The requested rows of the target buffer (point sources always get the gradient)."""
    r = {"gradient": out[:, 4:7]}
    if case["phi"]:
        r["potential"] = out[:, 3]
    if case["hess"]:
        r["hessian"] = out[:, 7:16]
    return r


def run(s):
    case, ctx, lib = s["case"], s["ctx"], L.lib()
    if case["entry"] == "host":
        # (the call also returns the interaction lists, whose lengths depend on the bodies)
        fm.fmm(s["system"], expansion_order=case["p"], leaf_size=case["leaf"], multipole_acceptance=case["mac"],
               scalar_potential=True, precision=case["precision"], context=ctx)
        return {"potential": s["system"].potential[:, 0], "gradient": s["system"].potential[:, 4:7]}
    if case["entry"] == "direct":
        prec = L.FMM_PRECISION_F64 if case["precision"] == "f64" else L.FMM_PRECISION_MIXED
        ctx.check(lib.fmm_direct(ctx.handle, C.byref(s["tgt"]), C.byref(s["src"]), int(case["phi"]), 1,
                                 int(case["hess"]), prec))
        return _rows(case, s["out"])
    if case["entry"] == "vjp":
        ctx.check(lib.fmm_vjp(ctx.handle, C.byref(s["tgt"]), C.byref(s["src"]), C.byref(s["opt"]), _dptr(s["cot"]),
                              _dptr(s["dq"]), _dptr(s["dx"]), _dptr(s["dy"]), C.byref(s["res"])))
        return dict(_rows(case, s["out"]), d_strength=s["dq"], d_position=s["dx"], d_target=s["dy"])
    ctx.check(lib.fmm_solve(ctx.handle, C.byref(s["tgt"]), C.byref(s["src"]), C.byref(s["opt"]), C.byref(s["res"])))
    return _rows(case, s["out"])


# ---------------------------------------------------------------------------
def work(case):
    """Bytes: every body read once, every requested row written once.  Flops: the pairwise sums and
    the multipole-to-local translations (M2L) that the interaction lists prescribe for the given
    leaf size and acceptance, estimated with a fit to list sizes of these distributions: per body
    60 leaf / mac^3 near-field pairs and per leaf 15 / mac^3 translations, both times
    1 / (1 + 16 leaf / (n mac^6)), the share left where the tree is shallow."""
    vortex = case["kind"] == "vortex"
    n, m, leaf, mac = case["n"], case["targets"] or case["n"], case["leaf"], case["mac"]
    width = 3 + (1 if case["phi"] else 0) + (9 if case["hess"] else 0)
    per_pair = (72 if case["hess"] else 30) if vortex else 20
    nbytes = 8 * ((7 if vortex else 5) * n + 3 * case["targets"] + width * m)
    if case["entry"] == "direct":
        return {"bytes": nbytes, "flops": per_pair * n * m}
    f = 1.0 / (1.0 + 16.0 * leaf / (n * mac ** 6))
    pairs = 0.4 * n * m if case["targets"] else n * min(n, f * 60.0 * leaf / mac ** 3)
    # order that the tolerance asks for; 2 (n + 1) (2 n + 1) per degree for each rotation, and the
    # translation along the axis
    p = case["p"] if not case["tol"] else max(4, min(case["p"], round(-1.2 * math.log10(case["tol"]))))
    per_m2l = 4.0 * sum(2 * (k + 1) * (2 * k + 1) + (k + 1) * (p + 1 - k / 2) for k in range(p + 1))
    flops = per_pair * pairs + f * 15.0 / mac ** 3 * m / leaf * per_m2l * (2 if vortex else 1)
    if case["entry"] == "vjp":  # the forward and the adjoint solve, and the gradients written
        flops, nbytes = 2 * flops, nbytes + 8 * (4 * n + 4 * m)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the largest difference measured on these ranges: in 64 bits between the
    solve and the CPU restatement of the same algorithm and, for the all-pairs sums, between two
    body orders (2.4e-14 in all, 1e-13 for single values); on the mixed path between it and the
    64-bit solve, i.e. FP32 coordinates relative to a leaf's centre (1.4e-6, single values 2.4e-4).
    Probes of the gradient solves come closer to a source than the FP32 coordinates resolve (1.2e-5),
    and the all-pairs sums hold theirs relative to one target of a block (9.9e-5, values 2.6e-3)."""
    if case["precision"] == "f64":
        return {"rel": 1e-13, "max": 1e-12}
    return {"solve": {"rel": 6e-6, "max": 1e-3}, "host": {"rel": 6e-6, "max": 1e-3}, "vjp": {"rel": 5e-5, "max": 2e-4},
            "direct": {"rel": 4e-4, "max": 1e-2}}[case["entry"]]


# ---------------------------------------------------------------------------
def _exact_fields(pos, bodies, case, hess):
    """All-pairs sums in 64 bits at pos: (potential, gradient / velocity, velocity gradient)."""
    m, n = len(pos), len(bodies)
    vortex = case["kind"] == "vortex"
    phi = torch.zeros(m, device=pos.device, dtype=torch.float64)
    grad = torch.zeros((m, 3), device=pos.device, dtype=torch.float64)
    jac = torch.zeros((m, 9), device=pos.device, dtype=torch.float64) if hess else None
    step = max(1, (1 << 27) // max(n, 1))
    x, s = bodies[:, :3], bodies[:, 4:]
    for a in range(0, m, step):
        d = [pos[a:a + step, k, None] - x[None, :, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        w = torch.where(r2 > 0, r2, 1.0).rsqrt()
        w = torch.where(r2 > 0, w, 0.0)
        if not vortex:
            phi[a:a + step] = w @ s[:, 0]
            w3 = w * w * w
            for k in range(3):
                grad[a:a + step, k] = (d[k] * w3) @ s[:, 0]
            continue
        w3 = w * w * w
        cross = [(1, 2), (2, 0), (0, 1)]  # (G x d)_j = G_i d_k - G_k d_i
        for j, (i, k) in enumerate(cross):
            # the reference's velocity is G x d / r^3
            grad[a:a + step, j] = (d[k] * w3) @ s[:, i] - (d[i] * w3) @ s[:, k]
        if hess:
            w5 = w3 * w * w
            e = [w3 @ s[:, k] for k in range(3)]
            for i in range(3):
                t = d[i] * w5
                for j, (u, v) in enumerate(cross):
                    q = (t * d[v]) @ s[:, u] - (t * d[u]) @ s[:, v]
                    jac[a:a + step, 3 * i + j] = -3.0 * q
            # + eps_jki G_k / r^3 in row 3 i + j
            for (i, j, k, sg) in ((0, 1, 2, 1), (0, 2, 1, -1), (1, 0, 2, -1), (1, 2, 0, 1), (2, 0, 1, 1), (2, 1, 0, -1)):
                jac[a:a + step, 3 * i + j] += sg * e[k]
    return phi / FOUR_PI, grad / FOUR_PI, (jac / FOUR_PI if hess else None)


def exact(case, seed):
    """The all-pairs sums the solve approximates (and the adjoint's exact gradients), in 64 bits."""
    m = case["targets"] or case["n"]
    if case["n"] * m > (2.5e10 if case["kind"] == "source" else 4e9):
        return None
    b = _bodies(case, seed)
    pos = _targets(case, seed, b) if case["targets"] else b[:, :3]
    phi, grad, jac = _exact_fields(pos, b, case, case["hess"])
    r = {"gradient": grad}
    if case["phi"]:
        r["potential"] = phi
    if case["hess"]:
        r["hessian"] = jac
    if case["entry"] == "vjp":
        g = torch.Generator(device="cuda").manual_seed(2_000_003 + int(seed))
        w = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
        adj = torch.zeros((m, 5), device="cuda", dtype=torch.float64)
        adj[:, :3], adj[:, 4] = pos, w
        psi, gpsi, _ = _exact_fields(b[:, :3], adj, case, False)
        r.update(d_strength=psi, d_position=-b[:, 4:5] * gpsi, d_target=-w[:, None] * grad)
    return r
