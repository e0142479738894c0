"""Performance cases of the regularisers, and their results in 64 bits.

A case is one call that a user's program makes, through the package's public
entry points: a regulariser on a torch tensor or on a numpy array, a batch of
uneven volumes, a set of served prox requests, a differentiated batch.
``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges,
``prepare``/``run`` execute one, ``exact`` restates it in plain float64 torch.

Parameters are those of the repository's parity cases and benchmark.  Inputs
are piecewise-constant phantoms of ellipses or ellipsoids with Gaussian noise
of standard deviation 0.05, the data that the regularisers are made for.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ccpi-regularisation-toolkit_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

OPS = ("rof", "fgp", "pd", "sb", "tgv", "ndf", "diff4th", "llt", "dtv")

# floating-point operations per voxel and iteration, (2D, 3D), counted from the update formulas
FLOPS = {"rof": (32, 66), "fgp": (24, 36), "pd": (24, 35), "sb": (56, 86), "tgv": (75, 165), "ndf": (20, 30),
         "diff4th": (50, 120), "llt": (46, 90), "dtv": (38, 58)}


def _case(op, nz, ny, nx, iterations, tolerance=0.0, api="device", aniso=False, nonneg=False, penalty=1, name=None):
    c = {"op": op, "api": api, "nz": nz, "ny": ny, "nx": nx, "iterations": iterations, "tolerance": tolerance,
         "aniso": aniso, "nonneg": nonneg, "penalty": penalty}
    if name is not None:
        c["name"] = name
    return c


def _group(kind, name=None, **values):
    c = {"op": kind, **values}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a thumbnail or a detector crop of odd size: the smallest calls, latency counts
        _case("fgp", 1, 181, 217, 100, name="fgp_2d_small"),
        # one 512^2 slice with the gradient flow's many short steps (the repository's 2D configuration)
        _case("rof", 1, 512, 512, 2000, name="rof_2d_slice"),
        # a slice as it leaves a reconstruction, odd on both sides
        _case("diff4th", 1, 701, 723, 300, name="diff4th_2d_odd"),
        # a detector frame, second-order model
        _case("tgv", 1, 1024, 1024, 200, name="tgv_2d_frame"),
        # a joint reconstruction's channel with its reference image and the stopping rule
        _case("dtv", 1, 640, 768, 300, tolerance=1e-6, nonneg=True, name="dtv_2d_stop"),
        # the repository's benchmark: a full volume with the stopping rule, the largest call
        _case("fgp", 512, 512, 512, 500, tolerance=1e-6, nonneg=True, name="fgp_3d_large"),
        # a numpy volume through the toolkit's own signature, copies included
        _case("pd", 256, 256, 256, 200, tolerance=1e-6, api="host", nonneg=True, name="pd_3d_host"),
        # an ordinary volume
        _case("sb", 256, 256, 256, 60, name="sb_3d"),
        # a cropped region of interest: ragged, odd rows
        _case("ndf", 143, 201, 255, 100, tolerance=1e-6, name="ndf_3d_odd"),
        # a medium volume with the fourth-order term
        _case("llt", 96, 160, 192, 100, name="llt_3d"),
        # volumes of uneven size regularised together
        _group("fgp_batch", volumes=12, smallest=48, largest=144, iterations=100, name="fgp_batch"),
        # a learned lambda: forward and adjoint of a batch
        _group("fgp_grad", volumes=4, nz=96, ny=96, nx=96, iterations=60, name="fgp_grad_batch"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(OPS * 3 + ("fgp_batch", "tgv_batch", "serve", "fgp_grad", "rof_grad"))
    if kind in ("fgp_batch", "tgv_batch"):
        return _group(kind, volumes=rng.randint(3, 12), smallest=rng.randint(24, 64), largest=rng.randint(65, 144),
                      iterations=rng.randint(40, 120))
    if kind in ("fgp_grad", "rof_grad"):
        two = rng.random() < 0.3
        return _group(kind, volumes=rng.randint(1, 4), nz=1 if two else rng.randint(24, 96),
                      ny=_log_int(rng, 64, 512) if two else rng.randint(40, 112),
                      nx=_log_int(rng, 64, 512) if two else rng.randint(40, 112), iterations=rng.randint(20, 60))
    if kind == "serve":
        # requests of an iterative reconstruction: FISTA steps over warm-started proxes
        return _group("serve", requests=rng.randint(2, 5), smallest=rng.randint(64, 96), largest=rng.randint(97, 160),
                      outer=rng.randint(3, 8), inner=rng.randint(5, 20))
    tolerance = rng.choice((0.0, 0.0, 1e-6, 1e-5))
    api = rng.choice(("device", "device", "device", "host"))
    opts = {"aniso": rng.random() < 0.3, "nonneg": rng.random() < 0.5, "penalty": rng.randint(1, 5)}
    if rng.random() < 0.5:
        ny, nx = _log_int(rng, 96, 3000), _log_int(rng, 96, 3000)
        iterations = _log_int(rng, 50, 1000)
        nz = 1
    else:
        nz, ny, nx = (_log_int(rng, 32, 400) for _ in range(3))
        iterations = _log_int(rng, 30, 300)
    # no more than an eighth of the largest listed case's voxel updates
    most = 500 * 512 ** 3 // 8 // (4 if kind in ("tgv", "sb") else 1)
    iterations = max(10, min(iterations, most // (nz * ny * nx)))
    return _case(kind, nz, ny, nx, iterations, tolerance, api, **opts)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _shape(case):
    return (case["ny"], case["nx"]) if case["nz"] == 1 else (case["nz"], case["ny"], case["nx"])


def _phantom(shape, seed, device, noise=0.05):
    """(noisy, clean) float32 phantoms of overlapping ellipses/ellipsoids."""
    rng = np.random.default_rng(seed)
    d = len(shape)
    img = torch.zeros(shape, dtype=torch.float32, device=device)
    axes = [((torch.arange(n, device=device, dtype=torch.float32) + 0.5) / n * 2 - 1).reshape(
        [-1 if a == b else 1 for b in range(d)]) for a, n in enumerate(shape)]
    for _ in range(12):
        centre, semi, value = rng.uniform(-0.7, 0.7, d), rng.uniform(0.05, 0.5, d), float(rng.uniform(0.1, 1.0))
        turn = np.linalg.qr(rng.normal(size=(d, d)))[0]
        r2 = 0.0
        for b in range(d):
            r2 = r2 + (sum(float(turn[a, b]) * (axes[a] - float(centre[a])) for a in range(d)) / float(semi[b])) ** 2
        img = torch.where(r2 <= 1.0, torch.full_like(img, value), img)
    g = torch.Generator(device=device).manual_seed(int(seed) + 1)
    return img + noise * torch.randn(shape, generator=g, device=device, dtype=torch.float32), img


def _uneven(case):
    """Shapes of the case's volumes, the same for every input seed; served requests are 2D one in four."""
    key = [case.get(k, 0) for k in ("volumes", "requests", "smallest", "largest")]
    rng = np.random.default_rng(key)
    lo, hi = case["smallest"], case["largest"]
    n = case.get("volumes", 0) or case.get("requests", 0)
    sizes = np.exp(rng.uniform(math.log(lo), math.log(hi), size=(n, 3))).astype(int)
    return [tuple(int(v) for v in (s * 3)[1:]) if case["op"] == "serve" and i % 4 == 1 else tuple(int(v) for v in s)
            for i, s in enumerate(sizes)]


LAM = {"rof": 0.02, "fgp": 0.03, "pd": 0.03, "sb": 0.03, "tgv": 0.03, "ndf": 0.02, "diff4th": 0.8, "llt": 0.02,
       "dtv": 0.05, "fgp_batch": 0.03, "tgv_batch": 0.03, "fgp_grad": 0.05, "rof_grad": 0.02}
SERVED = (("FGP", (0.03, 0, 0)), ("ROF", (0.02, 0.001)), ("SB", (0.05, 0)), ("NDF", (0.02, 0.05, 0.01, 1)))


def prepare(case, seed):
    state = {"case": case}
    op = case["op"]
    if op in ("fgp_batch", "tgv_batch"):
        state["volumes"] = [_phantom(s, seed * 97 + i, "cuda")[0] for i, s in enumerate(_uneven(case))]
        return state
    if op == "serve":
        from ccpi.filters.serving import ProxRequest, ProxServer

        state["server"] = ProxServer(slots=8)
        state["requests"] = [
            ProxRequest(i, SERVED[i % 4][0], _phantom(s, seed * 97 + i, "cuda")[0].cpu().numpy(), SERVED[i % 4][1],
                        outer=case["outer"], inner=case["inner"])
            for i, s in enumerate(_uneven(case))]
        return state
    if op in ("fgp_grad", "rof_grad"):
        state["f"] = torch.stack([_phantom(_shape(case), seed * 97 + i, "cuda")[0] for i in range(case["volumes"])])
        state["lam"] = torch.tensor(LAM[op], dtype=torch.float64)
        g = torch.Generator(device="cuda").manual_seed(seed)
        state["ybar"] = torch.randn(state["f"].shape, generator=g, device="cuda", dtype=torch.float32)
        return state
    noisy, clean = _phantom(_shape(case), seed, "cuda")
    state["f"] = noisy.cpu().numpy() if case["api"] == "host" else noisy
    if op == "dtv":  # the other channel: the same edges at other heights
        ref = 1.0 - 0.5 * clean
        state["ref"] = ref.cpu().numpy() if case["api"] == "host" else ref
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _run_device(case, state):
    from ccpi.filters import regularisersCuPy as R

    op, f, it, tol = case["op"], state["f"], case["iterations"], case["tolerance"]
    lam, aniso, nonneg = LAM[op], int(case["aniso"]), int(case["nonneg"])
    if op == "rof":
        return R.ROF_TV(f, lam, it, 0.001, tolerance_param=tol)
    if op == "fgp":
        return R.FGP_TV(f, lam, it, tol, aniso, nonneg)
    if op == "pd":
        return R.PD_TV(f, lam, it, tol, aniso, nonneg, 8.0)
    if op == "sb":
        return R.SB_TV(f, lam, it, tol, aniso)
    if op == "tgv":
        return R.TGV(f, lam, 1.0, 2.0, it, 12.0, tol)
    if op == "ndf":
        return R.NDF(f, lam, 0.05, it, 0.01, case["penalty"], tol)
    if op == "diff4th":
        return R.Diff4th(f, lam, 0.02, it, 0.0001, tol)
    if op == "llt":
        return R.LLT_ROF(f, lam, 0.01, it, 0.001, tol)
    return R.FGP_dTV(f, state["ref"], lam, it, tol, 0.2, aniso, nonneg)


def _run_host(case, state):
    from ccpi.filters import regularisers as R

    op, f, it, tol = case["op"], state["f"], case["iterations"], case["tolerance"]
    lam, aniso, nonneg = LAM[op], int(case["aniso"]), int(case["nonneg"])
    if op == "rof":
        return R.ROF_TV(f, lam, it, 0.001, tol, device="gpu")
    if op == "fgp":
        return R.FGP_TV(f, lam, it, tol, aniso, nonneg, device="gpu")
    if op == "pd":
        return R.PD_TV(f, lam, it, tol, 8.0, aniso, nonneg, device="gpu")
    if op == "sb":
        return R.SB_TV(f, lam, it, tol, aniso, device="gpu")
    if op == "tgv":
        return R.TGV(f, lam, 1.0, 2.0, it, 12.0, tol, device="gpu")
    if op == "ndf":
        return R.NDF(f, lam, 0.05, it, 0.01, case["penalty"], tol, device="gpu")
    if op == "diff4th":
        return R.Diff4th(f, lam, 0.02, it, 0.0001, tol, device="gpu")
    if op == "llt":
        return R.LLT_ROF(f, lam, 0.01, it, 0.001, tol, device="gpu")
    return R.FGP_dTV(f, state["ref"], lam, it, tol, 0.2, aniso, nonneg, device="gpu")


def run(state):
    case = state["case"]
    op, it = case["op"], case.get("iterations")
    if op == "fgp_batch":
        from ccpi.filters.batch import FGP_TV_batch

        return FGP_TV_batch(state["volumes"], LAM[op], it)
    if op == "tgv_batch":
        from ccpi.filters.batch import TGV_batch

        return TGV_batch(state["volumes"], LAM[op], 1.0, 2.0, it, 12.0)
    if op == "serve":
        return [r.output for r in state["server"].serve(state["requests"], realtime=False)]
    if op in ("fgp_grad", "rof_grad"):
        from ccpi.filters import autograd as A

        f, lam = state["f"].detach().requires_grad_(True), state["lam"].detach().requires_grad_(True)
        y = (A.fgp_tv(f, lam, it, batched=True) if op == "fgp_grad" else A.rof_tv(f, lam, it, 0.001, batched=True))
        y.backward(state["ybar"])
        return {"y": y.detach(), "f_grad": f.grad, "lam_grad": lam.grad}
    return _run_host(case, state) if case["api"] == "host" else _run_device(case, state)


def _voxels(case):
    if case["op"] in ("fgp_batch", "tgv_batch", "serve"):
        shapes = _uneven(case)
    else:
        shapes = [_shape(case)] * case.get("volumes", 1)
    return [(len(s), int(np.prod(s))) for s in shapes]


def work(case):
    op = case["op"]
    nbytes = flops = 0
    for i, (d, n) in enumerate(_voxels(case)):
        if op == "serve":
            alg = ("fgp", "rof", "sb", "ndf")[i % 4]
            steps, arrays = case["outer"] * case["inner"], 2
        elif op.endswith("_grad"):  # forward and its adjoint; f, ybar in, y, fbar out
            alg, steps, arrays = op[:3], 2 * case["iterations"], 4
        else:
            alg, steps, arrays = op.replace("_batch", ""), case["iterations"], 3 if op == "dtv" else 2
        nbytes += 4 * n * arrays
        flops += FLOPS[alg][d - 2] * n * steps
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _f32(v):
    return float(np.float32(v))


def _cut(a, axis, lo, hi):
    return a.narrow(axis, lo, hi - lo)


def _hi(a, axis):
    """a at the next index, mirrored at the last (an axis of length 1: a itself)."""
    n = a.shape[axis]
    return a if n == 1 else torch.cat([_cut(a, axis, 1, n), _cut(a, axis, n - 2, n - 1)], axis)


def _lo(a, axis):
    n = a.shape[axis]
    return a if n == 1 else torch.cat([_cut(a, axis, 1, 2), _cut(a, axis, 0, n - 1)], axis)


def _fwd0(a, axis):
    """a[i+1] - a[i], zero at the last index."""
    n = a.shape[axis]
    return torch.cat([_cut(a, axis, 1, n) - _cut(a, axis, 0, n - 1), torch.zeros_like(_cut(a, axis, 0, 1))], axis)


def _bwd0(a, axis):
    """a[i] - a[i-1] with a[-1] = 0."""
    n = a.shape[axis]
    return torch.cat([_cut(a, axis, 0, 1), _cut(a, axis, 1, n) - _cut(a, axis, 0, n - 1)], axis)


def _bwd_tgv(a, axis):
    """a[0] at 0, -a[n-2] at the last index, a[i] - a[i-1] between."""
    n = a.shape[axis]
    if n == 1:
        return a.clone()
    return torch.cat([_cut(a, axis, 0, 1), _cut(a, axis, 1, n - 1) - _cut(a, axis, 0, n - 2),
                      -_cut(a, axis, n - 2, n - 1)], axis)


class _Stop:
    """Every fifth iteration; stops at the fourth relative change below the tolerance."""

    def __init__(self, tolerance):
        self.tolerance, self.count = _f32(tolerance), 0

    def due(self, it):
        return self.tolerance != 0.0 and it % 5 == 0

    def now(self, u, before):
        re = float(torch.linalg.vector_norm(u - before) / torch.linalg.vector_norm(u))
        self.count += re < self.tolerance
        return self.count > 3


def _axes(f):
    return [-1, -2, -3][: f.dim()]


def _minmod(a, b):
    return 0.5 * (torch.sign(a) + torch.sign(b)) * torch.minimum(a.abs(), b.abs())


def _tv_div(u, eps):
    """Divergence of the minmod-normalised gradient (ROF flow)."""
    ax = _axes(u)
    hi = [_hi(u, a) - u for a in ax]
    m2 = [_minmod(h, u - _lo(u, a)) ** 2 for h, a in zip(hi, ax)]
    div = 0.0
    for c, a in enumerate(ax):
        flux = hi[c] / torch.sqrt(hi[c] ** 2 + sum(m2[k] for k in range(len(ax)) if k != c) + eps)
        div = div + (flux - _lo(flux, a))
    return div


def _rof(f, lam, it, tau, tol=0.0, u=None):
    u, stop = f.clone() if u is None else u, _Stop(tol)
    for k in range(it):
        before = u
        u = u + tau * (lam * _tv_div(u, 1e-8) - (u - f))
        if stop.due(k) and stop.now(u, before):
            break
    return u


def _project(p, aniso):
    if aniso:
        return [q / torch.clamp(q.abs(), min=1.0) for q in p]
    s = 1.0 / torch.sqrt(torch.clamp(sum(q * q for q in p), min=1.0))
    return [q * s for q in p]


def _fgp(f, lam, it, tol=0.0, aniso=False, nonneg=False, start=None, ref=None):
    """(U, P): fast gradient projection; `start`: the dual iterate of an earlier call; `ref`: the
    normalised reference gradient of directional TV."""
    ax, stop = _axes(f), _Stop(tol)
    multip = 1.0 / ((8.0 if len(ax) == 2 else 26.0 if ref is not None else 12.0) * lam)

    def across(v):
        if ref is None:
            return v
        ip = sum(a * b for a, b in zip(v, ref))
        return [a - ip * b for a, b in zip(v, ref)]

    r = [torch.zeros_like(f) for _ in ax] if start is None else start
    old, u, t = r, torch.zeros_like(f), 1.0
    for k in range(it):
        before = u
        r = across(r)
        u = f - lam * sum(_bwd0(q, a) for q, a in zip(r, ax))
        if nonneg:
            u = torch.clamp(u, min=0.0)
        p = _project([q - multip * g for q, g in zip(r, across([_fwd0(u, a) for a in ax]))], aniso)
        t_next = 0.5 * (1.0 + math.sqrt(1.0 + 4.0 * t * t))
        r = [a + (t - 1.0) / t_next * (a - b) for a, b in zip(p, old)]
        old, t = p, t_next
        if stop.due(k) and stop.now(u, before):
            break
    return u, old


def _dtv(f, ref, lam, it, tol, aniso, nonneg):
    ax, grad = _axes(f), []
    for a in ax:
        n = ref.shape[a]
        grad.append(torch.cat([_cut(ref, a, 1, n), torch.zeros_like(_cut(ref, a, 0, 1))], a) - ref)
    size = torch.sqrt(sum(g * g for g in grad) + _f32(0.2) ** 2)
    return _fgp(f, lam, it, tol, aniso, nonneg, ref=[g / size for g in grad])[0]


def _pd(f, lam, it, tol, aniso, nonneg):
    ax, stop = _axes(f), _Stop(tol)
    tau = lam * _f32(0.1)
    sigma, lt = 1.0 / (8.0 * tau), tau / lam
    u, p = f.clone(), [torch.zeros_like(f) for _ in ax]
    for k in range(it):
        p = [q + sigma * (_hi(u, a) - u) for q, a in zip(p, ax)]
        if nonneg:
            u = torch.clamp(u, min=0.0)
        p = _project(p, aniso)
        before = u
        u = (u + tau * sum(_bwd0(q, a) for q, a in zip(p, ax)) + lt * f) / (1.0 + lt)
        if stop.due(k) and stop.now(u, before):
            break
        u = 2.0 * u - before
    return u


def _sb(f, mu, it, tol=0.0, aniso=False, start=None):
    """(U, (D, B)): split Bregman with two Jacobi sweeps per iteration."""
    ax, stop = _axes(f), _Stop(tol)
    mu = 1.0 / mu
    lam = 2.0 * mu
    norm = 1.0 / (mu + 2.0 * len(ax) * lam)
    zero = [torch.zeros_like(f) for _ in ax]
    d, b = (zero, list(zero)) if start is None else start
    u = f.clone()
    for k in range(it):
        fixed = mu * f + lam * sum((_lo(x, a) - x) - (_lo(y, a) - y) for x, y, a in zip(d, b, ax))
        for _ in range(2):
            before = u
            u = norm * (fixed + lam * sum(_hi(u, a) + _lo(u, a) for a in ax))
        grad = [_hi(u, a) - u for a in ax]
        g = [x + y for x, y in zip(grad, b)]
        if aniso:
            d = [torch.sign(x) * torch.clamp(x.abs() - 1.0 / lam, min=0.0) for x in g]
        else:
            den = torch.sqrt(sum(x * x for x in g))
            m = torch.clamp(den - 1.0 / lam, min=0.0) / torch.where(den > 0, den, torch.ones_like(den))
            d = [m * x for x in g]
        b = [x - y for x, y in zip(g, d)]
        if stop.due(k) and stop.now(u, before):
            break
    return u, (d, b)


def _tgv(f, lam, it, tol=0.0, alpha1=1.0, alpha0=2.0, lipschitz=12.0):
    ax, stop = _axes(f), _Stop(tol)
    n = len(ax)
    tau = sigma = lipschitz ** -0.5
    pairs = [(a, a) for a in range(n)] + [(a, b) for a in range(n) for b in range(a + 1, n)]
    at = {}
    for i, (a, b) in enumerate(pairs):
        at[a, b] = at[b, a] = i
    u = f.clone()
    p, v = [torch.zeros_like(f) for _ in ax], [torch.zeros_like(f) for _ in ax]
    q = [torch.zeros_like(f) for _ in pairs]
    for k in range(it):
        p = [x + sigma * (_fwd0(u, a) - y) for x, y, a in zip(p, v, ax)]
        s = torch.clamp(torch.sqrt(sum(x * x for x in p)) / alpha1, min=1.0)
        p = [x / s for x in p]
        q = [x + sigma * 0.5 * (_fwd0(v[a], ax[b]) + _fwd0(v[b], ax[a])) for x, (a, b) in zip(q, pairs)]
        s = torch.clamp(torch.sqrt(sum((1.0 if a == b else 2.0) * x * x for x, (a, b) in zip(q, pairs))) / alpha0,
                        min=1.0)
        q = [x / s for x in q]
        before = u
        u = (lam * (u + tau * sum(_bwd_tgv(x, a) for x, a in zip(p, ax))) + tau * f) / (lam + tau)
        u = 2.0 * u - before
        v = [y + 2.0 * tau * (p[c] + sum(_bwd_tgv(q[at[c, b]], ax[b]) for b in range(n))) for c, y in enumerate(v)]
        if stop.due(k) and stop.now(u, before):
            break
    return u


def _ndf_flux(e, sg, penalty):
    a, zero = e.abs(), torch.zeros_like(e)
    if penalty == 1:
        return torch.where(a > sg, torch.sign(e), e / sg)
    if penalty == 2:
        return e / (1.0 + (e / sg) ** 2)
    if penalty == 3:
        return torch.where(a <= sg, e * (1.0 - (e / sg) ** 2) ** 2, zero)
    if penalty == 4:
        return torch.where(a > sg, zero, e)
    return torch.where(a <= 2.0 * sg, torch.where(a > sg, torch.sign(e), e / sg), zero)


def _ndf(f, lam, sigma, it, tau, penalty, tol=0.0, u=None):
    stop, sg = _Stop(tol), _f32(sigma / math.sqrt(2.0))
    u = f.clone() if u is None else u
    for k in range(it):
        before = u
        s = sum(_ndf_flux(_hi(u, a) - u, sg, penalty) + _ndf_flux(_lo(u, a) - u, sg, penalty) for a in _axes(f))
        u = u + tau * (lam * s - (u - f))
        if stop.due(k) and stop.now(u, before):
            break
    return u


def _diff4th(f, lam, sigma, it, tau, tol):
    ax, stop, u = _axes(f), _Stop(tol), f.clone()
    n = len(ax)
    for k in range(it):
        before = u
        g = [0.5 * (_lo(u, a) - _hi(u, a)) for a in ax]
        second = [_lo(u, a) + _hi(u, a) - 2.0 * u for a in ax]
        cross = 0.0
        for i in range(n):
            for j in range(i + 1, n):
                lo, hi = _lo(u, ax[i]), _hi(u, ax[i])
                cross = cross + 0.5 * g[i] * g[j] * (_lo(lo, ax[j]) + _hi(hi, ax[j]) - _hi(lo, ax[j]) - _lo(hi, ax[j]))
        den = sum(x * x for x in g)
        along = sum(x * y * y for x, y in zip(second, g)) + cross
        other = sum(x * (den - y * y) for x, y in zip(second, g)) - cross
        safe = torch.clamp(den, min=1e-7)
        c = 1.0 / (1.0 + den / (sigma * sigma))
        w = c * c * along / safe + c * other / safe
        lap = sum(_lo(w, a) + _hi(w, a) - 2.0 * w for a in ax)
        u = u + tau * (-lam * lap - (u - f))
        if stop.due(k) and stop.now(u, before):
            break
    return u


def _llt(f, lam_rof, lam_llt, it, tau, tol):
    ax, stop, u = _axes(f), _Stop(tol), f.clone()
    for k in range(it):
        before = u
        lap = 0.0
        for a in ax:
            dd = _hi(u, a) - 2.0 * u + _lo(u, a)
            dd = dd / (dd.abs() + 1e-12)
            lap = lap + _hi(dd, a) - 2.0 * dd + _lo(dd, a)
        u = u + tau * (lam_rof * _tv_div(u, 1e-12) - lam_llt * lap - (u - f))
        if stop.due(k) and stop.now(u, before):
            break
    return u


def _fista(request):
    f = torch.from_numpy(request.volume).cuda().double()
    prm = [_f32(p) for p in request.params]
    x, y, t, warm = f.clone(), f.clone(), 1.0, None
    for _ in range(request.outer):
        z = y - request.step * (y - f)
        if request.alg == "FGP":
            new, warm = _fgp(z, prm[0], request.inner, 0.0, prm[1] != 0, prm[2] == 1, start=warm)
        elif request.alg == "SB":
            new, warm = _sb(z, prm[0], request.inner, 0.0, prm[1] == 1, start=warm)
        elif request.alg == "ROF":
            new = warm = _rof(z, prm[0], request.inner, prm[1], u=warm)
        else:
            new = warm = _ndf(z, prm[0], prm[1], request.inner, prm[2], int(prm[3]), u=warm)
        t_next = 0.5 * (1.0 + math.sqrt(1.0 + 4.0 * t * t))
        y = new + (t - 1.0) / t_next * (new - x)
        x, t = new, t_next
    return x.cpu().numpy()


def exact(case, seed):
    op, it = case["op"], case.get("iterations")
    state = prepare(case, seed)
    lam = _f32(LAM[op]) if op in LAM else None
    if op == "fgp_batch":
        return [_fgp(v.double(), lam, it)[0] for v in state["volumes"]]
    if op == "tgv_batch":
        return [_tgv(v.double(), lam, it) for v in state["volumes"]]
    if op == "serve":
        return [_fista(r) for r in state["requests"]]
    if op in ("fgp_grad", "rof_grad"):
        ys, fs, lams = [], [], 0.0
        for f, ybar in zip(state["f"], state["ybar"]):
            f = f.double().requires_grad_(True)
            one = torch.tensor(lam, dtype=torch.float64, requires_grad=True)
            y = _fgp(f, one, it)[0] if op == "fgp_grad" else _rof(f, one, it, _f32(0.001))
            y.backward(ybar.double())
            ys.append(y.detach())
            fs.append(f.grad)
            lams = lams + one.grad
        return {"y": torch.stack(ys), "f_grad": torch.stack(fs), "lam_grad": lams}
    f = torch.as_tensor(state["f"]).cuda().double()
    tol, aniso, nonneg = case["tolerance"], case["aniso"], case["nonneg"]
    if op == "rof":
        u = _rof(f, lam, it, _f32(0.001), tol)
    elif op == "fgp":
        u = _fgp(f, lam, it, tol, aniso, nonneg)[0]
    elif op == "pd":
        u = _pd(f, lam, it, tol, aniso, nonneg)
    elif op == "sb":
        u = _sb(f, lam, it, tol, aniso)[0]
    elif op == "tgv":
        u = _tgv(f, lam, it, tol)
    elif op == "ndf":
        u = _ndf(f, lam, _f32(0.05), it, _f32(0.01), case["penalty"], tol)
    elif op == "diff4th":
        u = _diff4th(f, lam, _f32(0.02), it, _f32(0.0001), tol)
    elif op == "llt":
        u = _llt(f, lam, _f32(0.01), it, _f32(0.001), tol)
    else:
        u = _dtv(f, torch.as_tensor(state["ref"]).cuda().double(), lam, it, tol, aniso, nonneg)
    return u.cpu().numpy() if case["api"] == "host" else u
