"""The work this framework is timed on: solves, batches and gradients as a
user's program calls them.

Every case goes through a public entry point of ``reg_drot`` on inputs made
from a seed.  Solves run a budget of iterations (``iters``; even, so that the
quadratic solver hands back the plan itself) with a tolerance that the budget
ends before, as a call inside a training loop or a fixed-effort comparison
does; the smallest solve runs to its tolerance.

    kind       entry point
    qr         reg_drot.quadratic_drot (FP32 cost) / reg_drot.solve_qr (BF16-stored cost)
    gl         reg_drot.group_lasso_drot
    qr_batch   reg_drot.batch.QRBatch.solve
    qr_diff    reg_drot.cost.packed_sqeuclidean_cost -> reg_drot.autograd.batch_quadratic_drot_fn
               -> backward to the points
    gl_batch   reg_drot.batch.GLBatch.solve
    cost       reg_drot.cost.sqeuclidean_cost and its backward
"""
import math
import os
import random
import sys
import warnings

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "regularized-drot_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import reg_drot  # noqa: E402
from reg_drot.autograd import batch_quadratic_drot_fn  # noqa: E402
from reg_drot.batch import GLBatch, QRBatch  # noqa: E402
from reg_drot.cost import packed_sqeuclidean_cost, sqeuclidean_cost  # noqa: E402

# A gradient taken after a fixed budget of iterations warns once per call site.
warnings.filterwarnings("ignore", message=".*did not converge.*")

RHO = 2.0
NEVER = 1e-12  # a tolerance below FP32's reach: the budget of iterations ends the solve


def listed():
    return [
        # A call so small that launches and latency are all of it: an inner problem of a
        # larger method, solved to its tolerance.
        dict(name="qr_96x80", kind="qr", rows=96, cols=80, cost="clouds", alpha=1e-2,
             iters=5000, eps=1e-6, dtype="float32"),
        # The 1000 x 1000 problem on normalised squared distances of 2-D clouds.
        dict(name="qr_1000x1000", kind="qr", rows=1000, cols=1000, cost="clouds", alpha=1e-3,
             iters=600, eps=NEVER, dtype="float32"),
        # Odd sizes whose columns start off every vector boundary, Dirichlet marginals.
        dict(name="qr_777x1203", kind="qr", rows=777, cols=1203, cost="uniform", alpha=1e-3,
             iters=600, eps=NEVER, dtype="float32"),
        # The dense 3000 x 3000 workload: plan and cost fit the L2 cache.
        dict(name="qr_3000x3000", kind="qr", rows=3000, cols=3000, cost="uniform", alpha=1e-3,
             iters=600, eps=NEVER, dtype="float32"),
        # The dense 10000 x 10000 workload: 800 MB of plan and cost, beyond every cache.
        dict(name="qr_10000x10000", kind="qr", rows=10000, cols=10000, cost="uniform",
             alpha=1e-2, iters=200, eps=NEVER, dtype="float32"),
        # A cost stored in BF16 to halve its bytes, a rectangular problem.
        dict(name="qr_bf16_2600x4100", kind="qr", rows=2600, cols=4100, cost="uniform",
             alpha=1e-3, iters=400, eps=NEVER, dtype="bfloat16"),
        # Domain adaptation: 1500 labelled source points, 1000 target points, 2 classes.
        dict(name="gl_1500x1000", kind="gl", rows=1500, cols=1000, classes=2, weight=1e-3,
             iters=250, eps=NEVER),
        # A large adaptation problem, classes of 2000 rows.
        dict(name="gl_6000x5000", kind="gl", rows=6000, cols=5000, classes=3, weight=1e-3,
             iters=250, eps=NEVER),
        # Many uneven problems in one launch (rows and columns drawn from 64..2048).
        dict(name="qr_batch_32", kind="qr_batch", instances=32, low=64, high=2048, dim=8,
             alpha=1e-3, iters=400, shapes_seed=1, dtype="float32"),
        # A differentiable OT loss over point clouds: cost, solve, loss, gradient to the points.
        dict(name="qr_diff_8", kind="qr_diff", instances=8, low=512, high=2048, dim=16,
             alpha=1e-2, iters=400, shapes_seed=2),
        # Many uneven adaptation problems in one launch.
        dict(name="gl_batch_16", kind="gl_batch", instances=16, low=256, high=2048, classes=2,
             weight=1e-3, iters=300, shapes_seed=3),
        # The cost matrix of two clouds and its chain rule, as a loss on its own uses them.
        dict(name="cost_4000x3000", kind="cost", rows=4000, cols=3000, dim=16),
    ]


# --------------------------------------------------------------------------- draws
_MOST = 200 * 10000 * 10000  # element-iterations of the largest listed solve


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _iters(rng, elements, lo, hi):
    """An even budget within [lo, hi] that keeps the work below the largest solve's."""
    most = max(lo, min(hi, int(0.8 * _MOST / elements)))
    return max(2, _log(rng, lo, most) // 2 * 2)


def draw(rng):
    kind = rng.choice(("qr", "qr", "qr", "qr", "gl", "gl", "qr_batch", "qr_diff", "gl_batch",
                       "cost"))
    if kind == "qr":
        r, c = _log(rng, 64, 9000), _log(rng, 64, 9000)
        dtype = rng.choice(("float32", "float32", "float32", "bfloat16"))
        return dict(kind=kind, rows=r, cols=c, cost=rng.choice(("clouds", "uniform")),
                    alpha=rng.choice((1e-3, 1e-2)), iters=_iters(rng, r * c, 100, 600),
                    eps=NEVER, dtype=dtype)
    if kind == "gl":
        g = rng.choice((1, 2, 3, 5, 10))
        r = max(_log(rng, 64, 6000), 32 * g)
        c = _log(rng, 64, 6000)
        weight = rng.choice((1e-3, 5e-3)) if r * c < 2000 * 1000 else 1e-3
        return dict(kind=kind, rows=r, cols=c, classes=g, weight=weight,
                    iters=_iters(rng, r * c, 200, 300), eps=NEVER)
    if kind == "qr_batch":
        n = rng.randint(4, 40)
        return dict(kind=kind, instances=n, low=64, high=_log(rng, 256, 2048), dim=8,
                    alpha=rng.choice((1e-3, 1e-2)), iters=_log(rng, 100, 400) // 2 * 2,
                    shapes_seed=rng.randrange(1 << 20),
                    dtype=rng.choice(("float32", "float32", "bfloat16")))
    if kind == "qr_diff":
        return dict(kind=kind, instances=rng.randint(1, 10), low=_log(rng, 128, 512),
                    high=_log(rng, 768, 2048), dim=rng.choice((8, 16)), alpha=1e-2,
                    iters=_log(rng, 200, 400) // 2 * 2, shapes_seed=rng.randrange(1 << 20))
    if kind == "gl_batch":
        return dict(kind=kind, instances=rng.randint(2, 24), low=_log(rng, 64, 256),
                    high=_log(rng, 384, 2048), classes=rng.choice((1, 2, 3)), weight=1e-3,
                    iters=_log(rng, 200, 300) // 2 * 2, shapes_seed=rng.randrange(1 << 20))
    return dict(kind=kind, rows=_log(rng, 100, 6000), cols=_log(rng, 100, 6000),
                dim=rng.choice((8, 16, 24, 32)))


def _shapes(case):
    rng = random.Random(case["shapes_seed"])
    return [(rng.randint(case["low"], case["high"]), rng.randint(case["low"], case["high"]))
            for _ in range(case["instances"])]


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _sqdist(x, y):
    """[n, m] squared distances of x (m points) and y (n points), in FP64."""
    x, y = x.double(), y.double()
    return ((y * y).sum(1, keepdim=True) + (x * x).sum(1)[None, :] - 2.0 * (y @ x.T)).clamp_min_(0)


def _cloud_cost(g, m, n, dim):
    c = _sqdist(torch.randn(m, dim, generator=g, device="cuda"),
                torch.randn(n, dim, generator=g, device="cuda"))
    return (c / c.max()).float()


def _uniform(k):
    return torch.full((k,), 1.0 / k, device="cuda")


def _dirichlet(g, k):
    """Dirichlet(1): normalised exponentials."""
    e = -torch.log(1.0 - torch.rand(k, generator=g, device="cuda", dtype=torch.float64))
    return (e / e.sum()).float()


def _two_domains(g, m, n, classes, dim=2):
    """Source clouds of ``classes`` Gaussians in row order and targets under a random affine
    map; their normalised cost [n, m]."""
    def cloud(k, label):
        t = torch.randn(k, dim, generator=g, device="cuda")
        angle = label.float() * (2.0 * math.pi / classes)
        t[:, 0] += 2.0 * torch.cos(angle)
        t[:, 1] += 2.0 * torch.sin(angle)
        return t
    xs = cloud(m, torch.arange(m, device="cuda") * classes // m)
    xt = cloud(n, torch.randint(classes, (n,), generator=g, device="cuda"))
    a = torch.eye(dim, device="cuda") + 0.3 * torch.randn(dim, dim, generator=g, device="cuda")
    c = _sqdist(xs, xt @ a.T + torch.randn(dim, generator=g, device="cuda"))
    return (c / c.max()).float()


def prepare(case, seed):
    g = _gen(seed)
    s = dict(case)
    kind = case["kind"]
    if kind == "qr":
        m, n = case["rows"], case["cols"]
        if case["cost"] == "clouds":
            s["c"], s["p"], s["q"] = _cloud_cost(g, m, n, 2), _uniform(m), _uniform(n)
        else:
            s["c"] = torch.rand(n, m, generator=g, device="cuda")
            s["p"], s["q"] = _dirichlet(g, m), _dirichlet(g, n)
        if case["dtype"] == "bfloat16":
            s["c"] = s["c"].bfloat16()
    elif kind == "gl":
        m, n = case["rows"], case["cols"]
        s["c"] = _two_domains(g, m, n, case["classes"])
        s["p"], s["q"] = _uniform(m), _uniform(n)
        s["r_weight"] = _gl_weight(case)
    elif kind == "qr_batch":
        shapes = _shapes(case)
        s["batch"] = QRBatch(shapes, RHO, case["alpha"], NEVER, cols_per_tile=256)
        s["c"] = s["batch"].pack_c([_cloud_cost(g, m, n, case["dim"]) for m, n in shapes],
                                   getattr(torch, case["dtype"]))
        s["p"], s["q"] = s["batch"].pack_marginals([_uniform(m) for m, _ in shapes],
                                                   [_uniform(n) for _, n in shapes])
    elif kind == "qr_diff":
        shapes = _shapes(case)
        s["batch"] = QRBatch(shapes, RHO, case["alpha"], NEVER, cols_per_tile=256)
        s["x"], s["y"] = (torch.randn(sum(t[k] for t in shapes), case["dim"], generator=g,
                                      device="cuda", requires_grad=True) for k in (0, 1))
        s["p"], s["q"] = s["batch"].pack_marginals([_uniform(m) for m, _ in shapes],
                                                   [_uniform(n) for _, n in shapes])
        s["scale"] = 1.0 / (4.0 * case["dim"])
        s["w"] = 0.5
    elif kind == "gl_batch":
        shapes = _shapes(case)
        s["batch"] = GLBatch(shapes, case["classes"], RHO, case["weight"], NEVER,
                             cols_per_tile=256, convention="wrapper")
        s["c"] = s["batch"].pack_c([_two_domains(g, m, n, case["classes"]) for m, n in shapes])
        s["p"], s["q"] = s["batch"].pack_marginals([_uniform(m) for m, _ in shapes],
                                                   [_uniform(n) for _, n in shapes])
    else:
        s["x"] = torch.randn(case["rows"], case["dim"], generator=g, device="cuda",
                             requires_grad=True)
        s["y"] = torch.randn(case["cols"], case["dim"], generator=g, device="cuda",
                             requires_grad=True)
        s["up"] = torch.randn(case["cols"], case["rows"], generator=g, device="cuda")
    return s


def _gl_weight(case):
    """The weight whose operator threshold r sqrt(m // G) is weight / sqrt(m // G), the C++
    wrapper's."""
    return case["weight"] / (case["rows"] // case["classes"])


# --------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "qr":
        if s["dtype"] == "bfloat16":
            return reg_drot.solve_qr(s["c"], s["p"], s["q"], RHO, s["alpha"], s["iters"],
                                     s["eps"])[0]
        return reg_drot.quadratic_drot(s["c"], s["p"], s["q"], RHO, s["alpha"], s["iters"],
                                       s["eps"])
    if kind == "gl":
        return reg_drot.group_lasso_drot(s["c"], s["p"], s["q"], s["classes"], RHO,
                                         s["r_weight"], s["iters"], s["eps"])
    if kind in ("qr_batch", "gl_batch"):
        x, _ = s["batch"].solve(s["c"], s["p"], s["q"], s["iters"])
        return s["batch"].unpack(x)
    if kind == "qr_diff":
        b = s["batch"]
        c = packed_sqeuclidean_cost(b, s["x"], s["y"], s["scale"])
        x = batch_quadratic_drot_fn(b, c, s["p"], s["q"], s["iters"])
        plans, costs = b.unpack(x), b.unpack(c)
        loss = sum((ck * xk).sum() + s["w"] * (xk * xk).sum() for ck, xk in zip(costs, plans))
        gx, gy = torch.autograd.grad(loss, (s["x"], s["y"]))
        return {"loss": loss.detach(), "plans": [t.detach() for t in plans], "gx": gx, "gy": gy}
    c = sqeuclidean_cost(s["x"], s["y"], 1.0 / (4.0 * s["dim"]))
    gx, gy = torch.autograd.grad(c, (s["x"], s["y"]), s["up"])
    return {"c": c.detach(), "gx": gx, "gy": gy}


# --------------------------------------------------------------------------- work
_QR_FLOPS = 9   # per element and iteration: 3 adds, prox, divide, fold (half), 2 partial sums
_GL_FLOPS = 12  # the shrink and the group norm beside them


def work(case):
    kind = case["kind"]
    if kind in ("qr", "gl"):
        e = case["rows"] * case["cols"]
        iters = min(case["iters"], 500) if case["eps"] > NEVER else case["iters"]
        cb = 2 if case.get("dtype") == "bfloat16" else 4
        return {"bytes": e * (cb + 4), "flops": e * iters * (_QR_FLOPS if kind == "qr"
                                                             else _GL_FLOPS)}
    if kind == "cost":
        e = case["rows"] * case["cols"]
        # C written, its upstream gradient read; the Gram product and its two transposes
        return {"bytes": e * 8, "flops": e * 6 * case["dim"]}
    e = sum(m * n for m, n in _shapes(case))
    if kind == "qr_batch":
        cb = 2 if case["dtype"] == "bfloat16" else 4
        return {"bytes": e * (cb + 4), "flops": e * case["iters"] * _QR_FLOPS}
    if kind == "qr_diff":
        return {"bytes": e * 8, "flops": e * (case["iters"] * _QR_FLOPS + 6 * case["dim"])}
    return {"bytes": e * 8, "flops": e * case["iters"] * _GL_FLOPS}


# --------------------------------------------------------------------------- 64 bits
f32 = np.float32


def _step(m, n):
    return f32(RHO) / (f32(m) + f32(n))


def _warm(s, m, n):
    """The warm start's five constants, as the operators set them in 32 bits."""
    k = f32(f32(s * f32(m)) * f32(n)) - f32(2)
    t1, t2 = f32(k + f32(2)) / f32(m), f32(k + f32(2)) / f32(n)
    d = f32(n) + f32(m)
    return [float(v) for v in (t1 / d, t2 / d, f32(k + f32(1)) / f32(m),
                               f32(k + f32(1)) / f32(n), f32(k + f32(1)))]


class _Loop:
    """The iteration in 64 bits, as torch states it (cost [n, m], a plan of the same shape)."""

    def __init__(self, c, p, q):
        self.c, self.p, self.q = c.double(), p.double(), q.double()
        self.n, self.m = c.shape
        self.s = float(_step(self.m, self.n))
        v = _warm(_step(self.m, self.n), self.m, self.n)
        full = lambda k, t: torch.full((k,), t, dtype=torch.float64, device=c.device)  # noqa: E731
        self.x = torch.zeros_like(self.c)
        self.f1, self.f2 = full(self.m, v[0]), full(self.n, v[1])
        self.a, self.b = full(self.m, v[2]), full(self.n, v[3])
        self.alpha = full(1, v[4])

    def duals(self):
        x, m, n = self.x, self.m, self.n
        r, k = x.sum(0) - self.p, x.sum(1) - self.q
        total = x.sum()
        gamma = (2.0 * (total - 1.0) - self.alpha) / (m + n)
        self.a = self.a - r
        self.b = self.b - k
        self.f1 = ((self.a - r) + gamma) / n
        self.f2 = ((self.b - k) + gamma) / m
        self.alpha = self.alpha + 1.0 - total
        return (r * r).sum() + (k * k).sum()

    def ahead(self):
        t = self.x.add_(self.f1[None, :]).add_(self.f2[:, None])
        return t.add_(self.c, alpha=-self.s).clamp_min_(0.0)


def _qr_kappa(case, m, n):
    t = f32(_step(m, n) * f32(case["alpha"]))
    return float(f32(f32(1.0) + f32(t * f32(m + n))))


def _qr64(c, p, q, case):
    lp = _Loop(c, p, q)
    kappa = _qr_kappa(case, lp.m, lp.n)
    for it in range(case["iters"]):
        lp.x = lp.ahead().div_(kappa)
        res2 = lp.duals()
        # the residual is tested on every other iteration
        if it % 2 == 0 and case.get("eps", 0.0) > NEVER and \
                math.sqrt(float(res2)) < case["eps"]:
            break
    return lp


def _gl_bounds(m, classes):
    off = 0.49 if (m + classes - 1) // classes <= 256 else 0.49999
    per = f32(m) / f32(classes)
    return [int(float(per * f32(k)) + off) for k in range(classes + 1)]


def _gl64(lp, bounds, lam, iters):
    for _ in range(iters):
        y = lp.ahead()
        for lo, hi in zip(bounds, bounds[1:]):
            t = y[:, lo:hi]
            norm = t.square().sum(1, keepdim=True).sqrt_()
            t.mul_((1.0 - lam / (norm + 1e-9)).clamp_min_(0.0))
        lp.x = y
        lp.duals()
    return lp


def _mask_cg(mask, g, lam):
    """dL/dC through the plan for upstream g on the support mask ([n, m], 64 bits): the masked
    Laplacian's solution by conjugate gradients."""
    w = mask.double()
    dr, dc = w.sum(0), w.sum(1)
    gm = g * w
    rhs = torch.cat([gm.sum(0), gm.sum(1)])
    m = dr.numel()
    diag = torch.cat([dr, dc]).clamp_min(1.0)

    def mul(z):
        return torch.cat([dr * z[:m] + z[m:] @ w, dc * z[m:] + w @ z[:m]])
    z = torch.zeros_like(rhs)
    r = rhs.clone()
    y = r / diag
    d = y.clone()
    ry, r0 = r @ y, rhs.norm()
    for it in range(4000):
        t = mul(d)
        step = ry / (d @ t)
        z += step * d
        r -= step * t
        if it % 16 == 15 and float(r.norm()) < 1e-12 * float(r0):
            break
        y = r / diag
        new = r @ y
        d = y + (new / ry) * d
        ry = new
    return torch.where(mask, (z[:m][None, :] + z[m:][:, None] - g) / lam, torch.zeros_like(g))


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind == "qr":
        return _qr64(s["c"], s["p"], s["q"], case).x
    if kind == "gl":
        m = case["rows"]
        lam = float(f32(float(f32(s["r_weight"])) * math.sqrt(m // case["classes"])))
        return _gl64(_Loop(s["c"], s["p"], s["q"]), _gl_bounds(m, case["classes"]), lam,
                     case["iters"]).x
    if kind == "cost":
        x, y = (s[k].detach().double().requires_grad_(True) for k in ("x", "y"))
        c = torch.relu((y * y).sum(1, keepdim=True) + (x * x).sum(1)[None, :]
                       - 2.0 * (y @ x.T)) / (4.0 * case["dim"])
        gx, gy = torch.autograd.grad(c, (x, y), s["up"].double())
        return {"c": c.detach(), "gx": gx, "gy": gy}
    shapes = _shapes(case)
    if kind == "qr_batch":
        return [_qr64(c, s["p"][i:i + m], s["q"][j:j + n], case).x
                for c, (m, n), i, j in _each(s, shapes, s["batch"].unpack(s["c"]))]
    if kind == "qr_diff":
        loss, plans, gx, gy = 0.0, [], [], []
        for _, (m, n), i, j in _each(s, shapes, shapes):
            x, y = (s[k].detach()[o:o + t].double().requires_grad_(True)
                    for k, o, t in (("x", i, m), ("y", j, n)))
            c = torch.relu((y * y).sum(1, keepdim=True) + (x * x).sum(1)[None, :]
                           - 2.0 * (y @ x.T)) * s["scale"]
            cd = c.detach()
            lp = _qr64(cd, s["p"][i:i + m], s["q"][j:j + n], case)
            up = cd + 2.0 * s["w"] * lp.x
            mask = (lp.f1[None, :] + lp.f2[:, None] - lp.s * cd) > 0
            gc = lp.x + _mask_cg(mask, up, (_qr_kappa(case, m, n) - 1.0) / lp.s)
            a, b = torch.autograd.grad(c, (x, y), gc)
            gx.append(a)
            gy.append(b)
            loss = loss + (cd * lp.x).sum() + s["w"] * (lp.x * lp.x).sum()
            plans.append(lp.x)
        return {"loss": loss, "plans": plans, "gx": torch.cat(gx), "gy": torch.cat(gy)}
    plans = []
    for c, (m, n), i, j in _each(s, shapes, s["batch"].unpack(s["c"])):
        lam = float(f32(float(f32(case["weight"])) / math.sqrt(m // case["classes"])))
        plans.append(_gl64(_Loop(c, s["p"][i:i + m], s["q"][j:j + n]),
                           _gl_bounds(m, case["classes"]), lam, case["iters"]).x)
    return plans


def _each(s, shapes, things):
    i = j = 0
    for t, (m, n) in zip(things, shapes):
        yield t, (m, n), i, j
        i += m
        j += n
