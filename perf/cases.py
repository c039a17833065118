"""The performance cases of the inpainting framework: what a program that uses
it has it do, through the Python front end (`Context` and `autograd`).

Most cases are single layers of the path -- a PatchMatch call, an image
update, an update with its gradients -- because those are entry points of
their own and the multiscale driver is a sequence of them; three are whole
calls (one image, the flagship configuration, and a batch).  Sizes come from
the workloads of `workloads.py` and bench.py: the 256x256 NL-means, 512x512
NL-Poisson and 640x480 NL-depth configurations, the uneven batch (sides up to
1024) and the sizes that their pyramids pass through.

Images are piecewise-smooth Voronoi textures with oriented sinusoids, holes
unions of ellipses or brush strokes, as in `workloads.py` (built on the GPU
here where the numpy generators are slow).  The hole of a layer's image is
filled by the framework's own Poisson initialisation and its field found by a
short PatchMatch call, as the driver hands them to the layer.
"""
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.package()
from nli_gb300 import workloads  # noqa: E402
from nli_gb300.autograd import image_update  # noqa: E402

DISTANCES = {"l2combined": 0, "l2rgbd": 1, "l2": 2, "l1": 3}
FLOPS_PER_TAP = {"l2combined": lambda c: 10 * c + 1, "l2rgbd": lambda c: 44, "l2": lambda c: 3 * c, "l1": lambda c: 3 * c}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a coarse pyramid level: the smallest calls, where launches and latency count
        {"name": "pm-64x48", "kind": "pm", "w": 64, "h": 48, "c": 3, "dist": "l2combined", "patch": 9, "hole": 0.10},
        # the finest level of the flagship configuration
        {"name": "pm-512x512", "kind": "pm", "w": 512, "h": 512, "c": 3, "dist": "l2combined", "patch": 9, "hole": 0.15},
        # colour and depth together, brush strokes (640x480 RGB-D configuration)
        {"name": "pm-rgbd-640x480", "kind": "pm", "w": 640, "h": 480, "c": 4, "dist": "l2rgbd", "patch": 9, "hole": 0.12,
         "strokes": True},
        # another patch size and the plain L2 distance, a ragged size of the batch
        {"name": "pm-425x283-p7-l2", "kind": "pm", "w": 425, "h": 283, "c": 3, "dist": "l2", "patch": 7, "hole": 0.20},
        # the largest images of the batch, a ragged size
        {"name": "pm-1013x887", "kind": "pm", "w": 1013, "h": 887, "c": 3, "dist": "l2combined", "patch": 9, "hole": 0.25},
        # weighted medians, the command line's third update
        {"name": "medians-382x388", "kind": "update", "method": "nlmedians", "w": 382, "h": 388, "c": 3, "patch": 9,
         "hole": 0.15},
        # one NL-Poisson step at the flagship's finest level
        {"name": "poisson-512x512", "kind": "update", "method": "nlpoisson", "w": 512, "h": 512, "c": 3, "patch": 9,
         "hole": 0.15, "cg_tol": 1e-4},
        # a large NL-Poisson system: more unknowns than one thread-block cluster holds
        {"name": "poisson-1024x685", "kind": "update", "method": "nlpoisson", "w": 1024, "h": 685, "c": 3, "patch": 9,
         "hole": 0.25, "cg_tol": 1e-6},
        # the differentiation workload: a step and its gradients to the image, lambda and sigma
        {"name": "grad-poisson-512x512", "kind": "grad", "method": "nlpoisson", "w": 512, "h": 512, "c": 3, "patch": 9,
         "hole": 0.15, "cg_tol": 1e-12},
        # whole calls: the 256x256 NL-means configuration ...
        {"name": "process-means-256x256", "kind": "process", "method": "nlmeans", "w": 256, "h": 256, "c": 3, "hole": 0.05,
         "scales": 5, "coarse": 0.1},
        # ... the flagship: 512x512 NL-Poisson, eight scales ...
        {"name": "process-poisson-512x512", "kind": "process", "method": "nlpoisson", "w": 512, "h": 512, "c": 3,
         "hole": 0.15, "scales": 8, "coarse": 0.1, "cg_tol": 1e-4},
        # ... and a batch of small uneven images, NL-means and NL-Poisson alternating
        {"name": "batch-8x64-160", "kind": "batch", "count": 8, "low": 64, "high": 160, "hole": 0.10},
    ]


def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _sides(rng, low, high):
    side, aspect = _log(rng, low, high), _log(rng, 0.5, 2.0)
    w, h = (int(round(min(high, max(48, side * f)))) for f in (math.sqrt(aspect), 1 / math.sqrt(aspect)))
    return w, h


def draw(rng):
    kind = rng.choice(["pm", "pm", "pm", "update", "update", "update", "grad", "process", "process", "batch"])
    hole = round(rng.uniform(0.05, 0.25), 3)
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 8), "low": 64, "high": rng.randint(80, 160),
                "hole": round(rng.uniform(0.05, 0.12), 3)}
    if kind == "process":
        method = rng.choice(["nlmeans", "nlmedians", "nlpoisson", "nldepth"])
        w, h = _sides(rng, 96, 320)
        coarse = round(min(0.9, 64.0 / min(w, h)), 4)
        return {"kind": kind, "method": method, "w": w, "h": h, "c": 4 if method == "nldepth" else 3,
                "hole": round(rng.uniform(0.05, 0.12), 3), "scales": max(2, round(math.log(coarse) / math.log(0.75)) + 1),
                "coarse": coarse, "cg_tol": rng.choice([1e-4, 1e-6]), "strokes": rng.random() < 0.5}
    w, h = _sides(rng, 56, 1000)
    if kind == "pm":
        dist = rng.choice(["l2combined", "l2combined", "l2combined", "l2rgbd", "l2", "l1"])
        c = 4 if dist == "l2rgbd" else rng.choice([3, 3, 3, 1])
        return {"kind": kind, "w": w, "h": h, "c": c, "dist": dist, "patch": rng.choice([9, 9, 9, 7, 5]), "hole": hole,
                "strokes": rng.random() < 0.5}
    method = rng.choice(["nlmeans", "nlpoisson"] if kind == "grad" else ["nlmeans", "nlmedians", "nlpoisson", "nldepth"])
    return {"kind": kind, "method": method, "w": w, "h": h, "c": 4 if method == "nldepth" else 3,
            "patch": rng.choice([9, 9, 7]), "hole": hole, "cg_tol": 1e-12 if kind == "grad" else rng.choice([1e-4, 1e-6]),
            "strokes": rng.random() < 0.5}


# ----------------------------------------------------------------- inputs
_ctx = None


def context():
    """The one context a program keeps for all its calls."""
    global _ctx
    if _ctx is None:
        _ctx = pkg.Context(0)
    return _ctx


def _texture(w, h, cells, gen):
    """Voronoi cells of a uniform colour with an oriented sinusoid each, in [0, 255]."""
    def uniform(a, b, *shape):
        return a + (b - a) * torch.rand(*shape, generator=gen, device="cuda")
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    sx, sy = uniform(0, w, cells), uniform(0, h, cells)
    colour, theta = uniform(0, 255, cells, 3), uniform(0, math.pi, cells)
    period, amp = uniform(6, 20, cells), uniform(8, 30, cells)
    label = ((x[..., None] - sx) ** 2 + (y[..., None] - sy) ** 2).argmin(-1)
    phase = x * torch.cos(theta)[label] + y * torch.sin(theta)[label]
    texture = amp[label] * torch.sin(2 * math.pi * phase / period[label])
    return (colour[label] + texture[..., None]).clamp(0, 255).contiguous()


def _ellipses(w, h, count, coverage, gen):
    """Union of `count` ellipses of random centres, axes and angles, scaled
    together to cover `coverage` of the pixels."""
    r = torch.rand(count, 5, generator=gen, device="cuda")
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    dx = x[..., None] - w * (0.12 + 0.76 * r[:, 0])
    dy = y[..., None] - h * (0.12 + 0.76 * r[:, 1])
    ax, ay, th = 0.5 + r[:, 2], 0.5 + r[:, 3], math.pi * r[:, 4]
    u = (dx * torch.cos(th) + dy * torch.sin(th)) / ax
    v = (-dx * torch.sin(th) + dy * torch.cos(th)) / ay
    q = (u * u + v * v).amin(-1).reshape(-1)
    k = max(1, int(coverage * w * h))
    return (q <= q.kthvalue(k).values).reshape(h, w).to(torch.uint8)


def _image(case, seed, w, h, c):
    """(image, mask) of one input: RGB, one channel, or RGB and depth."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    img = _texture(w, h, 40, gen)
    if c == 1:
        img = img[..., :1].contiguous()
    if c == 4:
        depth = workloads.depth_planes(w, h, 60, np.random.default_rng(seed))
        img = torch.cat([img, torch.from_numpy(depth).cuda()[..., None]], -1).contiguous()
    if case.get("strokes"):
        width = (8, 24) if min(w, h) >= 200 else (4, 8)
        mask = workloads.stroke_mask(w, h, 10, width, np.random.default_rng(seed + 1), coverage=case["hole"])
        mask = torch.from_numpy(mask).cuda()
    else:
        mask = _ellipses(w, h, 6 if min(w, h) >= 200 else 2, case["hole"], gen)
    return img, mask


def _masks(ctx, mask, patch):
    """The domain a layer works on, as the driver builds it at one scale."""
    ext = ctx.extended_domain(mask, patch, patch)
    src, tgt, _ = ctx.scale_masks(ext, patch // 2, True)
    return ext, src, tgt


def _params(case, method):
    depth = method == "nldepth"
    return workloads.params(method, patch=case.get("patch", 9), scales=case.get("scales", 1),
                            coarse=case.get("coarse", 0.5), cg_tol=case.get("cg_tol", 1e-4),
                            lam_r=1.0 if depth else 0.05, lam_d=0.0 if depth else 0.05)


def prepare(case, seed):
    ctx = context()
    s = {"ctx": ctx, "kind": case["kind"], "seed": seed}
    if case["kind"] == "batch":
        rng = np.random.default_rng(case["count"])  # the sizes belong to the case, the images to the seed
        s["items"], s["params"] = [], []
        for i in range(case["count"]):
            side = math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"])))
            aspect = math.exp(rng.uniform(math.log(0.7), math.log(1.4)))
            w, h = max(48, int(round(side * math.sqrt(aspect)))), max(48, int(round(side / math.sqrt(aspect))))
            s["items"].append(_image(case, seed * 64 + i, w, h, 3))
            coarse = min(0.8, 56.0 / min(w, h))
            s["params"].append(workloads.params("nlmeans" if i % 2 == 0 else "nlpoisson", coarse=coarse, cg_tol=1e-4,
                                                scales=max(2, round(math.log(coarse) / math.log(0.75)) + 1)))
        return s
    w, h, c = case["w"], case["h"], case["c"]
    img, mask = _image(case, seed, w, h, c)
    if case["kind"] == "process":
        s.update(img=img, mask=mask, p=_params(case, case["method"]))
        return s
    method = case.get("method", "nlpoisson")
    p = _params(case, method)
    if case["kind"] == "pm":
        p.distance.kind = DISTANCES[case["dist"]]
        p.distance.lambda_ = 1.0 if case["dist"] == "l2rgbd" else 0.05
        p.distance.lambda_d = 0.0 if case["dist"] == "l2rgbd" else 0.05
    ext, src, tgt = _masks(ctx, mask, case["patch"])
    u = ctx.poisson_init(img, mask)
    s.update(p=p, u=u, src=src, tgt=tgt, mask=mask, ext=ext)
    if case["kind"] == "pm":
        return s
    # the field the layer starts from: three sweeps, as after a few iterations
    few = pkg.PatchMatchParams(3, 30, -1)
    ctx.set_seed(seed)
    s["nnf"] = ctx.patchmatch(p.distance, few, u, src, u, tgt)[0]
    s["conf"] = ctx.confidence_mask(mask, 5.0, 0.1)
    if case["kind"] == "grad":
        s["g"] = torch.randn(u.shape, generator=torch.Generator(device="cuda").manual_seed(seed + 3), device="cuda")
        s["lam"] = torch.tensor(0.05, requires_grad=True)
        s["sigma"] = torch.tensor(3.0, requires_grad=True)
        s["u"] = u.requires_grad_(True)
    return s


# -------------------------------------------------------------- one pass
def run(s):
    ctx = s["ctx"]
    if s["kind"] == "pm":
        ctx.set_seed(s["seed"])
        nnf, dist, energy = ctx.patchmatch(s["p"].distance, s["p"].patchmatch, s["u"], s["src"], s["u"], s["tgt"])
        return {"nnf": nnf, "dist": dist, "energy": energy}
    if s["kind"] == "update":
        out, total = ctx.update(s["p"].update, s["u"], s["u"], s["mask"], s["ext"], s["nnf"], s["conf"])
        return {"out": out, "total": total}
    if s["kind"] == "grad":
        out = image_update(ctx, s["p"].update, s["u"], s["lam"], s["sigma"], s["mask"], s["ext"], s["nnf"], s["conf"])
        gu, gl, gs = torch.autograd.grad(out, (s["u"], s["lam"], s["sigma"]), s["g"])
        return {"out": out.detach(), "grad_u": gu, "grad_lambda": gl, "grad_sigma": gs}
    ctx.set_seed(s["seed"])
    if s["kind"] == "process":
        out, stats = ctx.process_device(s["img"], s["mask"], s["p"])
        return {"out": out, "iterations": [int(i) for i in stats["iterations"]]}
    outs, stats = ctx.process_batch_device(s["items"], s["params"])
    return {"out": outs, "iterations": [int(i) for st in stats for i in st["iterations"]]}


# ------------------------------------------------------------------ work
def _pm_flops(case, w, h, targets):
    """Candidates of one call (the initial match, then per sweep two
    propagations and one draw per search window) times the distance."""
    windows = max(w, h).bit_length()
    taps = case.get("patch", 9) ** 2
    return targets * (1 + 10 * (2 + windows)) * taps * FLOPS_PER_TAP[case.get("dist", "l2combined")](case.get("c", 3))


def _update_flops(case, holes, c, method):
    taps = case.get("patch", 9) ** 2
    if method in ("nlmeans", "nlmedians"):
        return holes * taps * (2 * c + 1)
    # coefficients (value and two differences per tap), then CG: the
    # reference's runs take about 100 iterations a solve at these tolerances
    return holes * c * (taps * 6 + 100 * 20)


def work(case):
    if case["kind"] == "batch":
        side = math.sqrt(case["low"] * case["high"])
        one = {"kind": "process", "method": "nlpoisson", "w": int(side), "h": int(side), "c": 3, "hole": case["hole"],
               "scales": 3, "coarse": 56.0 / side}
        v = work(one)
        return {k: case["count"] * x for k, x in v.items()}
    w, h, c = case["w"], case["h"], case["c"]
    n = w * h
    holes = case["hole"] * n
    targets = 1.3 * holes  # with the band of patches that touch the hole
    if case["kind"] == "pm":
        return {"bytes": n * (4 * c + 2 + 8 + 4), "flops": _pm_flops(case, w, h, targets)}
    if case["kind"] in ("update", "grad"):
        method = case["method"]
        b = n * (4 * c * 2 + 2 + 8 + 4)  # image in and out, masks, field, confidence
        f = _update_flops(case, holes, c, method)
        return {"bytes": b, "flops": f} if case["kind"] == "update" else {"bytes": b + n * 8 * c, "flops": 3 * f}
    # one image in and out; per scale the iterations that such runs take on
    # average (about 60 in all of a level's 200 at most)
    flops, rate = 0.0, case["coarse"] ** (2.0 / max(1, case["scales"] - 1))
    for k in range(case["scales"]):
        a = rate ** k
        flops += 60 * (_pm_flops(case, w, h, targets * a) + _update_flops(case, holes * a, c, case["method"]))
    return {"bytes": n * (8 * c + 1), "flops": flops}


# ----------------------------------------------------------------- exact
def _weights64(sigma, patch):
    r = torch.arange(patch, dtype=torch.float64, device="cuda") - patch // 2
    e = torch.exp(-(r[:, None] ** 2 + r[None, :] ** 2) / (2 * sigma * sigma))
    return e / e.sum()


def _shifted(t, dx, dy, fill=0):
    """t at (x + dx, y + dy), `fill` outside the image."""
    h, w = t.shape[:2]
    out = torch.full_like(t, fill)
    y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
    if y0 < y1 and x0 < x1:
        out[y0:y1, x0:x1] = t[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
    return out


def _taps(s, patch):
    """Per window offset (dx, dy): the centre pixels' matches shifted to this
    pixel, as a flat source index, and whether there is one."""
    h, w = s["mask"].shape
    nnf = s["nnf"].long()
    for dy in range(-(patch // 2), patch // 2 + 1):
        for dx in range(-(patch // 2), patch // 2 + 1):
            q = _shifted(nnf, dx, dy, -1)
            has = _shifted(torch.ones_like(s["mask"]), dx, dy).bool()
            x, y = q[..., 0] - dx, q[..., 1] - dy
            ok = has & (x >= 0) & (y >= 0) & (x < w) & (y < h)
            yield dx, dy, q, ok, (y.clamp(0, h - 1) * w + x.clamp(0, w - 1))


def _means64(s, u, sigma, patch):
    """NL-means of the hole pixels: matches of the window's pixels, weights
    counted from the window's first pixel inside the image."""
    h, w, c = u.shape
    g, dom, conf = _weights64(sigma, patch), s["mask"].bool(), s["conf"].double()
    flat, r = u.reshape(-1, c), patch // 2
    xa = (torch.arange(w, device="cuda") - r).clamp(min=0)[None, :]
    ya = (torch.arange(h, device="cuda") - r).clamp(min=0)[:, None]
    x, y = torch.arange(w, device="cuda")[None, :], torch.arange(h, device="cuda")[:, None]
    num, den = torch.zeros_like(u), torch.zeros(h, w, dtype=u.dtype, device="cuda")
    for dx, dy, q, ok, at in _taps(s, patch):
        ok = ok & (q[..., 0] != -1)
        k = ((y + dy - ya) * patch + (x + dx - xa)).clamp(0, patch * patch - 1)
        wt = g.reshape(-1)[k] * torch.where(_shifted(dom, dx, dy), _shifted(conf, dx, dy), torch.ones_like(conf))
        wt = torch.where(ok, wt, torch.zeros_like(wt))
        den = den + wt
        num = num + wt[..., None] * flat[at]
    new = dom & (den > 0)
    return torch.where(new[..., None], num / torch.where(new, den, torch.ones_like(den))[..., None], u)


def _poisson64_system(s, u, lam, sigma, patch):
    """(b, diag, links) of the hole's system: links as (dx, dy, coefficient),
    everything on the image grid."""
    h, w, c = u.shape
    g, conf = _weights64(sigma, patch), s["conf"].double()
    ext = s["ext"].bool()
    gx = torch.cat([u[:, 1:] - u[:, :-1], torch.zeros_like(u[:, :1])], 1)
    gy = torch.cat([u[1:] - u[:-1], torch.zeros_like(u[:1])], 0)
    both = torch.cat([u, gx, gy], -1).reshape(h * w, 3 * c)
    S, F = torch.zeros(h, w, dtype=u.dtype, device="cuda"), torch.zeros(h, w, 3 * c, dtype=u.dtype, device="cuda")
    r = patch // 2
    for dx, dy, q, ok, at in _taps(s, patch):
        ok = ok & _shifted(ext, dx, dy)  # the tap's offset from its centre is (-dx, -dy)
        wt = torch.where(ok, g[r - dy, r - dx] * _shifted(conf, dx, dy), torch.zeros_like(S))
        S = S + wt
        F = F + wt[..., None] * both[at]
    U, GX, GY = F.split(c, -1)

    def before(t, dx, dy):  # t at (x + dx, y + dy), differentiable
        if dx:
            return torch.cat([torch.zeros_like(t[:, :1]), t[:, :-1]], 1) if dx < 0 else \
                torch.cat([t[:, 1:], torch.zeros_like(t[:, :1])], 1)
        return torch.cat([torch.zeros_like(t[:1]), t[:-1]], 0) if dy < 0 else \
            torch.cat([t[1:], torch.zeros_like(t[:1])], 0)

    x, y = torch.arange(w, device="cuda")[None, :], torch.arange(h, device="cuda")[:, None]
    right, down = (x != w - 1).expand(h, w), (y != h - 1).expand(h, w)
    zero = torch.zeros_like(S)
    links = [(-1, 0, before(S, -1, 0)), (0, -1, before(S, 0, -1)),
             (1, 0, torch.where(right, S, zero)), (0, 1, torch.where(down, S, zero))]
    div = torch.where(right[..., None], GX, torch.zeros_like(GX)) - before(GX, -1, 0) + \
        torch.where(down[..., None], GY, torch.zeros_like(GY)) - before(GY, 0, -1)
    b = lam * U - (1 - lam) * div - lam * S[..., None] * u
    for dx, dy, k in links:
        b = b + (1 - lam) * k[..., None] * (before(u, dx, dy) - u)
    return b, S, links, before


def _apply64(S, links, before, lam, hole, v):
    q = lam * S[..., None] * v
    for dx, dy, k in links:
        q = q - (1 - lam) * k[..., None] * (before(v, dx, dy) - v)
    return torch.where(hole, q, torch.zeros_like(q))


def _cg64(S, links, before, lam, hole, b, tol, limit):
    """The reference's conjugate gradient from zero, all channels at once,
    each until |r|^2 < tol |r0|^2."""
    def dot(a, c):
        return (a * c).sum((0, 1))
    x, r = torch.zeros_like(b), torch.where(hole, b, torch.zeros_like(b))
    d, rr = r.clone(), dot(r, r)
    r0, on, it = rr.clone(), rr > 0, 0
    while bool(on.any()):
        q = _apply64(S, links, before, lam, hole, d)
        a = torch.where(on, rr / dot(d, q).clamp(min=1e-300), torch.zeros_like(rr))
        x, r = x + a * d, r - a * q
        new = torch.where(on, dot(r, r), rr)
        d = torch.where(on, r + (new / rr.clamp(min=1e-300)) * d, d)
        rr = new
        on = on & ~((rr < tol * r0) | (it >= limit))
        it += 1
    return x


def exact(case, seed):
    if case["kind"] not in ("update", "grad") or case["method"] == "nlmedians":
        # the fields of a randomised search, and whole runs, have no value of
        # their own; the weighted median is one of its inputs
        return None
    with torch.no_grad():
        s = prepare(case, seed)
    u, patch = s["u"].detach().double(), case["patch"]
    hole = s["mask"].bool()[..., None]
    up = s["p"].update
    if case["kind"] == "update":
        if case["method"] == "nlmeans":
            out = _means64(s, u, float(up.sigma), patch)
        else:
            lam = torch.full((case["c"],), float(up.lambda_), dtype=torch.float64, device="cuda")
            if case["method"] == "nldepth":
                lam[3] = float(up.lambda_d)
            b, S, links, before = _poisson64_system(s, u, lam, float(up.sigma), patch)
            out = u + _cg64(S, links, before, lam, hole, b, float(up.cg_tol), int(up.cg_iters))
        d = torch.where(hole, out - u, torch.zeros_like(u))
        return {"out": out, "total": (d * d).sum()}
    # the gradient case: the same step, differentiated through its system
    u.requires_grad_(True)
    lam, sigma = (s[k].detach().double().cuda().requires_grad_(True) for k in ("lam", "sigma"))
    g = s["g"].double()
    if case["method"] == "nlmeans":
        out = _means64(s, u, sigma, patch)
        gu, gs = torch.autograd.grad(out, (u, sigma), g)
        return {"out": out.detach(), "grad_u": gu, "grad_lambda": torch.zeros((), dtype=torch.float64), "grad_sigma": gs}
    b, S, links, before = _poisson64_system(s, u, lam, sigma, patch)
    with torch.no_grad():
        delta = _cg64(S, links, before, lam, hole, b, 1e-24, 20000)
        z = _cg64(S, links, before, lam, hole, torch.where(hole, g, torch.zeros_like(g)), 1e-24, 20000)
    out = u + delta
    residual = (z * (b - _apply64(S, links, before, lam, hole, delta))).sum()
    gu, gl, gs = torch.autograd.grad((out * g).sum() + residual, (u, lam, sigma))
    return {"out": out.detach(), "grad_u": gu, "grad_lambda": gl, "grad_sigma": gs}
