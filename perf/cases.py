"""The work that users of this package have it do, as cases to measure.

A case names an entry point (``op``), a scan geometry, a data type and a batch:

* ``pair``       ``autograd.Projector`` forward, then its backward pass (A, A^T): a training step's share;
* ``bpair``      ``autograd.Backprojector`` forward and backward (B, B^T);
* ``gradient``   ``ops.data_gradient``: one iteration of a reconstruction without autograd;
* ``fidelity``   ``autograd.data_fidelity`` and the gradient of its loss;
* ``fbp``        ``fbp``: filtered backprojection of measured sinograms;
* ``ragged``     ``RaggedBatch``: projection, then fbp, of slices with geometries of their own;
* ``laplacian``  ``laplacian``: the kNN graph of a point set.

Images are sums of random ellipses with a fine texture, sinograms their line
integrals with photon noise: what scanners and phantom studies give. ``exact``
evaluates the operators in 64 bits by another route, from cumulative sums of
each image line (of each detector row) read at the projected boundaries.
"""

import math

import numpy as np
import torch

import ctlib_gb300 as ctlib
from ctlib_gb300 import autograd as ag
from ctlib_gb300 import ops
from ctlib_gb300.batched import RaggedBatch

ED, EA, PARA = 0, 1, 2
TWO_PI = 2 * math.pi
FOV = 340.0  # mm, the image side of the drawn geometries
# view-bin-lines of the largest listed case (8 slices of 1024^2, 2304 views, 1472 bins)
MOST = 8 * 2304 * 1472 * 1024


def _fan(op, scan, batch, views, dets, width, height, dImg, dDet, s2r, d2r, ang0=0.0, shift=0.0, dtype="float32"):
    return {"op": op, "scan": scan, "dtype": dtype, "batch": batch, "views": views, "dets": dets, "width": width,
            "height": height, "dImg": dImg, "dDet": dDet, "ang0": ang0, "dAng": TWO_PI / views, "s2r": s2r,
            "d2r": d2r, "shift": shift}


def _para(op, batch, views, dets, width, height, dImg, dDet, ang0=0.0, shift=0.0, dtype="float32"):
    c = _fan(op, PARA, batch, views, dets, width, height, dImg, dDet, 0.0, 0.0, ang0, shift, dtype)
    c["dAng"] = math.pi / views
    return c


def _ed512(op, batch):
    return _fan(op, ED, batch, 1152, 736, 512, 512, 0.6641, 1.2858, 595.0, 490.6)


def _ea512(op, batch):
    return _fan(op, EA, batch, 984, 888, 512, 512, 0.7, 0.0011, 541.0, 408.0)


def listed():
    return [
        # the smallest calls: one small parallel-beam slice, reconstructed and as a training step
        {"name": "fbp_para256_b1", **_para("fbp", 1, 360, 367, 256, 256, 1.0, 1.0)},
        {"name": "pair_para256_b1", **_para("pair", 1, 360, 367, 256, 256, 1.0, 1.0)},
        # one slice of the usual clinical size: an iteration of a reconstruction on its own
        {"name": "gradient_ed512_b1", **_ed512("gradient", 1)},
        # a training batch (the package's benchmark workload)
        {"name": "pair_ed512_b16", **_ed512("pair", 16)},
        # a batch of measured data in a learned reconstruction's data term
        {"name": "fidelity_ea512_b8", **_ea512("fidelity", 8)},
        # a few slices of a scan, reconstructed: a batch that is no power of two
        {"name": "fbp_ed512_b5", **_ed512("fbp", 5)},
        # reconstruction layer with gradients, one slice
        {"name": "bpair_ea512_b1", **_ea512("bpair", 1)},
        # the largest: high-resolution slices
        {"name": "pair_ed1024_b8", **_fan("pair", ED, 8, 2304, 1472, 1024, 1024, 0.33, 0.6429, 595.0, 490.6)},
        # nothing square, even or centred: a short odd scan with a detector shift
        {"name": "pair_ed400x363_b3", **_fan("pair", ED, 3, 491, 595, 400, 363, 0.85, 1.6, 595.0, 490.6, 0.3, 0.4)},
        # slices of different scanners together
        {"name": "ragged_24", "op": "ragged", "slices": 24, "mix": 4000},
        # double precision, as gradient checks and reference runs use it
        {"name": "pair_f64_ed256_b2", **_fan("pair", ED, 2, 576, 368, 256, 256, 1.3282, 2.5716, 595.0, 490.6,
                                             dtype="float64")},
        # the graph of a feature set
        {"name": "laplacian_16k", "op": "laplacian", "dtype": "float32", "points": 16384, "dim": 64, "k": 16},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["pair", "pair", "bpair", "gradient", "fidelity", "fbp", "fbp", "ragged", "laplacian", "f64"])
    if op == "laplacian":
        n = int(_log(rng, 1000, 16384))
        return {"op": op, "dtype": "float32", "points": n, "dim": int(_log(rng, 3, 128)), "k": int(_log(rng, 4, 40))}
    if op == "ragged":
        return {"op": op, "slices": rng.randint(3, 28), "mix": rng.randrange(1 << 20)}
    dtype = "float32"
    if op == "f64":
        op, dtype = rng.choice(["pair", "bpair", "gradient"]), "float64"
    big = 384 if dtype == "float64" else 1024
    width = int(_log(rng, 128 if dtype == "float64" else 200, big + 1))
    height = width if rng.random() < 0.6 else max(100, min(big, int(width * rng.uniform(0.75, 1.3))))
    size = max(width, height)
    views = int(_log(rng, 64, 2.25 * size))
    dets = int(size * rng.uniform(1.0, 1.75))
    batch = int(_log(rng, 1, 17 if dtype == "float32" else 4.5))
    batch = max(1, min(batch, MOST // (views * dets * size)))
    c = _geometry(rng.randrange(3), views, dets, width, height)
    c |= {"op": op, "dtype": dtype, "batch": batch}
    if rng.random() < 0.5:
        c["ang0"] = rng.uniform(0.0, 1.0)
        c["shift"] = c["dDet"] * rng.uniform(-0.5, 0.5)
    return c


def _geometry(scan, views, dets, width, height):
    """A scan whose detector covers the image's diagonal."""
    size = max(width, height)
    if scan == PARA:
        return _para("", 1, views, dets, width, height, FOV / size, FOV * 1.45 / dets)
    s2r, d2r = (595.0, 490.6) if scan == ED else (541.0, 408.0)
    half = math.asin(0.5 * FOV * 1.42 / s2r)
    dDet = 2 * (s2r + d2r) * math.tan(half) / dets if scan == ED else 2 * half / dets
    return _fan("", scan, 1, views, dets, width, height, FOV / size, dDet, s2r, d2r)


def _ragged_slices(c):
    """Sizes 256 to 768, 64 to 2304 views, 368 to 1024 bins, every geometry."""
    rng = np.random.default_rng(c["mix"])
    out = []
    for _ in range(c["slices"]):
        size = int(rng.choice([256, 384, 512, 640, 768]))
        views = int(rng.choice([64, 128, 360, 720, 1152, 2304]))
        g = _geometry(int(rng.integers(0, 3)), views, int(rng.integers(368, 1025)), size, size)
        out.append(g | {"dtype": "float32"})
    return out


# ------------------------------------------------------------------- inputs

def _options(c):
    """CTLIB's options vector."""
    o = [c["views"], c["dets"], c["width"], c["height"], c["dImg"], c["dDet"], c["ang0"], c["dAng"]]
    o += [] if c["scan"] == PARA else [c["s2r"], c["d2r"]]
    return torch.tensor(o + [c["shift"], c["scan"]], dtype=torch.float64)


def _dtype(c):
    return torch.float64 if c["dtype"] == "float64" else torch.float32


def _ellipses(c, seed):
    """B x 10 ellipses: centre, semi-axes, orientation, attenuation (1/mm)."""
    rng = np.random.default_rng(seed)
    fov, shape = c["width"] * c["dImg"], (c["batch"], 10)
    r, t = 0.45 * fov * np.sqrt(rng.uniform(size=shape)), rng.uniform(0, TWO_PI, shape)
    a, b = rng.uniform(0.05, 0.35, (2,) + shape) * fov
    p = np.stack([r * np.cos(t), r * np.sin(t), a, b, rng.uniform(0, math.pi, shape), rng.uniform(0, 0.02, shape)])
    return torch.from_numpy(p).cuda()


def _images(c, seed):
    """Phantoms B x 1 x H x W with a texture of 1e-3."""
    e = _ellipses(c, seed)
    x = (torch.arange(c["width"], dtype=torch.float64, device="cuda") - c["width"] / 2 + 0.5) * c["dImg"]
    y = ((c["height"] / 2 - 0.5 - torch.arange(c["height"], dtype=torch.float64, device="cuda")) * c["dImg"])[:, None]
    img = torch.zeros(c["batch"], 1, c["height"], c["width"], dtype=torch.float64, device="cuda")
    for b in range(c["batch"]):
        for cx, cy, sa, sb, phi, mu in e[:, b].T.tolist():
            u = ((x - cx) * math.cos(phi) + (y - cy) * math.sin(phi)) / sa
            v = ((y - cy) * math.cos(phi) - (x - cx) * math.sin(phi)) / sb
            img[b, 0] += mu * (u * u + v * v <= 1)
    return (img + 1e-3 * _randn(img.shape, seed + 1)).to(_dtype(c))


def _randn(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def _sinograms(c, seed):
    """Line integrals of the phantoms' ellipses through every bin's centre, B x 1
    x V x D, with the noise of 1e5 photons a ray."""
    kw = {"dtype": torch.float64, "device": "cuda"}
    ang = (torch.arange(c["views"], **kw) * c["dAng"] + c["ang0"])[:, None]
    t = torch.arange(c["dets"], **kw) + 0.5 - c["dets"] / 2
    cos, sin = torch.cos(ang), torch.sin(ang)
    if c["scan"] == PARA:
        s = t * c["dDet"] + c["shift"]
        ox, oy, dx, dy = s * cos, s * sin, -sin + 0 * s, cos + 0 * s
    else:
        ox, oy = -sin * c["s2r"] + 0 * t, cos * c["s2r"] + 0 * t
        if c["scan"] == ED:
            s = (t * c["dDet"] + c["shift"]) * c["s2r"] / (c["s2r"] + c["d2r"])
            dx, dy = s * cos - ox, s * sin - oy
            n = torch.hypot(dx, dy)
            dx, dy = dx / n, dy / n
        else:
            beta = t * c["dDet"] + c["shift"] + ang
            dx, dy = torch.sin(beta), -torch.cos(beta)
    e = _ellipses(c, seed)
    out = torch.zeros(c["batch"], 1, c["views"], c["dets"], **kw)
    for b in range(c["batch"]):
        for cx, cy, sa, sb, phi, mu in e[:, b].T.tolist():
            co, si = math.cos(phi), math.sin(phi)
            px, py = ((ox - cx) * co + (oy - cy) * si) / sa, ((oy - cy) * co - (ox - cx) * si) / sb
            qx, qy = (dx * co + dy * si) / sa, (dy * co - dx * si) / sb
            qq, pq = qx * qx + qy * qy, px * qx + py * qy
            out[b, 0] += 2 * mu * torch.sqrt(torch.clamp(pq * pq - qq * (px * px + py * py - 1), min=0)) / qq
    noise = _randn(out.shape, seed + 2) * torch.exp(0.5 * torch.clamp(out, max=8.0)) / math.sqrt(1e5)
    return (out + noise).to(_dtype(c))


def _residual(c, seed):
    """An upstream gradient: a sinogram's (image's) worth of noise."""
    shape = (c["height"], c["width"]) if c["op"] == "bpair" else (c["views"], c["dets"])
    return _randn((c["batch"], 1) + shape, seed + 3).to(_dtype(c))


def _points(c, seed):
    return _randn((c["points"], c["dim"]), seed).to(_dtype(c))


def prepare(case, seed):
    c, op = dict(case), case["op"]
    if op == "laplacian":
        return {"op": op, "points": _points(c, seed), "k": c["k"]}
    if op == "ragged":
        slices = _ragged_slices(c)
        return {"op": op, "batch": RaggedBatch([_options(s) for s in slices]),
                "images": [_images(s, seed + 10 * i) for i, s in enumerate(slices)]}
    s = {"op": op, "options": _options(c)}
    if op == "pair":
        s |= {"layer": ag.Projector(s["options"]), "x": _images(c, seed).requires_grad_(), "g": _residual(c, seed)}
    elif op == "bpair":
        s |= {"layer": ag.Backprojector(s["options"]), "x": _sinograms(c, seed).requires_grad_(),
              "g": _residual(c, seed)}
    elif op == "gradient":
        s |= {"x": _images(c, seed), "y": _sinograms(c, seed)}
    elif op == "fidelity":
        s |= {"x": _images(c, seed).requires_grad_(), "y": _sinograms(c, seed)}
    else:
        s |= {"y": _sinograms(c, seed)}
    return s


def run(s):
    op = s["op"]
    if op in ("pair", "bpair"):
        out = s["layer"](s["x"])
        (grad,) = torch.autograd.grad(out, s["x"], s["g"])
        return {"out": out, "grad": grad}
    if op == "gradient":
        grad, res = ops.data_gradient(s["x"], s["y"], s["options"], return_residual=True)
        return {"grad": grad, "residual": res}
    if op == "fidelity":
        loss = ag.data_fidelity(s["x"], s["y"], s["options"])
        (grad,) = torch.autograd.grad(loss, s["x"])
        return {"loss": loss, "grad": grad}
    if op == "fbp":
        return {"image": ctlib.fbp(s["y"], s["options"])}
    if op == "ragged":
        sinos = s["batch"].projection(s["images"])
        return {"sinos": sinos, "images": s["batch"].fbp(sinos)}
    w = ctlib.laplacian(s["points"], s["k"])
    return {"indices": w._indices(), "values": w._values()}


def work(case):
    c, op = case, case["op"]
    if op == "laplacian":
        n, dim, k = c["points"], c["dim"], c["k"]
        return {"bytes": 4.0 * n * dim + 20.0 * n * k, "flops": 2.0 * n * n * dim}
    if op == "ragged":
        parts = [work(s | {"op": o}) for s in _ragged_slices(c) for o in ("fbp", "projection")]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    img, sino = c["batch"] * c["height"] * c["width"], c["batch"] * c["views"] * c["dets"]
    es = 8.0 if c["dtype"] == "float64" else 4.0
    # per view and image line every pixel and every bin in the image ends one overlap: one multiply-add a slice
    size = max(c["width"], c["height"])
    pitch = c["dDet"] * {ED: c["s2r"] / max(1e-9, c["s2r"] + c["d2r"]), EA: c["s2r"], PARA: 1.0}[c["scan"]]
    flops = 2.0 * c["batch"] * c["views"] * size * (size + min(c["dets"], size * c["dImg"] / pitch))
    if op in ("pair", "bpair"):
        return {"bytes": es * 2 * (img + sino), "flops": 2 * flops}
    if op in ("gradient", "fidelity"):
        return {"bytes": es * 2 * (img + sino) if op == "gradient" else es * (2 * img + sino), "flops": 2 * flops}
    if op == "fbp":  # the ramp filter's non-zero taps, and the backprojection
        return {"bytes": es * (img + sino), "flops": flops + sino * c["dets"]}
    return {"bytes": es * (img + sino), "flops": flops}


# -------------------------------------------------------------------- exact

class _Scan:
    """The scan in 64 bits. Options and view angles are rounded to the data type
    first, as the operators define them: an angle picks the view's axis."""

    def __init__(self, c):
        T = np.float64 if c["dtype"] == "float64" else np.float32
        r = lambda k: float(T(c[k]))  # noqa: E731
        self.c, self.V, self.D, self.W, self.H, self.scan = c, c["views"], c["dets"], c["width"], c["height"], c["scan"]
        self.dImg, self.dDet, self.s2r, self.d2r, self.shift = (r(k) for k in ("dImg", "dDet", "s2r", "d2r", "shift"))
        self.dAng = r("dAng")
        self.ang = [float(T(v * self.dAng + r("ang0"))) for v in range(self.V)]
        groups = {}
        for v, a in enumerate(self.ang):
            x = abs(a - _round(a / math.pi) * math.pi) * 4 / math.pi <= 1
            e = (a - math.floor(a / TWO_PI) * TWO_PI) * 4 / math.pi
            groups.setdefault((x, 3 <= e < 7), []).append(v)
        self.groups = groups

    def chunks(self):
        """(views, rows are lines, detector order reversed) a few views at a time."""
        step = max(1, int(6e7 / (max(self.W, self.H) * (max(self.D, self.W, self.H) + 1))))
        for (x, flip), vs in self.groups.items():
            for i in range(0, len(vs), step):
                yield torch.tensor(vs[i:i + step], device="cuda"), x, flip

    def view(self, vs, x, flip):
        """Bin edges (n x D+1) on the view's axis, and each line's map of pixel
        edge k to the axis, alpha + sigma k (n x lines)."""
        kw = {"dtype": torch.float64, "device": "cuda"}
        a = torch.tensor(self.ang, **kw)[vs][:, None]
        c, s = torch.cos(a), torch.sin(a)
        t = (torch.arange(self.D + 1, **kw) - self.D / 2) * (-1 if flip else 1)
        sx, sy = -s * self.s2r, c * self.s2r
        m = self.s2r / (self.s2r + self.d2r) if self.scan != PARA else 1.0
        if self.scan == ED:
            d = t * (m * self.dDet) + m * self.shift
            dx, dy = d * c, d * s
            db = (sx * dy - sy * dx) / (dy - sy) if x else (sy * dx - sx * dy) / (dx - sx)
        elif self.scan == EA:
            beta = t * self.dDet + self.shift + a
            db = sx + torch.tan(beta) * sy if x else sy + sx / torch.tan(beta)
        else:
            db = (t * self.dDet + self.shift) / (c if x else s)
        x0, y0 = -self.W / 2 * self.dImg, -self.H / 2 * self.dImg
        p = self.line_pos(x)
        if self.scan == PARA:
            alpha = s / c * p + x0 if x else y0 + c / s * p
            sigma = torch.full_like(alpha, self.dImg)
        elif x:
            alpha, sigma = (sx * p - sy * x0) / (p - sy), -sy * self.dImg / (p - sy)
        else:
            alpha, sigma = (sy * p - sx * y0) / (p - sx), -sx * self.dImg / (p - sx)
        return sx, sy, db, alpha, sigma

    def line_pos(self, x):
        kw = {"dtype": torch.float64, "device": "cuda"}
        if x:
            return (self.H / 2 - 0.5 - torch.arange(self.H, **kw)) * self.dImg
        return (torch.arange(self.W, **kw) - self.W / 2 + 0.5) * self.dImg

    def weight(self, sx, sy, x):
        """The backprojector's pixel weight, n x lines x pixels (1 for parallel beams)."""
        if self.scan == PARA:
            return None
        kw = {"dtype": torch.float64, "device": "cuda"}
        n = self.W if x else self.H
        q, p = (torch.arange(n, **kw) - n / 2 + 0.5) * self.dImg, self.line_pos(x)[:, None]
        px, py = (q, p) if x else (p, q)
        sx, sy = sx[:, :, None], sy[:, :, None]
        if self.scan == ED:
            return (self.s2r ** 2 / (self.s2r ** 2 - sx * px - sy * py)) ** 2
        return 1 / ((sx - px) ** 2 + (sy - py) ** 2)

    def cbar(self, sx, sy, db, x):
        near, far = (sy, sx) if x else (sx, sy)
        cosb = near.abs() / torch.sqrt((db - far) ** 2 + near ** 2)
        return (cosb[:, 1:] + cosb[:, :-1]) / 2

    def norm(self, sx, sy, db, x):
        """A's factor per bin."""
        if self.scan == PARA:
            return torch.full_like(db[:, 1:], self.dImg / self.dDet)
        return self.dImg / (self.cbar(sx, sy, db, x) * (db[:, 1:] - db[:, :-1]))


def _round(v):
    return math.floor(v + 0.5) if v >= 0 else math.ceil(v - 0.5)


def _lines(img, x):
    """An image's lines along the walk: rows, or columns from the bottom up."""
    return img if x else img.flip(0).T.contiguous()


def _sums(v):
    return torch.nn.functional.pad(torch.cumsum(v, -1), (1, 0))


def _to_detector(sc, imgs, weighted):
    """A (or B^T) of images B x 1 x H x W."""
    out = torch.zeros(imgs.shape[0], 1, sc.V, sc.D, dtype=torch.float64, device="cuda")
    for vs, x, flip in sc.chunks():
        sx, sy, db, alpha, sigma = sc.view(vs, x, flip)
        N = sc.W if x else sc.H
        u = ((db[:, None, :] - alpha[:, :, None]) / sigma[:, :, None]).clamp_(0, N)
        k = u.floor().clamp_(max=N - 1)
        u -= k
        k = k.long()
        w = sc.weight(sx, sy, x) if weighted else None
        for b in range(imgs.shape[0]):
            ln = _lines(imgs[b, 0].double(), x)[None]
            ln = (ln * w if w is not None else ln).expand(len(vs), -1, -1)
            cum = _sums(ln if w is not None else ln[:1]).expand(len(vs), -1, -1)
            part = torch.gather(cum, 2, k) + u * torch.gather(ln, 2, k)
            edge = (part if weighted else part * sigma[:, :, None]).sum(1)
            val = edge[:, 1:] - edge[:, :-1]
            if not weighted:
                val = val * sc.norm(sx, sy, db, x)
            elif sc.scan == EA:
                val = val * sc.dImg / sc.cbar(sx, sy, db, x)
            out[b, 0, vs] = val.flip(1) if flip else val
    return out


def _to_image(sc, sinos, weighted):
    """A^T (or B) of sinograms B x 1 x V x D."""
    out = torch.zeros(sinos.shape[0], 1, sc.H, sc.W, dtype=torch.float64, device="cuda")
    for vs, x, flip in sc.chunks():
        sx, sy, db, alpha, sigma = sc.view(vs, x, flip)
        N = sc.W if x else sc.H
        kw = {"dtype": torch.float64, "device": "cuda"}
        e = alpha[:, :, None] + sigma[:, :, None] * torch.arange(N + 1, **kw)
        e = torch.minimum(torch.maximum(e, db[:, :1, None]), db[:, -1:, None])
        d = torch.searchsorted(db, e.reshape(len(vs), -1), right=True).sub_(1).clamp_(0, sc.D - 1)
        off = e.reshape(len(vs), -1) - torch.gather(db, 1, d)
        w = None
        if weighted:
            w = sc.weight(sx, sy, x)
            w = w / sigma[:, :, None] if w is not None else 1 / sc.dImg
        for b in range(sinos.shape[0]):
            q = sinos[b, 0, vs].double()
            q = q.flip(1) if flip else q
            if not weighted:
                q = q * sc.norm(sx, sy, db, x)
            cum = _sums(q * (db[:, 1:] - db[:, :-1]))
            val = (torch.gather(cum, 1, d) + off * torch.gather(q, 1, d)).reshape(e.shape)
            val = val[:, :, 1:] - val[:, :, :-1]
            val = (val * w if w is not None else val).sum(0)
            out[b, 0] += val if x else val.T.flip(0)
    return out


def _filtered(sc, sinos):
    """The ramp filter on pre-weighted rows."""
    kw = {"dtype": torch.float64, "device": "cuda"}
    t = torch.arange(sc.D, **kw) + 0.5 - sc.D / 2
    d = sc.dDet
    if sc.scan == ED:
        d = sc.dDet * sc.s2r / (sc.s2r + sc.d2r)
        pre = d * sc.s2r / torch.sqrt(sc.s2r ** 2 + (t * d) ** 2)
    elif sc.scan == EA:
        pre = torch.cos(t * d) * sc.s2r * d
    else:
        pre = torch.full_like(t, d)
    n = torch.arange(sc.D, **kw)[:, None] - torch.arange(sc.D, **kw)
    h = torch.where(n % 2 != 0, -1 / (math.pi * n * d).square().clamp(min=1e-300), torch.zeros_like(n))
    h.fill_diagonal_(1 / (4 * d * d))
    return (sinos.double() * pre) @ h


def _fbp(sc, sinos):
    return _to_image(sc, _filtered(sc, sinos), True) * (sc.dAng / 2)


def exact(case, seed):
    c, op = dict(case), case["op"]
    if op == "laplacian":
        x = _points(c, seed).double()
        n = (x * x).sum(1)
        d = torch.topk(n[:, None] + n - 2 * x @ x.T, c["k"], dim=1, largest=False)[0]
        w = torch.exp(-d / d.flatten().median())
        return {"indices": None, "values": (w / w.sum(1, keepdim=True)).reshape(-1)}
    if op == "ragged":
        sinos, images = [], []
        for i, s in enumerate(_ragged_slices(c)):
            sc = _Scan(s)
            sinos.append(_to_detector(sc, _images(s, seed + 10 * i), False))
            images.append(_fbp(sc, sinos[-1]))
        return {"sinos": sinos, "images": images}
    sc = _Scan(c)
    if op == "pair":
        return {"out": _to_detector(sc, _images(c, seed), False), "grad": _to_image(sc, _residual(c, seed), False)}
    if op == "bpair":
        return {"out": _to_image(sc, _sinograms(c, seed), True), "grad": _to_detector(sc, _residual(c, seed), True)}
    if op == "fbp":
        return {"image": _fbp(sc, _sinograms(c, seed))}
    res = _to_detector(sc, _images(c, seed), False) - _sinograms(c, seed).double()
    grad = _to_image(sc, res, False)
    return {"grad": grad, "residual": res} if op == "gradient" else {"loss": 0.5 * (res * res).sum(), "grad": grad}
