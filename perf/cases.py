"""The work this framework is timed on: calls of its public entry points at the sizes its users run.

Every case names a kind of call:

* ``train``: ``TileVoxelizer`` forward and backward, the hot path of a fit.  ``static`` takes the
  fixed-capacity voxelizer the graph-captured loops use, ``deterministic`` the fixed-order backward.
* ``render``: ``TileVoxelizer`` forward alone, as evaluations and exports call it.
* ``compat``: ``build_tile_pairs`` and ``_TileVoxelizeCUDA``, the reference's own call sequence.
* ``batch``: ``BatchedVoxelizer`` over volumes of uneven size, forward and backward.
* ``sense``: the SENSE data term and the magnitude TV of a volume, value and gradient.
* ``mlp``: the warm-start network, forward and (``backward``) the weight gradients.
* ``iter``: a whole fit iteration up to the gradients: voxelizer, SENSE data term, backward.

``exact`` restates each of them in 64 bits with plain torch.
"""
import math

import torch

from gs_tmi_b200 import TileVoxelizer, _TileVoxelizeCUDA, build_tile_pairs, sense
from gs_tmi_b200.batched import BatchedVoxelizer
from gs_tmi_b200.warmstart import WarmStartMLP

DEV = "cuda:0"
MAX_VOXELS = 256 * 256 * 160
MAX_GAUSSIANS = 2_000_000


def _vox(kind, name, d, h, w, n, **more):
    case = {"kind": kind, "d": d, "h": h, "w": w, "n": n, "tile": 8, "spread": "fit", "deterministic": False,
            "static": False, "coils": 0}
    case.update(more)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the smallest call: a toy volume, where launches and host work are everything
        _vox("train", "train_32c_500", 32, 32, 32, 500, spread="uniform"),
        # the voxelizer micro-benchmark: 64^3, 20,000 Gaussians of about 1.5 voxels
        _vox("train", "train_64c_20k", 64, 64, 64, 20_000, spread="uniform"),
        # a 128x128x96 fit at its start, on the workspace of the graph-captured loop
        _vox("train", "train_128x128x96_50k", 128, 128, 96, 50_000, static=True),
        # the same fit at its densification cap
        _vox("train", "train_128x128x96_500k", 128, 128, 96, 500_000),
        # the large fit at its cap, with the reproducible backward it runs with
        _vox("train", "train_det_256x256x160_2m", 256, 256, 160, 2_000_000, deterministic=True),
        # an evaluation's render of a volume whose sides are no multiple of anything
        _vox("render", "render_75x61x53_30k", 75, 61, 53, 30_000),
        # the other tile edge the tile-size tuner compares
        _vox("train", "train_tile4_96c_40k", 96, 96, 96, 40_000, tile=4),
        # a host that calls the reference's binning and autograd function itself
        _vox("compat", "compat_100x84x60_20k", 100, 84, 60, 20_000),
        # a study reconstructed as one batch of uneven volumes
        {"name": "batch_4_volumes", "kind": "batch", "count": 4, "d": 96, "h": 96, "w": 96, "n": 30_000,
         "grow": 1.2, "deterministic": False},
        # the loss of a 128x128x96 acquisition with 8 coils
        {"name": "sense_128x128x96_8c", "kind": "sense", "d": 128, "h": 128, "w": 96, "coils": 8},
        # a warm-start training step over the seeds of a 96^3 phantom
        {"name": "mlp_train_84k", "kind": "mlp", "rows": 84_375, "backward": True},
        # a whole iteration of the plain fit, up to the gradients
        _vox("iter", "iter_128x128x96_50k_8c", 128, 128, 96, 50_000, coils=8),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi):
    d, h, w = (_side(rng, lo, hi) for _ in range(3))
    if rng.random() < 0.5:  # half of the volumes are made of whole tiles
        d, h, w = (max(8, 8 * round(x / 8)) for x in (d, h, w))
    while d * h * w > MAX_VOXELS:
        d, h, w = max(8, d // 2), h, w
    return d, h, w


def _count(rng, voxels, lo=300, most=MAX_GAUSSIANS):
    hi = min(most, voxels // 3)  # the densest fits hold a Gaussian per three voxels
    return _side(rng, min(max(lo, voxels // 200), hi), hi)


def draw(rng):
    kind = rng.choices(["train", "render", "compat", "batch", "sense", "mlp", "iter"], [6, 2, 1, 1, 1, 1, 1])[0]
    if kind == "mlp":
        return {"kind": "mlp", "rows": _side(rng, 1000, 200_000), "backward": rng.random() < 0.5}
    if kind == "sense":
        d, h, w = _shape(rng, 32, 144)
        return {"kind": "sense", "d": d, "h": h, "w": w, "coils": rng.randint(2, 12)}
    if kind == "batch":
        side = _side(rng, 32, 112)
        return {"kind": "batch", "count": rng.randint(2, 6), "d": side, "h": side + rng.randint(-8, 8),
                "w": side + rng.randint(-8, 8), "n": _count(rng, side ** 3, most=60_000),
                "grow": round(rng.uniform(1.0, 1.2), 3), "deterministic": rng.random() < 0.3}
    if kind == "compat":
        d, h, w = _shape(rng, 24, 128)
        return _vox("compat", None, d, h, w, _count(rng, d * h * w, most=100_000), tile=rng.choice([8, 8, 4]))
    if kind == "iter":
        d, h, w = _shape(rng, 32, 128)
        return _vox("iter", None, d, h, w, _count(rng, d * h * w, most=200_000), coils=rng.randint(2, 8))
    d, h, w = _shape(rng, 24, 224)
    return _vox(kind, None, d, h, w, _count(rng, d * h * w), tile=rng.choice([8, 8, 8, 8, 4]),
                spread=rng.choice(["fit", "fit", "uniform"]), deterministic=rng.random() < 0.3,
                static=kind == "train" and rng.random() < 0.3)


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _spacing_sigma(n, shape):
    """The intensity-seeded init's scale: the mean distance to the nearest other seeds, in voxels."""
    d, h, w = shape
    return 0.75 * (d * h * w / n) ** (1.0 / 3.0)


def _gaussians(n, shape, spread, g):
    """Positions, scales, rotations, density re / im.  ``uniform``: the micro-benchmark's set.
    ``fit``: a fit's set, denser inside the object, scales that follow the seeds' spacing."""
    half = torch.tensor([0.5 * s for s in shape], device=DEV)
    pos = torch.rand(n, 3, generator=g, device=DEV) * 2 - 1
    quat = torch.randn(n, 4, generator=g, device=DEV)
    log_vox = torch.randn(n, 3, generator=g, device=DEV)
    if spread == "uniform":
        log_vox = math.log(1.5) + 0.3 * log_vox
    else:
        inside = torch.rand(n, generator=g, device=DEV) < 0.6
        ball = torch.randn(n, 3, generator=g, device=DEV)
        ball = ball / ball.norm(dim=-1, keepdim=True) * torch.rand(n, 1, generator=g, device=DEV) ** (1.0 / 3.0)
        pos = torch.where(inside[:, None], 0.75 * ball, pos)
        one = torch.randn(n, 1, generator=g, device=DEV)
        log_vox = math.log(_spacing_sigma(n, shape)) + 0.2 * log_vox + 0.2 * one
    den = 0.1 * torch.randn(2, n, generator=g, device=DEV)
    return [pos, torch.exp(log_vox) / half, quat, den[0].contiguous(), den[1].contiguous()]


def _complex_normal(shape, g):
    x = torch.randn(*shape, 2, generator=g, device=DEV)
    return torch.view_as_complex(x) / math.sqrt(2.0)


def _batch_shapes(case):
    out = []
    for i in range(case["count"]):
        f = case["grow"] ** i
        out.append(((int(case["d"] * f), int(case["h"] * f), int(case["w"] * f)), int(case["n"] * f ** 3)))
    return out


def _acquisition(shape, coils, g):
    """Smooth coil maps of unit sum of squares, a (ky, kz) mask at about R = 6 with a sampled centre,
    and noisy k-space of a smooth object."""
    d, h, w = shape
    zz, yy, xx = torch.meshgrid(*(torch.linspace(-1, 1, s, device=DEV) for s in shape), indexing="ij")
    maps = []
    for c in range(coils):
        a = 2 * math.pi * c / coils
        prof = torch.exp(-((yy - 1.3 * math.cos(a)) ** 2 + (xx - 1.3 * math.sin(a)) ** 2 + 0.5 * zz ** 2) / 1.62)
        maps.append(torch.polar(prof, a + 0.5 * (yy * math.sin(a) - xx * math.cos(a))))
    S = torch.stack(maps)
    S = S / torch.sqrt((S.abs() ** 2).sum(0, keepdim=True))
    plane = torch.rand(h, w, generator=g, device=DEV) < 1.0 / 7.0
    plane[h // 2 - h // 10:h // 2 + h // 10 + 1, w // 2 - w // 10:w // 2 + w // 10 + 1] = True
    mask = plane.float().expand(d, h, w).contiguous()
    obj = torch.polar(torch.exp(-2 * (zz ** 2 + yy ** 2 + xx ** 2)), 0.7 * zz + 0.4 * yy * xx)
    ku = _fft3c(S * obj)
    ku = (ku + 1e-3 * ku.abs().max() * _complex_normal(ku.shape, g)) * mask
    return S.to(torch.complex64).contiguous(), mask, ku.to(torch.complex64).contiguous()


def _fft3c(x):
    dims = (-3, -2, -1)
    return torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(x, dim=dims), dim=dims, norm="ortho"), dim=dims)


def _mlp_inputs(case, g):
    rows = case["rows"]
    x = torch.zeros(rows, 256, device=DEV)
    x[:, :250] = 0.5 * torch.randn(rows, 250, generator=g, device=DEV)
    x[:, 250] = 1.0 / 6.0
    x[:, 251] = math.log(2.0) + 0.2 * torch.randn(rows, generator=g, device=DEV)
    w = [torch.randn(o, i, generator=g, device=DEV) * math.sqrt(2.0 / i) for o, i in ((256, 256), (256, 256))]
    w.append(0.1 * torch.randn(16, 256, generator=g, device=DEV) * math.sqrt(2.0 / 256))
    b = [0.05 * torch.randn(o, generator=g, device=DEV) for o in (256, 256, 16)]
    dout = torch.randn(rows, 16, generator=g, device=DEV) / rows
    return x.bfloat16(), w + b, dout


def _inputs(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "mlp":
        return _mlp_inputs(case, g)
    if kind == "batch":
        return [(_gaussians(n, s, "fit", g), _complex_normal(s, g)) for s, n in _batch_shapes(case)]
    shape = (case["d"], case["h"], case["w"])
    if kind == "sense":
        smooth = torch.nn.functional.interpolate(torch.randn(1, 2, 9, 9, 9, generator=g, device=DEV), size=shape,
                                                 mode="trilinear", align_corners=True)[0]
        vol = torch.complex(smooth[0], smooth[1]) + 0.1 * _complex_normal(shape, g)
        return (vol.contiguous(), *_acquisition(shape, case["coils"], g))
    params = _gaussians(case["n"], shape, case["spread"], g)
    if kind == "iter":
        return (params, *_acquisition(shape, case["coils"], g))
    return params, _complex_normal(shape, g)


def _reference_preprocess(params, shape):
    """Center, inverse covariance, radius and half shape, as the reference's module computes them."""
    pos, scl, rot, _, _ = params
    size = torch.tensor(shape, dtype=pos.dtype, device=pos.device)
    center = (pos + 1.0) * 0.5 * size - 0.5
    q = rot / (rot.norm(dim=-1, keepdim=True) + 1e-8)
    t = _rotation(q) / (scl + 1e-8)[:, None, :]
    return center, t @ t.transpose(-1, -2), (scl * size * 0.5).max(-1).values * 3.0, size * 0.5


def _rotation(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([1 - 2 * y * y - 2 * z * z, 2 * x * y - 2 * z * w, 2 * x * z + 2 * y * w,
                        2 * x * y + 2 * z * w, 1 - 2 * x * x - 2 * z * z, 2 * y * z - 2 * x * w,
                        2 * x * z - 2 * y * w, 2 * y * z + 2 * x * w, 1 - 2 * x * x - 2 * y * y], -1).view(-1, 3, 3)


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

def _leaf(t):
    return t.clone().requires_grad_(True)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "mlp":
        x, weights, dout = _mlp_inputs(case, _gen(seed))
        s["net"] = WarmStartMLP(DEV)
        s["net"].load_state_dict({"params": weights})
        s.update(x=x, dout=dout)
        return s
    if kind == "batch":
        sets = _inputs(case, seed)
        s["vox"] = BatchedVoxelizer([v for v, _ in _batch_shapes(case)], device=DEV,
                                    deterministic=case["deterministic"])
        s["sets"] = [(_leaf(p[0]), _leaf(p[1]), _leaf(p[2]), _leaf(torch.complex(p[3], p[4]))) for p, _ in sets]
        s["grads"] = [g for _, g in sets]
        return s
    shape = (case["d"], case["h"], case["w"])
    if kind == "sense":
        vol, s["S"], s["mask"], s["ku"] = _inputs(case, seed)
        s.update(vol=_leaf(vol), ws=sense.sense_workspace(DEV), ws_tv=sense.sense_workspace(DEV))
        return s
    params, *rest = _inputs(case, seed)
    if kind == "compat":
        center, cov_inv, radius, half = _reference_preprocess(params, shape)
        s.update(center=_leaf(center), cov_inv=_leaf(cov_inv), radius=radius, half=half, dr=_leaf(params[3]),
                 di=_leaf(params[4]), grad=(rest[0].real.reshape(-1).contiguous(), rest[0].imag.reshape(-1).contiguous()))
        return s
    vox = TileVoxelizer(shape, tile_size=case["tile"], device=DEV, deterministic=case["deterministic"])
    if case["static"]:
        vox = vox.static(case["n"], vox.count_pairs(params[0], params[1]) + 4096)
    s["vox"] = vox
    if kind == "iter":
        s["S"], s["mask"], s["ku"] = rest
        s["ws"] = sense.sense_workspace(DEV)
        params = [params[0], torch.log(params[1]), *params[2:]]
    else:
        s["grad"] = rest[0]
        params = [*params[:3], torch.complex(params[3], params[4])]
    s["leaves"] = [p.clone() for p in params] if kind == "render" else [_leaf(p) for p in params]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("train", "render"):
        if kind == "render":
            with torch.no_grad():
                return s["vox"](*s["leaves"])
        vol = s["vox"](*s["leaves"])
        return (vol.detach(), *torch.autograd.grad(vol, s["leaves"], s["grad"]))
    if kind == "compat":
        shape = (case["d"], case["h"], case["w"])
        ranges, ids = build_tile_pairs(s["center"], s["radius"], shape, case["tile"])
        inputs = [s["center"], s["cov_inv"], s["dr"], s["di"]]
        vr, vi = _TileVoxelizeCUDA.apply(*inputs, ranges, ids, s["half"], case["tile"], *shape)
        return (ranges, vr.detach(), vi.detach(), *torch.autograd.grad([vr, vi], inputs, s["grad"]))
    if kind == "batch":
        vols = s["vox"](s["sets"])
        leaves = [t for ps in s["sets"] for t in ps]
        return ([v.detach() for v in vols], torch.autograd.grad(vols, leaves, s["grads"]))
    if kind == "sense":
        loss = sense.sense_data_term(s["vol"], s["S"], s["mask"], s["ku"], s["ws"])
        loss = loss + 0.1 * sense.magnitude_tv_fused(s["vol"], s["ws_tv"])
        return (loss.detach(), *torch.autograd.grad(loss, s["vol"]))
    if kind == "mlp":
        out, cache = s["net"].forward(s["x"])
        return (out, s["net"].backward(cache, s["dout"])) if case["backward"] else out
    pos, log_scales, rot, dr, di = s["leaves"]
    vol = s["vox"](pos, torch.exp(log_scales), rot, torch.complex(dr, di))
    loss = sense.sense_data_term(vol, s["S"], s["mask"], s["ku"], s["ws"])
    return (loss.detach(), vol.detach(), *torch.autograd.grad(loss, s["leaves"]))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _vox_work(n, voxels, sigma, backward):
    """Parameters in, volume out (and the upstream gradient in, the gradients out); 15 operations for
    each voxel within three sigma of a Gaussian forward, 33 backward."""
    included = n * min(voxels, 36.0 * math.pi * sigma ** 3)
    return {"bytes": 56 * n + 8 * voxels + (8 * voxels + 56 * n if backward else 0),
            "flops": included * (48 if backward else 15)}


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        rows, macs = case["rows"], 256 * 256 * 2 + 256 * 16
        bytes_ = rows * (512 + 64) + 4 * macs
        return {"bytes": bytes_ + (rows * 64 + 4 * macs if case["backward"] else 0),
                "flops": 2 * rows * macs + (2 * rows * (macs + 256 * 256 + 256 * 16) if case["backward"] else 0)}
    if kind == "batch":
        parts = [_vox_work(n, v[0] * v[1] * v[2], _spacing_sigma(n, v), True) for v, n in _batch_shapes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    voxels = case["d"] * case["h"] * case["w"]
    fft = 2 * case["coils"] * 5 * voxels * math.log2(max(voxels, 2))
    data = voxels * (8 * 2 + 4 + 16 * case["coils"])
    if kind == "sense":
        return {"bytes": data, "flops": fft + 40 * voxels * case["coils"]}
    sigma = 1.5 if case["spread"] == "uniform" else _spacing_sigma(case["n"], (case["d"], case["h"], case["w"]))
    w = _vox_work(case["n"], voxels, sigma, kind != "render")
    if kind == "iter":
        w = {"bytes": 112 * case["n"] + data, "flops": w["flops"] + fft + 20 * voxels * case["coils"]}
    return w


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------

class _Exact:
    """The voxelizer in 64 bits: for each Gaussian every voxel of its tile box with m <= 9."""

    CELLS = 1 << 24

    def __init__(self, center, cov_inv, radius, shape, tile):
        self.shape = shape
        size = torch.tensor(shape, dtype=torch.float64, device=DEV)
        half = 0.5 * size
        top = (size - 1).expand_as(center)
        lo = torch.minimum(torch.clamp(torch.floor(center - radius[:, None]), min=0), top)
        hi = torch.minimum(torch.clamp(torch.ceil(center + radius[:, None]), min=0), top)
        lo, hi = torch.floor(lo / tile) * tile, torch.minimum(torch.floor(hi / tile) * tile + tile, size) - 1
        self.q = cov_inv / (half[:, None] * half[None, :])
        reach = 3 * torch.sqrt(torch.diagonal(torch.linalg.inv(self.q), dim1=-2, dim2=-1)) + 1e-6
        lo = torch.maximum(lo, torch.ceil(center - reach))
        hi = torch.minimum(hi, torch.floor(center + reach))
        self.center, self.half = center, half
        self.first, self.count = lo, torch.clamp(hi - lo + 1, min=0)
        self.order = torch.argsort(self.count.prod(-1))

    def chunks(self):
        """(Gaussian, flat voxel, offset [3], weight) of the included pairs, a bounded number at a time."""
        d, h, w = self.shape
        cells = self.count.prod(-1)[self.order].cpu()
        n, at = self.order.numel(), 0
        while at < n:
            # Gaussians sorted by window size: take as many as fit when all are as large as the last
            lo, hi = 1, n - at
            while lo < hi:
                mid = (lo + hi + 1) // 2
                if float(cells[at + mid - 1]) * 1.5 * mid <= self.CELLS:
                    lo = mid
                else:
                    hi = mid - 1
            ids = self.order[at:at + lo]
            at += lo
            k = [int(x) for x in self.count[ids].max(0).values]
            if min(k) == 0:
                continue
            f, c, q = self.first[ids], self.count[ids], self.q[ids]
            step = [torch.arange(x, dtype=torch.float64, device=DEV) for x in k]
            e = [f[:, a, None] + step[a] - self.center[ids][:, a, None] for a in range(3)]
            e0, e1, e2 = e[0][:, :, None, None], e[1][:, None, :, None], e[2][:, None, None, :]
            qq = [[q[:, a, b, None, None, None] for b in range(3)] for a in range(3)]
            m = (qq[0][0] * e0 * e0 + 2 * qq[0][1] * e0 * e1 + qq[1][1] * e1 * e1
                 + 2 * (qq[0][2] * e0 + qq[1][2] * e1) * e2 + qq[2][2] * e2 * e2)
            ok = [step[a][None] < c[:, a, None] for a in range(3)]
            keep = (m <= 9) & ok[0][:, :, None, None] & ok[1][:, None, :, None] & ok[2][:, None, None, :]
            gi, i, j, l = torch.nonzero(keep, as_tuple=True)
            weight = torch.exp(-0.5 * m[keep])
            del m, keep
            fl = f.long()
            flat = ((fl[gi, 0] + i) * h + fl[gi, 1] + j) * w + fl[gi, 2] + l
            yield ids[gi], flat, (e[0][gi, i], e[1][gi, j], e[2][gi, l]), weight

    def forward(self, dr, di):
        d, h, w = self.shape
        vol = [torch.zeros(d * h * w, dtype=torch.float64, device=DEV) for _ in range(2)]
        for g, flat, _, weight in self.chunks():
            vol[0].index_add_(0, flat, weight * dr[g])
            vol[1].index_add_(0, flat, weight * di[g])
        return vol

    def backward(self, dr, di, gr, gi):
        """Gradients of (center, cov_inv, density re, density im)."""
        n = self.center.shape[0]
        mom = torch.zeros(11, n, dtype=torch.float64, device=DEV)
        for g, flat, e, weight in self.chunks():
            r, i = weight * gr[flat], weight * gi[flat]
            a = -0.5 * (r * dr[g] + i * di[g])
            rows = [r, i] + [a * x for x in e] + [a * e[j] * e[k] for j in range(3) for k in range(j, 3)]
            for k, x in enumerate(rows):
                mom[k].index_add_(0, g, x)
        g_center = -2 * torch.einsum("nab,bn->na", self.q, mom[2:5])
        second = mom[5:][[0, 1, 2, 1, 3, 4, 2, 4, 5]].t().view(n, 3, 3)
        return g_center, second / (self.half[:, None] * self.half[None, :]), mom[0], mom[1]


def _vox_exact(params, shape, tile, grad):
    """Volume and, with an upstream gradient (or a function of the volume that gives it), the
    gradients of positions, scales, rotations, density re / im."""
    params = [p.double() for p in params]
    leaves = [p.clone().requires_grad_(True) for p in params[:3]]
    center, cov_inv, radius, _ = _reference_preprocess([*leaves, None, None], shape)
    ex = _Exact(center.detach(), cov_inv.detach(), radius.detach(), shape, tile)
    vr, vi = ex.forward(params[3], params[4])
    vol = torch.complex(vr, vi).view(shape)
    if grad is None:
        return vol, None
    g = grad(vol) if callable(grad) else grad.to(torch.complex128)
    gc, gm, gdr, gdi = ex.backward(params[3], params[4], g.real.reshape(-1), g.imag.reshape(-1))
    return vol, [*torch.autograd.grad([center, cov_inv], leaves, [gc, gm]), gdr, gdi]


def _data_term(vol, S, mask, ku):
    r = _fft3c(vol.unsqueeze(0) * S.to(torch.complex128)) * mask.double() - ku.to(torch.complex128)
    return r.real.square().sum() + r.imag.square().sum()


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        x, wb, dout = _inputs(case, seed)
        p = [t.bfloat16().double() for t in wb[:3]] + [t.double() for t in wb[3:]]
        p = [t.requires_grad_(True) for t in p]
        y = x.double()
        for k in range(2):
            y = torch.nn.functional.gelu(y @ p[k].t() + p[3 + k], approximate="tanh")
        out = y @ p[2].t() + p[5]
        return (out.detach(), list(torch.autograd.grad(out, p, dout.double()))) if case["backward"] else out.detach()
    if kind == "batch":
        got = [_vox_exact(p, s, 8, g) for (s, _), (p, g) in zip(_batch_shapes(case), _inputs(case, seed))]
        return [v for v, _ in got], [t for _, q in got for t in (*q[:3], torch.complex(q[3], q[4]))]
    shape = (case["d"], case["h"], case["w"])
    if kind == "sense":
        vol, S, mask, ku = _inputs(case, seed)
        x = vol.to(torch.complex128).requires_grad_(True)
        m = x.abs()
        tv = sum(torch.diff(m, dim=a).abs().sum() for a in range(3))
        loss = _data_term(x, S, mask, ku) + 0.1 * tv
        return (loss.detach(), *torch.autograd.grad(loss, x))
    params, *rest = _inputs(case, seed)
    if kind == "compat":
        center, cov_inv, radius, _ = _reference_preprocess(params, shape)
        g = rest[0].to(torch.complex128)
        ex = _Exact(center.double(), cov_inv.double(), radius.double(), shape, case["tile"])
        dr, di = params[3].double(), params[4].double()
        return (None, *ex.forward(dr, di),
                *ex.backward(dr, di, g.real.reshape(-1).contiguous(), g.imag.reshape(-1).contiguous()))
    if kind == "iter":
        S, mask, ku = rest
        params[1] = torch.exp(torch.log(params[1]).double())  # the call is given log-scales
        said = []

        def upstream(vol):
            v = vol.clone().requires_grad_(True)
            loss = _data_term(v, S, mask, ku)
            said.append(loss.detach())
            return torch.autograd.grad(loss, v)[0]

        vol, q = _vox_exact(params, shape, case["tile"], upstream)
        return (said[0], vol, q[0], q[1] * params[1], *q[2:])
    vol, q = _vox_exact(params, shape, case["tile"], None if kind == "render" else rest[0])
    return vol if q is None else (vol, *q[:3], torch.complex(q[3], q[4]))
