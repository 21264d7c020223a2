"""The calls that a user of this package has it do, as cases that can be timed and checked.

Each case is one call (or one short chain of calls) of the public entry points on
inputs of a stated size: ``prepare`` makes what a program has in hand before the call
(data, trajectory, plan), ``run`` makes the call, ``exact`` gives its value in 64 bits
with plain torch and numpy, and ``work`` the bytes and operations that the call cannot do
without.  ``listed`` names the sizes that stand for the use, from a single-slice 2D radial
frame to a 3D acquisition of eight million samples on 32 coils; ``draw`` gives others of
the same ranges.
"""

import math

import numpy as np
import torch

import pyfourier_b200 as pf

GOLDEN = math.pi / ((1 + 5 ** 0.5) / 2)


def _nufft(name, op, shape, coils, views, samples, **kw):
    """A NUFFT call on a plan: ``op`` "fwd", "adj" or "both" (the normal operator)."""
    c = {"kind": "nufft", "op": op, "nz": shape[0] if len(shape) == 3 else 0, "ny": shape[-2], "nx": shape[-1],
         "coils": coils, "frames": 1, "views": views, "samples": samples, "traj": "radial", "width": 4,
         "osf": 1.25, "rank": 0, "segments": 0, "ragged": False, "weighted": False}
    c.update(kw)
    return {"name": name, **c} if name else c


def _train(name, n, coils, images, views, samples, osf):
    c = {"kind": "train", "nz": 0, "ny": n, "nx": n, "coils": coils, "images": images, "views": views,
         "samples": samples, "frames": 1, "traj": "spiral", "width": 4, "osf": osf, "rank": 0, "segments": 0,
         "ragged": False}
    return {"name": name, **c} if name else c


def _toeplitz(name, shape, coils, frames, rank, views, samples, traj):
    c = {"kind": "toeplitz", "nz": shape[0] if len(shape) == 3 else 0, "ny": shape[-2], "nx": shape[-1],
         "coils": coils, "frames": frames, "rank": rank, "views": views, "samples": samples, "traj": traj,
         "segments": 0, "ragged": False}
    return {"name": name, **c} if name else c


def _spfft(name, n, coils, share):
    c = {"kind": "spfft", "nz": n, "ny": n, "nx": n, "coils": coils, "share": share}
    return {"name": name, **c} if name else c


def _cgram(name, shape, slices, frames, rank):
    c = {"kind": "cgram", "nz": 0, "ny": shape[0], "nx": shape[1], "slices": slices, "frames": frames, "rank": rank}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one real-time 2D frame, 8 coils: a call whose latency and launches count
        _nufft("radial2d_fwd", "fwd", (128, 128), 8, 201, 256, osf=2.0),
        # the same frame gridded with its density weights (each displayed frame of a real-time scan)
        _nufft("radial2d_adj", "adj", (128, 128), 8, 201, 256, osf=2.0, weighted=True),
        # a full 3D golden-means acquisition, 32 coils: the predicted k-space of a reconstruction step
        _nufft("radial3d_fwd", "fwd", (200, 200, 200), 32, 20000, 400),
        # the same acquisition gridded (the right-hand side, and every gradient of a reconstruction)
        _nufft("radial3d_adj", "adj", (200, 200, 200), 32, 20000, 400, weighted=True),
        # an odd, anisotropic volume on few (compressed) coils with the wider, more accurate kernel:
        # the normal operator of one conjugate-gradient step
        _nufft("radial3d_odd", "both", (93, 111, 120), 5, 4001, 187, width=6, osf=1.5),
        # dynamic radial with off-resonance segments: 64 frames of uneven length in one call, forward
        # and adjoint
        _nufft("b0_dynamic", "both", (192, 192), 12, 55, 256, frames=64, segments=8, ragged=True),
        # a subspace reconstruction's right-hand side: 48 rotated spiral frames onto 4 coefficients
        _nufft("subspace_adj", "adj", (220, 220), 16, 16, 2048, frames=48, traj="spiral", rank=4, weighted=True),
        # one step of trajectory learning: the plan of the step's trajectory, forward, adjoint, and the
        # gradients with respect to the images and the trajectory
        _train("spiral_training", 256, 8, 32, 16, 4096, 2.0),
        # the Toeplitz normal operator of that subspace reconstruction (one call per iteration)
        _toeplitz("toeplitz2d", (220, 220), 16, 48, 4, 16, 2048, "spiral"),
        # the Toeplitz normal operator of a static 3D reconstruction
        _toeplitz("toeplitz3d", (128, 128, 128), 8, 1, 0, 8000, 256, "radial"),
        # Cartesian 3D with a quarter of the phase encodes: sampled FFT and its adjoint
        _spfft("cartesian3d", 128, 32, 0.25),
        # the Cartesian normal operator with a temporal subspace, one plane per readout position
        _cgram("cartesian_gram", (256, 256), 256, 48, 4),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _size(rng, a, b):
    """An image extent: an even one as protocols have it, or any."""
    n = _log(rng, a, b)
    return n if rng.random() < 0.4 else max(a, n // 4 * 4)


def _shape2(rng, a, b):
    n = _size(rng, a, b)
    return (n, n) if rng.random() < 0.6 else (n, _size(rng, a, b))


def draw(rng):
    kind = rng.choice(["2d", "2d", "3d", "3d", "b0", "subspace", "train", "toeplitz2d", "toeplitz3d", "spfft",
                       "cgram"])
    osf, width = rng.choice([(1.25, 4), (1.25, 4), (2.0, 4), (1.5, 6)])
    op = rng.choice(["fwd", "adj", "both"])
    top = work(listed()[2])
    while True:
        if kind == "2d":
            s = _shape2(rng, 64, 288)
            c = _nufft(None, op, s, _log(rng, 1, 32), _log(rng, 16, 600), _log(rng, 128, 640), osf=osf, width=width,
                       weighted=rng.random() < 0.5, traj=rng.choice(["radial", "spiral"]))
        elif kind == "3d":
            n = _size(rng, 48, 200)
            s = (n, n, n) if rng.random() < 0.5 else (_size(rng, 32, 160), n, _size(rng, 48, 200))
            c = _nufft(None, op, s, _log(rng, 1, 32), _log(rng, 1000, 20000), _log(rng, 64, 400), osf=osf,
                       width=width, weighted=rng.random() < 0.5)
        elif kind == "b0":
            c = _nufft(None, op, _shape2(rng, 96, 224), _log(rng, 2, 16), _log(rng, 16, 55), _log(rng, 128, 384),
                       frames=_log(rng, 4, 64), segments=rng.choice([4, 6, 8]), ragged=True)
        elif kind == "subspace":
            c = _nufft(None, op, _shape2(rng, 96, 256), _log(rng, 4, 24), rng.choice([4, 8, 16]),
                       _log(rng, 512, 3000), frames=_log(rng, 12, 64), traj="spiral", rank=rng.choice([3, 4, 5]),
                       weighted=rng.random() < 0.5)
        elif kind == "train":
            c = _train(None, _size(rng, 96, 256), _log(rng, 1, 8), _log(rng, 1, 32), rng.choice([8, 16]),
                       _log(rng, 512, 4096), rng.choice([1.25, 2.0]))
        elif kind == "toeplitz2d":
            c = _toeplitz(None, _shape2(rng, 96, 256), _log(rng, 1, 24), _log(rng, 8, 48), rng.choice([0, 3, 4, 5]),
                          8, _log(rng, 512, 2048), "spiral")
            if not c["rank"]:  # a static scan: one frame
                c["frames"] = 1
        elif kind == "toeplitz3d":
            n = _size(rng, 48, 144)
            s = (n, n, n) if rng.random() < 0.5 else (_size(rng, 32, 96), n, _size(rng, 48, 144))
            c = _toeplitz(None, s, _log(rng, 1, 12), 1, 0, _log(rng, 1000, 8000), _log(rng, 64, 256), "radial")
        elif kind == "spfft":
            c = _spfft(None, _size(rng, 48, 160), _log(rng, 4, 32), rng.choice([0.125, 0.25, 0.5]))
        else:
            c = _cgram(None, _shape2(rng, 96, 320), _log(rng, 8, 256), _log(rng, 12, 48), rng.choice([0, 3, 4, 5]))
            if not c["rank"]:
                c["frames"] = 1
        w = work(c)
        if w["bytes"] <= top["bytes"] and w["flops"] <= top["flops"] and (
                kind != "3d" or c["osf"] ** 3 * c["nz"] * c["ny"] * c["nx"] * c["coils"] < 5.2e8):
            return c


# ------------------------------------------------------------------------ trajectories
def _shape(c):
    return ((c["nz"],) if c["nz"] else ()) + (c["ny"], c["nx"])


def _frame_views(c):
    """Views of every frame: the same, or between a tenth and all of them (a gated scan)."""
    if not c["ragged"]:
        return [c["views"]] * c["frames"]
    rng = np.random.default_rng(c["views"])
    return [int(v) for v in rng.integers(max(1, c["views"] // 10), c["views"] + 1, c["frames"])]


def _frames(c):
    """One (views, samples, ndim) float32 tensor per frame, cycles per field of view, (x, y[, z])."""
    shape, ns = _shape(c), c["samples"]
    ext = torch.tensor(shape[::-1], dtype=torch.float64, device="cuda")
    out, first = [], 0
    for f, nv in enumerate(_frame_views(c)):
        v = torch.arange(first, first + nv, dtype=torch.float64, device="cuda")
        if c["traj"] == "spiral":
            tau = torch.linspace(0, 1, ns, dtype=torch.float64, device="cuda")
            r = 0.496 * tau ** 1.5
            th = 24 * math.pi * tau[None] + (2 * math.pi * (v - first) / nv + f * math.pi * (3 - 5 ** 0.5))[:, None]
            k = torch.stack([r * torch.cos(th), r * torch.sin(th)], -1)
        else:
            r = (torch.arange(ns, dtype=torch.float64, device="cuda") - ns // 2) / ns
            if len(shape) == 2:
                d = torch.stack([torch.cos(v * GOLDEN), torch.sin(v * GOLDEN)], -1)
            else:
                z, az = torch.remainder(v * 0.4656, 1.0), 2 * math.pi * torch.remainder(v * 0.6823, 1.0)
                s = torch.sqrt(1 - z * z)
                d = torch.stack([s * torch.cos(az), s * torch.sin(az), z], -1)
            k = d[:, None, :] * r[None, :, None]
        out.append((k * ext).to(torch.float32))
        first += nv
    return out


def _coord(c):
    """The trajectory as the plan takes it: one array, or a list of frames of uneven length."""
    fr = _frames(c)
    return fr if c["ragged"] else (torch.stack(fr) if c["frames"] > 1 else fr[0])


def _weights(c, coord):
    """Density weights: a ramp over the radius."""
    r = torch.linalg.norm(coord, dim=-1)
    return (r + 0.5) / (r.max() + 0.5)


def _basis(c):
    """(frames, rank) orthonormal temporal basis: the SVD of exponential recovery curves."""
    rng = np.random.default_rng(0)
    t = np.linspace(10.0, 3000.0, c["frames"])
    curves = 1 - 2 * np.exp(-t[None, :] / rng.uniform(200.0, 2000.0, 500)[:, None])
    _, _, vh = np.linalg.svd(curves, full_matrices=False)
    return torch.as_tensor(vh[:c["rank"]].T.astype(np.complex64), device="cuda")


def _field(c):
    """A smooth off-resonance map of up to 200 Hz and the sampling raster of a 5 ms readout."""
    yy, xx = np.mgrid[:c["ny"], :c["nx"]]
    yy, xx = yy / c["ny"] - 0.5, xx / c["nx"] - 0.5
    rng = np.random.default_rng(0)
    f = np.zeros((c["ny"], c["nx"]))
    for _ in range(6):
        m, s = rng.uniform(-0.3, 0.3, 2), rng.uniform(0.1, 0.3)
        f += rng.uniform(-1, 1) * np.exp(-((xx - m[0]) ** 2 + (yy - m[1]) ** 2) / (2 * s ** 2))
    return (f / np.abs(f).max() * 200.0).astype(np.float32), 5e-3 / c["samples"]


# ------------------------------------------------------------------------------- data
def _randn(g, *shape):
    return torch.complex(torch.randn(shape, generator=g, device="cuda"), torch.randn(shape, generator=g, device="cuda"))


def _images(g, lead, shape):
    """(*lead, *shape) complex64: ellipsoids of several intensities under smooth coil profiles, the
    contrasts of one coil (the second leading axis) of different weight, and a little noise."""
    ax = [(torch.arange(n, device="cuda", dtype=torch.float32) - n // 2) / n for n in shape]
    grid = torch.meshgrid(*ax, indexing="ij")
    obj = torch.zeros(shape, dtype=torch.complex64, device="cuda")
    for _ in range(8):
        m = (torch.rand(len(shape), generator=g, device="cuda") - 0.5) * 0.6
        r = 0.05 + 0.25 * torch.rand(len(shape), generator=g, device="cuda")
        a = _randn(g, 1)
        obj += a * (sum(((x - m[i]) / r[i]) ** 2 for i, x in enumerate(grid)) <= 1)
    out = torch.empty((*lead, *shape), dtype=torch.complex64, device="cuda")
    for b in range(lead[0]):
        m = 0.8 * (torch.rand(len(shape), generator=g, device="cuda") - 0.5)
        prof = torch.exp(-sum((x - m[i]) ** 2 for i, x in enumerate(grid)) / 0.32)
        w = _randn(g, *lead[1:], *([1] * len(shape)))
        out[b] = w * (prof * obj)
        out[b] += 0.01 * _randn(g, *out[b].shape)
    return out


def _kspace(g, coils, coord):
    """(coils, ...) complex64 with the decay over the radius that images of objects have."""
    r = torch.linalg.norm(coord, dim=-1)
    return _randn(g, coils, *r.shape) / (1 + r / 8) ** 1.5


def _image_shape(c):
    n = c["rank"] or c["frames"]
    return (c["coils"],) + ((n,) if c["rank"] or c["frames"] > 1 else ()), _shape(c)


def _inputs(c, seed):
    """The tensors of a case, made from the seed alone (the trajectory belongs to the protocol)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    d = {}
    if c["kind"] == "cgram":
        ky, kx = np.meshgrid(*[np.arange(n) - n // 2 for n in _shape(c)], indexing="ij")
        p = np.minimum(1.0, 0.02 + 0.5 * np.exp(-(ky ** 2 + kx ** 2) / (2 * 12.0 ** 2)))
        m = np.random.default_rng(0).random((c["frames"], *_shape(c))) < p[None]
        d["mask"] = torch.as_tensor(m.astype(np.float32), device="cuda")
        lead = (c["slices"],) + ((c["rank"],) if c["rank"] else ())
        d["x"] = _images(g, lead, _shape(c))
    elif c["kind"] == "spfft":
        n = c["nx"]
        pe = torch.as_tensor(np.random.default_rng(0).choice(n * n, max(1, int(c["share"] * n * n)), replace=False),
                             device="cuda")
        kx = torch.arange(n, device="cuda")
        idx = torch.stack(torch.broadcast_tensors(kx[None, :], (pe % n)[:, None], (pe // n)[:, None]), -1)
        d["index"] = idx.to(torch.float32)
        d["x"] = _images(g, (c["coils"],), _shape(c))
    elif c["kind"] == "train":
        k = _coord(c)
        d["coord"] = k + 0.1 * (torch.rand(k.shape, generator=g, device="cuda") - 0.5)  # a learned trajectory
        d["x"] = _images(g, (c["images"], c["coils"]), _shape(c))
    elif c["kind"] == "toeplitz":
        d["coord"] = _coord(c)
        d["weight"] = _weights(c, d["coord"])
        lead, shape = _image_shape(c)
        d["x"] = _images(g, lead, shape)
    else:
        d["coord"] = _coord(c)
        flat = torch.cat([f.reshape(-1, f.shape[-1]) for f in d["coord"]]) if c["ragged"] else d["coord"]
        lead, shape = _image_shape(c)
        if c["op"] == "adj":
            d["y"] = _kspace(g, c["coils"], flat)
        else:
            d["x"] = _images(g, lead, shape)
        if c["weighted"]:
            d["weight"] = _weights(c, flat)
    if c.get("rank"):
        d["basis"] = _basis(c)
    return d


def prepare(case, seed):
    c, s = case, _inputs(case, seed)
    s["case"] = c
    if c["kind"] == "nufft":
        kw = {}
        if c["segments"]:
            f, dt = _field(c)
            kw = {"zmap": torch.as_tensor(f, device="cuda"), "L": c["segments"], "nbins": 40, "dt": dt}
        s["plan"] = pf.plan_nufft(s["coord"], _shape(c), width=c["width"], oversamp=c["osf"], device="cuda:0", **kw)
    elif c["kind"] == "train":
        s["coord"].requires_grad_(True)
        s["x"].requires_grad_(True)
    elif c["kind"] == "toeplitz":
        s["gram"] = pf.plan_spgram(s["coord"], _shape(c), basis=s.get("basis"), weight=s["weight"], device="cuda:0")
    elif c["kind"] == "spfft":
        s["plan"] = pf.plan_spfft(s["index"], _shape(c), device="cuda:0")
    else:
        s["gram"] = pf.plan_gram(s["mask"], _shape(c), basis=s.get("basis"), device="cuda:0")
    return s


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "toeplitz":
        return pf.sparse_gram(s["x"], s["gram"])
    if c["kind"] == "cgram":
        return pf.gram(s["x"], s["gram"])
    if c["kind"] == "spfft":
        y = pf.sparse_fftn(s["x"], plan=s["plan"])
        return y, pf.sparse_ifftn(y, plan=s["plan"])
    if c["kind"] == "train":
        x, k = s["x"], s["coord"]
        plan = pf.plan_nufft(k.detach(), _shape(c), width=c["width"], oversamp=c["osf"])
        y = pf.nufft(x, k, nufft_plan=plan, norm="ortho")
        z = pf.nufft_adj(y, k, nufft_plan=plan, norm="ortho")
        loss = torch.sum(torch.abs(z - x) ** 2)
        gx, gk = torch.autograd.grad(loss, (x, k))
        return loss.detach(), gx, gk
    kw = {"nufft_plan": s["plan"], "basis": s.get("basis")}
    if c["op"] == "adj":
        return pf.nufft_adj(s["y"], weight=s.get("weight"), **kw)
    y = pf.nufft(s["x"], **kw)
    if c["op"] == "fwd":
        return y
    return y, pf.nufft_adj(y, weight=s.get("weight"), **kw)


# ------------------------------------------------------------------------------- work
def work(case):
    """Inputs read once and outputs written once, and the operations of the transform (5 n log2 n per
    complex point) and of the sample sums (4 per tap and complex value)."""
    c = case
    shape = _shape(c)
    vol = math.prod(shape)
    fft = lambda dims: 5.0 * math.prod(dims) * sum(math.log2(n) for n in dims)  # noqa: E731
    if c["kind"] == "cgram":
        planes = c["slices"] * max(1, c["rank"])
        k = max(1, c["rank"])
        return {"bytes": 16.0 * planes * vol + 8.0 * k * k * vol, "flops": planes * (2 * fft(shape) + 8.0 * k * vol)}
    if c["kind"] == "toeplitz":
        os = [2 * n for n in shape]
        k = max(1, c["rank"])
        planes = c["coils"] * k * (1 if c["rank"] else c["frames"])
        return {"bytes": 16.0 * planes * vol + 8.0 * k * k * math.prod(os),
                "flops": planes * (2 * fft(os) + 8.0 * k * math.prod(os))}
    if c["kind"] == "spfft":
        m = max(1, int(c["share"] * c["nx"] * c["nx"])) * c["nx"]
        return {"bytes": c["coils"] * (16.0 * vol + 16.0 * m) + 12.0 * m, "flops": 2.0 * c["coils"] * fft(shape)}
    nd = len(shape)
    os = [math.ceil(c["osf"] * n) for n in shape]
    m = sum(_frame_views(c)) * c["samples"]
    taps = 4.0 * c["width"] ** nd
    if c["kind"] == "train":
        ch = c["coils"] * c["images"]
        # images, gradients, trajectory; forward, adjoint and the gradients of both
        return {"bytes": 16.0 * ch * vol + 8.0 * nd * m, "flops": ch * (6 * fft(os) + (4 + 2 * (1 + nd)) * taps * m)}
    ch = c["coils"] * max(1, c["segments"])
    planes = ch * (c["rank"] or c["frames"])
    one = {"bytes": 8.0 * c["coils"] * ((c["rank"] or c["frames"]) * vol + m) + 4.0 * nd * m,
           "flops": planes * fft(os) + taps * ch * max(1, c["rank"]) * m}
    return {k: v * (2 if c["op"] == "both" else 1) for k, v in one.items()}


# ------------------------------------------------------------------------------ exact
def _beta(width, osf):
    w, o = np.int16(width), np.float32(osf)
    return float(np.float32(np.pi * (((w / o) * (o - 0.5)) ** 2 - 0.8) ** 0.5))


class _Grid:
    """The gridding NUFFT (Kaiser-Bessel kernel, oversampled grid, deapodisation) in 64 bits."""

    def __init__(self, coord, shape, width, osf):
        self.shape, self.width, self.beta = shape, width, _beta(width, osf)
        self.os = [int(np.ceil(np.float32(osf) * np.float32(n))) for n in shape]
        flat = coord.reshape(-1, coord.shape[-1])
        self.m = flat.shape[0]
        h, idx, val, scale = width / 2.0, [], [], 1.0
        for a, n, g in zip(range(len(shape)), shape[::-1], self.os[::-1]):
            # the grid position is stored in 32 bits (a plan does so), the rest is in 64
            f = float(np.float32(np.float32(g) / np.float32(n)))
            p = (flat[:, a].detach().float() * f + float(g // 2)).double()
            if flat.requires_grad:
                p = p + (flat[:, a] - flat[:, a].detach()) * f
            t = torch.ceil(p.detach() - h)[:, None] + torch.arange(width, device="cuda", dtype=torch.float64)
            u = (t - p[:, None]) / h
            q = 1 - u * u
            val.append(torch.where(q >= 0, torch.special.i0(self.beta * torch.sqrt(torch.where(q > 0, q, 1e-30))), 0.0))
            idx.append(torch.remainder(t, g).long())
            e = (math.ceil(-h) + np.arange(width)) / h
            scale *= float(np.sum(np.i0(self.beta * np.sqrt(np.maximum(0.0, 1 - e * e)))))
        self.idx, self.val, self.scale = idx, val, scale

    def taps(self):
        """Flat grid index and weight of every tap, one tap of all samples at a time."""
        nd, w = len(self.shape), self.width
        for t in range(w ** nd):
            i, v, f = 0, 1.0, 1
            for a in range(nd):
                e = t // w ** a % w
                i, v = i + self.idx[a][:, e] * f, v * self.val[a][:, e]
                f *= self.os[nd - 1 - a]
            yield i, v

    def apod(self, x):
        for a, (n, g) in enumerate(zip(self.shape[::-1], self.os[::-1])):
            i = torch.arange(n, dtype=torch.float64, device="cuda")
            r = torch.sqrt(self.beta ** 2 - (math.pi * self.width * (i - n // 2) / g) ** 2)
            r = torch.nan_to_num(r / torch.sinh(r) / (self.beta / math.sinh(self.beta)), nan=1.0)
            x = x * r.reshape([n] + [1] * a)
        return x

    def _axes(self):
        return tuple(range(1, 1 + len(self.shape)))

    def fwd(self, x, ortho=False):
        """(b, *shape) complex128 -> (b, samples)"""
        x = self.apod(x)
        for a, (n, g) in enumerate(zip(self.shape, self.os)):
            lo = max(g // 2 - n // 2, 0)
            z = [0, 0] * (len(self.shape) - 1 - a) + [lo, g - n - lo]
            x = torch.nn.functional.pad(x, z)
        ax = self._axes()
        k = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(x, ax), dim=ax, norm="ortho" if ortho else "backward"), ax)
        g = torch.view_as_real(k.reshape(k.shape[0], -1)).permute(1, 0, 2).reshape(-1, 2 * k.shape[0]).contiguous()
        y = 0
        for i, v in self.taps():
            y = y + g[i] * v[:, None]
        y = y.reshape(self.m, -1, 2).permute(1, 0, 2).contiguous()
        return torch.view_as_complex(y) / self.scale

    def adj(self, y, ortho=False):
        """(b, samples) complex128 -> (b, *shape)"""
        b = y.shape[0]
        r = torch.view_as_real(y).permute(1, 0, 2).reshape(self.m, 2 * b)
        g = torch.zeros((math.prod(self.os), 2 * b), dtype=torch.float64, device="cuda")
        for i, v in self.taps():
            g = g.index_add(0, i, r * v[:, None]) if r.requires_grad else g.index_add_(0, i, r * v[:, None])
        k = torch.view_as_complex(g.reshape(-1, b, 2).permute(1, 0, 2).contiguous()).reshape(b, *self.os)
        ax = self._axes()
        x = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(k / self.scale, ax), dim=ax, norm="ortho" if ortho else "backward"), ax)
        cut = tuple(slice(max(g // 2 - n // 2, 0), max(g // 2 - n // 2, 0) + n) for n, g in zip(self.shape, self.os))
        return self.apod(x[(slice(None), *cut)])


def _segments(field, dt, c):
    """Temporal and spatial coefficients of exp(-2 pi i f t) ~ sum_l B_l(t) C_l(r): a least-squares
    fit over the field's histogram."""
    t = (dt * np.arange(c["samples"], dtype=np.float32)).astype(np.float64)
    hk, edge = np.histogram(2 * math.pi * field.astype(np.float64).ravel(), bins=40)
    zk = 0.5j * (edge[1:] + edge[:-1])
    n = c["segments"]
    tl = np.linspace(0, n, n) / n * t[-1]
    w = np.diag(hk.astype(np.float64) ** 0.5)
    p = np.linalg.pinv(w @ np.exp(-tl[:, None] * zk[None, :]).T) @ w
    bt = p @ np.exp(-zk[:, None] * t[None, :])
    cr = np.exp(-tl[:, None, None] * (2j * math.pi * field.astype(np.float64))[None])
    return torch.as_tensor(bt, device="cuda"), torch.as_tensor(cr, device="cuda")


def _exact_nufft(c, d):
    frames, shape = _frames(c), _shape(c)
    grids = None if c["nz"] else [_Grid(f, shape, c["width"], c["osf"]) for f in frames]
    grids = grids or [_Grid(frames[0], shape, c["width"], c["osf"])]
    sizes = [g.m for g in grids]
    w = d["weight"].double().reshape(-1).split(sizes) if c["weighted"] else None
    seg = _segments(*_field(c), c) if c["segments"] else None
    bas = d["basis"].to(torch.complex128) if c["rank"] else None
    lead, _ = _image_shape(c)
    step = 4 if c["nz"] else c["coils"]
    fwd, adj = [], []
    for b in range(0, c["coils"], step):
        if c["op"] != "adj":
            x = d["x"][b:b + step].to(torch.complex128).reshape(-1, c["rank"] or c["frames"], *shape)
            ys = []
            for f, g in enumerate(grids):
                xf = torch.einsum("k,bk...->b...", bas[f], x) if c["rank"] else x[:, f]
                if seg is None:
                    ys.append(g.fwd(xf))
                else:
                    bt = seg[0].repeat(1, g.m // c["samples"])
                    ys.append(sum(bt[q] * g.fwd(seg[1][q] * xf) for q in range(c["segments"])))
            fwd.append(torch.cat(ys, 1))
        if c["op"] != "fwd":
            y = fwd[-1] if c["op"] == "both" else d["y"][b:b + step].to(torch.complex128).reshape(min(step, c["coils"] - b), -1)
            xs = 0 if c["rank"] else []
            for f, (g, yf) in enumerate(zip(grids, y.split(sizes, 1))):
                yf = yf * w[f] if w is not None else yf
                if seg is None:
                    xf = g.adj(yf)
                else:
                    bt = seg[0].conj().repeat(1, g.m // c["samples"])
                    xf = sum(seg[1][q].conj() * g.adj(bt[q] * yf) for q in range(c["segments"]))
                if c["rank"]:
                    xs = xs + bas[f].conj()[None, :, None, None] * xf[:, None]
                else:
                    xs.append(xf)
            xs = xs if c["rank"] else torch.stack(xs, 1)
            adj.append(xs.reshape(-1, *lead[1:], *shape))
    out = []
    if fwd:
        y = torch.cat(fwd)
        out.append(y if c["ragged"] else y.reshape(c["coils"], *((c["frames"],) if c["frames"] > 1 else ()), c["views"], c["samples"]))
    if adj:
        out.append(torch.cat(adj))
    return tuple(out) if c["op"] == "both" else out[0]


def _exact_train(c, d):
    shape = _shape(c)
    k = d["coord"].double().requires_grad_(True)
    x = d["x"].reshape(-1, *shape)
    loss, gk, gx = 0.0, 0.0, []
    for b in range(0, x.shape[0], 8):
        xb = x[b:b + 8].to(torch.complex128).requires_grad_(True)
        g = _Grid(k, shape, c["width"], c["osf"])
        r = torch.sum(torch.abs(g.adj(g.fwd(xb, True), True) - xb) ** 2)
        da, dk = torch.autograd.grad(r, (xb, k))
        loss, gk = loss + r.detach(), gk + dk
        gx.append(da)
    return loss, torch.cat(gx).reshape(d["x"].shape), gk


def _circulant(x, kern, os, rank):
    """Inverse FFT of the kernel times the FFT of the embedded images, cut back; x (b, [k,] *shape)."""
    nd = len(os)
    ax = tuple(range(-nd, 0))
    lo = [max(g // 2 - n // 2, 0) for n, g in zip(x.shape[-nd:], os)]
    z = []
    for a in range(nd - 1, -1, -1):
        z += [lo[a], os[a] - x.shape[a - nd] - lo[a]]
    f = torch.fft.fftn(torch.nn.functional.pad(x, z), dim=ax)
    f = torch.einsum("bj...,ij...->bi...", f, kern) if rank else f * kern
    y = torch.fft.ifftn(f, dim=ax)
    return y[(..., *(slice(a, a + n) for a, n in zip(lo, x.shape[-nd:])))]


def _exact_toeplitz(c, d):
    shape = _shape(c)
    nd, os = len(shape), [2 * n for n in shape]
    ax = tuple(range(-nd, 0))
    per = []
    coord = d["coord"].reshape(c["frames"], -1, nd)
    for f, w in zip(coord, d["weight"].double().reshape(c["frames"], -1)):
        per.append(_Grid(2 * f, os, 6, 1.25).adj(w.to(torch.complex128)[None])[0])
    per = torch.stack(per)
    if c["rank"]:
        bas = d["basis"].to(torch.complex128)
        psf = torch.einsum("fj,fi,f...->ij...", bas, bas.conj(), per)
    else:
        psf = per if c["frames"] > 1 else per[0]
    kern = torch.fft.fftn(torch.fft.ifftshift(psf, ax), dim=ax, norm="ortho")
    kern = kern / torch.mean(torch.abs(kern[kern != 0]))
    out = [_circulant(x[None].to(torch.complex128), kern, os, c["rank"]) for x in d["x"]]
    return torch.cat(out)


def _exact_spfft(c, d):
    n = c["nx"]
    i = d["index"].long()
    at = ((i[..., 2] * n + i[..., 1]) * n + i[..., 0]).reshape(-1)
    ax = (-3, -2, -1)
    ys, xs = [], []
    for x in d["x"]:
        k = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(x.to(torch.complex128), ax), dim=ax), ax).reshape(-1)
        y = k[at]
        g = torch.zeros_like(k)
        g[at] = y  # the phase encodes are drawn without repeats
        xs.append(torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(g.reshape(n, n, n), ax), dim=ax), ax))
        ys.append(y.reshape(i.shape[:-1]))
    return torch.stack(ys), torch.stack(xs)


def _exact_cgram(c, d):
    shape = _shape(c)
    m = torch.fft.ifftshift(d["mask"].to(torch.complex128), (-2, -1))
    if c["rank"]:
        bas = d["basis"].to(torch.complex128)
        kern = torch.einsum("fj,fi,f...->ij...", bas, bas.conj(), m)
    else:
        kern = m[0]
    return torch.cat([_circulant(x[None].to(torch.complex128), kern, list(shape), c["rank"]) for x in d["x"]])


def exact(case, seed):
    c, d = case, _inputs(case, seed)
    return {"nufft": _exact_nufft, "train": _exact_train, "toeplitz": _exact_toeplitz, "spfft": _exact_spfft,
            "cgram": _exact_cgram}[c["kind"]](c, d)
