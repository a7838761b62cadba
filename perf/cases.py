"""The work that users of pushpull_gb300 have it do, as timed cases.

Every case goes through the package's public entry points on data that is
already on the GPU: images and deformations of one registration, reconstruction
or resampling step.  A case is a dict of plain values:

    op            what is called (see ``run``)
    x, y, z       sample grid (the deformation's grid)
    ix, iy, iz    image grid
    ch, nb        channels, batch
    deg           spline degree of all three axes
    bnd           "circ", "dct2", "dst2" or "mixed" (circulant, DCT-II, DST-II along x, y, z)
    ext           extrapolate (1) or mask samples outside the image (0)
    amp           largest displacement of the deformation, in voxels
    fwhm          smoothness of the displacement field, in voxels
    scale         the sample grid is mapped onto the image grid and scaled by this about its centre
    volumes       number of volumes (op "batch" only)

Images are smoothed noise in [0, 1] (tissue-like contrast), cotangents of a
gradient are normal noise, deformations are the grid plus a smooth displacement.
"""
from __future__ import annotations

import math
import random

import torch

from __graft_entry__ import package

_BND = {"circ": (0, 0, 0), "dct2": (1, 1, 1), "dst2": (2, 2, 2), "mixed": (0, 1, 2)}


def _case(name, op, d, *, image=None, ch=1, nb=1, deg=3, bnd="dct2", ext=1, amp=5.0, fwhm=12.0, scale=1.0, volumes=0):
    i = image or d
    c = {"op": op, "x": d[0], "y": d[1], "z": d[2], "ix": i[0], "iy": i[1], "iz": i[2], "ch": ch, "nb": nb,
         "deg": deg, "bnd": bnd, "ext": ext, "amp": amp, "fwhm": fwhm, "scale": scale, "volumes": volumes}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the coarsest level of a registration pyramid: one pull and one push of a
        # tiny volume; the launch and the host path count
        _case("level_32", "normal", (32, 32, 32), amp=1.5, fwhm=8.0),
        # trilinear pull and push of a small periodic volume, samples outside masked
        _case("linear_64", "normal", (64, 64, 64), deg=1, bnd="circ", ext=0, amp=2.0, fwhm=8.0),
        # nearest-neighbour resampling of a label volume on an odd 1 mm template grid
        _case("labels_181", "labels", (181, 217, 181), deg=0, amp=3.0),
        # the headline: cubic pull of one volume ...
        _case("pull_192", "pull", (192, 192, 192)),
        # ... and its adjoint
        _case("push_192", "push", (192, 192, 192)),
        # rigid-plus-zoom resampling and its adjoint (super-resolution's forward model)
        _case("affine_192", "affine", (192, 192, 192), amp=0.0),
        # spatial gradients and their adjoint on an odd 1 mm template grid
        _case("gradient_181", "gradient", (181, 217, 181), amp=3.0),
        # a registration step by automatic differentiation: a pull and its backward
        # pass, two channels on an odd 1.5 mm template grid
        _case("backward_121", "backward", (121, 145, 121), ch=2, deg=2, amp=3.0),
        # the same as the fused least-squares step, mixed boundary conditions
        _case("fused_160", "fused", (160, 192, 160), deg=2, bnd="mixed", amp=3.0),
        # diffeomorphic shooting: the exponential of a velocity field (eight trilinear
        # self-compositions of three channels)
        _case("exp_128", "exp", (128, 128, 128), ch=3, deg=1, amp=8.0),
        # a batch of uneven volumes, pulled and pushed back by one plan
        _case("batch_8", "batch", (128, 128, 96), amp=3.0, volumes=8),
        # the largest: three channels pushed into a quarter of the field of view
        # (many samples per voxel)
        _case("contract_256", "push", (256, 256, 256), ch=3, amp=3.0, scale=0.25),
    ]


def draw(rng: random.Random):
    op = rng.choice(["normal", "normal", "pull", "push", "push", "labels", "affine", "gradient", "backward", "fused",
                     "exp", "batch"])
    ch = 3 if op == "exp" else rng.choice([1, 1, 1, 2, 3])
    nb = rng.choice([1, 1, 1, 2]) if op not in ("exp", "batch", "affine") else 1
    most = {"exp": 2.5e6, "batch": 2.0e6, "gradient": 7.5e6}.get(op, 9.0e6) / (1 if op == "exp" else ch * nb)
    while True:
        d = tuple(int(round(math.exp(rng.uniform(math.log(28), math.log(240))))) for _ in range(3))
        if d[0] * d[1] * d[2] <= most:
            break
    image = d
    if op in ("normal", "pull", "push", "affine", "gradient") and rng.random() < 0.3:
        image = tuple(max(24, min(240, int(round(n * rng.uniform(0.7, 1.4))))) for n in d)
    deg = {"labels": 0, "exp": 1}.get(op, rng.choice([1, 2, 2, 3, 3, 3, 4]))
    scale = 1.0
    if op == "push" and rng.random() < 0.35:
        scale = round(rng.uniform(0.25, 1.0), 3)
    return _case("", op, d, image=image, ch=ch, nb=nb, deg=deg, bnd=rng.choice(["circ", "dct2", "dct2", "dst2", "mixed"]),
                 ext=1 if op in ("fused", "backward", "exp", "batch") else rng.choice([1, 1, 1, 0]),
                 amp=0.0 if op == "affine" else round(rng.uniform(0.5, 5.0), 2), fwhm=round(rng.uniform(8.0, 16.0), 1),
                 scale=scale, volumes=rng.randint(3, 8) if op == "batch" else 0)


# ---- inputs -------------------------------------------------------------------
# Arrays are made as contiguous (..., z, y, x) tensors; ``_col`` views one as the
# package's column-major (x, y, z, ...) layout.
def _col(t):
    return t.permute(*range(t.dim() - 1, -1, -1))


def _smooth(v, fwhm):
    """Periodic Gaussian smoothing over the last three axes."""
    F = torch.fft.rfftn(v, dim=(-3, -2, -1))
    for ax in (-3, -2, -1):
        n = v.shape[ax]
        k = (torch.fft.rfftfreq if ax == -1 else torch.fft.fftfreq)(n, device=v.device)
        h = torch.exp(-2.0 * (math.pi * (fwhm / 2.3548) * k) ** 2)
        shape = [1, 1, 1]
        shape[ax] = -1
        F = F * h.view(shape)
    return torch.fft.irfftn(F, s=v.shape[-3:], dim=(-3, -2, -1))


def _image(g, ch, nb, d):
    v = torch.rand((nb, ch, d[2], d[1], d[0]), generator=g, device="cuda")
    return _smooth(v, 3.0).contiguous()


def _noise(g, shape):
    return torch.randn(shape, generator=g, device="cuda")


def _phi(g, nb, d, image, amp, fwhm, scale):
    """(nb, 3, z, y, x) 1-based sample positions in the image grid."""
    u = _smooth(torch.randn((nb, 3, d[2], d[1], d[0]), generator=g, device="cuda"), fwhm)
    u *= amp / u.abs().max()
    for k in range(3):
        n, m = d[k], image[k]
        p = 1.0 + torch.arange(n, dtype=torch.float64, device="cuda") * ((m - 1) / max(n - 1, 1))
        p = 0.5 * (m + 1) + scale * (p - 0.5 * (m + 1))
        shape = [1, 1, 1]
        shape[2 - k] = -1
        u[:, k] += p.float().view(shape)
    return u.contiguous()


def _affine(rng, d, image):
    """1-based 4 x 4 map of the sample grid onto the image grid: small rotations, zooms and a shift."""
    th = [rng.uniform(-math.pi / 18, math.pi / 18) for _ in range(3)]
    c, s = [math.cos(t) for t in th], [math.sin(t) for t in th]
    R = [torch.tensor(m, dtype=torch.float64) for m in (
        [[1, 0, 0], [0, c[0], -s[0]], [0, s[0], c[0]]], [[c[1], 0, s[1]], [0, 1, 0], [-s[1], 0, c[1]]],
        [[c[2], -s[2], 0], [s[2], c[2], 0], [0, 0, 1]])]
    M = R[0] @ R[1] @ R[2] @ torch.diag(torch.tensor(
        [rng.uniform(0.9, 1.1) * (image[k] - 1) / max(d[k] - 1, 1) for k in range(3)], dtype=torch.float64))
    A = torch.eye(4, dtype=torch.float64)
    A[:3, :3] = M
    src = torch.tensor([0.5 * (n + 1) for n in d], dtype=torch.float64)
    dst = torch.tensor([0.5 * (n + 1) for n in image], dtype=torch.float64)
    A[:3, 3] = dst - M @ src + torch.tensor([rng.uniform(-3, 3) for _ in range(3)], dtype=torch.float64)
    return A.float()


def _batch_items(case):
    """Sizes, channels and degrees of a batch: fixed by the case, uneven."""
    r = random.Random(case["volumes"] * 1000003 + case["x"] * 10007 + case["y"] * 101 + case["z"])
    out = []
    for _ in range(case["volumes"]):
        d = tuple(max(20, int(n * r.uniform(0.4, 1.0))) for n in (case["x"], case["y"], case["z"]))
        out.append((d, r.randint(1, 3), r.choice([1, 2, 3])))
    return out


def _raw(case, seed):
    """The arrays of a case from its seed, as contiguous tensors."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    d, image = (case["x"], case["y"], case["z"]), (case["ix"], case["iy"], case["iz"])
    ch, nb, op = case["ch"], case["nb"], case["op"]
    dz = (d[2], d[1], d[0])
    if op == "batch":
        items = []
        for dd, c, deg in _batch_items(case):
            items.append((dd, c, deg, _image(g, c, 1, dd), _phi(g, 1, dd, dd, case["amp"], case["fwhm"], 1.0)))
        return {"items": items}
    if op == "exp":
        v = _smooth(_noise(g, (1, 3) + dz), case["fwhm"])
        return {"v": (v * (case["amp"] / v.abs().max())).contiguous()}
    if op == "affine":
        return {"f": _image(g, ch, nb, image), "A": _affine(random.Random(seed), d, image)}
    r = {"phi": _phi(g, nb, d, image, case["amp"], case["fwhm"], case["scale"])}
    if op == "push":
        r["g"] = _image(g, ch, nb, d)
    elif op == "labels":
        r["f"] = torch.floor(8.0 * torch.sigmoid(40.0 * (_image(g, ch, nb, image) - 0.5)))
    else:
        r["f"] = _image(g, ch, nb, image)
    if op == "gradient":
        r["g"] = _noise(g, (nb, ch, 3) + dz)
    elif op == "backward":
        r["g"] = _noise(g, (nb, ch) + dz)
    elif op == "fused":
        r["g"] = _image(g, ch, nb, d)
    return r


def _give(t, ch_axis=None):
    """A (nb, ch, ...) tensor as a user holds it: no batch axis when there is one
    volume, and no channel axis when there is one channel."""
    if t.shape[0] == 1:
        t = t[0]
        if ch_axis is not None and t.shape[0] == 1:
            t = t[0]
    return _col(t)


def prepare(case, seed):
    pp = package()
    raw = _raw(case, seed)
    op = case["op"]
    s = {"op": op, "pp": pp, "d0": (case["ix"], case["iy"], case["iz"]), "d1": (case["x"], case["y"], case["z"])}
    if op == "batch":
        items, keep = [], []
        for dd, c, deg, f, phi in raw["items"]:
            f, phi = _give(f, 1), _give(phi)
            f1, out = _give(torch.empty((1, c) + dd[::-1], device="cuda"), 1), _give(torch.empty((1, c) + dd[::-1], device="cuda"), 1)
            items.append({"f0": f, "phi": phi, "f1": f1, "out": out,
                          "sett": pp.Settings(deg, _BND[case["bnd"]], bool(case["ext"]))})
            keep.append((f1, out))
        from pushpull_gb300.batch import BatchPlan
        s["plan"], s["outs"] = BatchPlan(items), keep
        return s
    s["sett"] = pp.Settings(case["deg"], _BND[case["bnd"]], bool(case["ext"]))
    for k in ("f", "g"):
        if k in raw:
            s[k] = _give(raw[k], 1)
    if "phi" in raw:
        s["phi"] = _give(raw["phi"])
    if "v" in raw:
        s["v"] = _give(raw["v"])
    if "A" in raw:
        s["A"] = raw["A"]
    if op == "backward":
        s["f"].requires_grad_(True)
        s["phi"].requires_grad_(True)
    return s


def run(state):
    pp, op, s = state["pp"], state["op"], state.get("sett")
    if op == "pull" or op == "labels":
        return pp.pull(state["f"], state["phi"], s)
    if op == "push":
        return pp.push(state["g"], state["phi"], state["d0"], s)
    if op == "normal":
        f1 = pp.pull(state["f"], state["phi"], s)
        return f1, pp.push(f1, state["phi"], state["d0"], s)
    if op == "affine":
        f1 = pp.affine_pull(state["f"], state["A"], state["d1"], s)
        return f1, pp.affine_push(f1, state["A"], state["d0"], s)
    if op == "gradient":
        return pp.pull_grad(state["f"], state["phi"], s), pp.push_grad(state["g"], state["phi"], state["d0"], s)
    if op == "backward":
        f1 = pp.autograd.pull(state["f"], state["phi"], s)
        return (f1.detach(),) + torch.autograd.grad(f1, (state["f"], state["phi"]), state["g"])
    if op == "fused":
        loss, df, dphi = pp.fused_step(state["f"], state["phi"], state["g"], s)
        return loss.float(), df, dphi          # the loss as a training loop adds it up
    if op == "exp":
        return pp.Exp(state["v"])
    state["plan"].run()
    return state["outs"]


def work(case):
    """Bytes: each input read once, each output written once.  Flops: two per tap
    and axis-separable pass of the patch (x rows, then y, then z)."""
    op = case["op"]

    def pull_flops(dp, grad=False):
        return (3 if grad else 1) * 2.0 * (dp ** 3 + dp ** 2 + dp)

    if op == "batch":
        b = f = 0.0
        for d, c, deg in _batch_items(case):
            n = d[0] * d[1] * d[2]
            b += n * (12 + 4 * c * 3)          # phi and f0 read, f1 and out written
            f += 2 * n * c * pull_flops(deg + 1)
        return {"bytes": b, "flops": f}
    n1 = case["x"] * case["y"] * case["z"] * case["nb"]
    n0 = case["ix"] * case["iy"] * case["iz"] * case["nb"]
    c, dp = case["ch"], case["deg"] + 1
    fl = n1 * c * pull_flops(dp)
    if op in ("pull", "labels", "push"):
        return {"bytes": 12.0 * n1 + 4 * c * (n0 + n1), "flops": fl}
    if op == "normal":
        return {"bytes": 2 * (12.0 * n1 + 4 * c * (n0 + n1)), "flops": 2 * fl}
    if op == "affine":
        return {"bytes": 2 * 4.0 * c * (n0 + n1), "flops": 2 * fl}
    if op == "gradient":
        return {"bytes": 2 * (12.0 * n1 + 4 * c * (n0 + 3 * n1)), "flops": 2 * n1 * c * pull_flops(dp, True)}
    if op == "backward":      # forward pull; push of the cotangent; contraction with the gradient
        return {"bytes": 3 * (12.0 * n1 + 4 * c * (n0 + n1)) + 12.0 * n1, "flops": 2 * fl + n1 * c * pull_flops(dp, True)}
    if op == "fused":
        return {"bytes": 24.0 * n1 + 4 * c * (2 * n0 + n1), "flops": fl + n1 * c * pull_flops(dp, True)}
    # exp: each squaring reads the field and writes the next, which depends on the whole of it
    return {"bytes": 8 * 24.0 * n1, "flops": 8 * fl}


# ---- the same in 64 bits ------------------------------------------------------
def _bspline(t, n):
    """Centred B-spline of degree n at t (Cox-de Boor)."""
    if n < 0:
        return torch.zeros_like(t)
    if n == 0:
        return ((t > -0.5) & (t <= 0.5)).to(t.dtype)
    h = 0.5 * (n + 1)
    return ((h + t) * _bspline(t + 0.5, n - 1) + (h - t) * _bspline(t - 0.5, n - 1)) / n


def _weights(x, o, i, deg, order):
    if deg == 0:
        return torch.ones_like(x) if order == 0 else torch.zeros_like(x)
    t = x - (o + i)
    if order == 0:
        return _bspline(t, deg)
    return _bspline(t + 0.5, deg - 1) - _bspline(t - 0.5, deg - 1)


def _fold(i, d, b):
    """(index, sign) of tap i on an axis of d voxels under boundary code b."""
    if b == 0:
        return torch.remainder(i, d), None
    r = torch.remainder(i, 2 * d)
    m = r >= d
    return torch.where(m, 2 * d - 1 - r, r), (torch.where(m, -1.0, 1.0).double() if b == 2 else None)


class _Samples:
    """Positions of one volume's samples and the taps they read."""

    def __init__(self, x, x32, d0, deg, bnd, ext):
        self.d0, self.deg = d0, deg
        self.bnd = bnd
        xs = x if x32 is None else x32
        ok = torch.isfinite(xs).all(0)
        if not ext:
            for k in range(3):
                hi = (torch.tensor(float(d0[k]), dtype=torch.float32) - torch.tensor(0.99, dtype=torch.float32)).item()
                lo = torch.tensor(-0.01, dtype=torch.float32).item()
                ok = ok & (xs[k] >= lo) & (xs[k] <= hi)
        self.ok = ok
        self.x = [x[k].double() for k in range(3)]
        self.o = [torch.ceil(xs[k] - 0.5 * (deg + 1)).double() for k in range(3)]

    def axis(self, k, order):
        taps = []
        for i in range(self.deg + 1):
            idx, sg = _fold(self.o[k].long() + i, self.d0[k], self.bnd[k])
            w = _weights(self.x[k], self.o[k], i, self.deg, order)
            taps.append((idx, w if sg is None else w * sg))
        return taps

    def taps(self, orders):
        ax = [self.axis(k, orders[k]) for k in range(3)]
        for iz, wz in ax[2]:
            for iy, wy in ax[1]:
                row, wyz = (iz * self.d0[1] + iy) * self.d0[0], wz * wy
                for ix, wx in ax[0]:
                    yield row + ix, wyz * wx

    def pull(self, f, orders=(0, 0, 0)):
        """f (C, n0) -> (C, n1); samples outside are NaN."""
        out = torch.zeros((f.shape[0], self.ok.numel()), dtype=torch.float64, device=f.device)
        for idx, w in self.taps(orders):
            for c in range(f.shape[0]):
                out[c] += w * f[c][idx]
        return torch.where(self.ok, out, torch.nan)

    def push(self, g, out, orders=(0, 0, 0)):
        """out (C, n0) += the adjoint of ``pull`` of g (C, n1); non-finite values are skipped."""
        keep = [torch.where(self.ok & torch.isfinite(v), v, 0.0) for v in g]
        for idx, w in self.taps(orders):
            for c, v in enumerate(keep):
                out[c].index_add_(0, idx, w * v)


_GRAD = ((1, 0, 0), (0, 1, 0), (0, 0, 1))


def _samples(phi, b, case, d0):
    x32 = (phi[b] - 1.0).reshape(3, -1)
    return _Samples(x32, x32, d0, case["deg"], _BND[case["bnd"]], case["ext"])


def _affine_samples(A, case, d0, d1):
    """Positions in float32, rounded operation by operation as the path defines them
    (the 1-based map's last column made 0-based first)."""
    A = A[:3].clone()
    A[:, 3] = A.sum(dim=1) - 1.0
    A = A.cuda()
    i, j, k = (torch.arange(n, dtype=torch.float32, device="cuda") for n in d1)
    x = []
    for r in range(3):
        xj = (A[r, 1] * j.view(1, -1, 1) + A[r, 2] * k.view(-1, 1, 1)) + A[r, 3]
        x.append((xj + A[r, 0] * i.view(1, 1, -1)).reshape(-1))
    x = torch.stack(x)
    return _Samples(x, x, d0, case["deg"], _BND[case["bnd"]], case["ext"])


def exact(case, seed):
    raw = _raw(case, seed)
    op, d0, d1 = case["op"], (case["ix"], case["iy"], case["iz"]), (case["x"], case["y"], case["z"])
    ch, nb = case["ch"], case["nb"]
    n0 = d0[0] * d0[1] * d0[2]
    z0, z1 = d0[::-1], d1[::-1]

    def flat(t):
        return t.double().reshape(t.shape[0], -1)

    def zero():
        return torch.zeros((ch, n0), dtype=torch.float64, device="cuda")

    def give(per_volume, tail, scalar_ch=True):
        t = torch.stack(per_volume)
        return _give(t.reshape(t.shape[:1] + tail), 1 if scalar_ch else None)

    if op == "batch":
        outs = []
        for dd, c, deg, f, phi in raw["items"]:
            s = _samples(phi, 0, dict(case, deg=deg), dd)
            f1 = s.pull(flat(f[0]))
            out = torch.zeros_like(flat(f[0]))
            s.push(f1, out)
            outs.append((_give(f1.reshape((1, c) + dd[::-1]), 1), _give(out.reshape((1, c) + dd[::-1]), 1)))
        return outs
    if op == "exp":
        u = flat(raw["v"][0]) / 256.0
        one = [torch.arange(n, dtype=torch.float64, device="cuda") for n in d1]
        idt = torch.stack([one[k].view([-1 if 2 - k == a else 1 for a in range(3)]).expand(z1).reshape(-1) for k in range(3)])
        for _ in range(8):
            x = idt + u
            u = torch.cat([_Samples(x, None, d1, 1, [2 if a == k else 1 for a in range(3)], 1).pull(u[k:k + 1])
                           for k in range(3)])
        return _give((u + idt + 1.0).reshape((1, 3) + z1))
    if op == "affine":
        s = _affine_samples(raw["A"], case, d0, d1)
        a, b = [], []
        for v in range(nb):
            f1 = s.pull(flat(raw["f"][v]))
            out = zero()
            s.push(f1, out)
            a.append(f1)
            b.append(out)
        return give(a, (ch,) + z1), give(b, (ch,) + z0)
    res = {"a": [], "b": [], "c": []}
    loss = 0.0
    for v in range(nb):
        s = _samples(raw["phi"], v, case, d0)
        if op in ("pull", "labels"):
            res["a"].append(s.pull(flat(raw["f"][v])))
        elif op == "push":
            out = zero()
            s.push(flat(raw["g"][v]), out)
            res["b"].append(out)
        elif op == "normal":
            f1, out = s.pull(flat(raw["f"][v])), zero()
            s.push(f1, out)
            res["a"].append(f1)
            res["b"].append(out)
        elif op == "gradient":
            f, g = flat(raw["f"][v]), raw["g"][v].double().reshape(ch, 3, -1)
            res["a"].append(torch.stack([s.pull(f, q) for q in _GRAD], 1))
            out = zero()
            fin = torch.isfinite(g).all(1)
            for k, q in enumerate(_GRAD):
                s.push(torch.where(fin, g[:, k], torch.nan), out, q)
            res["b"].append(out)
        else:
            f, g = flat(raw["f"][v]), flat(raw["g"][v])
            f1 = s.pull(f)
            up = g if op == "backward" else 2.0 * (f1 - g)
            out = zero()
            s.push(up, out)
            res["a"].append(f1)
            res["b"].append(out)
            res["c"].append(torch.stack([(up * s.pull(f, q)).sum(0) for q in _GRAD]))
            if op == "fused":
                loss = loss + ((f1 - g) ** 2).sum()
    if op in ("pull", "labels"):
        return give(res["a"], (ch,) + z1)
    if op == "push":
        return give(res["b"], (ch,) + z0)
    if op == "normal":
        return give(res["a"], (ch,) + z1), give(res["b"], (ch,) + z0)
    if op == "gradient":
        t = torch.stack(res["a"]).reshape((nb, ch, 3) + z1)
        return _give(t, 1), give(res["b"], (ch,) + z0)
    dphi = give(res["c"], (3,) + z1, False)
    if op == "backward":
        return give(res["a"], (ch,) + z1), give(res["b"], (ch,) + z0), dphi
    return loss, give(res["b"], (ch,) + z0), dphi
